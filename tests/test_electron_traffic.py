"""The electron traffic record adds one capture of each of the two electron
kernels (one kernel to a capture) and refuses anything else."""
import pytest

HEAD = '"ID","Kernel Name","Metric Name","Metric Unit","Metric Value"\n'


def _csv(path, kernel, read, write, ns, pipe=None):
    rows = [("dram__bytes_read.sum", read), ("dram__bytes_write.sum", write), ("gpu__time_duration.sum", ns)]
    if pipe is not None:
        rows.append(("sm__pipe_fp64_cycles_active.avg.pct_of_peak_sustained_active", pipe))
    path.write_text("==PROF== Connected\n" + HEAD
                    + "".join(f'"0","void {kernel}<16>(rrea_dev::ElectronArgs)","{m}","base","{v:,}"\n' for m, v in rows))
    return str(path)


def test_two_captures_are_summed(tmp_path):
    from rrea_feedback_warpx_amrex_geant4_gb300 import electron_traffic as et
    a = _csv(tmp_path / "a.csv", "electron_lean_kernel", 1_000_000, 2_000, 3_000, 85.5)
    b = _csv(tmp_path / "b.csv", "electron_step_kernel", 10, 20, 30, 50.0)
    for paths in ((a, b), (b, a)):
        v = et.read_capture(*paths)
        assert [v[m] for m in et.METRICS] == [1_000_010.0, 2_020.0, 3_030.0]
        assert v[et.FP64_PIPE] == 85.5
    rec = et.record([a, b], 10, out=str(tmp_path / "r.json"))
    assert rec["dram_bytes_per_particle_step"] == pytest.approx(100_203.0)


def test_one_capture_or_two_of_one_kernel_is_refused(tmp_path):
    from rrea_feedback_warpx_amrex_geant4_gb300 import electron_traffic as et
    a = _csv(tmp_path / "a.csv", "electron_lean_kernel", 1, 2, 3)
    c = _csv(tmp_path / "c.csv", "electron_lean_kernel", 1, 2, 3)
    for paths in ((a,), (a, c)):
        with pytest.raises(ValueError):
            et.read_capture(*paths)
