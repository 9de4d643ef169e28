// The common history of an electron: a survivor whose chords stay strictly
// inside an absorbing domain, that draws no discrete event, does not reach
// the cutoff and ends above the hard-Moller threshold.  Nineteen in twenty
// electrons of a runaway population are that, and the full loop
// (rrea_electron.cuh) makes them pay for the others: a warp with one event
// runs its samplers with one lane, the full loop's code (three quarters of a
// megabyte of instructions) never settles in the instruction caches, and its
// state lives in local memory.  This loop holds only what such an electron
// executes.  At the first condition it does not cover it records the state at
// the start of that substep (ResumeRec), commits nothing of the substep, and
// leaves the particle to the full kernel, launched over the records, which
// repeats the substep from the same state with the same counter-RNG draws.
// Measured, one resident phase of 2^21 scale-up electrons: 16.7 ms in the
// full loop, 11.0 ms here (10.1) and in the full loop over the recorded ones;
// the instruction-fetch stalls fall from 63 to 12 % of the issue interval and
// the FP64 pipe, the bound, is 85 % busy.
#pragma once

#include "rrea_electron.cuh"

namespace rrea_dev {

// TransportDensityRatioAtZ for a bound profile; NaN outside it.
static __device__ __noinline__ double lean_density(DensityProfile const& prof, double uniform, double z)
{
    Err err;
    double const v = density_ratio_at_z(prof, uniform, z, err);
    return err.code ? __longlong_as_double(0x7ff8000000000000LL) : positive_or(v, uniform);
}

// One electron through the outer step.  True when it is done (survived and
// written back); false with `rec` filled when the full loop must take over.
__device__ __forceinline__ bool transport_lean(StepConstants const& C, ElectronArgs const& A, int64_t ip,
                                               uint64_t& subcycles_out, IonPairCache& ion_pairs, ResumeRec& rec)
{
    constexpr double q = -1.0;
    const double* __restrict__ arena = A.arena;
    rrea_gpu_config const& cfg = C.cfg;
    Geom const g = make_geom(C);
    double const cutoff = cfg.low_energy_cutoff_eV;
    double const hm_thr = C.hm_threshold_eV;
    double const dt_s = C.dt_s;
    rec.sub = kResumeFromStart;
    rec.subcycles = 0;

    int32_t const cpu = A.cpu ? A.cpu[ip] : 0;
    uint64_t const key = static_cast<uint64_t>(llabs(A.id[ip])) ^ (static_cast<uint64_t>(cpu) << 40);
    FieldView const fv = A.fv.for_instance(cpu);
    double const weight = A.w[ip];
    double const r0 = A.prev_r[ip], z0 = A.prev_z[ip];
    double dx = A.prev_ux[ip], dy = A.prev_uy[ip], dz = A.prev_uz[ip];
    double k = kinetic_from_proper_velocity(dx, dy, dz);
    normalize(dx, dy, dz);
    if (le0(weight) || !finite_bits(weight) || lt0(r0) || !(k >= cutoff)) return false;
    double run_x, run_y, run_z = z0;
    {
        double s, c;
        fsincos(arena, A.prev_theta[ip], s, c);
        run_x = r0 * c;
        run_y = r0 * s;
    }
    RngStream rng;
    rng.init(cfg.rng_seed, key, C.step_key);
    RateCache rc;
    Err err;
    double const rho = C.density_ratio;
    constexpr uint32_t kRates = 1u << RREA_RATE_COLLISION | 1u << RREA_RATE_SOFT | 1u << RREA_RATE_HARD
        | 1u << RREA_RATE_BREMS;
    // the two open channels' rates at energy e (competing_rates), row in rc
    auto channels = [&](double e, double& s0, double& s1) {
        s0 = C.hm_enabled && gt0(hm_thr) && e > 2.0 * hm_thr ? max0(row_value(rc.hit, RREA_RATE_HARD)) : 0.0;
        s1 = e > C.photon_cutoff_eV ? max0(row_value(rc.hit, RREA_RATE_BREMS)) : 0.0;
        // an open channel of rate zero counts as one per 1e99 m
        if (eq0(s0) && C.hm_enabled && gt0(hm_thr) && e > 2.0 * hm_thr) s0 = 1.0e-99;
        if (eq0(s1) && e > C.photon_cutoff_eV) s1 = 1.0e-99;
    };
    auto density = [&](Path<1> const& p) {
        return A.prof.n == 0 ? rho : lean_density(A.prof, rho, fma(0.5, p.dz, p.sz));
    };
    double gb = 0.0;
    auto chord = [&](double dt, Path<1>& p) {
        double const sc = charged_speed(k, gb) * dt;
        double const ex = fma(sc, dx, run_x), ey = fma(sc, dy, run_y), ez = fma(sc, dz, run_z);
        return clip_inside<1, true>(run_x, run_y, run_z, 0.0, ex, ey, ez, fma(ex, ex, ey * ey), g, p);
    };
    // every later chord starts where one that lay inside ended
    if (!strictly_inside(g, fma(run_x, run_x, run_y * run_y), run_z)) return false;

    // ---- substep count, O/RreaElectronTransport.cpp:187-279, of a chord
    // that lies inside: its uniform slices never exceed the target by more
    // than the reference's tolerance while the count is below a thousand
    uint32_t subcycles;
    {
        Path<1> path;
        if (!chord(dt_s, path)) return false;
        if (!rate_bracket(C, arena, rc, k, err) || row_flags(rc.hit) & (kRates | 1u << RREA_RATE_ELASTIC)) return false;
        double const dpath = path.full * density(path);
        FieldRange const dfw = path_field_work(fv, g, path, q, 0.0, 1.0, err);
        double s0, s1;
        channels(k, s0, s1);
        double const target = cfg.max_optical_depth_per_substep;
        double const by_tau = ceil(((s0 * dpath) + (s1 * dpath)) / target);
        double const gs_n = row_value(rc.hit, RREA_RATE_ELASTIC) * dpath;
        double const drag = (max0(row_value(rc.hit, RREA_RATE_COLLISION)) + max0(row_value(rc.hit, RREA_RATE_SOFT))) * dpath;
        double const impulse = fmax(cfg.max_field_impulse_fraction * k, fmax(cfg.field_impulse_floor_eV, 1.0));
        double const by_gs =
            ceil(fmin(gs_n, cfg.gs_total_collision_cap) / fmax(cfg.max_gs_collisions_per_substep, 1.0));
        double const by_impulse = ceil((fabs(dfw.work) + drag) / impulse);
        double const most = fmax(1.0, fmax(by_tau, fmax(by_gs, by_impulse)));
        if (err.code || !(most < 1000.0) || !(most < static_cast<double>(cfg.max_subcycles)) || !(dpath > 0.0)) return false;
        subcycles = static_cast<uint32_t>(most);
    }
    subcycles_out = subcycles;
    rec.subcycles = subcycles;
    double const sub_dt = dt_s / static_cast<double>(subcycles);
    double const pairs_per_eV = weight / fmax(C.tix.w_air_eV_per_pair, 1.0);
    double dpath_sum = 0.0, length_sum = 0.0;

    for (uint32_t sub = 0;; ++sub) {
        // the state the full loop resumes from
        rec.k = k;
        rec.dx = dx;
        rec.dy = dy;
        rec.dz = dz;
        rec.sub = sub;
        if (sub >= subcycles) break;
        Path<1> path;
        bool go = chord(sub_dt, path);
        double pair_weight = 0.0;
        if (go) {
            double const rho_s = density(path);
            FieldRange const field = path_field_work(fv, g, path, q, 0.0, 1.0, err);
            half_kick(field, 0.5 * sub_dt, q, gb, k, dx, dy, dz);
            go = k >= cutoff && rate_bracket(C, arena, rc, k, err) && !(row_flags(rc.hit) & kRates);
            if (go) {
                double const dpath = path.full * rho_s;
                double s0, s1;
                channels(k, s0, s1);
                double const tau = s0 * dpath + s1 * dpath;
                uint64_t index;
                go = finite_bits(tau) && live_hazard_index(0, sub, 0, index);
                // (select_hazard's test: no event whatever the roundings)
                double const u1 = rng.uniform(index, kChElectronCompetingOpticalDepth);
                go = go && __double2hiint(u1) > max(__double2hiint(tau) + 1, 0x3e100000);
                // drag to the end of the substep, short of the cutoff
                double const sc = max0(row_value(rc.hit, RREA_RATE_COLLISION));
                double const ss = max0(row_value(rc.hit, RREA_RATE_SOFT));
                double const room = k - cutoff;
                double const raw = sc * dpath;
                double const drag = fmin(raw + ss * dpath, room);
                go = go && (sc + ss) * dpath < room && !err.code;
                pair_weight = pairs_per_eV * fmin(raw, drag);
                k -= drag;
                // elastic deflection, O/RreaTransportStep.H:371-423
                go = go && rate_bracket(C, arena, rc, k, err) && !(row_flags(rc.hit) >> RREA_RATE_ELASTIC & 1u);
                if (go) {
                    double const gs_n = row_value(rc.hit, RREA_RATE_ELASTIC) * dpath;
                    // (sample_gs_cos' checks; the rows cover the certified energies)
                    go = gs_n >= C.tix.gs_few_collision_threshold && gs_n < C.tix.gs_isotropic_above_n;
                    if (go) {
                        bool const wentzel = !(k <= C.tix.gs_wentzel_transition_eV);
                        double const ct = sample_gs_angle_rows(
                            C, arena, rc, wentzel ? C.tix.wentzel[0] : C.tix.gs[0], 0, wentzel ? 1 : 0, k, gs_n,
                            rng.uniform(static_cast<uint64_t>(sub) << 8, kChElectronGsAngle), err);
                        double nx, ny, nz;
                        cone_unit(arena, dx, dy, dz, ct, rng.uniform(static_cast<uint64_t>(sub) << 8, kChElectronGsAzimuth),
                                  nx, ny, nz);
                        dx = nx;
                        dy = ny;
                        dz = nz;
                        half_kick(field, 0.5 * sub_dt, q, gamma_beta(k), k, dx, dy, dz);
                        go = k >= cutoff && !err.code;
                    }
                }
                dpath_sum += go ? dpath : 0.0;
                length_sum += go ? path.full : 0.0;
            }
        }
        if (!go) break;
        // the substep stands: its ion pairs and the new position
        if (gt0(pair_weight)) {
            double const x = fma(0.5, path.dx, path.sx), y = fma(0.5, path.dy, path.sy);
            ion_pairs.add(C, A.cells, fsqrt(fma(x, x, y * y)), fma(0.5, path.dz, path.sz),
                          pair_weight);
        }
        run_x = path.sx + path.dx;
        run_y = path.sy + path.dy;
        run_z = path.sz + path.dz;
    }
    // a low-energy survivor's gate needs the field and the mean drag
    if (rec.sub == subcycles && k > hm_thr && gt0(hm_thr) && k <= C.tix.charged_max_eV) {
        // CommitSurvivorChargedWriteback, O/RreaTransportStep.H:874-905
        double const um = proper_velocity_from_kinetic(k);
        double const r = rz_radius(run_x, run_y);
        A.ux[ip] = um * dx;
        A.uy[ip] = um * dy;
        A.uz[ip] = um * dz;
        A.r[ip] = r;
        A.theta[ip] = fatan2(arena, run_y, run_x);
        A.z[ip] = run_z;
        if (A.segments) {
            SegmentRec& s = A.segments[ip];
            s.a[0] = r0;
            s.a[1] = z0;
            s.a[2] = r;
            s.a[3] = run_z;
            s.a[4] = q * weight;
            s.faces = 0u;
            s.kind = 1;
        }
        return true;
    }
    rec.x = run_x;
    rec.y = run_y;
    rec.z = run_z;
    rec.dpath = dpath_sum;
    rec.length = length_sum;
    return false;
}

// The common-history kernel: every valid electron is either finished or
// recorded in A.resume, in warp-aggregated order.
template <int MinBlocks>
__global__ void __launch_bounds__(128, MinBlocks) electron_lean_kernel(const __grid_constant__ ElectronArgs A)
{
    StepConstants const& C = c_step;
    __shared__ IonPairSlot ion_slots[128];
    IonPairSlot* const my_slot = ion_slots + threadIdx.x;
    unsigned int moved = 0;
    for_each_particle(A.n, A.work, [&](int64_t ip) {
        bool const valid = A.id[ip] > 0;
        if (A.segments) A.segments[ip].kind = 0;
        if (A.sec_per_parent) A.sec_per_parent[ip] = 0;
        if (!valid) {
            if (A.diag_disposition) A.diag_disposition[ip] = -1;
            if (A.diag_subcycles) A.diag_subcycles[ip] = 0;
            if (A.diag_events) A.diag_events[ip] = 0;
            return;
        }
        ++moved;
        IonPairCache ion_pairs;
        ion_pairs.init(my_slot, 0.5 * C.cfg.low_energy_cutoff_eV, C.tix.w_air_eV_per_pair);
        uint64_t sub = 0;
        ResumeRec rec;
        bool const done = transport_lean(C, A, ip, sub, ion_pairs, rec);
        ion_pairs.flush(C, A.cells);
        if (!done) {
            rec.ip = ip;
            A.resume[atomicAdd(A.resume_count, 1ULL)] = rec;
            return;
        }
        if (A.diag_disposition) A.diag_disposition[ip] = 0;
        if (A.diag_subcycles) A.diag_subcycles[ip] = sub;
        if (A.diag_events) A.diag_events[ip] = sub;   // one hazard draw per substep
    }, A.order);
    unsigned int const warp_total = __reduce_add_sync(0xffffffffu, moved);
    if ((threadIdx.x & 31) == 0 && warp_total) atomicAdd(A.transported, static_cast<unsigned long long>(warp_total));
}

}  // namespace rrea_dev
