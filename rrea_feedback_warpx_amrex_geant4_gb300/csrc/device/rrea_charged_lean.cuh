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
// full loop, 11.0 ms here (10.1) and in the full loop over the recorded ones
// (1.3e5 positrons 1.37 ms, 1.14);
// the instruction-fetch stalls fall from 63 to 12 % of the issue interval and
// the FP64 pipe, the bound, is 85 % busy.
#pragma once

#include "rrea_electron.cuh"

namespace rrea_dev {

// One electron (POS: positron) through the outer step.  True when it is done
// (survived and written back); false with `rec` filled when the full loop must
// take over.
template <bool POS>
__device__ __forceinline__ bool transport_lean(StepConstants const& C, ElectronArgs const& A, int64_t ip,
                                               uint64_t& subcycles_out, IonPairCache& ion_pairs, ResumeRec& rec)
{
    constexpr double q = POS ? 1.0 : -1.0;
    constexpr int species = POS ? 1 : 0;
    constexpr int base = POS ? RREA_T_P_COLLISION : RREA_T_E_COLLISION;
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
        | 1u << RREA_RATE_BREMS | (POS ? 1u << RREA_RATE_ANNIHILATION : 0u);
    // every later chord starts where one that lay inside ended
    if (!strictly_inside(g, fma(run_x, run_x, run_y * run_y), run_z)) return false;

    // ---- substep count, O/RreaElectronTransport.cpp:187-279 and
    // O/RreaPositronTransport.cpp:168-230, of a chord
    // that lies inside: its uniform slices never exceed the target by more
    // than the reference's tolerance while the count is below a thousand
    uint32_t subcycles;
    {
        Path<1> path;
        double gb;
        double const sc = charged_speed(k, gb) * dt_s;
        double const ex = fma(sc, dx, run_x), ey = fma(sc, dy, run_y), ez = fma(sc, dz, run_z);
        if (!clip_inside<1, true>(run_x, run_y, run_z, 0.0, ex, ey, ez, fma(ex, ex, ey * ey), g, path)) return false;
        if (!rate_bracket(C, arena, rc, k, err, base) || row_flags(rc.hit) & (kRates | 1u << RREA_RATE_ELASTIC)) return false;
        double const dpath = path.full
            * (A.prof.n == 0 ? rho : common_density(A.prof, rho, fma(0.5, path.dz, path.sz)));
        FieldRange const dfw = path_field_work(fv, g, path, q, 0.0, 1.0, err);
        double s0, s1, s2;
        common_rates<POS>(C, rc, k, s0, s1, s2);
        double const target = cfg.max_optical_depth_per_substep;
        double const by_tau = ceil((POS ? ((s0 + s1) + s2) * dpath : (s0 * dpath) + (s1 * dpath)) / target);
        double const gs_n = row_value(rc.hit, RREA_RATE_ELASTIC) * dpath;
        double const col = max0(row_value(rc.hit, RREA_RATE_COLLISION));
        double const drag = (POS ? col : col + max0(row_value(rc.hit, RREA_RATE_SOFT))) * dpath;
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

    Running p{run_x, run_y, run_z, dx, dy, dz, k};
    uint32_t sub = 0;
    for (; sub < subcycles; ++sub) {
        uint64_t hazard;
        Path<1> path;
        double dpath;
        if (!live_hazard_index(species, sub, 0, hazard)) break;
        SubstepDraws const draws{hazard, static_cast<uint64_t>(sub) << 8,
                                 POS ? kChPositronCompetingOpticalDepth : kChElectronCompetingOpticalDepth,
                                 POS ? kChPositronGsAngle : kChElectronGsAngle,
                                 POS ? kChPositronGsAzimuth : kChElectronGsAzimuth};
        if (!common_substep<POS>(C, A, g, fv, rng, draws, sub_dt, pairs_per_eV, ion_pairs, rc, p, path, dpath)) {
            break;
        }
        dpath_sum += dpath;
        length_sum += path.full;
    }
    // a low-energy electron's gate needs the field and the mean drag
    if (sub == subcycles && (POS || (p.k > hm_thr && gt0(hm_thr) && p.k <= C.tix.charged_max_eV))) {
        // CommitSurvivorChargedWriteback, O/RreaTransportStep.H:874-905
        double const um = proper_velocity_from_kinetic(p.k);
        double const r = rz_radius(p.x, p.y);
        A.ux[ip] = um * p.dx;
        A.uy[ip] = um * p.dy;
        A.uz[ip] = um * p.dz;
        A.r[ip] = r;
        A.theta[ip] = fatan2(arena, p.y, p.x);
        A.z[ip] = p.z;
        if (A.segments) {
            SegmentRec& s = A.segments[ip];
            s.a[0] = r0;
            s.a[1] = z0;
            s.a[2] = r;
            s.a[3] = p.z;
            s.a[4] = q * weight;
            s.faces = 0u;
            s.kind = 1;
        }
        return true;
    }
    rec.x = p.x;
    rec.y = p.y;
    rec.z = p.z;
    rec.dx = p.dx;
    rec.dy = p.dy;
    rec.dz = p.dz;
    rec.k = p.k;
    rec.sub = sub;
    rec.dpath = dpath_sum;
    rec.length = length_sum;
    return false;
}

// The common-history kernels: every valid particle is either finished or
// recorded in A.resume.
template <bool POS>
__device__ __forceinline__ void lean_step_body(ElectronArgs const& A)
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
        ion_pairs.init(my_slot, POS ? 0.0 : 0.5 * C.cfg.low_energy_cutoff_eV, C.tix.w_air_eV_per_pair);
        uint64_t sub = 0;
        ResumeRec rec;
        bool const done = transport_lean<POS>(C, A, ip, sub, ion_pairs, rec);
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

template <int MinBlocks>
__global__ void __launch_bounds__(128, MinBlocks) electron_lean_kernel(const __grid_constant__ ElectronArgs A)
{
    lean_step_body<false>(A);
}

// (1.3e5 positrons: 1.14 ms with 16 resident blocks, 1.15 with 8)
static __global__ void __launch_bounds__(128, 16) positron_lean_kernel(const __grid_constant__ ElectronArgs A)
{
    lean_step_body<true>(A);
}

}  // namespace rrea_dev
