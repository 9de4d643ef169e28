// Pathwise adjoint of the charged push with respect to an axial field
// profile E_z(z): the gradient pattern built on the kinetic step.
//
// The differentiated model is the continuous part of the charged substep
// (O/RreaChargedInterleave.H:100-138 and :218-292 with the two-node field
// work of O/RreaPathFieldWork.H:57-150), with every discrete outcome frozen:
//
//   chord     L = v(K) h along d from z (h = dt / substeps), z1 = z + L d_z
//   work      W = q d_z L <E>,  <E> = (E(z + a L d_z) + E(z + b L d_z)) / 2
//             (two-point Gauss-Legendre, a, b = 1/2 -+ 1/(2 sqrt 3))
//   kick      d <- (u(K) d + s <E> z^) / |.|,  K <- K + W / 2,
//             s = q (c^2 / m c^2) h / 2  (the half kick without B)
//   drag      K <- K - rho S(K) L, S the tables' collision plus soft
//             radiative stopping power (log-log, as the transport reads them)
//   kick      as above, with the same <E> and W
//   scatter   d <- R d, R a rotation drawn once from the counter RNG of
//             (seed, particle, step, substep): the frozen elastic deflection
//
// E(z) interpolates the profile nodes linearly (clamped outside).  A
// particle whose drag would take it below the cutoff stops there (a frozen
// topology: it stops at the same substep in the reverse pass).  The loss is
// the smoothed runaway count plus the smoothed net charge crossing the
// plane z_p (the time integral of J_z through the plane, by charge
// conservation):
//   J = sum_i w_i [ sig((K_i(T) - K_th) / tau_K)
//                   - lambda (sig((z_i(T) - z_p) / tau_z) - sig((z_i(0) - z_p) / tau_z)) ]
// with sig the logistic function (the electron charge is -e; lambda counts
// it in elementary charges).
//
// Forward: one thread per particle, the state checkpointed every C steps.
// Reverse: per checkpoint segment, last to first, from a tape of substep
// inputs that the forward pass left or, for segments and nodes it did not, that
// is computed again from the checkpoint (with each substep's
// stopping power, its derivative and the frozen rotation, so the adjoint
// evaluates neither tables nor the RNG again), then the adjoint runs back
// through it.  A substep moves a particle a small part of a node spacing, so
// the two nodes' gradient terms gather in registers while the node pair stays
// and go to the block's shared memory when it changes; the block's sums are
// added to the output once per block and node.
//
// What bounds both kernels is the FP64 pipe (two multiply-adds per clock per
// SM; a division or square root is ten of them, a library logarithm 39).
// Velocities are in units of c (|v| = gamma beta, one inverse root per kick
// and one each for gamma beta and 1/gamma), the stopping power and its
// derivative come from interval polynomials (device/rrea_rate_rows.cuh), and
// the rotation's sines from a table or a series.  Measured, 100,003
// electrons, 96 steps of 4 substeps in three segments: forward 36.2 -> 17.9 ms
// (16.8 without the tape it leaves), reverse 71.9 -> 15.4 ms.
#include "rrea_kernels.h"
#include "device/rrea_device_path.cuh"
#include "host/adjoint_tape.hpp"

#include <cuda_runtime.h>

namespace rrea_dev {
namespace adj {

constexpr double kGlA = 0.21132486540518711775;   // 1/2 - 1/(2 sqrt 3)
constexpr double kGlB = 0.78867513459481288225;   // 1/2 + 1/(2 sqrt 3)
constexpr int kMaxNodes = 2048;

struct Params {
    int64_t n;
    int n_nodes;
    double z0, dz_node;     // node k at z0 + k dz_node
    int steps, substeps, ckpt_every;
    double h;               // substep duration
    double rho;             // density ratio of the stopping power
    double cutoff;          // eV
    double scatter_rms;     // rad
    double k_th, tau_k, z_p, tau_z, lambda;
    uint64_t seed;
    RreaTable1DIndex col, soft;
    RreaRowIndex rows;      // their interval polynomials (columns RREA_RATE_COLLISION and _SOFT)
    double inv_dz;          // 1 / dz_node
    double kick;            // q (c / m c^2) h / 2: change of v per volt per metre in half a substep
    // each particle's end: (global substep << 1) | kind (0 stopped in the
    // drag, 1 below the cutoff after the second kick), -1 for none.  A
    // recording forward writes it; a replaying one (and the reverse pass)
    // ends every particle exactly there, so a perturbed profile keeps the
    // topology of the recorded run.
    int32_t* ends;
    int replay;
};

struct State {
    double z, dx, dy, dz, k;
    int alive;
};

__device__ __forceinline__ double sig(double x) { return 1.0 / (1.0 + exp(-x)); }
__device__ __forceinline__ double dsig(double x)
{
    double const s = sig(x);
    return s * (1.0 - s);
}

// E(z) and dE/dz of the profile; node weights for the reverse pass.
__device__ __forceinline__ double field(Params const& p, const double* __restrict__ e, double z, double& slope, int& k0,
                                       double& f)
{
    double const x = (z - p.z0) * p.inv_dz;
    if (!gt0(x)) {
        slope = 0.0;
        k0 = 0;
        f = 0.0;
        return e[0];
    }
    if (!(x < static_cast<double>(p.n_nodes - 1))) {
        slope = 0.0;
        k0 = p.n_nodes - 2;
        f = 1.0;
        return e[p.n_nodes - 1];
    }
    split_cell<false>(z - p.z0, Divisor{p.dz_node, p.inv_dz}, k0, f);
    // x just below a node can round onto it
    k0 = max(0, min(k0, p.n_nodes - 2));
    double const e0 = e[k0], de = e[k0 + 1] - e0;
    slope = de * p.inv_dz;
    return fma(f, de, e0);
}

// rho S(K) and its K-derivative from the two log-log hot tables, where the
// rows are flagged (two nodes within 1e-9 of one another).
static __device__ __noinline__ double2 drag_power_fallback(Params const& p, const double* __restrict__ arena, double k)
{
    double total = 0.0;
    double dk = 0.0;
    for (RreaTable1DIndex const* h : {&p.col, &p.soft}) {
        Err err;
        Bracket b;
        if (!bracket_hot(arena, *h, k, b, err)) continue;
        double const v = eval_hot(arena, *h, b, err);
        total += v;
        if (b.kind != 3) continue;   // constant beyond the grid (a node itself has measure zero)
        // d/dK in the table's mode: log-log between positive nodes, linear
        // in the log-energy fraction otherwise (the zero-threshold rule)
        const double* y = arena + h->y;
        double const ylo = __ldg(y + b.hi - 1), yhi = __ldg(y + b.hi);
        double const ilx = __ldg(arena + h->ilx + b.hi);
        if (h->mode == RREA_INTERP_LOGLOG || (ylo > 0.0 && yhi > 0.0)) {
            const double* ly = arena + h->ly;
            dk += v * (__ldg(ly + b.hi) - __ldg(ly + b.hi - 1)) * ilx / k;
        } else {
            dk += (yhi - ylo) * ilx / k;
        }
    }
    return make_double2(p.rho * total, p.rho * dk);
}

// rho S(K) and, when asked for, its K-derivative (0 outside the tables, as
// there).
__device__ __forceinline__ double drag_power(Params const& p, const double* __restrict__ arena, double k,
                                             bool derivative, double& dk)
{
    dk = 0.0;
    RowHit h;
    if (!find_row(arena, p.rows, k, h)) return 0.0;
    if (row_flags(h) & (1u << RREA_RATE_COLLISION | 1u << RREA_RATE_SOFT)) {
        double2 const r = drag_power_fallback(p, arena, k);
        dk = r.y;
        return r.x;
    }
    if (derivative) dk = p.rho * ((row_slope(h, RREA_RATE_COLLISION) + row_slope(h, RREA_RATE_SOFT)) * h.rec[1]);
    return p.rho * (max0(row_value(h, RREA_RATE_COLLISION)) + max0(row_value(h, RREA_RATE_SOFT)));
}

// gamma beta, gamma and their inverses at kinetic energy K: gamma beta is
// the velocity in units of c, its K-derivative gamma / (gamma beta) / mc^2,
// the speed beta = gamma beta / gamma, whose K-derivative is 1 / (gamma^2
// gamma beta) / mc^2.
struct Motion {
    double gb, igb, g, ig;
};
__device__ __forceinline__ Motion motion(double k)
{
    double const t = k * kInvMeC2;
    double const w = t * (t + 2.0);
    double const igb = frsqrt(w);
    return Motion{w * igb, igb, 1.0 + t, frsqrt(w + 1.0)};
}

// The frozen rotation of (particle, step, substep): axis uniform on the
// sphere, angle Gaussian with the configured rms.
__device__ __forceinline__ void rotation(Params const& p, const double* __restrict__ arena, uint64_t id, int step,
                                         int sub, double n[3], double& c, double& s)
{
    uint64_t const key = splitmix64(p.seed ^ splitmix64(id * 0x9e3779b97f4a7c15ULL + 0x5eed))
        ^ (static_cast<uint64_t>(step) << 20) ^ static_cast<uint64_t>(sub);
    auto uni = [&](int k) {
        return (static_cast<double>(splitmix64(key * 4 + k) >> 11) + 0.5) * 0x1.0p-53;
    };
    double const mu = 2.0 * uni(0) - 1.0;
    double const st = fsqrt(max0(1.0 - mu * mu));
    double sp, cp, sg, cg;
    sincos_turn(arena, uni(1), sp, cp);
    n[0] = st * cp;
    n[1] = st * sp;
    n[2] = mu;
    sincos_turn(arena, uni(3), sg, cg);
    double const th = p.scatter_rms * (fsqrt(-2.0 * flog(arena, uni(2))) * cg);
    double const t2 = th * th;
    if (__double2hiint(t2) < 0x3fb00000) {
        // |theta| < 1/4: the series' next terms are below 2^-56
        s = th * fma(t2, fma(t2, fma(t2, fma(t2, fma(t2, -1.0 / 39916800.0, 1.0 / 362880.0), -1.0 / 5040.0), 1.0 / 120.0),
                             -1.0 / 6.0), 1.0);
        c = fma(t2, fma(t2, fma(t2, fma(t2, fma(t2, fma(t2, 1.0 / 479001600.0, -1.0 / 3628800.0), 1.0 / 40320.0),
                                        -1.0 / 720.0), 1.0 / 24.0), -0.5), 1.0);
    } else {
        sincos(th, &s, &c);
    }
}

// Rodrigues: v cos + (n x v) sin + n (n.v) (1 - cos); its transpose is the
// same with -sin.
__device__ __forceinline__ void rotate(double const n[3], double c, double s, double v[3])
{
    double const nv = n[0] * v[0] + n[1] * v[1] + n[2] * v[2];
    double const cx = n[1] * v[2] - n[2] * v[1], cy = n[2] * v[0] - n[0] * v[2], cz = n[0] * v[1] - n[1] * v[0];
    double const m = nv * (1.0 - c);
    double const r[3] = {v[0] * c + cx * s + n[0] * m, v[1] * c + cy * s + n[1] * m, v[2] * c + cz * s + n[2] * m};
    v[0] = r[0];
    v[1] = r[1];
    v[2] = r[2];
}

__device__ __forceinline__ int32_t end_code(Params const& p, int step, int sub, int kind)
{
    return ((step * p.substeps + sub) << 1) | kind;
}

// Values of one substep that the reverse pass reads back instead of
// evaluating them again: the stopping power and its K-derivative at K1, and
// the frozen rotation (axis, cos, sin).  kAux columns of n per tape entry.
constexpr int kAux = 7;

// One substep forward; `end` is the particle's end record (see Params).
// With `aux` (column stride n, particle i) the drag and rotation go to the
// tape beside the substep's input state.
__device__ __forceinline__ void substep(Params const& p, const double* __restrict__ e,
                                        const double* __restrict__ arena, uint64_t id, int step, int sub, State& st,
                                        int32_t& end, double* __restrict__ aux, int64_t i)
{
    if (!st.alive) return;
    double const q = -1.0;
    Motion mo = motion(st.k);
    double const L = (kC * p.h) * (mo.gb * mo.ig);
    double const ldz = L * st.dz;
    double sl;
    int k0;
    double f;
    double const e1 = field(p, e, fma(kGlA, ldz, st.z), sl, k0, f);
    double const e2 = field(p, e, fma(kGlB, ldz, st.z), sl, k0, f);
    double const eavg = 0.5 * (e1 + e2);
    double const w = q * ldz * eavg;
    double const s = p.kick * eavg;
    // kick 1
    double m[3] = {mo.gb * st.dx, mo.gb * st.dy, fma(mo.gb, st.dz, s)};
    double inv = frsqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
    double d[3] = {m[0] * inv, m[1] * inv, m[2] * inv};
    double k1 = st.k + 0.5 * w;
    double const z1 = st.z + ldz;
    // drag
    double ds;
    double const sp = drag_power(p, arena, k1, aux != nullptr, ds);
    double const loss = sp * L;
    if (aux) {
        aux[i] = sp;
        aux[p.n + i] = ds;
    }
    bool const stop = p.replay ? end == end_code(p, step, sub, 0) : !(k1 - loss > p.cutoff);
    if (stop) {
        st.z = z1;
        st.k = p.cutoff;
        st.alive = 0;
        if (!p.replay) end = end_code(p, step, sub, 0);
        return;
    }
    double const k2 = k1 - loss;
    // kick 2
    double const gb2 = gamma_beta(k2);
    m[0] = gb2 * d[0];
    m[1] = gb2 * d[1];
    m[2] = fma(gb2, d[2], s);
    inv = frsqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
    d[0] = m[0] * inv;
    d[1] = m[1] * inv;
    d[2] = m[2] * inv;
    double const k3 = k2 + 0.5 * w;
    double n[3], c, sn;
    rotation(p, arena, id, step, sub, n, c, sn);
    if (aux) {
        aux[2 * p.n + i] = n[0];
        aux[3 * p.n + i] = n[1];
        aux[4 * p.n + i] = n[2];
        aux[5 * p.n + i] = c;
        aux[6 * p.n + i] = sn;
    }
    rotate(n, c, sn, d);
    st.z = z1;
    st.k = k3;
    st.dx = d[0];
    st.dy = d[1];
    st.dz = d[2];
    bool const below = p.replay ? end == end_code(p, step, sub, 1) : !(k3 > p.cutoff);
    if (below) {
        st.alive = 0;
        if (!p.replay) end = end_code(p, step, sub, 1);
    }
}

struct Adj {
    double z, dx, dy, dz, k;
};

// The gradient terms of the node pair (node, node + 1) a particle is in.
struct NodeSums {
    int node = -1;
    double lo = 0.0, hi = 0.0;
    __device__ __forceinline__ void flush(double* g)
    {
        if (node < 0) return;
        if (ne0(lo)) atomicAdd(g + node, lo);
        if (ne0(hi)) atomicAdd(g + node + 1, hi);
        lo = hi = 0.0;
    }
    __device__ __forceinline__ void add(double* g, int n, double v, double f)
    {
        if (n != node) {
            flush(g);
            node = n;
        }
        double const up = v * f;
        hi += up;
        lo += v - up;
    }
};

// One substep backward: `in` is the substep's input state and `aux` its
// tape values (column stride n, particle i); `a` holds the output adjoint
// and becomes the input adjoint; node gradients go to g through `sums`.
__device__ __forceinline__ void substep_adjoint(Params const& p, const double* __restrict__ e,
                                                const double* __restrict__ aux, int64_t i, int step, int sub,
                                                State const& in, int32_t end, Adj& a, NodeSums& sums, double* g)
{
    if (!in.alive) return;   // frozen: nothing moved
    double const q = -1.0;
    Motion const m0 = motion(in.k);
    double const ch = kC * p.h;
    double const L = ch * (m0.gb * m0.ig);
    // dL/dK = h c / (gamma^2 gamma beta mc^2)
    double const dL = (ch * kInvMeC2) * (m0.ig * m0.ig * m0.igb);
    double const ldz = L * in.dz;
    double sl1, sl2, f1, f2;
    int n1, n2;
    double const e1 = field(p, e, fma(kGlA, ldz, in.z), sl1, n1, f1);
    double const e2 = field(p, e, fma(kGlB, ldz, in.z), sl2, n2, f2);
    double const eavg = 0.5 * (e1 + e2);
    double const w = q * ldz * eavg;
    double const kick = p.kick * eavg;
    double const v1[3] = {m0.gb * in.dx, m0.gb * in.dy, fma(m0.gb, in.dz, kick)};
    double const inv1 = frsqrt(v1[0] * v1[0] + v1[1] * v1[1] + v1[2] * v1[2]);
    double const d1[3] = {v1[0] * inv1, v1[1] * inv1, v1[2] * inv1};
    double const k1 = in.k + 0.5 * w;
    double const sp = aux[i], dsp = aux[p.n + i];
    double const loss = sp * L;
    if (end == end_code(p, step, sub, 0)) {
        // stopped in the drag: z1 = z + L d_z, K the constant cutoff, d as it came
        a = Adj{a.z, a.dx, a.dy, a.dz + a.z * L, a.z * in.dz * dL};
        return;
    }
    double ez_bar = 0.0, l_bar = 0.0, w_bar = 0.0;
    double d1_bar[3];
    double const z1_bar = a.z;
    double const k2 = k1 - loss;
    Motion const m2 = motion(k2);
    double const v2[3] = {m2.gb * d1[0], m2.gb * d1[1], fma(m2.gb, d1[2], kick)};
    double const inv2 = frsqrt(v2[0] * v2[0] + v2[1] * v2[1] + v2[2] * v2[2]);
    double const d2[3] = {v2[0] * inv2, v2[1] * inv2, v2[2] * inv2};
    // scatter: d3 = R d2 -> d2_bar = R^T d3_bar
    double const n[3] = {aux[2 * p.n + i], aux[3 * p.n + i], aux[4 * p.n + i]};
    double const c = aux[5 * p.n + i], sn = aux[6 * p.n + i];
    double d2_bar[3] = {a.dx, a.dy, a.dz};
    rotate(n, c, -sn, d2_bar);
    // kick 2: d2 = v2 / |v2|, v2 = gb(K2) d1 + kick z, K3 = K2 + W/2
    double const dd = d2[0] * d2_bar[0] + d2[1] * d2_bar[1] + d2[2] * d2_bar[2];
    double v2_bar[3];
    for (int c3 = 0; c3 < 3; ++c3) v2_bar[c3] = (d2_bar[c3] - d2[c3] * dd) * inv2;
    double const gb2_bar = v2_bar[0] * d1[0] + v2_bar[1] * d1[1] + v2_bar[2] * d1[2];
    for (int c3 = 0; c3 < 3; ++c3) d1_bar[c3] = m2.gb * v2_bar[c3];
    ez_bar += p.kick * v2_bar[2];
    double const k2_bar = a.k + gb2_bar * (kInvMeC2 * (m2.g * m2.igb));
    w_bar += 0.5 * a.k;
    // drag: K2 = K1 - rho S(K1) L
    double const k1_bar = k2_bar * (1.0 - dsp * L);
    l_bar -= k2_bar * sp;
    // kick 1: d1 = v1 / |v1|, K1 = K + W/2
    double const dd1 = d1[0] * d1_bar[0] + d1[1] * d1_bar[1] + d1[2] * d1_bar[2];
    double v1_bar[3];
    for (int c3 = 0; c3 < 3; ++c3) v1_bar[c3] = (d1_bar[c3] - d1[c3] * dd1) * inv1;
    double const gb0_bar = v1_bar[0] * in.dx + v1_bar[1] * in.dy + v1_bar[2] * in.dz;
    Adj r{0.0, m0.gb * v1_bar[0], m0.gb * v1_bar[1], m0.gb * v1_bar[2],
          k1_bar + gb0_bar * (kInvMeC2 * (m0.g * m0.igb))};
    ez_bar += p.kick * v1_bar[2];
    w_bar += 0.5 * k1_bar;
    // W = q dz L <E>
    double const we = w_bar * q * eavg;
    r.dz += we * L;
    l_bar += we * in.dz;
    ez_bar += w_bar * q * ldz;
    // <E> = (E(za) + E(zb)) / 2
    double const e_bar = 0.5 * ez_bar;
    sums.add(g, n1, e_bar, f1);
    sums.add(g, n2, e_bar, f2);
    double const za_bar = e_bar * sl1, zb_bar = e_bar * sl2;
    r.z += za_bar + zb_bar + z1_bar;
    double const ldz_bar = za_bar * kGlA + zb_bar * kGlB + z1_bar;
    l_bar += ldz_bar * in.dz;
    r.dz += ldz_bar * L;
    // L = v(K) h
    r.k += l_bar * dL;
    a = r;
}

__device__ __forceinline__ State load(const double* __restrict__ s, int64_t n, int64_t i)
{
    return State{s[i], s[n + i], s[2 * n + i], s[3 * n + i], s[4 * n + i], s[5 * n + i] != 0.0 ? 1 : 0};
}
__device__ __forceinline__ void store(double* __restrict__ s, int64_t n, int64_t i, State const& st)
{
    s[i] = st.z;
    s[n + i] = st.dx;
    s[2 * n + i] = st.dy;
    s[3 * n + i] = st.dz;
    s[4 * n + i] = st.k;
    s[5 * n + i] = st.alive ? 1.0 : 0.0;
}

// Blocks of 64 threads, one particle per thread, registers for eleven blocks
// per SM: the SMs' shares of 1e5 particles then differ by 7 % where blocks of
// 128 in a grid of 4 per SM left a fifth of the threads a second particle
// (forward and reverse of 96 steps: 50.6 ms with those, 48.8 with these; with
// registers for eight or six blocks, or blocks of 32, 50.3 to 51.7).
constexpr int kThreads = 64;
constexpr int kResident = 11;

// Forward over every step: checkpoints ckpt[c] (6 x n each) at the steps
// c * C; from step tape_from on the tape of the reverse pass (its entries
// start there); final state and the loss.
__global__ void __launch_bounds__(kThreads, kResident) forward_kernel(Params p, const double* __restrict__ e, const double* __restrict__ arena,
                               const double* __restrict__ seeds, const double* __restrict__ w,
                               const uint64_t* __restrict__ id, double* __restrict__ ckpt,
                               double* __restrict__ final_state, double* __restrict__ partials, int tape_from,
                               double* __restrict__ tape, double* __restrict__ aux)
{
    double acc = 0.0;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < p.n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        State st = load(seeds, p.n, i);
        double const z_init = st.z;
        int32_t end = p.replay ? p.ends[i] : -1;
        for (int t = 0; t < p.steps; ++t) {
            if (t % p.ckpt_every == 0) store(ckpt + static_cast<int64_t>(t / p.ckpt_every) * 6 * p.n, p.n, i, st);
            for (int q = 0; q < p.substeps; ++q) {
                // one call for both, so that a taped run takes the steps of an untaped one to the bit
                bool const taped = t >= tape_from;
                int64_t const k = static_cast<int64_t>(t - tape_from) * p.substeps + q;
                if (taped) store(tape + k * 6 * p.n, p.n, i, st);
                substep(p, e, arena, id[i], t, q, st, end, taped ? aux + k * kAux * p.n : nullptr, i);
            }
        }
        if (!p.replay) p.ends[i] = end;
        store(final_state, p.n, i, st);
        acc += w[i] * (sig((st.k - p.k_th) / p.tau_k)
                       - p.lambda * (sig((st.z - p.z_p) / p.tau_z) - sig((z_init - p.z_p) / p.tau_z)));
    }
    // the loss is summed in a fixed order (warp tree, the warps of a block
    // in turn, then the blocks by sum_partials_kernel), so the same
    // nodes give the same loss to the bit and finite differences of the loss
    // carry only its rounding
    __shared__ double warp_sums[32];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0.0;
        for (int k = 0; k < static_cast<int>(blockDim.x >> 5); ++k) b += warp_sums[k];
        partials[blockIdx.x] = b;
    }
}

// The block partials summed in a fixed order with Neumaier's compensation (a
// warp's lanes each over every 32nd, then the lanes in turn), so the loss is the
// correctly rounded sum of the partials to within an ulp or two and a
// difference of two losses carries only their final roundings.
__global__ void sum_partials_kernel(const double* __restrict__ partials, int count, double* loss)
{
    double s = 0.0, c = 0.0;
    auto add = [&](double x) {
        double const t = s + x;
        c += fabs(s) >= fabs(x) ? (s - t) + x : (x - t) + s;
        s = t;
    };
    for (int k = threadIdx.x; k < count; k += 32) add(partials[k]);
    for (int lane = 1; lane < 32; ++lane) {
        double const other = __shfl_sync(0xffffffffu, s, lane), low = __shfl_sync(0xffffffffu, c, lane);
        if (threadIdx.x == 0) {
            add(other);
            c += low;
        }
    }
    if (threadIdx.x == 0) *loss = s + c;
}

// tape[0]: whether this reverse pass can use the tape: it is still the forward
// pass's (tape[1]) and the field nodes are the forward pass's, to the bit.  A
// pass that cannot overwrites the tape, as does one with segments that need a
// slot of it (`overwritten`).
__global__ void tape_usable_kernel(const double* __restrict__ a, const double* __restrict__ b, int n, int overwritten,
                                   int* tape)
{
    __shared__ int differ;
    if (threadIdx.x == 0) differ = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        if (__double_as_longlong(a[k]) != __double_as_longlong(b[k])) differ = 1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        tape[0] = tape[1] && !differ;
        if (!tape[0] || overwritten) tape[1] = 0;
    }
}

// Reverse pass over one checkpoint segment [t0, t1): unless the forward pass
// left the segment's tape and it is usable (taped, *taped != 0), recompute onto the tape (substep inputs, 6 x n per entry); then run the
// adjoint back through it.
__global__ void __launch_bounds__(kThreads, kResident) reverse_segment_kernel(Params p, const double* __restrict__ e, const double* __restrict__ arena,
                                       const uint64_t* __restrict__ id, const double* __restrict__ ckpt, int t0,
                                       int t1, double* __restrict__ tape, double* __restrict__ aux,
                                       double* __restrict__ adj, double* __restrict__ grad,
                                       const int* __restrict__ taped)
{
    extern __shared__ double g[];
    for (int k = threadIdx.x; k < p.n_nodes; k += blockDim.x) g[k] = 0.0;
    __syncthreads();
    int64_t const entries = static_cast<int64_t>(t1 - t0) * p.substeps;
    bool const kept = taped && *taped != 0;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < p.n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        int32_t end = p.ends[i];
        State st{};
        if (!kept) st = load(ckpt, p.n, i);
        for (int t = t0; t < t1 && !kept; ++t) {
            for (int q = 0; q < p.substeps; ++q) {
                int64_t const k = static_cast<int64_t>(t - t0) * p.substeps + q;
                store(tape + k * 6 * p.n, p.n, i, st);
                substep(p, e, arena, id[i], t, q, st, end, aux + k * kAux * p.n, i);
            }
        }
        Adj a{adj[i], adj[p.n + i], adj[2 * p.n + i], adj[3 * p.n + i], adj[4 * p.n + i]};
        NodeSums sums;
        for (int64_t k = entries - 1; k >= 0; --k) {
            int const t = t0 + static_cast<int>(k / p.substeps), q = static_cast<int>(k % p.substeps);
            State const in = load(tape + k * 6 * p.n, p.n, i);
            substep_adjoint(p, e, aux + k * kAux * p.n, i, t, q, in, end, a, sums, g);
        }
        sums.flush(g);
        adj[i] = a.z;
        adj[p.n + i] = a.dx;
        adj[2 * p.n + i] = a.dy;
        adj[3 * p.n + i] = a.dz;
        adj[4 * p.n + i] = a.k;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < p.n_nodes; k += blockDim.x) {
        if (g[k] != 0.0) atomicAdd(grad + k, g[k]);
    }
}

// The loss adjoint at the final state.
__global__ void seed_adjoint_kernel(Params p, const double* __restrict__ final_state, const double* __restrict__ w,
                                    double* __restrict__ adj)
{
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < p.n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        double const z = final_state[i], k = final_state[4 * p.n + i];
        adj[i] = -w[i] * p.lambda * dsig((z - p.z_p) / p.tau_z) / p.tau_z;
        adj[p.n + i] = 0.0;
        adj[2 * p.n + i] = 0.0;
        adj[3 * p.n + i] = 0.0;
        adj[4 * p.n + i] = w[i] * dsig((k - p.k_th) / p.tau_k) / p.tau_k;
    }
}

}  // namespace adj
}  // namespace rrea_dev

namespace rrea_launch {

// Device memory a staged problem's tape may take where it is more than the one
// segment every reverse pass needs.
constexpr int64_t kTapeBytes = int64_t{8} << 30;

struct AdjointState {
    rrea_dev::adj::Params p{};
    int64_t cap = 0;
    double* seeds = nullptr;   // 6 x n
    double* w = nullptr;
    uint64_t* id = nullptr;
    double* ckpt = nullptr;    // n_ckpt x 6 x n
    double* final_state = nullptr;
    double* tape = nullptr;    // kept x C x substeps x 6 x n
    double* aux = nullptr;     // kept x C x substeps x kAux x n
    int kept = 1;              // segments the tape holds, the last ones
    double* nodes = nullptr;   // field nodes of the last recording forward
    int* tape_state = nullptr; // tape_usable_kernel's two words
    bool taped = false;        // the last forward left a tape
    double* adj = nullptr;     // 5 x n
    double* loss = nullptr;
    double* partials = nullptr;   // one loss partial per forward block
    int32_t* ends = nullptr;   // n end records (Params::ends)
    bool recorded = false;     // a recording forward has run
    int blocks = 1;
    int segments() const { return (p.steps + p.ckpt_every - 1) / p.ckpt_every; }
    int first_kept() const { return segments() > kept ? segments() - kept : 0; }
};

void adjoint_free(AdjointState* s)
{
    if (!s) return;
    for (void* ptr : {static_cast<void*>(s->seeds), static_cast<void*>(s->w), static_cast<void*>(s->id),
                      static_cast<void*>(s->ckpt), static_cast<void*>(s->final_state), static_cast<void*>(s->tape),
                      static_cast<void*>(s->aux), static_cast<void*>(s->nodes), static_cast<void*>(s->tape_state),
                      static_cast<void*>(s->adj), static_cast<void*>(s->loss), static_cast<void*>(s->partials),
                      static_cast<void*>(s->ends)}) {
        if (ptr) cudaFree(ptr);
    }
    delete s;
}

cudaError_t adjoint_stage(AdjointSetup const& in, const double* seeds6, const double* w, const uint64_t* id,
                          int num_sms, AdjointState*& out)
{
    adjoint_free(out);
    out = nullptr;
    auto* s = new AdjointState();
    rrea_dev::adj::Params& p = s->p;
    p.n = in.n;
    p.n_nodes = in.n_nodes;
    p.z0 = in.z0;
    p.dz_node = in.dz_node;
    p.steps = in.steps;
    p.substeps = in.substeps;
    p.ckpt_every = in.ckpt_every;
    p.h = in.dt / in.substeps;
    p.rho = in.rho;
    p.cutoff = in.cutoff;
    p.scatter_rms = in.scatter_rms;
    p.k_th = in.k_th;
    p.tau_k = in.tau_k;
    p.z_p = in.z_p;
    p.tau_z = in.tau_z;
    p.lambda = in.lambda;
    p.seed = in.seed;
    p.col = in.col;
    p.soft = in.soft;
    p.rows = in.rows;
    p.inv_dz = 1.0 / in.dz_node;
    p.kick = -(rrea_dev::kC * rrea_dev::kInvMeC2) * 0.5 * p.h;
    int64_t const want = (in.n + rrea_dev::adj::kThreads - 1) / rrea_dev::adj::kThreads;
    s->blocks = static_cast<int>(want < 1 ? 1 : want < num_sms * 64 ? want : num_sms * 64);
    int64_t const n = in.n;
    int64_t const n_ckpt = (in.steps + in.ckpt_every - 1) / in.ckpt_every;
    cudaError_t e = cudaSuccess;
    auto alloc = [&](auto** ptr, int64_t count) {
        if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(ptr), sizeof(**ptr) * static_cast<size_t>(count > 0 ? count : 1));
    };
    alloc(&s->seeds, 6 * n);
    alloc(&s->w, n);
    alloc(&s->id, n);
    alloc(&s->ckpt, n_ckpt * 6 * n);
    alloc(&s->final_state, 6 * n);
    alloc(&s->nodes, in.n_nodes);
    alloc(&s->tape_state, 2);
    alloc(&s->adj, 5 * n);
    alloc(&s->loss, 1);
    alloc(&s->partials, s->blocks);
    alloc(&s->ends, n);
    // The forward pass leaves the tape of the last segments, as many as
    // kept_segments allows (at least one, which the reverse pass needs for any
    // other), so that those are not computed a second time: 1e5 electrons
    // over 96 steps in three segments, forward 16.1 to 17.0 and reverse 32.4
    // to 15.4 ms (an entry is written and read once, 4 GB in all, where
    // computing it again took half of the reverse pass).  It comes last,
    // and gives way to one segment where it does not fit.
    int64_t const entries = static_cast<int64_t>(in.ckpt_every) * in.substeps;
    int64_t const segment_bytes = (6 + rrea_dev::adj::kAux) * static_cast<int64_t>(sizeof(double)) * entries * n;
    size_t free_bytes = 0, total_bytes = 0;
    if (e == cudaSuccess) e = cudaMemGetInfo(&free_bytes, &total_bytes);
    s->kept = rrea_host::kept_segments(n_ckpt, segment_bytes, kTapeBytes, static_cast<int64_t>(free_bytes));
    alloc(&s->tape, s->kept * entries * 6 * n);
    alloc(&s->aux, s->kept * entries * rrea_dev::adj::kAux * n);
    if (e == cudaErrorMemoryAllocation && s->kept > 1) {
        cudaGetLastError();
        if (s->tape) cudaFree(s->tape);
        s->tape = nullptr;
        s->kept = 1;
        e = cudaSuccess;
        alloc(&s->tape, entries * 6 * n);
        alloc(&s->aux, entries * rrea_dev::adj::kAux * n);
    }
    p.ends = s->ends;
    p.replay = 0;
    if (e == cudaSuccess && n > 0) {
        e = cudaMemcpy(s->seeds, seeds6, sizeof(double) * 6 * n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(s->w, w, sizeof(double) * n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(s->id, id, sizeof(uint64_t) * n, cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess) {
        adjoint_free(s);
        return e;
    }
    out = s;
    return cudaSuccess;
}

cudaError_t adjoint_forward(AdjointState& s, const double* arena, const double* e_nodes, bool replay, double& loss,
                            cudaStream_t stream)
{
    cudaError_t e = cudaSuccess;
    rrea_dev::adj::Params p = s.p;
    p.replay = replay ? 1 : 0;
    // a frozen forward moves the checkpoints but leaves no tape
    s.taped = false;
    if (!replay) {
        e = cudaMemcpyAsync(s.nodes, e_nodes, sizeof(double) * static_cast<size_t>(p.n_nodes), cudaMemcpyDeviceToDevice,
                            stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(s.tape_state + 1, 1, sizeof(int), stream);
        if (e != cudaSuccess) return e;
    }
    int const tape_from = replay ? p.steps : s.first_kept() * p.ckpt_every;
    note_launch();
    rrea_dev::adj::forward_kernel<<<s.blocks, rrea_dev::adj::kThreads, 0, stream>>>(
        p, e_nodes, arena, s.seeds, s.w, s.id, s.ckpt, s.final_state, s.partials, tape_from, s.tape, s.aux);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    note_launch();
    rrea_dev::adj::sum_partials_kernel<<<1, 32, 0, stream>>>(s.partials, s.blocks, s.loss);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (!replay) s.recorded = s.taped = true;
    e = cudaMemcpyAsync(&loss, s.loss, sizeof(double), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    return e;
}

bool adjoint_recorded(AdjointState const& s) { return s.recorded; }

cudaError_t adjoint_backward(AdjointState& s, const double* arena, const double* e_nodes, double* grad,
                             cudaStream_t stream)
{
    rrea_dev::adj::Params p = s.p;
    p.replay = 1;   // the reverse pass follows the recorded ends
    cudaError_t e = cudaMemsetAsync(grad, 0, sizeof(double) * p.n_nodes, stream);
    if (e != cudaSuccess) return e;
    note_launch();
    rrea_dev::adj::seed_adjoint_kernel<<<s.blocks, 256, 0, stream>>>(p, s.final_state, s.w, s.adj);
    int const n_ckpt = s.segments();
    if (s.taped) {
        note_launch();
        rrea_dev::adj::tape_usable_kernel<<<1, 256, 0, stream>>>(e_nodes, s.nodes, p.n_nodes, s.first_kept() > 0 ? 1 : 0,
                                                               s.tape_state);
    }
    int64_t const entries = static_cast<int64_t>(p.ckpt_every) * p.substeps;
    size_t const shmem = sizeof(double) * static_cast<size_t>(p.n_nodes);
    for (int c = n_ckpt - 1; c >= 0; --c) {
        int const t0 = c * p.ckpt_every;
        int const t1 = t0 + p.ckpt_every < p.steps ? t0 + p.ckpt_every : p.steps;
        // a segment without a tape takes the first slot: its segment is done by then
        int64_t const slot = c > s.first_kept() ? c - s.first_kept() : 0;
        note_launch();
        rrea_dev::adj::reverse_segment_kernel<<<s.blocks, rrea_dev::adj::kThreads, shmem, stream>>>(
            p, e_nodes, arena, s.id, s.ckpt + static_cast<int64_t>(c) * 6 * p.n, t0, t1, s.tape + slot * entries * 6 * p.n,
            s.aux + slot * entries * rrea_dev::adj::kAux * p.n, s.adj, grad, s.taped && c >= s.first_kept() ? s.tape_state : nullptr);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t adjoint_final_state(AdjointState const& s, double* host6)
{
    return cudaMemcpy(host6, s.final_state, sizeof(double) * 6 * static_cast<size_t>(s.p.n), cudaMemcpyDeviceToHost);
}

int adjoint_max_nodes() { return rrea_dev::adj::kMaxNodes; }

}  // namespace rrea_launch
