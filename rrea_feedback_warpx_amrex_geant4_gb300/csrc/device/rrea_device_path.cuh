// Device transport geometry and kinematics: chord construction and RZ
// clipping, material path, path field work, half kick, cone sampling and
// the competing-hazard selection.  Register-resident, fixed-capacity
// structures replace the reference's heap vectors; the arithmetic follows the
// cited reference primitives operation for operation.
#pragma once

#include "rrea_device_common.cuh"

namespace rrea_dev {

// I/RreaTransportPath.H:13-73
struct Piece {
    double begin, end, length, shift;
};

// NP is the piece capacity: 1 for an absorbing z domain (a clipped chord
// has exactly one in-domain piece), RREA_ARENA_MAX_PIECES for periodic z.
template <int NP>
struct Path {
    double sx, sy, sz, ex, ey, ez;
    double dx, dy, dz;  // end - start
    double full, in_begin, in_end, in_length;
    double inv_full;    // 1 / full
    bool exits;
    int npieces;
    Piece pieces[NP];
};

struct Geom {
    double rlo, rhi, zlo, zhi;
    bool periodic;
    double r2_in, z_in_lo, z_in_hi;  // a billionth of the domain inside its faces
};
__device__ __forceinline__ Geom make_geom(StepConstants const& C)
{
    rrea_gpu_config const& c = C.cfg;
    return Geom{c.r_lo, c.r_hi, c.z_lo, c.z_hi, c.periodic_z != 0, C.r2_inner, C.z_inner_lo, C.z_inner_hi};
}

// The wrap into [zlo, zhi) of a periodic domain.  Out of line: the
// remainder's code would otherwise sit at every point of the transport loop,
// which no absorbing domain ever reaches.
static __device__ __noinline__ double periodic_wrap(double z, double zlo, double zhi)
{
    double const len = zhi - zlo;
    if (!(gt0(len))) return z;
    double w = fmod(z - zlo, len);
    if (lt0(w)) w += len;
    return zlo + w;
}
// S/RreaTransportPath.cpp:13-27
__device__ __forceinline__ double wrap_z(Geom const& g, double z)
{
    return g.periodic ? periodic_wrap(z, g.zlo, g.zhi) : z;
}
// S/RreaTransportPath.cpp:42-52
template <int NP>
__device__ __forceinline__ void point_at_full(Path<NP> const& p, Geom const& g, double f, double& x, double& y, double& z)
{
    f = max0(fmin(1.0, f));
    x = p.sx + f * p.dx;
    y = p.sy + f * p.dy;
    z = wrap_z(g, p.sz + f * p.dz);
}
// S/RreaTransportPath.cpp:54-71
template <int NP>
__device__ __forceinline__ void point_at_piece(Path<NP> const& p, Geom const& g, Piece const& pc, double f, double& x,
                                               double& y, double& z)
{
    if constexpr (NP == 1) {
        // an absorbing domain's one piece: its callers pass fractions inside
        // it, its shift is zero, and a z an ulp past a face reads the edge cell
        x = p.sx + f * p.dx;
        y = p.sy + f * p.dy;
        z = p.sz + f * p.dz;
        return;
    }
    f = fmax(pc.begin, fmin(pc.end, f));
    x = p.sx + f * p.dx;
    y = p.sy + f * p.dy;
    z = p.sz + f * p.dz + pc.shift;
    z = fmax(g.zlo, fmin(g.zhi, z));
}
// S/RreaTransportPath.cpp:29-40
__device__ __forceinline__ bool outside_certified(Geom const& g, double r, double z)
{
    if (!finite_bits(r) || !finite_bits(z)) return true;
    if (r < g.rlo || r >= g.rhi) return true;
    return !g.periodic && (z < g.zlo || z >= g.zhi);
}

// A chord with both ends strictly inside an absorbing domain, a convex body:
// nothing is clipped, its one piece is [0, 1].  Almost every microchord of
// the transport loops is one, and skips two radii, three divisions and a
// square root.  False (p unset) when an end is within a billionth of a face,
// outside, or not finite: clip_chord decides those.
__device__ __forceinline__ bool strictly_inside(Geom const& g, double r2, double z)
{
    // a NaN or negative-zero-free non-negative r2 orders as its bits
    return dbits(r2) < dbits(g.r2_in) && z > g.z_in_lo && z < g.z_in_hi;
}
// StartInside: the caller knows it of the start (r02 is not read).
template <int NP, bool StartInside = false>
__device__ __forceinline__ bool clip_inside(double x0, double y0, double z0, double r02, double x1, double y1, double z1,
                                            double r12, Geom const& g, Path<NP>& p)
{
    if constexpr (NP != 1) return false;
    if (!StartInside && !strictly_inside(g, r02, z0)) return false;
    if (!strictly_inside(g, r12, z1)) return false;
    double const dx = x1 - x0, dy = y1 - y0, dz = z1 - z0;
    double const n2 = dx * dx + dy * dy + dz * dz;
    if (!gt0(n2)) return false;
    double const inv = frsqrt(n2);
    p.sx = x0;
    p.sy = y0;
    p.sz = z0;
    p.ex = x1;
    p.ey = y1;
    p.ez = z1;
    p.dx = dx;
    p.dy = dy;
    p.dz = dz;
    p.full = n2 * inv;
    p.inv_full = inv;
    p.in_begin = 0.0;
    p.in_end = 1.0;
    p.in_length = p.full;
    p.exits = false;
    p.npieces = 1;
    p.pieces[0] = Piece{0.0, 1.0, p.full, 0.0};
    return true;
}

// S/RreaTransportPath.cpp:73-295 on Cartesian chord ends (x0, y0, z0) ->
// (x1, y1, z1) with their radii r0, r1.  Periodic seams use double
// arithmetic where the host reference uses long double.
// Out of line: the chords that reach it are at a face (clip_inside).
template <int NP>
__device__ __noinline__ void clip_chord(double x0, double y0, double z0, double r0, double x1, double y1, double z1,
                                           double r1, bool ends_finite, Geom const& g, Path<NP>& p, Err& err)
{
    if (!ends_finite || !finite_bits(r0) || !finite_bits(z0) || !finite_bits(r1) || !finite_bits(z1) || lt0(r0) || lt0(r1)) {
        err.set(RREA_GPU_ERR_GEOMETRY);
        p.npieces = 0;
        p.full = 0.0;
        p.inv_full = 0.0;
        p.in_begin = p.in_end = p.in_length = 0.0;
        p.exits = false;
        return;
    }
    p.sx = x0;
    p.sy = y0;
    p.sz = z0;
    p.ex = x1;
    p.ey = y1;
    p.ez = z1;
    double const dx = p.ex - p.sx, dy = p.ey - p.sy, dz = p.ez - p.sz;
    p.dx = dx;
    p.dy = dy;
    p.dz = dz;
    p.full = sqrt(dx * dx + dy * dy + dz * dz);
    p.inv_full = 1.0 / p.full;
    p.in_begin = 0.0;
    double const scale = fmax(1.0, fmax(g.rhi, fmax(fabs(g.zlo), fabs(g.zhi))));
    double const tol = 64.0 * kEps * scale;
    if (r0 < g.rlo - tol || r0 > g.rhi + tol || z0 < g.zlo - tol || z0 > g.zhi + tol) {
        err.set(RREA_GPU_ERR_GEOMETRY);
    }
    double exit_fraction = 1.0;
    if (!g.periodic) {
        if (gt0(dz)) {
            double const c = (g.zhi - z0) / dz;
            if (ge0(c) && c < exit_fraction) exit_fraction = c;
        } else if (lt0(dz)) {
            double const c = (g.zlo - z0) / dz;
            if (ge0(c) && c < exit_fraction) exit_fraction = c;
        }
    }
    double const a = dx * dx + dy * dy;
    if (gt0(a)) {
        double const b = 2.0 * (p.sx * dx + p.sy * dy);
        for (int cyl = 0; cyl < 2; ++cyl) {
            bool const outer = cyl == 0;
            double const radius = outer ? g.rhi : g.rlo;
            if (!outer && !(gt0(g.rlo))) break;
            double const c = p.sx * p.sx + p.sy * p.sy - radius * radius;
            double const disc = b * b - 4.0 * a * c;
            if (lt0(disc)) continue;
            double const root = sqrt(max0(disc));
            double const inv2a = 0.5 / a;
            double const roots[2] = {(-b - root) * inv2a, (-b + root) * inv2a};
            for (int q = 0; q < 2; ++q) {
                double const cand = roots[q];
                if (le0(cand) || cand > 1.0) continue;
                double const deriv = 2.0 * a * cand + b;
                bool const leaves = outer ? gt0(deriv) : deriv < 0.0;
                if (leaves && ge0(cand) && cand < exit_fraction) exit_fraction = cand;
            }
        }
    }
    p.in_end = max0(fmin(1.0, exit_fraction));
    p.in_length = p.full * (p.in_end - p.in_begin);
    p.exits = p.in_end < 1.0 - 64.0 * kEps;

    if constexpr (NP == 1) {
        // Absorbing z: no seams, so the breakpoints are [in_begin, in_end]
        // (already sorted); deduplication drops the piece when the two are
        // within the tolerance.  Static indices keep the path in registers.
        double const l = p.in_begin, r = p.in_end;
        bool const dup = fabs(l - r) <= 128.0 * kEps * fmax(1.0, fmax(fabs(l), fabs(r)));
        p.npieces = 0;
        if (!dup && r > l) {
            p.pieces[0] = Piece{l, r, p.full * (r - l), 0.0};
            p.npieces = 1;
        }
        return;
    }
    // Breakpoints: [in_begin, seams..., in_end], sorted and deduplicated.
    double bp[NP + 1];
    int nb = 0;
    bp[nb++] = p.in_begin;
    if (g.periodic && fabs(dz) > 0.0 && p.in_end > p.in_begin) {
        double const zend = z0 + dz * p.in_end;
        double const period = g.zhi - g.zlo;
        double const low = fmin(z0, zend), high = fmax(z0, zend);
        double const first = floor((low - g.zlo) / period) + 1.0;
        double const last = ceil((high - g.zlo) / period) - 1.0;
        for (double image = first; image <= last; image += 1.0) {
            double const seam = g.zlo + image * period;
            double const frac = (seam - z0) / dz;
            double const ftol = 128.0 * kEps * fmax(1.0, fabs(frac));
            if (frac > p.in_begin + ftol && frac < p.in_end - ftol) {
                if (nb >= NP) {
                    err.set(RREA_GPU_ERR_CAPACITY);
                    break;
                }
                bp[nb++] = frac;
            }
        }
    }
    bp[nb++] = p.in_end;
    // insertion sort (tiny)
    for (int i = 1; i < nb; ++i) {
        double const v = bp[i];
        int j = i - 1;
        while (j >= 0 && bp[j] > v) {
            bp[j + 1] = bp[j];
            --j;
        }
        bp[j + 1] = v;
    }
    // std::unique with a relative tolerance
    int nu = 0;
    for (int i = 0; i < nb; ++i) {
        if (nu > 0) {
            double const l = bp[nu - 1], r = bp[i];
            if (fabs(l - r) <= 128.0 * kEps * fmax(1.0, fmax(fabs(l), fabs(r)))) continue;
        }
        bp[nu++] = bp[i];
    }
    double const period_m = g.zhi - g.zlo;
    p.npieces = 0;
    for (int i = 1; i < nu; ++i) {
        double const b0 = bp[i - 1], e0 = bp[i];
        if (!(e0 > b0)) continue;
        double shift = 0.0;
        if (g.periodic) {
            double const mid = 0.5 * (b0 + e0);
            double const mid_z = z0 + mid * dz;
            double const image = floor((mid_z - g.zlo) / period_m);
            shift = -image * period_m;
        }
        p.pieces[p.npieces++] = Piece{b0, e0, p.full * (e0 - b0), shift};
    }
}

// ClipRz as the reference calls it, on cylindrical ends (r, theta, z).
template <int NP>
__device__ __forceinline__ void clip_rz(const double* __restrict__ arena, double r0, double th0, double z0, double r1,
                                        double th1, double z1, Geom const& g, Path<NP>& p, Err& err)
{
    bool const finite = finite_bits(th0) && finite_bits(th1);
    double s0 = 0.0, c0 = 1.0, s1 = 0.0, c1 = 1.0;
    if (finite) {
        fsincos(arena, th0, s0, c0);
        fsincos(arena, th1, s1, c1);
    }
    double const x0 = r0 * c0, y0 = r0 * s0, x1 = r1 * c1, y1 = r1 * s1;
    if (finite && !lt0(r0) && !lt0(r1) && clip_inside(x0, y0, z0, r0 * r0, x1, y1, z1, r1 * r1, g, p)) return;
    Path<NP> out;   // the out-of-line call's, so that p stays in registers
    Err e;
    clip_chord(x0, y0, z0, r0, x1, y1, z1, r1, finite, g, out, e);
    p = out;
    if (e.code) err.set(e.code);
}

// The chords the transport loops build run between Cartesian points, which
// the reference passes through ClipRz's (r, theta, z) interface as
// (hypot(x, y), atan2(y, x), z) and turns back into r cos(theta),
// r sin(theta).  Clipping the Cartesian ends directly gives the same chord to
// within an ulp of each coordinate and saves an atan2 and a sincos per end.
// True for a chord inside the domain (clip_inside).
template <int NP>
__device__ __forceinline__ bool clip_xyz(double x0, double y0, double z0, double x1, double y1, double z1, Geom const& g,
                                         Path<NP>& p, Err& err)
{
    if (clip_inside(x0, y0, z0, fma(x0, x0, y0 * y0), x1, y1, z1, fma(x1, x1, y1 * y1), g, p)) return true;
    bool const finite = finite_bits(x0) && finite_bits(y0) && finite_bits(x1) && finite_bits(y1);
    Path<NP> out;   // the out-of-line call's, so that p stays in registers
    Err e;
    clip_chord(x0, y0, z0, rz_radius(x0, y0), x1, y1, z1, rz_radius(x1, y1), finite, g, out, e);
    p = out;
    if (e.code) err.set(e.code);
    return false;
}

// ------------------------------------------------------------ kinematics
// I/RreaSeedSchedule.H:31-43
__device__ __forceinline__ double proper_velocity_from_kinetic(double k)
{
    if (le0(k)) return 0.0;
    double const gm = 1.0 + k * kInvMeC2;
    return kC * sqrt(max0(gm * gm - 1.0));
}
// O/RreaParticleInteraction.H:1494-1506
__device__ __forceinline__ double kinetic_from_proper_velocity(double ux, double uy, double uz)
{
    double const u2 = ux * ux + uy * uy + uz * uz;
    double const gm = sqrt(1.0 + u2 / (kC * kC));
    return u2 * kMeC2 / ((kC * kC) * (gm + 1.0));
}
// gamma beta = sqrt(gamma^2 - 1) of kinetic energy k, from gamma^2 - 1 =
// (k/mc^2)(k/mc^2 + 2) (no cancellation); 0 for k <= 0.
__device__ __forceinline__ double gamma_beta(double k)
{
    double const t = k * kInvMeC2;
    return le0(k) ? 0.0 : fsqrt(t * (t + 2.0));
}
// Speed c beta (O/RreaParticleInteraction.H:92-105: c sqrt(1 - 1/gamma^2)) as
// c (gamma beta) / gamma, with gamma beta handed on; NaN for k < 0 or not
// finite, as there.
__device__ __forceinline__ double charged_speed(double k, double& gb)
{
    if (!finite_bits(k) || lt0(k)) {
        gb = 0.0;
        return __longlong_as_double(0x7ff8000000000000LL);
    }
    gb = gamma_beta(k);
    double const t = k * kInvMeC2;
    return (kC * gb) * frsqrt(fma(t, t + 2.0, 1.0));
}
// O/RreaChargedInterleave.H:294-307.  The reference divides by sqrt(n2);
// scaling by rsqrt(n2) (within an ulp of 1/sqrt(n2)) gives the same unit
// vector to within two ulps per component for a third of the FP64
// instructions.  A zero norm falls back to +z as in the reference.
__device__ __forceinline__ void normalize(double& x, double& y, double& z)
{
    double const n2 = x * x + y * y + z * z;
    if (!(gt0(n2))) {
        x = 0.0; y = 0.0; z = 1.0;
        return;
    }
    double const inv = frsqrt(n2);
    x *= inv; y *= inv; z *= inv;
}
// O/RreaChargedInterleave.H:309-364 about a unit axis d, for cos_t in [-1, 1].
// The reference normalises the axis, a copy of it, both basis vectors and
// the result.  With b1 = e x d / rho (e the z axis, or x where |d_z| > 0.9;
// rho = |e x d|) and b2 = d x b1 the rotated vector is, component by
// component,
//   along e:      d_e cos + B rho^2
//   across, a, b: a (cos - B d_e) - A b,  b (cos - B d_e) + A a
// with A, B = (sin / rho) (cos phi, sin phi) and sin / rho = sin^2 / sqrt(sin^2
// rho^2), one inverse root; the direction differs from the reference's by
// ulps (and is renormalised by the next half kick).
__device__ __forceinline__ void cone_unit(const double* __restrict__ arena, double dx, double dy, double dz, double cos_t,
                                          double u_phi, double& ox, double& oy, double& oz)
{
    bool const about_x = (dbits(dz) & 0x7fffffffffffffffull) > 0x3feccccccccccccdull;  // |d_z| > 0.9
    double const pole = about_x ? dx : dz, a = about_x ? dy : dx, b = about_x ? dz : dy;
    // cos^2 is rounded on its own before the subtraction, as the reference's
    // x86-64 build rounds it: a fused 1 - cos^2 differs by up to an ulp of 1,
    // which a small-angle deflection (cos near 1, the Wentzel-VI energies)
    // amplifies by 1/sin^2 in sin and then in every later direction.
    double const s2 = 1.0 - __dmul_rn(cos_t, cos_t);
    double const rho2 = fma(a, a, b * b);
    double const q = gt0(s2) ? s2 * frsqrt(s2 * rho2) : 0.0;
    double sp, cp;
    sincos_turn(arena, u_phi, sp, cp);
    double const A = q * cp, B = q * sp;
    double const h = fma(-B, pole, cos_t);
    double const op = fma(pole, cos_t, B * rho2);
    double const oa = fma(a, h, -(A * b));
    double const ob = fma(b, h, A * a);
    ox = about_x ? op : oa;
    oy = about_x ? oa : ob;
    oz = about_x ? ob : op;
}
// The same about any axis and for any cos_t (clamped), u_phi in [0, 1).
__device__ __forceinline__ void cone_direction(const double* __restrict__ arena, double ax, double ay, double az,
                                               double cos_t, double u_phi, double& ox, double& oy, double& oz)
{
    normalize(ax, ay, az);
    cone_unit(arena, ax, ay, az, fmin(1.0, fmax(-1.0, cos_t)), u_phi, ox, oy, oz);
}
// O/RreaChargedInterleave.H:371-389
__device__ __forceinline__ int poisson_capped(double mean, double u, int kmax)
{
    if (le0(mean)) return 0;
    double p = exp(-mean);
    double cum = p;
    int k = 0;
    while (u > cum && k < kmax) {
        ++k;
        p *= mean / static_cast<double>(k);
        cum += p;
    }
    return k;
}
__device__ __forceinline__ double unit_cycle(double u)
{
    u -= floor(u);
    return lt0(u) ? u + 1.0 : u;
}
// O/RreaChargedInterleave.H:391-463
__device__ __forceinline__ double moller_cos(double kp, double ks_or_scat)
{
    double const v = ks_or_scat * (kp + 2.0 * kMeC2) / (kp * (ks_or_scat + 2.0 * kMeC2));
    return sqrt(fmin(1.0, max0(v)));
}
__device__ __forceinline__ void moller_lab_directions(const double* __restrict__ arena, double px, double py, double pz, double kp, double ks,
                                                      double u_az, double& opx, double& opy, double& opz,
                                                      double& osx, double& osy, double& osz)
{
    normalize(px, py, pz);
    u_az = unit_cycle(u_az);
    double cs;
    {
        double const a = max0(kp), b = max0(ks);
        cs = (le0(a) || le0(b)) ? 1.0 : moller_cos(a, b);
    }
    double cpm;
    {
        double const scat = max0(kp - ks);
        cpm = (le0(kp) || le0(scat)) ? 1.0 : moller_cos(kp, scat);
    }
    cone_unit(arena, px, py, pz, cs, u_az, osx, osy, osz);
    cone_unit(arena, px, py, pz, cpm, unit_cycle(u_az + 0.5), opx, opy, opz);
}
// O/RreaChargedInterleave.H:465-496
__device__ __forceinline__ void photon_recoil(double k0, double eg, double gx, double gy, double gz, double& cx,
                                              double& cy, double& cz)
{
    eg = max0(eg);
    if (le0(k0) || le0(eg)) return;
    normalize(cx, cy, cz);
    normalize(gx, gy, gz);
    double const p0 = sqrt(max0(k0 * (k0 + 2.0 * kMeC2)));
    double const px = p0 * cx - eg * gx, py = p0 * cy - eg * gy, pz = p0 * cz - eg * gz;
    double const n = sqrt(px * px + py * py + pz * pz);
    if (gt0(n)) {
        Divisor const d = make_divisor(n);
        cx = quot(px, d); cy = quot(py, d); cz = quot(pz, d);
        normalize(cx, cy, cz);
    }
}

struct FieldRange {
    double work, ex, ey, ez, bx, by, length;  // B is azimuthal: no z component
};

// O/RreaChargedInterleave.H:100-138 with the Boris rotation of
// I/RreaLorentzPush.H:21-46, in units of c: v = u/c with |v| = gb at energy k.
// The rotation keeps |v|, so the norm of the kicked vector (needed for its
// gamma) normalises the result; without B nothing rotates.
__device__ __forceinline__ void half_kick(FieldRange const& f, double half_dt, double q, double gb, double& k, double& dx,
                                          double& dy, double& dz)
{
    double const s = q * (kC / kMeC2) * half_dt;
    double vx = fma(gb, dx, s * f.ex);
    double vy = fma(gb, dy, s * f.ey);
    double vz = fma(gb, dz, s * f.ez);
    double const v2 = vx * vx + vy * vy + vz * vz;
    if (ne0(f.bx) || ne0(f.by)) {
        // t = q B dt / (2 m gamma), w = 2 t / (1 + t^2)
        double const h = (0.5 * kC) * s * frsqrt(1.0 + v2);
        double const tx = h * f.bx, ty = h * f.by;
        double const t2 = tx * tx + ty * ty;
        // 1 / (1 + t^2): below t^2 = 2^-18 the series' next term is below 2^-54
        double const d = 2.0 * (__double2hiint(t2) < 0x3ed00000 ? fma(t2, t2 - 1.0, 1.0) : 1.0 / (1.0 + t2));
        double const wx = tx * d, wy = ty * d;
        double const px = vx - vz * ty;
        double const py = vy + vz * tx;
        double const pz = vz + vx * ty - vy * tx;
        vx -= pz * wy;
        vy += pz * wx;
        vz += px * wy - py * wx;
    }
    if (gt0(v2) && finite_bits(v2)) {
        double const inv = frsqrt(v2);
        dx = vx * inv;
        dy = vy * inv;
        dz = vz * inv;
    }
    k = max0(k + 0.5 * f.work);
}

// ------------------------------------------------------------ field gather
// Cell-centred total field (Maxwell + ambient face averages, computed once
// per step by a prep kernel exactly as S/RreaAmrexAdvance.cpp:556-565 forms
// them) and the corner Btheta of the replicated Maxwell vectors.
struct FieldView {
    Divisor div_dr, div_dz;
    const double* __restrict__ cell_er;  // nr*nz, i + nr*j
    const double* __restrict__ cell_ez;  // nr*nz
    const double* __restrict__ bt;       // (nr+1)*(nz+1), i + (nr+1)*j
    int nr, nz;
    double dr, dz, r_lo, z_lo;
    bool periodic;
    bool has_b;
    // ensemble mode: instance k's fields follow instance k-1's at these
    // strides (0: one field for every particle)
    int64_t inst_cells, inst_bt;

    // The field of one ensemble instance (the particle's cpu ordinal).
    __device__ __forceinline__ FieldView for_instance(int64_t inst) const
    {
        FieldView v = *this;
        if (inst_cells) {
            v.cell_er += inst * inst_cells;
            v.cell_ez += inst * inst_cells;
            v.bt += inst * inst_bt;
        }
        return v;
    }
};

// x / d - offset (0 or 1/2) split into a whole cell and the fraction in it:
// the whole part is read from the low word of a sum (a floor and two
// conversions otherwise, 3 to 4 FP64 slots).  Within an ulp of a cell's edge
// the split may name either neighbour with a fraction of 1 or 0 (to an ulp):
// the weights on either are the same.
template <bool Centred>
__device__ __forceinline__ void split_cell(double x, Divisor const& d, int& cell, double& fraction)
{
    constexpr double magic = 6755399441055744.0;   // 1.5 2^52: the sum's low word is the nearest integer
    if constexpr (Centred) {
        double const t = fma(x, d.y, magic - 1.0);   // nearest of (x/d - 1/2) - 1/2
        cell = __double2loint(t);
        fraction = fma(x, d.y, -0.5) - (t - magic);
    } else {
        double const t = fma(x, d.y, magic);
        cell = __double2loint(t);
        fraction = fma(x, d.y, magic - t);
        if (lt0(fraction)) {
            cell -= 1;
            fraction += 1.0;
        }
    }
}

// S/RreaAmrexAdvance.cpp:532-579 with I/RreaFieldGatherStencil.H:49-133 and
// MaxwellBthetaAt :511-530
__device__ __forceinline__ void gather(FieldView const& fv, double r, double z, double& er, double& ez, double& bth)
{
    int ir0, iz0;
    double tx, tz;
    double const zr = z - fv.z_lo;
    split_cell<true>(r - fv.r_lo, fv.div_dr, ir0, tx);
    split_cell<true>(zr, fv.div_dz, iz0, tz);
    int const i0 = max(0, min(fv.nr - 1, ir0));
    int const i1 = max(0, min(fv.nr - 1, ir0 + 1));
    int j0, j1;
    if (fv.periodic) {
        j0 = (iz0 + fv.nz) % fv.nz;
        j1 = (iz0 + 1 + fv.nz) % fv.nz;
    } else {
        j0 = max(0, min(fv.nz - 1, iz0));
        j1 = max(0, min(fv.nz - 1, iz0 + 1));
    }
    size_t const r0 = static_cast<size_t>(fv.nr) * j0, r1 = static_cast<size_t>(fv.nr) * j1;
    auto bilinear = [](double v00, double v01, double v10, double v11, double a, double b) {
        double const lo = fma(b, v01 - v00, v00), hi = fma(b, v11 - v10, v10);
        return fma(a, hi - lo, lo);
    };
    er = bilinear(__ldg(fv.cell_er + i0 + r0), __ldg(fv.cell_er + i0 + r1), __ldg(fv.cell_er + i1 + r0),
                  __ldg(fv.cell_er + i1 + r1), tx, tz);
    ez = bilinear(__ldg(fv.cell_ez + i0 + r0), __ldg(fv.cell_ez + i0 + r1), __ldg(fv.cell_ez + i1 + r0),
                  __ldg(fv.cell_ez + i1 + r1), tx, tz);
    // inside the first cell centre Er falls linearly to the axis
    if (ir0 < 0) er *= max0(2.0 * quot(r - fv.r_lo, fv.div_dr));
    if (!fv.has_b || le0(r)) {
        bth = 0.0;
        return;
    }
    int a0, b0;
    double tr, tzz;
    split_cell<false>(r, fv.div_dr, a0, tr);
    split_cell<false>(zr, fv.div_dz, b0, tzz);
    // the corners' range, clamped as r <= nr dr and 0 <= z - z_lo <= nz dz are
    if (a0 < 0) { a0 = 0; tr = 0.0; }
    if (a0 > fv.nr - 1) { a0 = fv.nr - 1; tr = 1.0; }
    if (b0 < 0) { b0 = 0; tzz = 0.0; }
    if (b0 > fv.nz - 1) { b0 = fv.nz - 1; tzz = 1.0; }
    size_t const w = static_cast<size_t>(fv.nr + 1);
    const double* const corner = fv.bt + a0 + w * b0;
    bth = bilinear(__ldg(corner), __ldg(corner + w), __ldg(corner + 1), __ldg(corner + w + 1), tr, tzz);
}

// O/RreaPathFieldWork.H:57-150 with the two-node rule of
// I/RreaGaussLegendre8.H:24-60
template <int NP>
__device__ __forceinline__ FieldRange path_field_work(FieldView const& fv, Geom const& g, Path<NP> const& p, double q,
                                                      double begin, double end, Err& err)
{
    FieldRange res{0, 0, 0, 0, 0, 0, 0};
    if (!(gt0(p.full))) return res;
    begin = fmax(p.in_begin, begin);
    end = fmin(p.in_end, end);
    if (!(end > begin)) return res;
    double const pdx = p.dx * p.inv_full, pdy = p.dy * p.inv_full, pdz = p.dz * p.inv_full;
#pragma unroll
    for (int ip = 0; ip < NP; ++ip) {
        if (ip >= p.npieces) break;
        Piece const& pc = p.pieces[ip];
        double const pb = NP == 1 ? begin : fmax(begin, pc.begin);
        double const pe = NP == 1 ? end : fmin(end, pc.end);
        if (NP != 1 && !(pe > pb)) continue;
        double const mid = 0.5 * (pb + pe);
        double const half = 0.5 * (pe - pb);
        double const off = half * kGl2Node;
        double acc[6];
#pragma unroll
        for (int node = 0; node < 2; ++node) {
            double const f = node == 0 ? mid - off : mid + off;
            double x, y, z;
            point_at_piece(p, g, pc, f, x, y, z);
            // r and the radial unit vector from one rsqrt of r^2 (within two
            // ulps of hypot and of the quotients by it)
            double const r2 = fma(x, x, y * y);
            double r = 0.0, rad = 0.0, rc = 1.0, rs = 0.0;
            if (gt0(r2)) {
                double const inv = frsqrt(r2);
                r = r2 * inv;
                rc = x * inv;
                rs = y * inv;
                rad = pdx * rc + pdy * rs;
            }
            double er, ez, bth;
            gather(fv, r, z, er, ez, bth);
            double const work = er * rad + ez * pdz;
            if (!finite_bits(work) || !finite_bits(er) || !finite_bits(ez) || !finite_bits(bth)) {
                err.set(RREA_GPU_ERR_INVALID_STATE);
            }
            double const v[4] = {work, er * rc, er * rs, ez};
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[c] = node == 0 ? v[c] : acc[c] + v[c];
            if (fv.has_b) {
                acc[4] = node == 0 ? -bth * rs : acc[4] - bth * rs;
                acc[5] = node == 0 ? bth * rc : acc[5] + bth * rc;
            }
        }
        if (!fv.has_b) acc[4] = acc[5] = 0.0;
        double const w = p.full * half;
        res.work += (q * w) * acc[0];
        if constexpr (NP == 1) {
            // one piece: the mean over the path is the mean of its two nodes
            res.ex = 0.5 * acc[1];
            res.ey = 0.5 * acc[2];
            res.ez = 0.5 * acc[3];
            res.bx = 0.5 * acc[4];
            res.by = 0.5 * acc[5];
        } else {
            res.ex += w * acc[1];
            res.ey += w * acc[2];
            res.ez += w * acc[3];
            res.bx += w * acc[4];
            res.by += w * acc[5];
        }
        res.length += p.full * (pe - pb);
    }
    if (NP != 1 && gt0(res.length)) {
        Divisor const dl = make_divisor(res.length);
        res.ex = quot(res.ex, dl); res.ey = quot(res.ey, dl); res.ez = quot(res.ez, dl);
        res.bx = quot(res.bx, dl); res.by = quot(res.by, dl);
    }
    return res;
}

// ------------------------------------------------------------ material path
// O/RreaMaterialPath.H:47-199: one interval per in-domain piece, with the
// piece's density ratio taken at its midpoint.
template <int NP>
struct Intervals {
    int n;
    double begin[NP], end[NP], length[NP], density[NP];
};

__device__ __forceinline__ double positive_or(double v, double fb) { return gt0(v) ? v : fb; }

// The altitude density profile bound to the context
// (rrea.air_density_model=altitude_profile); n == 0 is the uniform ratio.
struct DensityProfile {
    const double* alt;  // n strictly increasing altitudes above mean sea level (m)
    const double* val;  // n densities (kg/m^3), strictly positive
    int n;
    double alt0;        // altitude of z = 0 (ProfileAltitudeMslAtZ, O/RreaWarpXCoupling.cpp:67-71)
    double ref;         // the tables' reference density (kg/m^3)
};

// TransportDensityRatioAtZ (O/RreaWarpXCoupling.cpp:79-95) with
// RreaAltitudeProfile::Interpolate (S/RreaAltitudeProfile.cpp:125-147): the
// uniform ratio without a profile; with one, the density interpolated
// linearly at alt0 + z over the reference density.  An altitude outside the
// profile fails the step (the reference throws).  The interpolation is
// evaluated without contraction so it rounds as the reference does.
__device__ __forceinline__ double density_ratio_at_z(DensityProfile const& d, double uniform, double z, Err& err)
{
    if (d.n == 0) return uniform;
    double const a = d.alt0 + z;
    if (!(a >= __ldg(d.alt) && a <= __ldg(d.alt + d.n - 1))) {
        err.set(RREA_GPU_ERR_RANGE);
        return uniform;
    }
    // std::upper_bound: the first node above a
    long long const ak = order_key(a);
    const long long* __restrict__ xk = reinterpret_cast<const long long*>(d.alt);
    int up = 0, count = d.n;
    while (count > 0) {
        int const step = count >> 1;
        if (__ldg(xk + up + step) <= ak) {
            up += step + 1;
            count -= step + 1;
        } else {
            count = step;
        }
    }
    double v;
    if (up == 0) {
        v = __ldg(d.val);
    } else if (up == d.n) {
        v = __ldg(d.val + d.n - 1);
    } else {
        int const lo = up - 1;
        double const span = __ldg(d.alt + up) - __ldg(d.alt + lo);
        double const t = gt0(span) ? (a - __ldg(d.alt + lo)) / span : 0.0;
        v = __dadd_rn(__dmul_rn(1.0 - t, __ldg(d.val + lo)), __dmul_rn(t, __ldg(d.val + up)));
    }
    return v / d.ref;
}

// :60-114
template <int NP>
__device__ __forceinline__ void build_intervals(Path<NP> const& p, double rho, Intervals<NP>& iv)
{
    iv.n = 0;
    if constexpr (NP == 1) {
        Piece const& pc = p.pieces[0];
        if (p.npieces < 1 || !(gt0(pc.length))) return;
        iv.begin[0] = pc.begin;
        iv.end[0] = pc.end;
        iv.length[0] = pc.length;
        // the reference's (length * rho) / length, to within an ulp
        iv.density[0] = rho;
        iv.n = 1;
    } else {
        for (int i = 0; i < p.npieces; ++i) {
            Piece const& pc = p.pieces[i];
            if (!(gt0(pc.length))) continue;
            double dl = 0.0;
            if (pc.end > pc.begin && gt0(p.full)) dl = p.full * (pc.end - pc.begin) * positive_or(rho, rho);
            iv.begin[iv.n] = pc.begin;
            iv.end[iv.n] = pc.end;
            iv.length[iv.n] = pc.length;
            iv.density[iv.n] = positive_or(dl / pc.length, rho);
            ++iv.n;
        }
    }
}
// :60-114 with the density profile: each piece's ratio at its midpoint
// (integrate_density_piece_m's midpoint rule); `rho` is the step's ratio,
// the fallback of a non-positive value.
// Kept out of line: the uniform-density transport never calls it, and its
// code stays out of the transport loop.
template <int NP>
__device__ __noinline__ void build_intervals_profile(Path<NP> const& p, Geom const& g, DensityProfile const& dp,
                                                     double rho, Intervals<NP>& iv, Err& err)
{
    iv.n = 0;
#pragma unroll 1
    for (int i = 0; i < p.npieces; ++i) {
        Piece const& pc = p.pieces[i];
        if (!(gt0(pc.length))) continue;
        double dl = 0.0;
        if (pc.end > pc.begin && gt0(p.full)) {
            double x, y, z;
            point_at_piece(p, g, pc, 0.5 * (pc.begin + pc.end), x, y, z);
            dl = p.full * (pc.end - pc.begin) * positive_or(density_ratio_at_z(dp, rho, z, err), rho);
        }
        iv.begin[iv.n] = pc.begin;
        iv.end[iv.n] = pc.end;
        iv.length[iv.n] = pc.length;
        iv.density[iv.n] = positive_or(dl / pc.length, rho);
        ++iv.n;
    }
}
template <int NP>
__device__ __forceinline__ void build_intervals(Path<NP> const& p, Geom const& g, DensityProfile const& dp,
                                                double rho, Intervals<NP>& iv, Err& err)
{
    if (dp.n == 0) build_intervals(p, rho, iv);
    else build_intervals_profile(p, g, dp, rho, iv, err);
}
// :117-136
template <int NP>
__device__ __forceinline__ double density_path(Intervals<NP> const& iv, Path<NP> const& p, double b, double e)
{
    if constexpr (NP == 1) {
        // the one interval is the path's inside, and every caller's [b, e] lies in it
        return iv.n > 0 && e > b ? p.full * (e - b) * iv.density[0] : 0.0;
    }
    b = fmax(p.in_begin, b);
    e = fmin(p.in_end, e);
    if (!(e > b)) return 0.0;
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        if (i >= iv.n) break;
        double const bb = fmax(b, iv.begin[i]), ee = fmin(e, iv.end[i]);
        if (ee > bb) s += p.full * (ee - bb) * iv.density[i];
    }
    return s;
}
// :142-170
template <int NP>
__device__ __forceinline__ double fraction_at_density_path(Intervals<NP> const& iv, Path<NP> const& p, double b, double e,
                                                           double target, Err& err)
{
    b = fmax(p.in_begin, b);
    e = fmin(p.in_end, e);
    if (!finite_bits(target) || lt0(target)) {
        err.set(RREA_GPU_ERR_INVALID_STATE);
        return e;
    }
    double rem = target;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        if (i >= iv.n) break;
        double const bb = fmax(b, iv.begin[i]), ee = fmin(e, iv.end[i]);
        if (!(ee > bb) || !(gt0(iv.density[i]))) continue;
        double const c = p.full * (ee - bb) * iv.density[i];
        if (rem <= c) return bb + rem / (p.full * iv.density[i]);
        rem -= c;
    }
    return e;
}
// :175-199
template <int NP>
__device__ __forceinline__ double max_uniform_slice(Intervals<NP> const& iv, Path<NP> const& p, uint64_t n)
{
    double const span = p.in_end - p.in_begin;
    double const d = static_cast<double>(n);
    double m = 0.0;
    for (uint64_t i = 0; i < n; ++i) {
        m = fmax(m, density_path(iv, p, p.in_begin + static_cast<double>(i) / d * span,
                                 p.in_begin + static_cast<double>(i + 1U) / d * span));
    }
    return m;
}

// ------------------------------------------------------------ hazards
// O/RreaParticleInteraction.H:1402-1454
struct Selection {
    bool valid, event;
    int channel;
    double sampled, total;
};
// `draw_u2` gives the channel draw, taken only for an event.  Most hazards
// end without one, and -log(1 - u) >= u: a draw above the total depth (by
// more than every rounding: its high word above the total's, and above
// 2^-30) settles that on the integer pipe, without the logarithm.
template <class Draw>
__device__ __forceinline__ Selection select_hazard(const double* __restrict__ arena, double t0, double t1, double t2,
                                                  int count, double u1, Draw&& draw_u2)
{
    Selection r{false, false, -1, 0.0, 0.0};
    double const taus[3] = {t0, t1, t2};
    if (count < 1 || count > 3 || !finite_bits(u1)) return r;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (i >= count) break;
        if (!finite_bits(taus[i]) || lt0(taus[i])) return r;
        r.total += taus[i];
    }
    r.valid = finite_bits(r.total);
    if (!r.valid) return r;
    if (__double2hiint(u1) > max(__double2hiint(r.total) + 1, 0x3e100000)) return r;
    u1 = max0(fmin(1.0, u1));
    r.sampled = -flog(arena, fmax(1.0e-30, 1.0 - u1));
    if (!(r.sampled < r.total)) return r;
    double const u2 = max0(fmin(1.0, draw_u2()));
    r.event = finite_bits(u2);
    if (!r.event) {
        r.valid = false;
        return r;
    }
    double const target = u2 * r.total;
    double cum = 0.0;
    int last_open = -1;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (i >= count) break;
        if (gt0(taus[i])) last_open = i;
        cum += taus[i];
        if (target < cum) {
            r.channel = i;
            return r;
        }
    }
    r.channel = last_open;
    r.valid = r.channel >= 0;
    r.event = r.valid;
    return r;
}

// ------------------------------------------------------------ terminal helpers
// O/RreaParticleInteraction.H:318-354
__device__ __forceinline__ bool cartesian_half_open(Geom const& g, double x, double y, double z)
{
    if (!finite_bits(x) || !finite_bits(y)) return false;
    double const r = rz_radius(x, y);
    return finite_bits(r) && finite_bits(z) && g.rhi > g.rlo && g.zhi > g.zlo && r >= g.rlo && r < g.rhi && z >= g.zlo
        && z < g.zhi;
}
// RreaChargedBoundaryCrossingForPath (O/RreaParticleInteraction.H:468-540):
// the exact absorbing-face point of the final microchord and the crossed
// faces (bits 1 r_hi, 2 z_lo, 4 z_hi).  Returns false when no face is
// certified.
template <int NP>
__device__ __forceinline__ bool charged_crossing(Path<NP> const& p, Geom const& g, double& sr, double& sz, double& cr,
                                                 double& cz, uint32_t& faces)
{
    double cx, cy;
    point_at_full(p, g, p.in_end, cx, cy, cz);
    cz = wrap_z(g, cz);
    cr = rz_radius(cx, cy);
    sr = rz_radius(p.sx, p.sy);
    sz = wrap_z(g, p.sz);
    double const scale = fmax(1.0, fmax(g.rhi, fmax(fabs(g.zlo), fabs(g.zhi))));
    double const tol = 512.0 * kEps * scale;
    bool const on_r = fabs(cr - g.rhi) <= tol;
    bool const on_zlo = !g.periodic && fabs(cz - g.zlo) <= tol;
    bool const on_zhi = !g.periodic && fabs(cz - g.zhi) <= tol;
    double const dx = p.ex - p.sx, dy = p.ey - p.sy, dz = p.ez - p.sz;
    double const outward = cx * dx + cy * dy;
    faces = 0u;
    if (on_r && outward > -tol * scale) { faces |= 1u; cr = g.rhi; }
    if (on_zlo && lt0(dz)) { faces |= 2u; cz = g.zlo; }
    if (on_zhi && gt0(dz)) { faces |= 4u; cz = g.zhi; }
    if (faces == 0u) {
        if (on_r) { faces |= 1u; cr = g.rhi; }
        if (on_zhi) { faces |= 4u; cz = g.zhi; }
    }
    return faces != 0u && finite_bits(sr) && finite_bits(sz) && finite_bits(cr) && finite_bits(cz);
}

// O/RreaParticleInteraction.H:409-452 (clipped policy: RREA owns every escape)
template <int NP>
__device__ __forceinline__ void clipped_escape_policy(Path<NP> const& p, Geom const& g, double er, double ez,
                                                      bool& escapes, bool& invalidate)
{
    if (!finite_bits(er) || !finite_bits(ez)) {
        escapes = true;
        invalidate = true;
        return;
    }
    double const cz = wrap_z(g, ez);
    bool const outside = outside_certified(g, er, cz);
    escapes = p.exits || outside;
    invalidate = escapes;
}

}  // namespace rrea_dev
