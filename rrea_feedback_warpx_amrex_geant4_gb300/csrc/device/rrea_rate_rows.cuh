// Table values from interval polynomials.
//
// Every table the charged loops query with a continuous argument (energy,
// path length, CDF node) is smooth between two of its nodes: a power of x
// (log-log), linear in log x, the inverse of that, or the fraction of log x
// between two nodes.  Evaluated as the reference does, each value costs a
// binary search, a logarithm and an exponential, 35 slots of the FP64 pipe
// and a dozen dependent loads.  The loader instead cuts the axis at every
// node and every 1/256 octave and stores the Taylor polynomial of each
// column about each row's middle, so a value is four FP64 multiply-adds:
// with |d| <= 2^-9, d = (q - xc) / xc, the terms from d^4 on are below 2^-36
// of the value and are summed in FP32 (their rounding is below 2^-59 of it).
// The polynomial is the interpolant itself to within an ulp (a row whose
// bound exceeds that is flagged and the caller interpolates as before).
//
// Lookup: the top bits of q (exponent and 8 mantissa bits) name a cell, the
// cell its first row, and the row is the first with q <= hi, the same
// half-open rule as std::lower_bound on the nodes.  Most cells have one row.
#pragma once

#include "../rrea_arena.h"

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define RREA_HD __host__ __device__ __forceinline__
#else
#define RREA_HD inline
#endif

namespace rrea_dev {

RREA_HD long long row_bits(double x)
{
#if defined(__CUDA_ARCH__)
    return __double_as_longlong(x);
#else
    long long b;
    memcpy(&b, &x, sizeof(b));
    return b;
#endif
}
RREA_HD double row_double(long long b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double(b);
#else
    double x;
    memcpy(&x, &b, sizeof(x));
    return x;
#endif
}
RREA_HD float row_float(uint32_t u)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, sizeof(f));
    return f;
#endif
}
RREA_HD uint32_t row_float_bits(float f)
{
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, sizeof(u));
    return u;
#endif
}

// FP64 <-> FP32 on the integer pipe (a conversion instruction takes as long
// as an FP64 multiply-add).  Narrowing truncates, and both flush magnitudes
// below 2^-126 to zero (narrowing keeps the sign, which the quadrant of an
// angle needs); magnitudes from 2^128 on are the caller's to keep out.  They
// are for the small terms of a sum.
RREA_HD float narrow_f32(double x)
{
    long long const b = row_bits(x);
    uint32_t const hi = static_cast<uint32_t>(static_cast<unsigned long long>(b) >> 32);
    uint32_t const lo = static_cast<uint32_t>(b);
    uint32_t const mag = hi & 0x7fffffffu;
    uint32_t const u = ((mag - 0x38000000u) << 3) | (lo >> 29);
    return row_float((mag < 0x38100000u ? 0u : u) | (hi & 0x80000000u));
}
RREA_HD double widen_f32(float f)
{
    uint32_t const u = row_float_bits(f);
    uint32_t const hi = (((u & 0x7fffffffu) >> 3) + 0x38000000u) | (u & 0x80000000u);
    unsigned long long const b = (static_cast<unsigned long long>(hi) << 32) | (u << 29);
    return row_double((u & 0x7f800000u) == 0u ? 0LL : static_cast<long long>(b));
}

// A row's record and the argument's offset in it.
struct RowHit {
    const double* rec;
    double d;
    float df;
};

RREA_HD uint64_t row_meta(RowHit const& h) { return static_cast<uint64_t>(row_bits(h.rec[2])); }
RREA_HD uint32_t row_flags(RowHit const& h) { return static_cast<uint32_t>(row_meta(h)); }
RREA_HD int row_index(RowHit const& h) { return static_cast<int>(row_meta(h) >> 32); }

// The row of q; false when q is outside the rows' range (or not finite).
RREA_HD bool find_row(const double* __restrict__ arena, RreaRowIndex const& ix, double q, RowHit& h)
{
    long long const b = row_bits(q);
    // (an object without rows has a negative span and lo_key 0)
    unsigned long long const off = static_cast<unsigned long long>(b) - static_cast<unsigned long long>(ix.lo_key);
    if (ix.span_key < 0 || off > static_cast<unsigned long long>(ix.span_key)) return false;
    int const cell = static_cast<int>((b >> RREA_ROW_CELL_SHIFT) - ix.first_cell);
    const int32_t* start = reinterpret_cast<const int32_t*>(arena + ix.start);
    const long long* hi = reinterpret_cast<const long long*>(arena + ix.hi);
    int row = start[cell];
    while (hi[row] < b) ++row;   // ends: a cell's last row reaches its upper edge
    const double* rec = arena + ix.rec + static_cast<int64_t>(row) * ix.stride;
    h.rec = rec;
    h.d = (q - rec[0]) * rec[1];
    h.df = narrow_f32(h.d);
    return true;
}

// Column c of the row: c0 + d (c1 + d (c2 + d (c3 + tail))), the tail
// d (c4 + d (c5 + d c6)) in FP32.
RREA_HD double row_value(RowHit const& h, int c)
{
    const double* p = h.rec + RREA_ROW_HEADER + RREA_ROW_COLUMN * c;
    const float* t = reinterpret_cast<const float*>(p + 4);
    float const tail = h.df * (t[0] + h.df * (t[1] + h.df * t[2]));
    double const c3 = p[3] + widen_f32(tail);
    double const c0 = p[0], c1 = p[1], c2 = p[2];
    return fma(h.d, fma(h.d, fma(h.d, c3, c2), c1), c0);
}

// d (column c) / d d = c1 + d (2 c2 + d (3 c3 + d (4 c4 + d (5 c5 + 6 d c6)))); divided by xc it is the
// derivative by the argument.
RREA_HD double row_slope(RowHit const& h, int c)
{
    const double* p = h.rec + RREA_ROW_HEADER + RREA_ROW_COLUMN * c;
    const float* t = reinterpret_cast<const float*>(p + 4);
    float const tail = h.df * (4.0f * t[0] + h.df * (5.0f * t[1] + h.df * 6.0f * t[2]));
    double const c3 = 3.0 * p[3] + widen_f32(tail);
    double const c1 = p[1], c2 = p[2];
    return fma(h.d, fma(h.d, c3, 2.0 * c2), c1);
}

}  // namespace rrea_dev
