// Builds the interval-polynomial rows that the device reads in place of a
// search, a logarithm and an exponential per table value
// (device/rrea_rate_rows.cuh): the axis cut at every node and every 1/256
// octave, each piece's interpolant as a Taylor polynomial about its middle.
#pragma once

#include "../rrea_arena.h"

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

namespace rrea_host {

// One column of interval-polynomial rows: a table on nodes x (n of them).
struct RowColumn {
    enum Kind { Table, InverseSemilog, LogFraction } kind = Table;
    int mode = 0;                // RreaInterpMode of a Table
    const double* x = nullptr;
    const double* y = nullptr;   // values (LogFraction: none)
    int n = 0;
    bool index = false;          // its lower node index goes into the rows' meta
};

// Taylor coefficients of the column about xc on a row (lo, hi]; false
// when the truncated polynomial is not the interpolant to within an ulp.
inline bool row_polynomial(RowColumn const& col, double lo, double hi, double xc, double c[7], int& lower)
{
    // the interval (x[up - 1], x[up]] the row lies in (std::lower_bound's rule)
    int up = static_cast<int>(std::lower_bound(col.x, col.x + col.n, hi) - col.x);
    if (up == 0) up = 1;
    if (up >= col.n) return false;
    lower = up - 1;
    double const x0 = col.x[up - 1], x1 = col.x[up];
    double const dl = std::log1p((x1 - x0) / x0);
    double const l0 = std::log1p((xc - x0) / x0);
    if (!(dl > 1.0e-9) || hi > x1 || lo < x0) return false;
    auto log_series = [&](double a, double m) {  // a + m log(x / xc)
        c[0] = a;
        for (int k = 1; k < 7; ++k) c[k] = (k % 2 ? m : -m) / k;
    };
    double const y0 = col.y ? col.y[up - 1] : 0.0, y1 = col.y ? col.y[up] : 1.0;
    bool linear = true;
    if (col.kind == RowColumn::LogFraction) {
        log_series(l0 / dl, 1.0 / dl);
    } else if (col.kind == RowColumn::InverseSemilog) {
        // 1 / (y0 + (y1 - y0) log(x / x0) / dl): reciprocal of the series
        double g[7];
        log_series(y0 + (y1 - y0) * (l0 / dl), (y1 - y0) / dl);
        for (int k = 0; k < 7; ++k) g[k] = c[k];
        if (!(y0 > 0.0) || !(y1 > 0.0)) return false;
        linear = false;
        c[0] = 1.0 / g[0];
        for (int k = 1; k < 7; ++k) {
            double sum = 0.0;
            for (int i = 1; i <= k; ++i) sum += g[i] * c[k - i];
            c[k] = -sum / g[0];
        }
    } else if (col.mode == RREA_INTERP_LINEAR) {
        double const m = (y1 - y0) / (x1 - x0);
        c[0] = y0 + m * (xc - x0);
        c[1] = m * xc;
        for (int k = 2; k < 7; ++k) c[k] = 0.0;
    } else if (col.mode == RREA_INTERP_LOGX_LINEAR
               || (col.mode == RREA_INTERP_LOGLOG_ZERO_THRESHOLD && !(y0 > 0.0 && y1 > 0.0))) {
        log_series(y0 + (y1 - y0) * (l0 / dl), (y1 - y0) / dl);
    } else {
        if (!(y0 > 0.0) || !(y1 > 0.0)) return false;
        // y0 (x / x0)^s about xc: the binomial series
        linear = false;
        double const s = std::log(y1 / y0) / dl;
        c[0] = y0 * std::exp(s * l0);
        for (int k = 1; k < 7; ++k) c[k] = c[k - 1] * (s - (k - 1)) / k;
    }
    // what is dropped (the seventh term, bounded by the sixth's growth) and
    // the FP32 rounding of the tail, against the largest value on the row (of
    // a piece linear in x or log x, and of a fraction: on its interval, whose
    // ends the reference's t in [0, 1] weights)
    double const d = std::max(std::fabs(lo - xc), std::fabs(hi - xc)) / xc;
    double top = std::max(std::fabs(c[0] + d * c[1]), std::fabs(c[0] - d * c[1]));
    if (linear) top = std::max(top, std::max(y0, y1));
    double const d4 = d * d * d * d;
    double const tail = d4 * (std::fabs(c[4]) + d * (std::fabs(c[5]) + d * std::fabs(c[6])));
    for (int k = 0; k < 7; ++k) {
        if (!std::isfinite(c[k])) return false;
    }
    if (top != 0.0 && top < 1.0e-25) return false;   // the tail's coefficients would leave FP32
    return std::fabs(c[6]) * d4 * d * d * d <= 2.0e-17 * top && tail * 1.2e-7 <= 1.2e-16 * top;
}

// Rows over [x_min, x_max]: cut at every node of every column and at the
// cells' edges.  `columns[c]` lists the tables that serve column c, each on
// its own range (the angle tables hand over at the transition energy).
inline void push_rows(std::vector<double>& arena, RreaRowIndex& ix, double x_min, double x_max, std::vector<std::vector<RowColumn>> const& columns)
{
    auto bits = [](double v) {
        int64_t b;
        std::memcpy(&b, &v, sizeof(b));
        return b;
    };
    auto value = [](int64_t b) {
        double v;
        std::memcpy(&v, &b, sizeof(v));
        return v;
    };
    std::vector<double> nodes;
    for (auto const& alternatives : columns) {
        for (RowColumn const& col : alternatives) nodes.insert(nodes.end(), col.x, col.x + col.n);
    }
    std::sort(nodes.begin(), nodes.end());
    nodes.erase(std::unique(nodes.begin(), nodes.end()), nodes.end());
    int const ncol = static_cast<int>(columns.size());
    ix.stride = (RREA_ROW_HEADER + RREA_ROW_COLUMN * ncol + 3) / 4 * 4;
    ix.lo_key = bits(x_min);
    ix.span_key = bits(x_max) - ix.lo_key;
    ix.first_cell = ix.lo_key >> RREA_ROW_CELL_SHIFT;
    int64_t const cells = (bits(x_max) >> RREA_ROW_CELL_SHIFT) - ix.first_cell + 1;
    std::vector<int32_t> start;
    std::vector<double> hi, rec;
    auto add_row = [&](double lo, double top) {
        std::vector<double> r(static_cast<std::size_t>(ix.stride), 0.0);
        double const xc = lo + 0.5 * (top - lo);
        r[0] = xc;
        r[1] = 1.0 / xc;
        uint32_t flags = 0;
        int32_t index = 0;
        for (int c = 0; c < ncol; ++c) {
            bool good = columns[c].empty();   // an unused column stays zero
            for (RowColumn const& col : columns[c]) {
                if (good || !(col.x[0] <= lo && top <= col.x[col.n - 1])) continue;
                double p[7];
                int lower = 0;
                if (!row_polynomial(col, lo, top, xc, p, lower)) continue;
                good = true;
                if (col.index) index = lower;
                double* const out = r.data() + RREA_ROW_HEADER + RREA_ROW_COLUMN * c;
                for (int k = 0; k < 4; ++k) out[k] = p[k];
                float const t[4] = {static_cast<float>(p[4]), static_cast<float>(p[5]), static_cast<float>(p[6]), 0.0f};
                std::memcpy(out + 4, t, sizeof(t));
            }
            if (!good) flags |= 1u << c;
        }
        uint64_t const meta = (static_cast<uint64_t>(static_cast<uint32_t>(index)) << 32) | flags;
        std::memcpy(&r[2], &meta, sizeof(meta));
        hi.push_back(top);
        rec.insert(rec.end(), r.begin(), r.end());
    };
    std::size_t node = 0;
    for (int64_t k = 0; k < cells; ++k) {
        start.push_back(static_cast<int32_t>(hi.size()));
        int64_t const first = (ix.first_cell + k) << RREA_ROW_CELL_SHIFT;
        int64_t const last = ((ix.first_cell + k + 1) << RREA_ROW_CELL_SHIFT) - 1;
        double lo = std::max(value(first), x_min);
        while (node < nodes.size() && nodes[node] < lo) ++node;
        for (; node < nodes.size() && bits(nodes[node]) <= last; ++node) {
            if (nodes[node] < x_min || nodes[node] > x_max) continue;
            add_row(lo, nodes[node]);
            lo = nodes[node];
        }
        // arguments above the cell's last node; the open edge is the next cell's
        if (lo < value(last) || hi.empty() || bits(hi.back()) < last) {
            double const top = std::min(value(last), x_max);
            if (top > lo) add_row(lo, top);
            if (bits(hi.back()) < last) hi.back() = value(last);   // past x_max: never reached, ends the search
        }
    }
    ix.rows = static_cast<int32_t>(hi.size());
    std::vector<double> packed((start.size() + 1) / 2, 0.0);
    std::memcpy(packed.data(), start.data(), start.size() * sizeof(int32_t));
    auto push = [&](std::vector<double> const& v) {
        int64_t const off = static_cast<int64_t>(arena.size());
        arena.insert(arena.end(), v.begin(), v.end());
        while (arena.size() % 4 != 0) arena.push_back(0.0);   // records stay 32-byte aligned
        return off;
    };
    ix.start = push(packed);
    ix.hi = push(hi);
    ix.rec = push(rec);
}

}  // namespace rrea_host
