// Interval-polynomial rows of the loaded tables (device/rrea_rate_rows.cuh)
// against the reference's interpolation formulas in extended precision.
//
//   rate_rows <transport_physics.json>
//
// For every rows object: each node of its columns, the doubles on either
// side of it, the cells' edges and 20,000 seeded arguments.  Prints, per
// column, the number of values compared, the number on flagged rows and the
// largest error in units of the allowed one; exits 1 when a value is outside
// it, a row search leaves its cell, or the lower node index is wrong.
//
// Allowed error: the polynomial is the interpolant to one rounding of the
// row's largest value; its Horner form adds two more; the row's
// constants are built in double with about three roundings each, which the
// exponent s log(xc / x0) of a log-log value carries into it by the factor
// |log(y1 / y0)|; a reciprocal adds one more.  Together 2^-53 x (6 + 4 |log
// (y1 / y0)|) of the interval's larger end.
#include "../../rrea_feedback_warpx_amrex_geant4_gb300/csrc/device/rrea_rate_rows.cuh"
#include "../../rrea_feedback_warpx_amrex_geant4_gb300/csrc/host/table_set.hpp"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

using namespace rrea_host;
using namespace rrea_dev;

namespace {

int failures = 0;

struct Column {
    int kind;  // 0 table, 1 inverse semilog, 2 log fraction
    int mode;
    const double* x;
    const double* y;
    int n;
};

struct Truth {
    long double value, scale;
    int lower;
    bool defined;
};

Truth truth(Column const& c, double q)
{
    Truth t{0, 0, 0, false};
    if (q < c.x[0] || q > c.x[c.n - 1]) return t;
    int up = static_cast<int>(std::lower_bound(c.x, c.x + c.n, q) - c.x);
    if (up == 0) up = 1;
    long double const x0 = c.x[up - 1], x1 = c.x[up];
    t.lower = up - 1;
    if (!(x1 / x0 > 1.0L + 0.9e-9L)) return t;
    long double const f = std::log(static_cast<long double>(q) / x0) / std::log(x1 / x0);
    t.defined = true;
    if (c.kind == 2) {
        t.value = f;
        t.scale = 1.0L;
        return t;
    }
    long double const y0 = c.y[up - 1], y1 = c.y[up];
    long double const top = std::max(y0, y1);
    if (c.kind == 1) {
        t.value = 1.0L / (y0 + f * (y1 - y0));
        t.scale = 1.0L / std::min(y0, y1);
    } else if (c.mode == RREA_INTERP_LINEAR) {
        t.value = y0 + (q - x0) / (x1 - x0) * (y1 - y0);
        t.scale = top;
    } else if (c.mode == RREA_INTERP_LOGX_LINEAR
               || (c.mode == RREA_INTERP_LOGLOG_ZERO_THRESHOLD && !(y0 > 0 && y1 > 0))) {
        t.value = y0 + f * (y1 - y0);
        t.scale = top;
    } else if (!(y0 > 0 && y1 > 0)) {
        t.defined = false;
    } else {
        t.value = y0 * std::exp(f * std::log(y1 / y0));
        t.scale = top * (1.0L + std::fabs(std::log(y1 / y0)) * (4.0L / 6.0L));
    }
    return t;
}

void check(TableSet const& set, RreaRowIndex const& ix, std::vector<std::vector<Column>> const& cols, bool has_index,
           char const* name)
{
    const double* arena = set.arena().data();
    double const x_min = row_double(ix.lo_key), x_max = row_double(ix.lo_key + ix.span_key);
    std::vector<double> q;
    auto around = [&](double v) {
        for (double w : {v, std::nextafter(v, 0.0), std::nextafter(v, 1.0e300)}) {
            if (w >= x_min && w <= x_max) q.push_back(w);
        }
    };
    for (auto const& alt : cols) {
        for (Column const& c : alt) {
            for (int i = 0; i < c.n; ++i) around(c.x[i]);
        }
    }
    std::size_t const nodes = q.size();
    long long const first = ix.lo_key >> RREA_ROW_CELL_SHIFT, last = (ix.lo_key + ix.span_key) >> RREA_ROW_CELL_SHIFT;
    for (long long k = first; k <= last + 1; ++k) around(row_double(k << RREA_ROW_CELL_SHIFT));
    std::mt19937_64 gen(11);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    for (int i = 0; i < 20000; ++i) q.push_back(std::min(x_max, std::max(x_min, x_min * std::pow(x_max / x_min, u(gen)))));
    const int32_t* start = reinterpret_cast<const int32_t*>(arena + ix.start);
    const double* hi = arena + ix.hi;
    for (long long k = first; k <= last; ++k) {
        // every cell's search ends inside the cell
        int const b = start[k - first], e = k < last ? start[k - first + 1] : ix.rows;
        if (!(b < e) || row_bits(hi[e - 1]) < (((k + 1) << RREA_ROW_CELL_SHIFT) - 1)) {
            std::printf("%s: cell %lld has rows [%d, %d) and does not reach its edge\n", name, k, b, e);
            ++failures;
        }
    }
    if (failures) return;
    RowHit out;
    for (double w : {std::nextafter(x_min, 0.0), std::nextafter(x_max, 1.0e300), -x_max, 0.0, -0.0, HUGE_VAL, -HUGE_VAL,
                     std::nan("")}) {
        if (find_row(arena, ix, w, out)) {
            std::printf("%s: %g accepted\n", name, w);
            ++failures;
        }
    }
    std::vector<double> worst(cols.size(), 0.0);
    std::vector<long> compared(cols.size(), 0), flagged(cols.size(), 0), between(cols.size(), 0);
    for (std::size_t k = 0; k < q.size(); ++k) {
        double const v = q[k];
        RowHit h;
        if (!find_row(arena, ix, v, h)) {
            std::printf("%s: %.17g refused\n", name, v);
            ++failures;
            continue;
        }
        for (std::size_t c = 0; c < cols.size(); ++c) {
            if (cols[c].empty()) continue;
            if (row_flags(h) >> c & 1u) {
                ++flagged[c];
                between[c] += k >= nodes;
                continue;
            }
            double const got = row_value(h, static_cast<int>(c));
            // at a node two alternatives may serve (the angle tables hand over): any of them
            double best = HUGE_VAL;
            bool lower_ok = !has_index || c + 1 != cols.size();
            for (Column const& a : cols[c]) {
                Truth const t = truth(a, v);
                if (!t.defined) continue;
                // a table that is zero over its interval stays exactly zero
                double const e = t.scale == 0.0L ? (got == 0.0 ? 0.0 : HUGE_VAL)
                                                 : static_cast<double>(std::fabs(got - t.value)
                                                                       / (t.scale * 6.0L * 1.1102230246251565e-16L));
                if (e < best) best = e;
                if (t.lower == row_index(h) && e <= 1.0) lower_ok = true;
            }
            ++compared[c];
            worst[c] = std::max(worst[c], best);
            if (!(best <= 1.0) || !lower_ok) {
                if (++failures < 20) {
                    std::printf("%s column %zu at %.17g: %.17g, %g of the allowed error, lower %d\n", name, c, v, got,
                                best, row_index(h));
                }
            }
        }
    }
    for (std::size_t c = 0; c < cols.size(); ++c) {
        std::printf("%s rows %d column %zu: %ld compared, %ld flagged (%ld between nodes), worst %.3f of the allowed "
                    "error\n", name, ix.rows, c, compared[c], flagged[c], between[c], worst[c]);
        // only the gaps of rounded node pairs and the steep pieces at a
        // threshold may be flagged: under 5 % of the axis
        if (between[c] * 20 > static_cast<long>(q.size() - nodes)) ++failures;
    }
}

}  // namespace

int main(int argc, char** argv)
{
    if (argc != 2) return 2;
    TableSet set;
    set.Load(argv[1]);
    RreaArenaIndex const& ix = set.index();
    auto table = [&](int t) {
        RreaTable1DIndex const& h = ix.hot[t];
        return Column{0, h.mode, set.at(h.x), set.at(h.y), h.n};
    };
    for (int s = 0; s < 2; ++s) {
        int const base = s == 0 ? RREA_T_E_COLLISION : RREA_T_P_COLLISION;
        std::vector<std::vector<Column>> cols(RREA_RATE_COLUMNS);
        for (int c = 0; c < 4; ++c) cols[c].push_back(table(base + c));
        if (s == 1) cols[RREA_RATE_ANNIHILATION].push_back(table(RREA_T_P_ANNIHILATION));
        RreaElasticIndex const& el = ix.elastic[s];
        cols[RREA_RATE_ELASTIC].push_back(Column{1, 0, set.at(el.x), set.at(el.mfp), el.n});
        for (RreaAngleIndex const* a : {&ix.gs[s], &ix.wentzel[s]}) {
            cols[RREA_RATE_ANGLE_ENERGY].push_back(Column{2, 0, set.at(a->e), nullptr, a->ne});
        }
        check(set, ix.rate_rows[s], cols, true, s == 0 ? "electron rates" : "positron rates");
    }
    std::vector<std::vector<Column>> photon(RREA_PHOTON_COLUMNS);
    for (int c = 0; c < RREA_PHOTON_COLUMNS; ++c) photon[c].push_back(table(RREA_T_PH_COMPTON + c));
    check(set, ix.photon_rows, photon, false, "photon rates");
    for (RreaAngleIndex const* a : {&ix.gs[0], &ix.gs[1], &ix.wentzel[0], &ix.wentzel[1]}) {
        check(set, a->p_rows, {{Column{2, 0, set.at(a->p), nullptr, a->np}}}, true, "path");
        check(set, a->u_rows, {{Column{2, 0, set.at(a->u + 1), nullptr, a->nu - 2}}}, true, "cdf");
    }
    std::printf(failures ? "FAILED %d\n" : "ok\n", failures);
    return failures ? 1 : 0;
}
