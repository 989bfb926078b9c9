// necg_maps.h -- host-side tables of a symmetry set: the inverse of each term and the
// sparse map of the ket's raw sums (RawMap).
#pragma once
#include <math.h>

#include <utility>
#include <vector>

#include "necg_lanes.cuh"

namespace necg {

// pinv[p]: the term whose coordinate and shift maps are the inverses of p's; false if
// the set is not closed under inverse.
inline bool inverse_terms(int n, int nst, const double *sml, const double *sms, std::vector<int> &pinv) {
    const int m = 3 * n;
    auto inverse = [](const double *a, const double *b, int d) {  // a b = 1
        for (int i = 0; i < d; ++i)
            for (int j = 0; j < d; ++j) {
                double s = 0.0;
                for (int k = 0; k < d; ++k) s += a[i * d + k] * b[k * d + j];
                if (!(fabs(s - (i == j)) < 1e-12)) return false;
            }
        return true;
    };
    pinv.assign(nst, -1);
    for (int p = 0; p < nst; ++p) {
        for (int q = 0; q < nst && pinv[p] < 0; ++q)
            if (inverse(sml + (size_t)p * n * n, sml + (size_t)q * n * n, n) &&
                inverse(sms + (size_t)p * m * m, sms + (size_t)q * m * m, m))
                pinv[p] = q;
        if (pinv[p] < 0) return false;
    }
    return true;
}

// Host arrays of a RawMap.
struct RawMapTable {
    std::vector<int> cnt, src;
    std::vector<double> coef;
    int maxnz = 1, fold = 0;
};

// sl slots per (P, matrix), slot(f) of field f (KetSlots<n>).
template <typename SLOT>
RawMapTable raw_map_table(int n, int nst, const double *sml, const double *sms, int sl, const SLOT &slot) {
    const int m = 3 * n, T = n * (n + 1) / 2;
    RawMapTable t;
    // e' = A' s' maps as e = A s does when each shift map is that of its coordinate
    // map, sms = kron(sml^-1, I3), i.e. sms kron(sml, I3) = 1; the kets' raw sums
    // are then mapped and summed as they are, else folded in P's frame first
    for (int p = 0; p < nst && !t.fold; ++p)
        for (int r = 0; r < m && !t.fold; ++r)
            for (int j = 0; j < n && !t.fold; ++j)
                for (int c = 0; c < 3 && !t.fold; ++c) {  // column (j, c) of sms kron(sml, I3)
                    double v = 0.0;
                    for (int k = 0; k < n; ++k) v += sms[(size_t)p * m * m + r * m + 3 * k + c] * sml[(size_t)p * n * n + k * n + j];
                    t.fold = fabs(v - (r == 3 * j + c ? 1.0 : 0.0)) > 1e-12;
                }
    std::vector<std::vector<std::pair<int, double>>> rows((size_t)nst * sl);
    for (int p = 0; p < nst; ++p) {
        const double *P = sml + (size_t)p * n * n, *S = sms + (size_t)p * m * m;
        auto row = [&](int f) -> std::vector<std::pair<int, double>> & { return rows[(size_t)p * sl + slot(f)]; };
        for (int a = 0; a < n; ++a)
            for (int b = 0; b <= a; ++b) {
                std::vector<double> coef(T, 0.0);
                for (int cc = 0; cc < n; ++cc)
                    for (int d = 0; d < n; ++d) coef[sx(cc, d)] += P[a * n + cc] * P[b * n + d];
                for (int s = 0; s < T; ++s)
                    if (coef[s] != 0.0) row(sx(a, b)).push_back({slot(s), coef[s]});
            }
        row(T).push_back({slot(T), 1.0});
        for (int r = 0; r < m; ++r)
            if (t.fold) {  // dF/ds: (sms^T g')_r
                for (int c = 0; c < m; ++c)
                    if (S[c * m + r] != 0.0) row(T + 1 + r).push_back({slot(T + 1 + c), S[c * m + r]});
            } else {  // dF/de: (sml g')_r
                for (int k = 0; k < n; ++k)
                    if (P[(r / 3) * n + k] != 0.0) row(T + 1 + r).push_back({slot(T + 1 + 3 * k + r % 3), P[(r / 3) * n + k]});
            }
    }
    for (const auto &r : rows) t.maxnz = (int)r.size() > t.maxnz ? (int)r.size() : t.maxnz;
    t.cnt.resize(rows.size());
    t.src.assign(rows.size() * t.maxnz, 0);
    t.coef.assign(rows.size() * t.maxnz, 0.0);
    for (size_t e = 0; e < rows.size(); ++e) {
        t.cnt[e] = (int)rows[e].size();
        for (size_t i = 0; i < rows[e].size(); ++i) {
            t.src[e * t.maxnz + i] = rows[e][i].first;
            t.coef[e * t.maxnz + i] = rows[e][i].second;
        }
    }
    return t;
}

}  // namespace necg
