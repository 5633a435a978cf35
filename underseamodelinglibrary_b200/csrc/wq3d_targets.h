/*
 * wq3d_targets.h -- the CPA search's view of a queue's targets, formed on
 * the host: clusters of targets near one another, whose extents the search's
 * bounds trust (k_cpa).
 */
#pragma once

#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

namespace wq3d {

/* 32 targets of the CPA search: the middle of their ranges of rho, theta,
 * phi and rho sin(theta), and the half-widths (rounded up) */
struct TgtCluster {
    double R, T, P, RS;
    float dR, dT, dP, dRS;
    int32_t branch; /* holds a target with QueueDev::de_branch set */
    int32_t pad;
};

/* the CPA search's view of the targets (QueueDev::clusters, cpa_tgt,
 * cpa_index, tgt_box).  A target with a NaN or infinite coordinate is left
 * out: its distance2 is NaN or infinite for every ray, so it has no eigenray,
 * and extents that held it would bound none of its neighbours. */
struct CpaTargets {
    std::vector<TgtCluster> clusters;
    std::vector<double> tgt;
    std::vector<uint32_t> index;
    double box[6] = {0, 0, 0, 0, 0, 0};
};

/* the clusters of the targets in the given order, and the sum of their
 * extents in metres */
inline double make_clusters(const std::vector<double>& r, const std::vector<double>& th,
                            const std::vector<double>& ph, const std::vector<double>& sn,
                            const std::vector<uint8_t>& branch, const std::vector<uint32_t>& order,
                            std::vector<TgtCluster>* out) {
    out->clear();
    double total = 0.0;
    for (size_t b = 0; b < order.size(); b += 32) {
        const size_t e = std::min(order.size(), b + 32);
        double lo[4] = {}, hi[4] = {};
        for (size_t j = b; j < e; ++j) {
            const uint32_t t = order[j];
            const double v[4] = {r[t], th[t], ph[t], r[t] * sn[t]};
            for (int k = 0; k < 4; ++k) {
                if (j == b || v[k] < lo[k]) lo[k] = v[k];
                if (j == b || v[k] > hi[k]) hi[k] = v[k];
            }
        }
        TgtCluster c{};
        for (size_t j = b; j < e; ++j) c.branch |= branch[order[j]];
        double mid[4], half[4];
        for (int k = 0; k < 4; ++k) {
            mid[k] = 0.5 * (lo[k] + hi[k]);
            half[k] = std::max(hi[k] - mid[k], mid[k] - lo[k]) * 1.000001;
        }
        c.R = mid[0];
        c.T = mid[1];
        c.P = mid[2];
        c.RS = mid[3];
        c.dR = (float)half[0];
        c.dT = (float)half[1];
        c.dP = (float)half[2];
        c.dRS = (float)half[3];
        total += half[0] + std::abs(mid[0]) * half[1] + std::abs(mid[3]) * half[2];
        out->push_back(c);
    }
    return total;
}

/* Clusters of 32 consecutive targets, in the caller's order or along a
 * Morton curve, whichever has the smaller extents: a range x depth table's
 * columns are already compact (1.5 of 32 clusters survive a warp's bounds on
 * the sloped workload, 3 along the curve), random targets are not (27 of 128
 * on the reverberation workload, 126 in their own order). */
inline void cpa_targets(const std::vector<double>& r, const std::vector<double>& th,
                        const std::vector<double>& ph, const std::vector<double>& sn,
                        const std::vector<uint8_t>& branch, CpaTargets* o) {
    o->index.clear();
    double lo[3] = {}, hi[3] = {};
    for (size_t t = 0; t < r.size(); ++t) {
        const double v[3] = {r[t], th[t], ph[t]};
        if (!std::isfinite(v[0]) || !std::isfinite(v[1]) || !std::isfinite(v[2])) continue;
        for (int k = 0; k < 3; ++k) {
            if (o->index.empty() || v[k] < lo[k]) lo[k] = v[k];
            if (o->index.empty() || v[k] > hi[k]) hi[k] = v[k];
        }
        o->index.push_back((uint32_t)t);
    }
    const size_t nt = o->index.size();
    for (int k = 0; k < 3 && nt; ++k) {
        o->box[2 * k] = lo[k];
        o->box[2 * k + 1] = hi[k];
    }
    const double own = make_clusters(r, th, ph, sn, branch, o->index, &o->clusters);
    if (nt > 32) {
        const double size = std::max({hi[0] - lo[0], hi[0] * (hi[1] - lo[1]), hi[0] * (hi[2] - lo[2])});
        if (size > 0.0 && size < 1e30) {
            std::vector<uint32_t> key(r.size());
            for (const uint32_t t : o->index) {
                const double x[3] = {r[t] - lo[0], hi[0] * (th[t] - lo[1]), hi[0] * sn[t] * (ph[t] - lo[2])};
                uint32_t m = 0;
                for (int k = 0; k < 3; ++k) {
                    const uint32_t c = (uint32_t)std::min(1023.0, std::max(0.0, 1023.0 * x[k] / size));
                    for (int b = 0; b < 10; ++b) m |= ((c >> b) & 1u) << (3 * b + k);
                }
                key[t] = m;
            }
            /* by key, then index, ten bits at a time (10,000 targets: 0.1 ms;
             * a comparison sort of pairs took 0.9) */
            std::vector<uint32_t> order(o->index), next(nt), start(1025);
            for (int shift = 0; shift < 30; shift += 10) {
                std::fill(start.begin(), start.end(), 0u);
                for (const uint32_t t : order) ++start[((key[t] >> shift) & 1023u) + 1];
                for (int d = 0; d < 1024; ++d) start[d + 1] += start[d];
                for (const uint32_t t : order) next[start[(key[t] >> shift) & 1023u]++] = t;
                order.swap(next);
            }
            std::vector<TgtCluster> cl;
            if (make_clusters(r, th, ph, sn, branch, order, &cl) < own) {
                o->index.swap(order);
                o->clusters.swap(cl);
            }
        }
    }
    o->tgt.resize(4 * nt);
    for (size_t j = 0; j < nt; ++j) {
        const uint32_t t = o->index[j];
        o->tgt[4 * j] = r[t];
        o->tgt[4 * j + 1] = th[t];
        o->tgt[4 * j + 2] = ph[t];
        o->tgt[4 * j + 3] = sn[t];
    }
}

/* the most patches of 32 rays that a fan is cut into (cpa_patches) */
inline size_t cpa_patch_bound(size_t nde, size_t naz) {
    size_t most = 0;
    for (int s = 0; s <= 5; ++s) {
        const size_t rows = 32 >> s, cols = (size_t)1 << s;
        most = std::max(most, ((nde + rows - 1) / rows) * ((naz + cols - 1) / cols));
    }
    return most;
}

/* Room for the search's items (a patch and a target whose 32 pairs the
 * bounds leave).  A few a patch in fans whose rays lie close, and two a ray
 * are room enough; but patches of a coarse fan span kilometres and keep most
 * targets, so there is room for every patch and target up to 2^18.  (k_cpa
 * decides those that find none, one after another: 69 x 8 rays and 1500
 * targets took 137 us a step with room for 4096 items, 43 with room for all.) */
inline size_t cpa_item_capacity(size_t nde, size_t naz, size_t nt) {
    return std::max({(size_t)4096, std::min((size_t)1 << 20, 2 * nde * naz),
                     std::min((size_t)1 << 18, cpa_patch_bound(nde, naz) * nt)});
}

/* Blocks of four warps for them: one per 256 rays as for the eigenrays, up to
 * four an SM, and at most 16 items a warp where 24 patches keep every target,
 * which a coarse fan's do, up to the seven an SM that are resident; the count
 * is not known when the launch is made. */
inline int cpa_item_blocks(size_t n, size_t patches, size_t nt, size_t sms) {
    return (int)std::max({sms, std::min(4 * sms, (n + 255) / 256),
                          std::min(7 * sms, std::min<size_t>(patches, 24) * nt / 64)});
}

}  // namespace wq3d
