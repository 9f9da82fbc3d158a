/*
 * cluster_plan.cpp — splits one graph's slices over the CTAs of a thread-block cluster for
 * the cluster solver (pcg_cluster.cu): slice ranges, CTA-local columns, and for every row
 * the CTAs that read it. Host code, once per graph.
 */
#include <algorithm>

#include "cluster_plan.h"

namespace {

/* contiguous ranges of at most `cap` slices over exactly `ctas` CTAs, none empty, each of
 * at most `bound` slots unless a single slice is larger; false if they do not suffice */
bool fill(const gslam_structure &S, int sl0, int sl1, int ctas, int cap, int64_t bound, std::vector<int> *out) {
    int used = 1, nsl = 0;
    int64_t cur = 0;
    if (out) out->assign(1, sl0);
    for (int sl = sl0; sl < sl1; sl++) {
        const int64_t w = S.slice_ptr[sl + 1] - S.slice_ptr[sl];
        /* the CTAs still to come need a slice each */
        const bool must = nsl > 0 && sl1 - sl <= ctas - used;
        if (must || (nsl > 0 && (cur + w > bound || nsl == cap))) {
            if (++used > ctas) return false;
            if (out) out->push_back(sl);
            cur = 0;
            nsl = 0;
        }
        cur += w;
        nsl++;
    }
    if (out) out->push_back(sl1);
    return used == ctas;
}

}  // namespace

bool gslam_cluster_plan(const gslam_structure &S, int sl0, int sl1, int ctas, unsigned shapes, int elem, int64_t budget,
                        gslam_cluster_part *part, std::vector<int> *lcol, std::vector<int> *keep, std::vector<int> *pos) {
    const int ns = sl1 - sl0;
    if (ns < ctas || ns > ctas * GSLAM_CLUSTER_SLICES) return false;
    part->ctas = ctas;
    static const int slices[] = { 12, 16, 20, GSLAM_CLUSTER_SLICES };
    part->shape = 0;
    while (!(shapes >> part->shape & 1) || ns > slices[part->shape] * ctas) part->shape++;
    const int cap = slices[part->shape];
    int64_t lo = 0, hi = S.slice_ptr[sl1] - S.slice_ptr[sl0];
    for (int sl = sl0; sl < sl1; sl++) lo = std::max(lo, S.slice_ptr[sl + 1] - S.slice_ptr[sl]);
    while (lo < hi) {
        const int64_t mid = lo + (hi - lo) / 2;
        if (fill(S, sl0, sl1, ctas, cap, mid, nullptr)) hi = mid;
        else lo = mid + 1;
    }
    if (!fill(S, sl0, sl1, ctas, cap, lo, &part->bounds)) return false;
    int most = 0;
    for (int r = 0; r < ctas; r++) most = std::max(most, part->bounds[r + 1] - part->bounds[r]);
    part->threads = 32 * (part->shape == 3 ? (most + 1) / 2 : most);
    /* local columns and halos; the rows each CTA reads from others */
    part->n_halo.assign(ctas, 0);
    std::vector<std::vector<int>> halo(ctas);
    const int row_base = 32 * sl0, n_rows = 32 * ns;
    part->exp_ptr.assign((size_t)n_rows + 1, 0);
    part->halo_max = 0;
    for (int r = 0; r < ctas; r++) {
        const int row0 = 32 * part->bounds[r], row1 = 32 * part->bounds[r + 1], nloc = row1 - row0;
        const int64_t a0 = S.slice_ptr[part->bounds[r]], a1 = S.slice_ptr[part->bounds[r + 1]];
        std::vector<int> &rem = halo[r];
        for (int64_t t = a0; t < a1; t++) {
            const int c = S.col[t];
            if (c >= 0 && (c < row0 || c >= row1)) rem.push_back(c);
        }
        std::sort(rem.begin(), rem.end());
        rem.erase(std::unique(rem.begin(), rem.end()), rem.end());
        for (int64_t t = a0; t < a1; t++) {
            const int c = S.col[t];
            if (c < 0) (*lcol)[t] = 0;
            else if (c >= row0 && c < row1) (*lcol)[t] = c - row0;
            else (*lcol)[t] = nloc + (int)(std::lower_bound(rem.begin(), rem.end(), c) - rem.begin());
        }
        for (int c : rem) {
            if (c < row_base || c >= row_base + n_rows) return false; /* a block that leaves the graph's rows */
            part->exp_ptr[c - row_base + 1]++;
        }
        part->n_halo[r] = (int)rem.size();
        part->halo_max = std::max(part->halo_max, (int)rem.size());
    }
    for (int i = 0; i < n_rows; i++) part->exp_ptr[i + 1] += part->exp_ptr[i];
    part->exp.resize(part->exp_ptr[n_rows]);
    std::vector<int> at(part->exp_ptr.begin(), part->exp_ptr.end() - 1);
    for (int r = 0; r < ctas; r++)
        for (int h = 0; h < part->n_halo[r]; h++)
            part->exp[at[halo[r][h] - row_base]++] = (unsigned)r << 20 | (unsigned)h;
    /* shared memory, and what sets the iteration's time */
    part->smem = 0;
    part->positions = part->left = part->sent = part->width = 0;
    for (int r = 0; r < ctas; r++) {
        const int64_t n_slots = S.slice_ptr[part->bounds[r + 1]] - S.slice_ptr[part->bounds[r]];
        const ClusterSmem m = cluster_smem_layout(elem, n_slots, part->bounds[r + 1] - part->bounds[r], part->n_halo[r],
                                                  part->halo_max, budget);
        if (m.val_cap < 0) return false;
        /* block positions that do not fit are left out evenly: the last one of every slice,
         * then of every slice that still has one, and so on */
        const int a = part->bounds[r], b = part->bounds[r + 1];
        int64_t out = std::max<int64_t>(0, (9 * n_slots - m.val_cap) / 288);
        for (int sl = a; sl < b; sl++) (*keep)[sl] = (int)((S.slice_ptr[sl + 1] - S.slice_ptr[sl]) / 32);
        while (out > 0)
            for (int sl = a; sl < b && out > 0; sl++)
                if ((*keep)[sl] > 0) { (*keep)[sl]--; out--; }
        int positions = 0, kept = 0;
        for (int sl = a; sl < b; sl++) {
            const int width = (int)((S.slice_ptr[sl + 1] - S.slice_ptr[sl]) / 32);
            positions += width;
            kept += (*keep)[sl];
            part->width = std::max(part->width, width);
        }
        part->positions = std::max(part->positions, positions);
        part->left = std::max(part->left, positions - kept);
        part->sent = std::max(part->sent, part->exp_ptr[32 * (b - sl0)] - part->exp_ptr[32 * (a - sl0)]);
        (*pos)[a] = 0;
        for (int sl = a + 1; sl < b; sl++) (*pos)[sl] = (*pos)[sl - 1] + (*keep)[sl - 1];
        part->smem = std::max(part->smem, (size_t)m.end);
    }
    /* one mbarrier phase counts at most 2^20 - 1 bytes; halo slots are 20-bit */
    if (16 * GSLAM_CLUSTER_CTAS + 24 * (int64_t)part->halo_max >= (1 << 20) - 1) return false;
    return true;
}

/*
 * Least-squares fits to measured times per iteration: 190 plans (walks, walks with up to 40 near
 * or 8 random closures per pose, landmark logs of 10 to 40 observations per landmark; 100 to 20,000
 * poses, 1 to 16 CTAs), within 7 % of the measured time (root mean square), 26 % at most. A CTA's
 * positions are its SpMV, a position left to L2 costs about as much again, a halo row sent costs
 * a store to another SM, and the widest slice is the longest chain of one warp. With two rows per
 * thread, D^-1 and the left-out positions come from L2 one after another, along the widest slice.
 */
double gslam_cluster_us(const gslam_cluster_part &p, int elem) {
    const bool two_rows = p.shape == 3;
    if (elem == 8) {
        if (two_rows) return 2.6 + 0.019 * p.positions + 0.0021 * p.sent + 0.236 * p.width;
        if (p.ctas == 1) return 1.1 + 0.022 * p.positions + 0.004 * p.left;
        return 1.7 + 0.014 * p.positions + 0.017 * p.left + 0.0019 * p.sent + 0.020 * p.width;
    }
    if (two_rows) return 3.2 + 0.0053 * p.positions + 0.0098 * p.left + 0.0009 * p.sent + 0.067 * p.width;
    return 2.0 + 0.0086 * p.positions + 0.007 * p.left + 0.001 * p.sent + 0.024 * p.width;
}

/* The same for the resident solver on the whole GPU (70 of these graphs up to 7,168 poses; 8 % at
 * most): two reductions over 148 CTAs, a few slices per CTA and the halo rows it polls. */
double gslam_resident_us(int positions, int left, int halo) {
    return 2.8 + 0.035 * positions + 0.08 * left + 0.00155 * halo;
}

/* The grid-wide batch solver, which streams the matrix (100 batches of 1 to 30 graphs; 9 % root
 * mean square, 38 % too low at most): its barriers, the widest slice's chain of loads, and the
 * bytes. */
double gslam_batch_us(int width, int64_t positions, int elem) {
    return elem == 8 ? 7.6 + 0.447 * width + 1.08e-3 * (double)positions
                     : 8.0 + 0.320 * width + 0.63e-3 * (double)positions;
}
