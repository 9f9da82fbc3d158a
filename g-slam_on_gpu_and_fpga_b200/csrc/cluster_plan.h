/* cluster_plan.h — host-side plan of the cluster solver (internal). */
#ifndef GSLAM_CLUSTER_PLAN_H
#define GSLAM_CLUSTER_PLAN_H

#include <cstddef>
#include <vector>

#include "gslam_internal.h"
#include "kernels.cuh"

/* one graph's split over a cluster */
struct gslam_cluster_part {
    int ctas = 0, threads = 0, shape = 0; /* shape: launch_pcg_cluster */
    int halo_max = 0;
    size_t smem = 0;                     /* dynamic shared memory of the largest CTA */
    /* what an iteration's time follows: the most block positions (288 values) a CTA owns and
     * leaves to L2, the most halo rows it sends, and the widest slice */
    int positions = 0, left = 0, sent = 0, width = 0;
    std::vector<int> bounds;             /* [ctas + 1] slices */
    std::vector<int> n_halo;             /* [ctas] */
    std::vector<int> exp_ptr;            /* [rows of the graph + 1] */
    std::vector<unsigned> exp;           /* rank << 20 | halo slot */
};

/* Splits the slices [sl0, sl1) over a cluster of `ctas` CTAs for values of `elem` bytes, in the
 * first of the allowed shapes (bits of `shapes`; the last one always is) that has room;
 * lcol (all slots of the layout) gets the graph's CTA-local columns, keep and pos (all its
 * slices) the block positions in shared memory and where they start. False when the graph
 * does not fit (more rows than the threads own, or the fixed parts of a CTA's shared
 * memory exceed the budget); *part and the graph's part of the arrays are then undefined. */
bool gslam_cluster_plan(const gslam_structure &S, int sl0, int sl1, int ctas, unsigned shapes, int elem, int64_t budget,
                        gslam_cluster_part *part, std::vector<int> *lcol, std::vector<int> *keep, std::vector<int> *pos);

/* Estimated us per iteration of the cluster solver for a plan in values of `elem` bytes, and of
 * the grid-wide FP64 resident solver for the most positions, left-out positions and halo rows of
 * its CTAs. */
double gslam_cluster_us(const gslam_cluster_part &p, int elem);
double gslam_resident_us(int positions, int left, int halo);
/* The same for the grid-wide batch solver: the widest slice and all positions of the batch. */
double gslam_batch_us(int width, int64_t positions, int elem);

#endif
