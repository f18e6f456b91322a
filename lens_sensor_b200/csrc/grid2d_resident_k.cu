// One row template of the resident 2D grid step (grid2d_resident.cuh), in both register
// splits: compiled once per RS_RM (rows of a lean band) and RS_GEN (rows of a band in
// the general form), so that the templates build side by side.
#include "grid2d_resident.cuh"

#define RS_CAT_(a, b) a##b
#define RS_CAT(a, b) RS_CAT_(a, b)

__attribute__((visibility("hidden"))) const void *RS_CAT(lens_grid2d_rs_k, RS_RM)(bool wide) {
    return wide ? (const void *)grid2d_rs<RS_RM, 384, RS_GEN> : (const void *)grid2d_rs<RS_RM, 256, RS_GEN>;
}
