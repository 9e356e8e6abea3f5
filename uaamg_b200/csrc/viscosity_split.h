// viscosity_split.h -- how k_vbottom (viscosity_bottom.cuh) splits its passes
// over the row CTAs of its cluster, and how many values a pass exchanges.
// Host and device, without CUDA.
//
// A pass updates one group of rows (or, the prolongation, all of them).  Every
// row CTA sends something to every row CTA in every pass: its rows' values, or
// one word that nobody reads where it has no row of the group.  So a CTA that
// has received a whole pass knows that every CTA has finished the pass before,
// also where a group is too small for all of them (4 rows over 3 CTAs are
// 2 + 2 + 0).
#pragma once

#ifdef __CUDACC__
#define VB_HD __host__ __device__ __forceinline__
#else
#define VB_HD inline
#endif

namespace uaamg {

constexpr int VB_GROUPS = 6;  // channel * 2 + colour

struct VbPart {
    int lo, cnt;  // first row and rows of a CTA
};
// CTA j's part of `size` rows over NC CTAs
VB_HD VbPart vb_part(int size, int NC, int j) {
    const int s = (size + NC - 1) / NC;
    const int lo = j * s < size ? j * s : size;
    return VbPart{lo, lo + s < size ? s : size - lo};
}
// CTAs with a row of `size` rows: the first ones
VB_HD int vb_busy(int size, int NC) {
    const int s = (size + NC - 1) / NC;
    return s ? (size + s - 1) / s : 0;
}
// Values every row CTA receives in a pass over group g (VB_GROUPS: all rows);
// gs[g]: first row of group g, gs[VB_GROUPS] the number of rows.
VB_HD int vb_values(const int* gs, int NC, int g) {
    if (g < VB_GROUPS) return gs[g + 1] - gs[g] + NC - vb_busy(gs[g + 1] - gs[g], NC);
    int busy = 0;
    for (int k = 0; k < VB_GROUPS; ++k) {
        const int b = vb_busy(gs[k + 1] - gs[k], NC);
        busy = b > busy ? b : busy;
    }
    return gs[VB_GROUPS] + NC - busy;
}
// Threads of a CTA that take part in its passes: the warps with a row of any
// group (cnt: its rows of each), at least one.
VB_HD int vb_threads(const int* cnt, int block) {
    int most = 1;
    for (int g = 0; g < VB_GROUPS; ++g) most = cnt[g] > most ? cnt[g] : most;
    return most < block ? (most + 31) / 32 * 32 : block;
}

}  // namespace uaamg
