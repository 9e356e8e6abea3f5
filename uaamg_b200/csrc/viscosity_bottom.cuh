// viscosity_bottom.cuh -- the bottom of the viscosity mu-cycle in one launch.
//
// simd_viscosity3d::mucycle (SIMD_UAAMG/simd_viscosity3d.cpp:3837-3884) visits
// the level next to the coarsest (level lb) twice per visit of the level above
// it: each visit is 24 one-colour passes of one channel, the residual and its
// restriction, the coarsest CG and the prolongation.  Level lb holds few DOFs
// spread thinly over its leaves (128^3: 5,812 DOF in 52 leaves of 3 x 512
// voxels), so as leaf kernels the passes cost their launches and load chains
// (2.2 us per fused red-black step, 123 us per pair of visits there).
//
// k_vbottom does both visits in one thread-block cluster over the DOFs alone.
// A row per DOF (14 off-diagonal coefficients, the indices of the values they
// multiply, diag, 1/diag), ordered by (channel, colour), so a pass is one
// contiguous group of rows.  The groups' rows are split over the row CTAs and
// stay in their shared memory; every row CTA has a copy of the whole solution
// vector.  A pass: gather from the own copy, update, and send the new value to
// every copy with st.async, whose bytes complete a phase of the receiver's
// mbarrier.  So one one-way trip through the cluster separates two passes; no
// barrier of the cluster and no fence is on that path.
//
// Measured (events around the launch): 128^3, two visits with their CG 68 us,
// 54 launches of 2.2 us in a graph before; 44^3 (15,496 DOF over 2,017) 99 us
// against 57 launches, whole solve 7.4 -> 4.8 ms as a graph.
//
// Why this is safe without one: a warp sends pass p + 1 only when all of pass p
// has arrived, and a row's value is sent after its gathers; so when a value of
// pass p + 1 arrives anywhere, every gather of pass p is done.  Every CTA sends
// in every pass, one word that nobody reads where it has no row of the group
// (viscosity_split.h), so all of a pass arrives only when every CTA is in it.
// Two mbarriers, a parity bit each, alternate: a warp has to see pass p's phase
// before pass p + 2's ends.  The warps of a CTA that have rows (the others take
// no part) meet at a named barrier after each pass, so none of them sends p + 1
// while another still waits for p.  (That and the words: 65.6 -> 68.2 us a
// launch at 128^3, 98.5 -> 98.6 at 44^3.  A barrier after every second pass
// would do, but 68.6 and 100.7: the warps drift apart.)
//
// The coarsest CG runs in a CTA of its own while its rows fit that CTA's
// registers (up to 1024 DOF, k_vcoarsest_cg's form), above that over eight
// CTAs (vcg8_solve).  Operations and their order are those of the leaf
// kernels, so results are bit-identical to the launch sequence.
#pragma once
#include <cooperative_groups.h>

#include "viscosity_kernels.cuh"
#include "viscosity_split.h"

namespace uaamg {

#define VB_THREADS 256
#define VB_COEF 14
#define VB_MAX_CLUSTER 16  // non-portable cluster size limit
#define VB_CG8 8           // CTAs of the distributed CG: one warp of k_vcoarsest_cg's 256 lanes each

struct VBotRows {        // level lb by DOF, rows sorted by group channel * 2 + colour
    int n, nc;           // rows; coarsest DOFs
    int gs[7];           // first row of each group
    int val[7];          // values a row CTA receives in a pass over the group (vb_values; [6]: over all rows)
    const float* coef;   // [14][n]: neg +x, -x, +y, -y, +z, -z; T of channel d2: 00 01 10 11; T of channel d1: the same
    const unsigned* idx; // [7][n] rows of the values they multiply, two 16-bit ones per word; n = no DOF
    const float* iv;     // [n] 1/diag
    const float* dg;     // [n] diag
    const int* slot;     // [n] position in the leaf-dense vectors
    const uint16_t* cdst;  // [n] coarse DOF * 8 + octant in it
    const int* rcount;   // [8] rows whose coarse DOF each CTA of the distributed CG holds
};
struct VbLimit {            // of the waits of a cluster's CTAs for one another
    unsigned long long ns;  // 0: every wait gives up at once
    int* error;
};
struct VBotArgs {
    VBotRows R;
    DCoarsestV C;
    int NC;            // row CTAs
    int visits;        // 2, or 1 when level lb is the top
    const float* rhs;  // level lb
    float* lhs;
    VbLimit lim;
};

// ---- building the rows -----------------------------------------------------
// bits of mask word x (bit 8y + z) whose voxel has colour par: (x + y + z) & 1 == par
__host__ __device__ __forceinline__ uint64_t vcolour_mask(int x, int par) {
    return ((x + par) & 1) ? 0x55AA55AA55AA55AAull : 0xAA55AA55AA55AA55ull;
}
// row of voxel (X, Y, Z) relative to the leaf whose neighbours nbrow lists (n where it is no DOF of channel c);
// base: [nl][6] first row of each leaf and group
__device__ __forceinline__ int vrow_of(const VLevel& L, const int* base, const int* nbrow, int c, int X, int Y, int Z,
                                       int n) {
    const int lf = nbrow[vnb_index(X, Y, Z)];
    if (lf < 0) return n;
    const int off = voff3(X, Y, Z);
    const uint64_t* m = L.dof + ((long long)c * L.nl + lf) * 8;
    if (!((m[off >> 6] >> (off & 63)) & 1ull)) return n;
    const int par = ((off >> 6) + (off >> 3) + off) & 1;
    int r = base[lf * 6 + c * 2 + par];
    for (int w = 0; w < (off >> 6); ++w) r += __popcll(m[w] & vcolour_mask(w, par));
    return r + __popcll(m[off >> 6] & vcolour_mask(off >> 6, par) & ((1ull << (off & 63)) - 1ull));
}
// coefficient as the applier reads it: the default where the leaf does not exist
__device__ __forceinline__ float vrow_coef(const VLevel& L, const int* nbrow, int c, int a, int X, int Y, int Z) {
    const int lf = nbrow[vnb_index(X, Y, Z)];
    if (lf < 0) return L.app[c * VNA + a];
    return L.coef[(long long)(c * VNA + a) * L.nl * UAAMG_LEAF + (long long)lf * UAAMG_LEAF + voff3(X, Y, Z)];
}
// grid (nl, 3, 4): one voxel per thread
__global__ void __launch_bounds__(128) k_vbot_rows(VLevel L, VLevel C, const int* base, const int* cdof_base, int n,
                                                   float* coef, unsigned* idx, float* iv, float* dg, int* slot,
                                                   uint16_t* cdst, int* rcount) {
    griddep_wait();
    griddep_launch();
    const int leaf = blockIdx.x, c = blockIdx.y, t = threadIdx.x;
    const int X = t >> 4, Y = (t >> 1) & 7, Z = (t & 1) * 4 + blockIdx.z;
    const int* nb = L.nb + (long long)leaf * 27;
    const int r = vrow_of(L, base, nb, c, X, Y, Z, n);
    if (r == n) return;
    const int d0 = c, d1 = (c + 1) % 3, d2 = (c + 2) % 3;
    int e0[3] = {d0 == 0, d0 == 1, d0 == 2}, e1[3] = {d1 == 0, d1 == 1, d1 == 2}, e2[3] = {d2 == 0, d2 == 1, d2 == 2};
    const int Xm = X - e0[0], Ym = Y - e0[1], Zm = Z - e0[2];
    auto put = [&](int k, float v) { coef[(long long)k * n + r] = v; };
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int px = ax == 0, py = ax == 1, pz = ax == 2;
        put(2 * ax, vrow_coef(L, nb, c, VA_NEGX + ax, X + px, Y + py, Z + pz));
        put(2 * ax + 1, vrow_coef(L, nb, c, VA_NEGX + ax, X, Y, Z));
        const unsigned a = (unsigned)vrow_of(L, base, nb, c, X + px, Y + py, Z + pz, n);
        const unsigned b = (unsigned)vrow_of(L, base, nb, c, X - px, Y - py, Z - pz, n);
        idx[(long long)ax * n + r] = a | (b << 16);
    }
    put(6, vrow_coef(L, nb, d2, VA_T00, X, Y, Z));
    put(7, vrow_coef(L, nb, d2, VA_T01, X, Y, Z));
    put(8, vrow_coef(L, nb, d2, VA_T10, Xm, Ym, Zm));
    put(9, vrow_coef(L, nb, d2, VA_T11, Xm, Ym, Zm));
    put(10, vrow_coef(L, nb, d1, VA_T00, X, Y, Z));
    put(11, vrow_coef(L, nb, d1, VA_T01, Xm, Ym, Zm));
    put(12, vrow_coef(L, nb, d1, VA_T10, X, Y, Z));
    put(13, vrow_coef(L, nb, d1, VA_T11, Xm, Ym, Zm));
    const unsigned u0 = (unsigned)vrow_of(L, base, nb, d1, X, Y, Z, n);
    const unsigned u1 = (unsigned)vrow_of(L, base, nb, d1, X + e1[0], Y + e1[1], Z + e1[2], n);
    const unsigned u2 = (unsigned)vrow_of(L, base, nb, d1, Xm, Ym, Zm, n);
    const unsigned u3 = (unsigned)vrow_of(L, base, nb, d1, Xm + e1[0], Ym + e1[1], Zm + e1[2], n);
    const unsigned v0 = (unsigned)vrow_of(L, base, nb, d2, X, Y, Z, n);
    const unsigned v1 = (unsigned)vrow_of(L, base, nb, d2, Xm, Ym, Zm, n);
    const unsigned v2 = (unsigned)vrow_of(L, base, nb, d2, X + e2[0], Y + e2[1], Z + e2[2], n);
    const unsigned v3 = (unsigned)vrow_of(L, base, nb, d2, Xm + e2[0], Ym + e2[1], Zm + e2[2], n);
    idx[3LL * n + r] = u0 | (u1 << 16);
    idx[4LL * n + r] = u2 | (u3 << 16);
    idx[5LL * n + r] = v0 | (v1 << 16);
    idx[6LL * n + r] = v2 | (v3 << 16);
    iv[r] = vrow_coef(L, nb, c, VA_INV, X, Y, Z);
    dg[r] = vrow_coef(L, nb, c, VA_DIAG, X, Y, Z);
    const int off = voff3(X, Y, Z);
    slot[r] = (c * L.nl + leaf) * UAAMG_LEAF + off;
    // the coarse voxel: a DOF, since this child is one
    const int P = L.parent[leaf], o = L.octant[leaf];
    const int coff = voff3(((o >> 2) & 1) * 4 + (X >> 1), ((o >> 1) & 1) * 4 + (Y >> 1), (o & 1) * 4 + (Z >> 1));
    const uint64_t* cm = C.dof + ((long long)c * C.nl + P) * 8;
    int cr = cdof_base[c * C.nl + P];
    for (int w = 0; w < (coff >> 6); ++w) cr += __popcll(cm[w]);
    cr += __popcll(cm[coff >> 6] & ((1ull << (coff & 63)) - 1ull));
    cdst[r] = (uint16_t)(cr * 8 + (X & 1) * 4 + (Y & 1) * 2 + (Z & 1));
    atomicAdd(rcount + ((cr & 255) >> 5), 1);
}

// ---- the cluster's exchange ------------------------------------------------
__device__ __forceinline__ unsigned vb_map(unsigned a, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// v to the word at (this CTA's) shared address a in CTA `rank`, counted by that CTA's mbarrier at bar
__device__ __forceinline__ void vb_send(unsigned a, unsigned bar, unsigned rank, float v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(
                     vb_map(a, rank)),
                 "f"(v), "r"(vb_map(bar, rank))
                 : "memory");
}
__device__ __forceinline__ bool vb_try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, "
        "0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void vb_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned long long vb_now() {  // ns
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Waits for a phase, within the limit (each poll blocks briefly).  A wait that
// gives up sets the kernel's error word and `dead` in the thread, which from
// then on neither waits, arms nor sends; nor do the launches after it, until
// the word is cleared for the next solve.
__device__ __forceinline__ void vb_wait(unsigned bar, unsigned parity, const VbLimit& lim, bool& dead) {
    if (dead) return;
    if (lim.ns && vb_try_wait(bar, parity)) return;
    for (const unsigned long long t0 = vb_now(); vb_now() - t0 < lim.ns;)
        if (vb_try_wait(bar, parity)) return;
    dead = true;
    *lim.error = 1;
}
// The last thing a CTA does: nobody sends into a CTA that has left.  After a
// wait that gave up, values may still be under way to it when all have met.
__device__ __forceinline__ void vb_leave(bool dead) {
    __syncthreads();
    vb_cluster_sync();
    if (dead) __nanosleep(100000);
}
__device__ __forceinline__ void vb_arm(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// ---- the coarsest CG over eight CTAs ----------------------------------------
// k_vcoarsest_cg's CG with its 256 lanes split over VB_CG8 CTAs: CTA j has
// lanes 32 j .. 32 j + 31, i.e. warp j of the eight, and thread (w, l) of it
// the rows 32 j + l + 256 k for k = w and w + 8.  The products of a lane's
// rows are added in a chain over k by one warp, lanes by shfl_down, the eight
// sums in the same tree.  For 1025 - 4000 DOF one CTA's registers do not hold
// the rows, and reading them from L2 in each of the ten iterations took
// several microseconds an iteration.
struct VCg8Smem {  // in each CTA's shared memory, at the same place in all eight
    float* p;         // [nc] p by row (all rows); the solution afterwards
    float* zero;      // a zero, for absent entries
    float *ca, *cb;   // [kmax][32] factors of this CTA's rows' products
    float *s1, *s2;   // [8], [16] sums (16-byte aligned)
    uint64_t* bar;    // [3] p, first sum, second sums
};
__host__ __device__ __forceinline__ int vcg8_kmax(int nc) { return (nc + VCG_THREADS - 1) / VCG_THREADS; }
__host__ __device__ __forceinline__ size_t vcg8_smem_bytes(int nc) {  // a multiple of 16
    return 4 * (((size_t)nc + 1 + 3) / 4 * 4 + 64 * (size_t)vcg8_kmax(nc) + 24) + 32;
}
__device__ __forceinline__ VCg8Smem vcg8_smem(unsigned char* m, int nc) {  // m: 16-byte aligned
    VCg8Smem S;
    S.p = reinterpret_cast<float*>(m);
    S.zero = S.p + nc;
    S.ca = S.p + (nc + 1 + 3) / 4 * 4;
    S.cb = S.ca + 32 * vcg8_kmax(nc);
    S.s1 = S.cb + 32 * vcg8_kmax(nc);
    S.s2 = S.s1 + 8;
    S.bar = reinterpret_cast<uint64_t*>(S.s2 + 16);
    return S;
}
struct VCg8Rows {
    float val[2][VCG_W];
    unsigned col[2][8];  // byte offsets into p, two per word
    float iv[2];
    int row[2];          // -1: no row
};
__device__ __forceinline__ void vcg8_load(const DCoarsestV& C, int j, VCg8Rows& M) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int i = 32 * j + l + VCG_THREADS * (w + 8 * q);
        const bool ok = i < C.n;
        M.row[q] = ok ? i : -1;
        M.iv[q] = ok ? C.invd[i] : 0.f;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int cc = ok && e < VCG_W ? __ldg(C.col + (long long)i * VCG_W + (e < VCG_W ? e : 0)) : -1;
            const unsigned o = 4u * (unsigned)(cc >= 0 ? cc : C.n);  // S.zero follows p
            M.col[q][e >> 1] = (e & 1) ? (M.col[q][e >> 1] | (o << 16)) : o;
            if (e < VCG_W) M.val[q][e < VCG_W ? e : 0] = cc >= 0 ? __ldg(C.val + (long long)i * VCG_W + (e < VCG_W ? e : 0)) : 0.f;
        }
    }
}
// called by one thread of each CTA before the cluster's first barrier
__device__ __forceinline__ void vcg8_init(const VCg8Smem& S) {
    for (int i = 0; i < 3; ++i) mbar_init(&S.bar[i], 1);
    *S.zero = 0.f;
}
// this CTA's sums of ca * fb over its lanes' chains (and, second, of ca * cb): to every CTA
__device__ __forceinline__ void vcg8_sum(const VCg8Smem& S, int kmax, int j, bool squares, bool products, float* dst,
                                         unsigned bar, unsigned rank0, bool dead) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int nsum = (int)squares + (int)products;
    if (w >= nsum) return;
    const bool sq = squares && w == 0;
    float acc = 0.f;
    for (int k = 0; k < kmax; ++k) {
        const float a = S.ca[32 * k + l];
        acc = __fmaf_rn(a, sq ? a : S.cb[32 * k + l], acc);
    }
    acc = cg_warp_partial(acc);
    acc = __shfl_sync(FULLMASK, acc, 0);
    if (l < VB_CG8 && !dead) vb_send(smem_u32(dst + 8 * w + j), bar, rank0 + (unsigned)l, acc);
}
// x of this thread's rows for the rhs r (0 in rows it does not have); every thread of the eight CTAs.
// ph: phases of the three mbarriers used so far (they advance together with the solves).  Once a wait of one of its
// threads gives up, a CTA's threads leave together (stop): the barriers inside are the whole block's.
__device__ __forceinline__ void vcg8_solve(const DCoarsestV& C, const VCg8Rows& M, const VCg8Smem& S, int j, unsigned rank0,
                                           float (&r)[2], float (&x)[2], unsigned (&ph)[3], const VbLimit& lim,
                                           bool& dead) {
    const int t = threadIdx.x, w = t >> 5, l = t & 31;
    const int kmax = vcg8_kmax(C.n);
    const unsigned bp = smem_u32(&S.bar[0]), b1 = smem_u32(&S.bar[1]), b2 = smem_u32(&S.bar[2]);
    const unsigned pb = smem_u32(S.p);
    auto factors = [&](const float (&a)[2], const float (&b)[2]) {
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (w + 8 * q < kmax) {
                S.ca[32 * (w + 8 * q) + l] = a[q];
                S.cb[32 * (w + 8 * q) + l] = b[q];
            }
        __syncthreads();
    };
    auto wait = [&](unsigned bar, int i) {
        vb_wait(bar, ph[i] & 1u, lim, dead);
        ph[i]++;
    };
    auto stop = [&]() {
        dead = __syncthreads_or(dead) != 0;
        return dead;
    };
    float p[2] = {0.f, 0.f}, z[2];
    x[0] = x[1] = 0.f;
    // r.r, then r.z with z = invd r
    if (t == 0 && !dead) vb_arm(b2, 64);
#pragma unroll
    for (int q = 0; q < 2; ++q) z[q] = __fmul_rn(M.iv[q], r[q]);
    factors(r, z);
    vcg8_sum(S, kmax, j, true, true, S.s2, b2, rank0, dead);
    wait(b2, 2);
    if (stop()) return;
    const float rhsNorm2 = cg_tree_sum<8>(S.s2);
    float absNew = cg_tree_sum<8>(S.s2 + 8);
    const float threshold = fmaxf(__fmul_rn(__fmul_rn(FLT_EPSILON, FLT_EPSILON), rhsNorm2), FLT_MIN);
    if (rhsNorm2 == 0.f || rhsNorm2 < threshold) return;
    p[0] = z[0];
    p[1] = z[1];
    for (int it = 0; it < 10; ++it) {
        if (t == 0 && !dead) {
            vb_arm(bp, 4u * (unsigned)C.n);
            vb_arm(b1, 32);
            vb_arm(b2, 64);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (M.row[q] >= 0 && !dead)
#pragma unroll
                for (unsigned k = 0; k < VB_CG8; ++k) vb_send(pb + 4u * (unsigned)M.row[q], bp, rank0 + k, p[q]);
        wait(bp, 0);
        float tq[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            float s = 0.f;
#pragma unroll
            for (int e = 0; e < VCG_W; ++e) {
                const unsigned o = (e & 1) ? (M.col[q][e >> 1] >> 16) : (M.col[q][e >> 1] & 0xffffu);
                s = __fmaf_rn(M.val[q][e], lds_f32(pb + o), s);
            }
            tq[q] = s;
        }
        factors(p, tq);
        vcg8_sum(S, kmax, j, false, true, S.s1, b1, rank0, dead);
        wait(b1, 1);
        const float alpha = __fdiv_rn(absNew, cg_tree_sum<8>(S.s1));
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            x[q] = __fmaf_rn(alpha, p[q], x[q]);
            r[q] = __fmaf_rn(-alpha, tq[q], r[q]);
            z[q] = __fmul_rn(M.iv[q], r[q]);
        }
        factors(r, z);
        vcg8_sum(S, kmax, j, true, true, S.s2, b2, rank0, dead);
        wait(b2, 2);
        if (stop()) return;
        const float rr = cg_tree_sum<8>(S.s2);
        if (rr < threshold) break;
        const float absOld = absNew;
        absNew = cg_tree_sum<8>(S.s2 + 8);
        const float beta = __fdiv_rn(absNew, absOld);
#pragma unroll
        for (int q = 0; q < 2; ++q) p[q] = __fmaf_rn(beta, p[q], z[q]);
    }
}

// the coarsest solve alone, for hierarchies whose level lb does not fit k_vbottom: one cluster of VB_CG8 CTAs
__global__ void __launch_bounds__(VB_THREADS, 1) k_vcoarsest_cg8(DCoarsestV C, const float* rhs, float* out, VbLimit lim) {
    extern __shared__ __align__(16) unsigned char cg8_mem[];
    const VCg8Smem S = vcg8_smem(cg8_mem, C.n);
    const int j = (int)cooperative_groups::this_cluster().block_rank();
    VCg8Rows M;
    vcg8_load(C, j, M);
    long long sl[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) sl[q] = M.row[q] >= 0 ? C.slot[M.row[q]] : -1;
    if (threadIdx.x == 0) vcg8_init(S);
    __syncthreads();
    vb_cluster_sync();
    griddep_wait();
    griddep_launch();
    float r[2], x[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) r[q] = sl[q] >= 0 ? rhs[sl[q]] : 0.f;
    unsigned ph[3] = {0, 0, 0};
    bool dead = __ldcg(lim.error) != 0;
    vcg8_solve(C, M, S, j, 0, r, x, ph, lim, dead);
#pragma unroll
    for (int q = 0; q < 2; ++q)
        if (sl[q] >= 0) out[sl[q]] = x[q];
    vb_leave(dead);
}

// ---- both visits ------------------------------------------------------------
// Shared memory of a row CTA (cap rows of its own), in this order.
struct VBotLayout {
    size_t x, xc, coef, iv, dg, b, idx, cdst, rbuf, cg, total;
};
template <int ROWS>
__host__ __device__ inline VBotLayout vbot_layout(int n, int nc, int cap) {
    VBotLayout o;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t a = at;
        at = (at + bytes + 15) & ~(size_t)15;
        return a;
    };
    o.x = take(4 * ((size_t)n + 1));
    o.coef = take(4 * (size_t)VB_COEF * cap);
    o.iv = take(4 * (size_t)cap);
    o.dg = take(4 * (size_t)cap);
    o.b = take(4 * (size_t)cap);
    o.idx = take(4 * (size_t)(VB_COEF / 2) * cap);
    o.cdst = take(2 * (size_t)cap);
    // coarse solution (the distributed CG's p, whose last readers are done when the solution is sent)
    o.xc = ROWS ? take(4 * (size_t)nc) : 0;
    // residuals by coarse DOF and octant: all of them in the CG's CTA (which holds nothing else), or an eighth
    o.rbuf = ROWS ? 0 : take(4 * 8 * 32 * (size_t)vcg8_kmax(nc));
    o.cg = ROWS ? 0 : take(vcg8_smem_bytes(nc));
    o.total = at;
    const size_t own = 4 * 8 * (size_t)ROWS * VCG_THREADS;  // the CG's CTA
    if (ROWS && own > o.total) o.total = own;
    return o;
}

struct VbRow {  // a row's static data
    float k[VB_COEF], iv, b;
    unsigned ix[VB_COEF / 2];
};
struct VbSm {  // pointers into a row CTA's shared memory
    const float *coef, *iv, *b;
    const unsigned* idx;
    int cap;
};
__device__ __forceinline__ void vb_row(const VbSm& s, int li, VbRow& w) {
#pragma unroll
    for (int k = 0; k < VB_COEF; ++k) w.k[k] = s.coef[k * s.cap + li];
#pragma unroll
    for (int k = 0; k < VB_COEF / 2; ++k) w.ix[k] = s.idx[k * s.cap + li];
    w.iv = s.iv[li];
    w.b = s.b[li];
}
// off-diagonal sum of a row (voffdiag's operations)
__device__ __forceinline__ float vb_off(const VbRow& w, const float* x) {
    float u[VB_COEF];
#pragma unroll
    for (int k = 0; k < VB_COEF / 2; ++k) {
        u[2 * k] = x[w.ix[k] & 0xffffu];
        u[2 * k + 1] = x[w.ix[k] >> 16];
    }
    float p[VB_COEF];
#pragma unroll
    for (int k = 0; k < VB_COEF; ++k) p[k] = __fmul_rn(u[k], w.k[k]);
    const float td2 = __fadd_rn(__fadd_rn(p[6], p[7]), __fadd_rn(p[8], p[9]));
    const float td1 = __fadd_rn(__fadd_rn(p[10], p[11]), __fadd_rn(p[12], p[13]));
    return vsum_off(p[0], p[1], p[2], p[3], p[4], p[5], td2, td1);
}

// restriction (:2353-2413) of a coarse DOF's eight children (0 where there is none: s + 0 is s)
__device__ __forceinline__ float vb_restrict8(float4 a, float4 b) {
    float s = 0.f;
    s = __fadd_rn(s, a.x);
    s = __fadd_rn(s, a.y);
    s = __fadd_rn(s, a.z);
    s = __fadd_rn(s, a.w);
    s = __fadd_rn(s, b.x);
    s = __fadd_rn(s, b.y);
    s = __fadd_rn(s, b.z);
    s = __fadd_rn(s, b.w);
    return __fmul_rn(__fmul_rn(__fmul_rn(s, 0.125f), 0.5f), 2.0f);
}

// ROWS 4: CTA 0 does the CG, ROWS rows a thread (vcg_solve); 0: the CG over CTAs 0-7 (at least as many row CTAs)
template <int ROWS>
__global__ void __launch_bounds__(VB_THREADS, 1) k_vbottom(VBotArgs A) {
    extern __shared__ __align__(16) unsigned char vsm[];
    __shared__ uint64_t bars[4];                  // x (two that alternate), residuals, coarse solution
    __shared__ int g_row[6], g_cnt[7], g_loc[6];  // this CTA's rows of each group: first, count, local position
    __shared__ float g_word;                      // where the words of CTAs without rows arrive
    constexpr unsigned R0 = ROWS ? 1u : 0u;       // first row CTA
    const unsigned rank = cooperative_groups::this_cluster().block_rank();
    const int t = threadIdx.x, n = A.R.n, nc = A.R.nc, NC = A.NC;
    int cap = 0;
#pragma unroll
    for (int g = 0; g < 6; ++g) cap += (A.R.gs[g + 1] - A.R.gs[g] + NC - 1) / NC;
    const VBotLayout o = vbot_layout<ROWS>(n, nc, cap);
    const unsigned bx = smem_u32(&bars[0]), bres = smem_u32(&bars[2]), bxc = smem_u32(&bars[3]);
    bool dead = false;
    if (t < 4) mbar_init(&bars[t], 1);

    if constexpr (ROWS > 0) {
        if (rank == 0) {  // ---- the coarsest CG's CTA
            __shared__ float ps[VCG_THREADS * ROWS + 4];
            __shared__ __align__(16) float red[3][64];
            float* rbuf = reinterpret_cast<float*>(vsm);
            VCgRows<ROWS> M;
            vcg_load<ROWS>(A.C, M, ps);
            for (int i = t; i < 8 * ROWS * VCG_THREADS; i += VB_THREADS) rbuf[i] = 0.f;  // absent children
            __syncthreads();
            vb_cluster_sync();
            griddep_wait();
            griddep_launch();
            dead = __ldcg(A.lim.error) != 0;
            const unsigned xcb = smem_u32(vsm + o.xc);
#pragma unroll 1
            for (int visit = 0; visit < A.visits; ++visit) {
                if (t == 0 && !dead) vb_arm(bres, 4u * (unsigned)n);
                vb_wait(bres, visit & 1, A.lim, dead);
                float r[ROWS], x[ROWS];
#pragma unroll
                for (int k = 0; k < ROWS; ++k) {
                    const float4* c8 = reinterpret_cast<const float4*>(rbuf + 8 * (t + k * VCG_THREADS));
                    r[k] = vb_restrict8(c8[0], c8[1]);
                }
                vcg_solve<ROWS>(M, r, x, ps, red);
#pragma unroll
                for (int k = 0; k < ROWS; ++k) {
                    const int i = t + k * VCG_THREADS;
                    if (i < nc && !dead)
                        for (int q = 0; q < NC; ++q) vb_send(xcb + 4u * (unsigned)i, bxc, R0 + (unsigned)q, x[k]);
                }
            }
            vb_leave(dead);
            return;
        }
    }
    // ---- a row CTA
    const int j = (int)(rank - R0);
    if (t == 0) {
        int at = 0;
        for (int g = 0; g < 6; ++g) {
            const VbPart part = vb_part(A.R.gs[g + 1] - A.R.gs[g], NC, j);
            g_row[g] = A.R.gs[g] + part.lo;
            g_cnt[g] = part.cnt;
            g_loc[g] = at;
            at += part.cnt;
        }
        g_cnt[6] = at;
    }
    float* x = reinterpret_cast<float*>(vsm + o.x);
    float* xc = reinterpret_cast<float*>(vsm + o.xc);
    float* scoef = reinterpret_cast<float*>(vsm + o.coef);
    float* siv = reinterpret_cast<float*>(vsm + o.iv);
    float* sdg = reinterpret_cast<float*>(vsm + o.dg);
    float* sb = reinterpret_cast<float*>(vsm + o.b);
    unsigned* sidx = reinterpret_cast<unsigned*>(vsm + o.idx);
    uint16_t* scd = reinterpret_cast<uint16_t*>(vsm + o.cdst);
    float* rbuf = reinterpret_cast<float*>(vsm + o.rbuf);
    const VCg8Smem cg = vcg8_smem(vsm + o.cg, nc);
    if constexpr (ROWS == 0) xc = cg.p;
    const bool cg8 = ROWS == 0 && rank < VB_CG8;
    __syncthreads();
    // static data, before the wait for the previous kernel
    for (int i = t; i <= n; i += VB_THREADS) x[i] = 0.f;
    for (int g = 0; g < 6; ++g) {
        const int row0 = g_row[g], loc = g_loc[g];
        for (int i = t; i < g_cnt[g]; i += VB_THREADS) {
#pragma unroll
            for (int k = 0; k < VB_COEF; ++k) scoef[k * cap + loc + i] = A.R.coef[(long long)k * n + row0 + i];
#pragma unroll
            for (int k = 0; k < VB_COEF / 2; ++k) sidx[k * cap + loc + i] = A.R.idx[(long long)k * n + row0 + i];
            siv[loc + i] = A.R.iv[row0 + i];
            sdg[loc + i] = A.R.dg[row0 + i];
            scd[loc + i] = A.R.cdst[row0 + i];
        }
    }
    VCg8Rows M;
    unsigned ph[3] = {0, 0, 0};
    int rexp = 0;
    if constexpr (ROWS == 0) {
        if (cg8) {
            vcg8_load(A.C, (int)rank, M);
            rexp = A.R.rcount[rank];
            for (int i = t; i < 8 * 32 * vcg8_kmax(nc); i += VB_THREADS) rbuf[i] = 0.f;  // absent children
        }
        if (t == 0) vcg8_init(cg);
    }
    griddep_wait();
    griddep_launch();
    dead = __ldcg(A.lim.error) != 0;
    for (int g = 0; g < 6; ++g)
        for (int i = t; i < g_cnt[g]; i += VB_THREADS) sb[g_loc[g] + i] = A.rhs[A.R.slot[g_row[g] + i]];
    __syncthreads();
    vb_cluster_sync();  // every CTA has started, its mbarriers and its copy are set up

    const int nthr = vb_threads(g_cnt, VB_THREADS);
    const bool active = t < nthr;  // (uniform in a warp)
    const VbSm s{scoef, siv, sb, sidx, cap};
    const unsigned xb = smem_u32(x);
    int pass = 0;  // exchanges of x so far
    VbRow nx;      // this thread's first row of the next pass
    auto fetch = [&](int g) {
        if (t < g_cnt[g]) vb_row(s, g_loc[g] + t, nx);
    };
    auto arm = [&](int g) {  // a pass over group g (6: all rows) begins
        if (t == 0 && !dead) vb_arm(bx + 8u * (pass & 1), 4u * (unsigned)A.R.val[g]);
    };
    auto put = [&](unsigned a, float v) {
        if (dead) return;
        for (int q = 0; q < NC; ++q) vb_send(a, bx + 8u * (pass & 1), R0 + (unsigned)q, v);
    };
    auto send = [&](int row, float v) { put(xb + 4u * (unsigned)row, v); };
    auto sent = [&](int cnt) {  // the rows' values are sent; a CTA without rows sends its word
        if (cnt == 0 && t == 0) put(smem_u32(&g_word), 0.f);
    };
    auto wait = [&]() {
        vb_wait(bx + 8u * (pass & 1), (pass >> 1) & 1, A.lim, dead);
        ++pass;
        asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
    };
    // one Gauss-Seidel pass over group g; next: the group whose first row to fetch meanwhile (-1: none)
    auto gauss_seidel = [&](int g, int next) {
        arm(g);
        const int cnt = g_cnt[g], row0 = g_row[g], loc = g_loc[g];
        for (int i = t; i < cnt; i += VB_THREADS) {
            if (i != t) vb_row(s, loc + i, nx);
            send(row0 + i, vgs_update(nx.b, vb_off(nx, x), nx.iv, 1.0f, 0.0f, x[row0 + i]));
        }
        sent(cnt);
        if (next >= 0) fetch(next);
        wait();
    };
#pragma unroll 1
    for (int visit = 0; visit < A.visits; ++visit) {
        if constexpr (ROWS == 0) {
            if (cg8 && t == 0 && !dead) vb_arm(bres, 4u * (unsigned)rexp);
        }
        if (active) {
            fetch(0);
#pragma unroll 1
            for (int q = 0; q < 12; ++q) gauss_seidel(q % 6, q < 11 ? (q + 1) % 6 : -1);  // x, y, z: red, black
            // residuals to where they are restricted
#pragma unroll 1
            for (int g = 0; g < 6; ++g) {
                const int cnt = g_cnt[g], row0 = g_row[g], loc = g_loc[g];
                for (int i = t; i < cnt; i += VB_THREADS) {
                    VbRow w;
                    vb_row(s, loc + i, w);
                    const float res = __fsub_rn(w.b, __fmaf_rn(x[row0 + i], sdg[loc + i], vb_off(w, x)));
                    const int cd = scd[loc + i];
                    if (dead) break;
                    if constexpr (ROWS > 0) {
                        vb_send(smem_u32(vsm) + 4u * (unsigned)cd, bres, 0u, res);
                    } else {
                        const int cr = cd >> 3, pos = (((cr >> 8) << 5) | (cr & 31)) * 8 + (cd & 7);
                        vb_send(smem_u32(rbuf) + 4u * (unsigned)pos, bres, (unsigned)((cr & 255) >> 5), res);
                    }
                }
            }
            if (t == 0 && !dead) vb_arm(bxc, 4u * (unsigned)nc);
        }
        if constexpr (ROWS == 0) {
            if (cg8) {  // the whole block
                vb_wait(bres, visit & 1, A.lim, dead);
                const int w = t >> 5, l = t & 31;
                float r[2], cx[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float4* c8 = reinterpret_cast<const float4*>(rbuf + 8 * (32 * (w + 8 * q) + l));
                    r[q] = M.row[q] >= 0 ? vb_restrict8(c8[0], c8[1]) : 0.f;
                }
                vcg8_solve(A.C, M, cg, (int)rank, R0, r, cx, ph, A.lim, dead);
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    if (M.row[q] >= 0 && !dead)
                        for (int k = 0; k < NC; ++k)
                            vb_send(smem_u32(xc) + 4u * (unsigned)M.row[q], bxc, (unsigned)k, cx[q]);
            }
        }
        if (!active) continue;
        vb_wait(bxc, visit & 1, A.lim, dead);
        // prolongation: x += x_c of the coarse voxel
        arm(6);
#pragma unroll 1
        for (int g = 0; g < 6; ++g)
            for (int i = t; i < g_cnt[g]; i += VB_THREADS)
                send(g_row[g] + i, __fadd_rn(x[g_row[g] + i], xc[scd[g_loc[g] + i] >> 3]));
        sent(g_cnt[6]);
        fetch(5);
        wait();
#pragma unroll 1
        for (int q = 0; q < 12; ++q) gauss_seidel(5 - q % 6, q < 11 ? 5 - (q + 1) % 6 : -1);  // z, y, x: black, red
    }
    for (int g = 0; g < 6; ++g)
        for (int i = t; i < g_cnt[g]; i += VB_THREADS) A.lhs[A.R.slot[g_row[g] + i]] = x[g_row[g] + i];
    vb_leave(dead);
}

}  // namespace uaamg
