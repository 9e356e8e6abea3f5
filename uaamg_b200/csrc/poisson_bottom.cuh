// poisson_bottom.cuh -- the bottom of the Poisson W-cycle in one launch.
//
// In muCyclePreconditioner<2> (SIMD_UAAMG/simd_vdb_poisson.cpp:1844-1977) the
// level next to the coarsest (level lb) is visited twice per visit of the
// level above it, and each visit is seven smoothing / transfer passes over a
// few dozen leaves plus the coarsest CG: fourteen small launches that are
// bound by launch latency, not by their bytes.  k_bottom runs both visits in
// one launch of one thread-block cluster.  CTA 0 holds the coarsest level and
// does its CG; the other CTAs hold level lb, P leaves each (leaf i in CTA
// 1 + i / P, slot i % P), a thread four voxels of NL leaves.  What another
// thread reads (the two smoothing vectors) lives in shared memory, everything
// else (rhs, coefficients, the thread's own values, the addresses of its
// neighbours' values) in registers for the whole launch.
//
// Measured at 128^3 (40 leaves, 1,916 DOF below them; events around the
// launch): 40.3 us, 47.7 us when the leaves' pointers were read and tested in
// every pass and CTA 0 held leaves too.
// What bounds a pass is one chain: neighbour loads (distributed shared memory
// across CTAs), the stencil's arithmetic, the store, the cluster barrier.  The
// loads are unconditional (an absent neighbour's address is a zero slot), so
// they are in flight together; with the leaf's pointers read and tested per
// pass they queued one after another.  The CG is a CTA of its own because the
// registers of its matrix rows and of a leaf's stencil do not fit one thread
// together, and so the rows are loaded once for both visits.
//
// The per-voxel arithmetic is that of the unfused kernels (sweep_value_s,
// restrict_leaf, k_materialize with SrcFirstJacobi / SrcProlong,
// cg_rows_solve), so the results are bit-identical to the launch sequence it
// replaces.
#pragma once
#include <cooperative_groups.h>

#include "poisson_kernels.cuh"

namespace uaamg {

namespace cgx = cooperative_groups;

constexpr int BOT_THREADS = CG_THREADS;  // the coarsest CG's block; four 128-thread leaf groups
constexpr int BOT_GROUPS = BOT_THREADS / 128;
constexpr int BOT_MAX_CLUSTER = 16;      // non-portable cluster size limit
constexpr int BOT_MAX_NL = 2;            // leaves per thread: more do not fit its registers

struct BottomArgs {
    DLevel L;              // level lb
    const float* rhs;      // level lb rhs (written by the restriction of level lb - 1)
    float* lhs;            // level lb lhs (read by the prolongation into level lb - 1)
    DCoarsest C;           // coarsest level (lb + 1) system
    int nlc;               // coarsest level leaves (held by CTA 0)
    int P;                 // level-lb leaves per CTA
    float w[3];            // pre-smoothing weights (post-smoothing uses them reversed)
};

__device__ __forceinline__ float4 mask_out(float4 v, unsigned m) {
    if (!(m & 1)) v.x = 0.f;
    if (!(m & 2)) v.y = 0.f;
    if (!(m & 4)) v.z = 0.f;
    if (!(m & 8)) v.w = 0.f;
    return v;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// loads and stores at shared-memory addresses of the cluster (this CTA's own included)
__device__ __forceinline__ unsigned dsm_map(const void* p, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 dsm_ld4(unsigned a) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(a)
                 : "memory");
    return v;
}
__device__ __forceinline__ float2 dsm_ld2(unsigned a) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float dsm_ld1(unsigned a) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void dsm_st1(unsigned a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// Shared memory of a leaf CTA: per leaf slot the vectors x and t, then a slot
// of zeros.  Offsets in bytes.
constexpr unsigned BOT_X = 0, BOT_T = UAAMG_LEAF * 4, BOT_SLOT = 2 * UAAMG_LEAF * 4;

// One thread's part of one leaf of level lb.
struct BotLeaf {
    bool on;                                     // the leaf exists
    int leaf;
    unsigned m;                                  // DOF bits
    unsigned own, xp, xm, yp, ym, zn;            // addresses of the thread's float4, its neighbours', the +-z neighbour
    unsigned cr, cp, cm;                         // coarse rhs word it restricts to, coarse pair it prolongs, child bits
    float4 b, dg, iv, cxp, cxm, cyp, cym, czo;   // rhs and coefficients (sweep_static)
    float czp3;
    float4 v;                                    // the thread's values of the vector written last
};

// the leaf's static data, before the wait for the previous kernel
__device__ __forceinline__ void bot_load(const BottomArgs& A, BotLeaf& B, unsigned char* sm, int leaf, int slot, int t,
                                         const float* bc, const float* xc) {
    const DLevel& L = A.L;
    const int P = A.P, X = t >> 4, Y = (t >> 1) & 7, zh = t & 1;
    const unsigned zero = smem_u32(sm) + (unsigned)P * BOT_SLOT;
    B.leaf = leaf;
    B.on = slot < P && leaf < L.nl;
    B.m = 0;
    if (!B.on) return;
    PStatic S;
    stencil_static(L, leaf, t, S);
    B.cxp = S.cxp; B.cxm = S.cxm; B.cyp = S.cyp; B.cym = S.cym; B.czo = S.czo;
    const float pcz = __shfl_xor_sync(FULLMASK, S.czo.x, 1);
    B.czp3 = zh == 0 ? pcz : S.czp3;
    B.dg = (S.fl & TRIM_DIAG) ? f4splat(L.def_diag) : ld4(L.diag, leaf, t);
    B.iv = (S.fl & TRIM_DIAG) ? f4splat(L.def_invdiag) : ld4(L.invdiag, leaf, t);
    B.m = mask4(L.mask, leaf, t);
    B.own = smem_u32(sm) + (unsigned)slot * BOT_SLOT + 16u * t;
    // a neighbour leaf's slot, as the cluster addresses it
    auto at = [&](int n, int off) {
        return n < 0 ? zero : dsm_map(sm + (size_t)(n % P) * BOT_SLOT, 1u + (unsigned)(n / P)) + 4u * off;
    };
    B.xp = X < 7 ? B.own + 16u * 16 : at(S.nxp, 4 * (t - 112));
    B.xm = X > 0 ? B.own - 16u * 16 : at(S.nxm, 4 * (t + 112));
    B.yp = Y < 7 ? B.own + 16u * 2 : at(S.nyp, 4 * (t - 14));
    B.ym = Y > 0 ? B.own - 16u * 2 : at(S.nym, 4 * (t + 14));
    B.zn = zh == 0 ? at(S.nzm, 4 * t + 7) : at(S.nzp, 4 * t - 4);
    const int par = L.parent[leaf], o = L.octant[leaf];
    const int cX = ((o >> 2) & 1) * 4, cY = ((o >> 1) & 1) * 4, cZ = (o & 1) * 4;
    B.cp = dsm_map(xc + (size_t)par * UAAMG_LEAF + (cX + (X >> 1)) * 64 + (cY + (Y >> 1)) * 8 + cZ + 2 * zh, 0);
    // t < 64: coarse voxel (i, j, k) of the octant, its eight fine voxels
    const int i = (t >> 4) & 3, j = (t >> 2) & 3, k = t & 3;
    B.cr = dsm_map(bc + (size_t)par * UAAMG_LEAF + ((cX + i) << 6) + ((cY + j) << 3) + cZ + k, 0);
    B.cm = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int fo = ((2 * i + (q >> 2)) << 6) | ((2 * j + ((q >> 1) & 1)) << 3) | (2 * k + (q & 1));
        B.cm |= (unsigned)((L.mask[(long long)leaf * 8 + (fo >> 6)] >> (fo & 63)) & 1ull) << q;
    }
}

__device__ __forceinline__ void bot_store(const BotLeaf& B, unsigned dst) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(B.own + dst), "f"(B.v.x), "f"(B.v.y), "f"(B.v.z),
                 "f"(B.v.w)
                 : "memory");
}

// stencil_dyn: the 6-neighbour sum of the thread's float4 (B.v) over the vector at byte offset src
__device__ __forceinline__ float4 bot_stencil(const BotLeaf& B, unsigned src, int zh) {
    const float4 xp = dsm_ld4(B.xp + src), xm = dsm_ld4(B.xm + src);
    const float4 yp = dsm_ld4(B.yp + src), ym = dsm_ld4(B.ym + src);
    const float zn = dsm_ld1(B.zn + src);
    const float4 xc = B.v;
    const float px = __shfl_xor_sync(FULLMASK, xc.x, 1);
    const float pw = __shfl_xor_sync(FULLMASK, xc.w, 1);
    const float zp[4] = {xc.y, xc.z, xc.w, zh == 0 ? px : zn};
    const float zm[4] = {zh == 0 ? zn : pw, xc.x, xc.y, xc.z};
    const float czp[4] = {B.czo.y, B.czo.z, B.czo.w, B.czp3};
    float4 off;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float f1 = __fmul_rn(f4get(xp, j), f4get(B.cxp, j));
        float f2 = __fmul_rn(f4get(xm, j), f4get(B.cxm, j));
        float f3 = __fmul_rn(f4get(yp, j), f4get(B.cyp, j));
        float f4 = __fmul_rn(f4get(ym, j), f4get(B.cym, j));
        float f5 = __fmul_rn(zp[j], czp[j]);
        float f6 = __fmul_rn(zm[j], f4get(B.czo, j));
        f1 = __fadd_rn(f1, f2);
        f3 = __fadd_rn(f3, f4);
        f5 = __fadd_rn(f5, f6);
        f1 = __fadd_rn(f1, f3);
        f1 = __fadd_rn(f1, f5);
        f4set(off, j, f1);
    }
    return off;
}
// weighted Jacobi (sweep_value_s<M_JACOBI>): v = x + w invdiag (b - A x)
__device__ __forceinline__ void bot_jacobi(BotLeaf& B, unsigned src, float w, int zh) {
    const float4 off = bot_stencil(B, src, zh);
    float4 res;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float r = __fsub_rn(f4get(B.b, j), __fmaf_rn(f4get(B.v, j), f4get(B.dg, j), f4get(off, j)));
        r = __fmul_rn(r, f4get(B.iv, j));
        f4set(res, j, __fmaf_rn(w, r, f4get(B.v, j)));
    }
    B.v = mask_out(res, B.m);
}
// residual of t restricted into the coarsest rhs of CTA 0 (restrict_leaf<true>);
// the leaf's x, which nobody reads in this pass, carries the residual.  Called by
// the whole 128-thread group.
__device__ __forceinline__ void bot_restrict(const BotLeaf& B, int t, int group) {
    const float4 off = bot_stencil(B, BOT_T, t & 1);
    float4 res;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        f4set(res, j, __fsub_rn(f4get(B.b, j), __fmaf_rn(f4get(B.v, j), f4get(B.dg, j), f4get(off, j))));
    res = mask_out(res, B.m);
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(B.own + BOT_X), "f"(res.x), "f"(res.y), "f"(res.z),
                 "f"(res.w)
                 : "memory");
    asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
    if (t < 64) {
        const int i = t >> 4, j = (t >> 2) & 3, k = t & 3;
        const unsigned rs = B.own - 16u * t + 4u * (((2 * i) << 6) | ((2 * j) << 3) | (2 * k));
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 u = dsm_ld2(rs + 4u * (64 * (q >> 1) + 8 * (q & 1)));
            if ((B.cm >> (2 * q)) & 1) s = __fadd_rn(s, u.x);
            if ((B.cm >> (2 * q + 1)) & 1) s = __fadd_rn(s, u.y);
        }
        dsm_st1(B.cr, __fmul_rn(s, 0.125f));
    }
}
// v += x_c(parent voxel) on the DOF (SrcProlong with alpha 1)
__device__ __forceinline__ void bot_prolong(BotLeaf& B) {
    const float2 c = dsm_ld2(B.cp);
    const float c0 = __fmul_rn(1.0f, c.x), c1 = __fmul_rn(1.0f, c.y);
    if (B.m & 1) B.v.x = __fadd_rn(B.v.x, c0);
    if (B.m & 2) B.v.y = __fadd_rn(B.v.y, c0);
    if (B.m & 4) B.v.z = __fadd_rn(B.v.z, c1);
    if (B.m & 8) B.v.w = __fadd_rn(B.v.w, c1);
    B.v = mask_out(B.v, B.m);
}

// dynamic shared memory of every CTA: CTA 0's coarse vectors and CG storage, or the leaf slots
template <int ROWS, int NT>
constexpr size_t bottom_smem_bytes(int P, int nlc) {
    const size_t cg = (size_t)CgShape<ROWS, NT>::SMEM_FLOATS * 4 + (size_t)nlc * UAAMG_LEAF * 4 * 2;
    const size_t leaves = (size_t)(P + 1) * BOT_SLOT;
    return cg > leaves ? cg : leaves;
}

// Barriers of the cluster, the same for every CTA: start; per visit the two
// (first visit; else three) sweeps, the restriction, the CG, the prolongation
// and three sweeps.
template <int ROWS, int NT, int NL>
__global__ void __launch_bounds__(BOT_THREADS, 1) k_bottom(BottomArgs A) {
    extern __shared__ __align__(16) unsigned char bsm[];
    __shared__ __align__(16) float red[3][64];
    const unsigned rank = cgx::this_cluster().block_rank();
    // CTA 0's layout: the CG's storage, the coarsest lhs and rhs
    float* ps = reinterpret_cast<float*>(bsm);
    float* xc = ps + CgShape<ROWS, NT>::SMEM_FLOATS;
    float* bc = xc + (size_t)A.nlc * UAAMG_LEAF;
    if (rank == 0) {
        CgRows<ROWS, NT> M;
        cg_rows_load<ROWS, NT>(A.C, M, ps);
        griddep_wait();
        griddep_launch();
        cluster_sync_all();
#pragma unroll 1
        for (int visit = 0; visit < 2; ++visit) {
#pragma unroll 1
            for (int i = 0; i < 3 + visit; ++i) cluster_sync_all();
            cg_rows_solve<ROWS, NT>(A.C, M, bc, xc, ps, red);
#pragma unroll 1
            for (int i = 0; i < 5; ++i) cluster_sync_all();
        }
        return;
    }
    const int group = threadIdx.x >> 7, t = threadIdx.x & 127, zh = t & 1;
    BotLeaf B[NL];
#pragma unroll
    for (int q = 0; q < NL; ++q) {
        const int slot = group + q * BOT_GROUPS;
        bot_load(A, B[q], bsm, ((int)rank - 1) * A.P + slot, slot, t, bc, xc);
    }
    if (threadIdx.x < BOT_SLOT / 16) reinterpret_cast<float4*>(bsm + (size_t)A.P * BOT_SLOT)[threadIdx.x] = f4zero();
    griddep_wait();
    griddep_launch();
    const float w0 = A.w[0], w1 = A.w[1], w2 = A.w[2];
#define BOT_EACH(body)                 \
    _Pragma("unroll")                  \
    for (int q = 0; q < NL; ++q)       \
        if (B[q].on) { body; }         \
    cluster_sync_all();
    // rhs; t = first sweep from zero, w invdiag b.  The barrier: every CTA has started and filled its leaves
    BOT_EACH(B[q].b = ld4(A.rhs, B[q].leaf, t);
             B[q].v = mask_out(make_float4(__fmul_rn(w0, __fmul_rn(B[q].iv.x, B[q].b.x)),
                                           __fmul_rn(w0, __fmul_rn(B[q].iv.y, B[q].b.y)),
                                           __fmul_rn(w0, __fmul_rn(B[q].iv.z, B[q].b.z)),
                                           __fmul_rn(w0, __fmul_rn(B[q].iv.w, B[q].b.w))), B[q].m);
             bot_store(B[q], BOT_T));
#pragma unroll 1
    for (int visit = 0; visit < 2; ++visit) {
        // pre-smoothing, ends in t
        if (visit) { BOT_EACH(bot_jacobi(B[q], BOT_X, w0, zh); bot_store(B[q], BOT_T)); }
        BOT_EACH(bot_jacobi(B[q], BOT_T, w1, zh); bot_store(B[q], BOT_X));
        BOT_EACH(bot_jacobi(B[q], BOT_X, w2, zh); bot_store(B[q], BOT_T));
        BOT_EACH(bot_restrict(B[q], t, group));
        cluster_sync_all();  // the coarsest solve (its second visit in the W-cycle re-solves the same system: skipped)
        // post-smoothing with reversed weights: t += P x_c, x = J(t), t = J(x), x = J(t)
        BOT_EACH(bot_prolong(B[q]); bot_store(B[q], BOT_T));
        BOT_EACH(bot_jacobi(B[q], BOT_T, w2, zh); bot_store(B[q], BOT_X));
        BOT_EACH(bot_jacobi(B[q], BOT_X, w1, zh); bot_store(B[q], BOT_T));
        // the last barrier also keeps this CTA's shared memory until nobody reads it
        BOT_EACH(bot_jacobi(B[q], BOT_T, w0, zh); if (visit) st4(A.lhs, B[q].leaf, t, B[q].v); else bot_store(B[q], BOT_X));
    }
#undef BOT_EACH
}

}  // namespace uaamg
