// poisson_march.cuh -- sweeps of the 7-point operator over one level, for FP32
// and 16-bit storage: sixteen lanes march through a leaf plane by plane.
//
// Lane q of a half-warp owns the four z-consecutive voxels of row Y = q >> 1,
// half zh = q & 1, in every plane x of its part of a leaf (NP planes).  A
// plane is then 64 consecutive values per array and half-warp, every address
// is a per-lane base plus a constant, and what a voxel reads along x stays in
// registers from plane to plane.  Rows above and below come from the leaf's own
// (just loaded) lines or a neighbour's, the z neighbours inside a leaf by
// shuffle; a missing neighbour is a page of zeros, so no load is predicated.
// The next plane's loads are issued before the current plane is computed and
// stored.
//
// In a leaf whose voxels are all DOF and whose coefficients, with those read
// from its neighbours, are the level's defaults (most leaves of a large
// domain), the coefficients are constants and each voxel's product with the
// face coefficient serves its neighbours along x and z: about 60 instructions
// per four voxels, so the bytes of x, b and the result bound the sweep.  (With
// a leaf per 128-thread block, its arrays and halos staged in shared memory,
// the same took 330 instructions and the issue slots bounded it.)  On the
// 124,644 leaves of a 512^3 level 0, 0.77 GB a sweep: Jacobi 256 -> 177 us, A p
// with p.q 275 -> 168, residual + restriction (0.51 GB) 263 -> 142; a 320^3
// level 0 in FP16 (0.09 GB): Jacobi 65 -> 49.
//
// The per-voxel operations are those of sweep_value_s / restrict_leaf in the
// same order, so results are theirs bit for bit.
#pragma once
#include "poisson_kernels.cuh"

namespace uaamg {

// ---- storage element traits
template <typename E> struct MarchE;
template <> struct MarchE<float> {
    static __device__ __forceinline__ float4 q(const float* p) { return *reinterpret_cast<const float4*>(p); }
    static __device__ __forceinline__ float v(const float* p) { return *p; }
    static __device__ __forceinline__ void st(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
    static __device__ __forceinline__ void st2(float* p, float a, float b) {
        *reinterpret_cast<float2*>(p) = make_float2(a, b);
    }
};

// ---- level traits.  A 16-bit level (poisson_mixed.cuh) stores its coefficients
// and rhs divided by a power of two cs and 1/diag multiplied by it; since
// scaling by a power of two is exact, these kernels compute in the stored units
// -- off-diagonal sum, diagonal term and residual all come out divided by cs,
// and the product with the stored 1/diag is the true value -- with the defaults
// of trimmed leaves brought to the same units (def_face / cs, def_diag / cs,
// def_invdiag * cs).  Each result equals the one computed from rescaled values.
template <class LV> struct MarchLv;
template <> struct MarchLv<DLevel> {
    using E = float;
    static constexpr bool SCALED = false;
    static __device__ __forceinline__ float def_face(const DLevel& L) { return L.def_face; }
    static __device__ __forceinline__ float def_diag(const DLevel& L) { return L.def_diag; }
    static __device__ __forceinline__ float def_invdiag(const DLevel& L) { return L.def_invdiag; }
    static __device__ __forceinline__ const float* spai0(const DLevel& L) { return L.spai0; }
    static __device__ __forceinline__ float def_spai0(const DLevel& L) { return L.def_spai0; }
};

__device__ float4 g_zero_leaf[UAAMG_LEAF4];  // what a missing neighbour reads (never written)

// what a plane reads besides x along x
struct MarchPlane {
    float4 yp, ym, b;
    float z;
};
__device__ __forceinline__ float4 f4mul(float4 a, float s) {
    return make_float4(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s), __fmul_rn(a.w, s));
}
__device__ __forceinline__ float4 f4mul(float4 a, float4 b) {
    return make_float4(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z), __fmul_rn(a.w, b.w));
}
__device__ __forceinline__ float4 f4add(float4 a, float4 b) {
    return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}

// the mode's result from the off-diagonal sum (sweep_value_s), four voxels
template <int MODE>
__device__ __forceinline__ float4 march_value(float4 xc, float4 off, float4 bb, float4 dg, float4 iv, float w,
                                              float wsor, float one_minus_wsor, int xy) {
    float4 res;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float x = f4get(xc, j), o = f4get(off, j);
        float v;
        if (MODE == M_RED || MODE == M_BLACK) {
            const int par = (xy + j) & 1;  // z = 4 zh + j has the parity of j
            const bool upd = (MODE == M_RED) ? (par == 0) : (par == 1);
            float r = __fsub_rn(f4get(bb, j), o);
            r = __fmul_rn(r, f4get(iv, j));
            r = __fmul_rn(r, wsor);
            v = upd ? __fmaf_rn(x, one_minus_wsor, r) : x;
        } else if (MODE == M_LAPLACIAN) {
            v = __fmaf_rn(x, f4get(dg, j), o);
        } else {
            v = __fsub_rn(f4get(bb, j), __fmaf_rn(x, f4get(dg, j), o));
            if (MODE == M_JACOBI) v = __fmaf_rn(w, __fmul_rn(v, f4get(iv, j)), x);
            if (MODE == M_SPAI0) v = __fmaf_rn(f4get(iv, j), v, x);
        }
        f4set(res, j, v);
    }
    return res;
}

// sets LEAF_PLAIN
__global__ void k_plain_leaves(DLevel L, uint32_t* flags) {
    const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
    if (leaf >= L.nl) return;
    constexpr unsigned ALL = TRIM_X | TRIM_Y | TRIM_Z | TRIM_DIAG;
    bool plain = (flags[leaf] & ALL) == ALL;
    for (int w = 0; w < 8 && plain; ++w) plain = L.mask[(long long)leaf * 8 + w] == ~0ull;
    for (int c = 0; c < 3 && plain; ++c) {
        const int n = L.nbr[(long long)leaf * 6 + 2 * c + 1];
        plain = n < 0 || (flags[n] & (TRIM_X << c));
    }
    if (plain) flags[leaf] |= LEAF_PLAIN;  // (bits that other threads read do not change)
}

constexpr int MARCH_THREADS = 128;
// CTAs per SM: the sweeps are bound by the loads in flight, so a few spilled
// words of the general path cost less than warps (512^3 level 0, Jacobi: 183 us
// at 5, 177 at 6, 175 at 7, 190 at 8; 250^3: 35.0, 35.8, 35.8, 39.0)
constexpr int MARCH_MINB = 6;
constexpr int MARCH_MINB16 = 7;  // 16-bit storage, 320^3: 58.6 us at 5, 54.4 at 6, 48.6 at 7, 51.7 at 8
// CTAs of a launch over nl leaves, NP planes per half-warp
__host__ __device__ __forceinline__ unsigned march_grid(int nl, int NP) {
    return (unsigned)(((long long)nl * (8 / NP) + 7) / 8);
}

// NP planes from X0 on of a leaf, by the 16 lanes q of a half-warp: a sweep
// (RESTRICT false: out[leaf] = value, optionally scaled by *zscale; returns the
// lane's part of the dot product, if dot.r) or residual + restriction (RESTRICT
// true, MODE M_RESIDUAL: coarse = 0.125 * sum of the active fine residuals of
// each 2x2x2 block, times coarse_scale on 16-bit levels).  RED and BLACK may run
// in place: what an update reads of its own colour is its own voxel.  on: the
// half-warp has a leaf (else it follows the other half); gate: nothing is
// written if this word is zero.  DOTK: 0 z.r with the b of a level-0 sweep or
// dot.r, 1 p.q with p the swept vector.
template <int MODE, class LV, typename TOut, bool RESTRICT, int NP, int DOTK = 0>
__device__ __forceinline__ double march_leaf(const LV& L, int leaf, int X0, bool on,
                                             const typename MarchLv<LV>::E* x, const typename MarchLv<LV>::E* b, TOut* out,
                                             float w, float wsor, float one_minus_wsor, const DotOut& dot,
                                             const float* zscale, float coarse_scale, const unsigned* gate = nullptr) {
    using T = MarchLv<LV>;
    using E = typename T::E;
    using P = MarchE<E>;
    const int lane = threadIdx.x & 31, q = lane & 15, Y = q >> 1, zh = q & 1;
    const long long l0 = (long long)leaf * UAAMG_LEAF;
    // ---- static data, before the wait for the previous kernel
    const int2* nbp = reinterpret_cast<const int2*>(L.nbr + (long long)leaf * 6);
    const int2 nx = nbp[0], ny = nbp[1], nz = nbp[2];  // (-, +) neighbours
    const unsigned fl = L.flags[leaf];
    int par = 0, oct = 0;
    if constexpr (RESTRICT) {
        par = L.parent[leaf];
        oct = L.octant[leaf];
    }
    const E* zero = reinterpret_cast<const E*>(g_zero_leaf);
    const E* px = x + l0 + 64 * X0 + 4 * q;
    const E* pxp = X0 + NP < 8 ? px + 64 * NP : (nx.y >= 0 ? x + (long long)nx.y * UAAMG_LEAF : zero) + 4 * q;
    const E* pxm = X0 > 0 ? px - 64 : (nx.x >= 0 ? x + (long long)nx.x * UAAMG_LEAF : zero) + 448 + 4 * q;
    const E* pyp = Y < 7 ? px + 8 : (ny.y >= 0 ? x + (long long)ny.y * UAAMG_LEAF : zero) + 64 * X0 + 4 * zh;
    const E* pym = Y > 0 ? px - 8 : (ny.x >= 0 ? x + (long long)ny.x * UAAMG_LEAF : zero) + 64 * X0 + 56 + 4 * zh;
    const int nzn = zh ? nz.y : nz.x;
    const E* pz = (nzn >= 0 ? x + (long long)nzn * UAAMG_LEAF : zero) + 64 * X0 + 8 * Y + (zh ? 0 : 7);
    const E* pb = MODE == M_LAPLACIAN ? zero : b + l0 + 64 * X0 + 4 * q;
    TOut* po = out;
    if constexpr (RESTRICT)
        po += (long long)par * UAAMG_LEAF + ((((oct >> 2) & 1) * 4 + (X0 >> 1)) << 6) +
              ((((oct >> 1) & 1) * 4 + (Y >> 1)) << 3) + (oct & 1) * 4 + 2 * zh;
    else
        po += l0 + 64 * X0 + 4 * q;
    const float df = T::def_face(L), ddg = T::def_diag(L);
    float div;
    if constexpr (MODE == M_SPAI0) div = T::def_spai0(L);
    else div = T::def_invdiag(L);
    griddep_wait();
    griddep_launch();
    if (gate) {
        on = on && *gate != 0;
        if (!__any_sync(FULLMASK, on)) return 0.0;
    }

    auto plane = [&](int i) {
        MarchPlane r;
        r.yp = P::q(pyp + 64 * i);
        r.ym = P::q(pym + 64 * i);
        r.z = P::v(pz + 64 * i);
        if (MODE != M_LAPLACIAN) r.b = P::q(pb + 64 * i);
        return r;
    };
    double sum = 0.0;
    float4 keep = f4zero();  // RESTRICT: the even plane's residual
    auto finish = [&](int i, float4 res, float4 bb, float4 xc) {
        if constexpr (RESTRICT) {
            if ((i & 1) == 0) {
                keep = res;
            } else {
                float4 up0, up1;  // the row above, both planes (even rows use it)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    f4set(up0, j, __shfl_down_sync(FULLMASK, f4get(keep, j), 2));
                    f4set(up1, j, __shfl_down_sync(FULLMASK, f4get(res, j), 2));
                }
                float s[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {  // the order of restrict_leaf; a voxel that is no DOF holds 0
                    float a = __fadd_rn(0.f, f4get(keep, 2 * k));
                    a = __fadd_rn(a, f4get(keep, 2 * k + 1));
                    a = __fadd_rn(a, f4get(up0, 2 * k));
                    a = __fadd_rn(a, f4get(up0, 2 * k + 1));
                    a = __fadd_rn(a, f4get(res, 2 * k));
                    a = __fadd_rn(a, f4get(res, 2 * k + 1));
                    a = __fadd_rn(a, f4get(up1, 2 * k));
                    a = __fadd_rn(a, f4get(up1, 2 * k + 1));
                    s[k] = __fmul_rn(a, 0.125f);
                    if (T::SCALED) s[k] = __fmul_rn(s[k], coarse_scale);
                }
                if (on && (Y & 1) == 0) MarchE<TOut>::st2(po + 64 * (i >> 1), s[0], s[1]);
            }
        } else {
            if constexpr (T::SCALED) {
                if (zscale) res = f4mul(res, *zscale);
            }
            if (on) MarchE<TOut>::st(po + 64 * i, res);
            if (dot.r) {  // z.r or p.q
                float4 rr = DOTK == 1 ? xc : bb;
                if constexpr (T::SCALED && DOTK == 0) rr = ld4(dot.r, leaf, (X0 + i) * 16 + q);
                const double s = (double)res.x * rr.x + (double)res.y * rr.y + (double)res.z * rr.z +
                                 (double)res.w * rr.w;
                if (on) sum = NP == 1 ? s : sum + s;
            }
        }
    };
    // two planes ahead: x along x, the rest of a plane one ahead
    float4 xc = P::q(px), xp = NP > 1 ? P::q(px + 64) : P::q(pxp);
    MarchPlane A = plane(0);
    float4 xm = P::q(pxm);
    constexpr unsigned PLAIN = LEAF_PLAIN | (MODE == M_SPAI0 ? TRIM_SPAI0 : 0u);
    if (__all_sync(FULLMASK, (fl & PLAIN) == PLAIN)) {
        const float4 dg4 = f4splat(ddg), iv4 = f4splat(div);
        float4 Pm = f4mul(xm, df), Pc = f4mul(xc, df);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            float4 xn = xp;
            MarchPlane B = A;
            if (i + 1 < NP) {
                xn = i + 2 < NP ? P::q(px + 64 * (i + 2)) : P::q(pxp);
                B = plane(i + 1);
            }
            const float4 Pp = f4mul(xp, df);
            const float up = __shfl_xor_sync(FULLMASK, Pc.x, 1), dn = __shfl_xor_sync(FULLMASK, Pc.w, 1);
            const float zs = __fmul_rn(A.z, df);
            const float4 zp = make_float4(Pc.y, Pc.z, Pc.w, zh == 0 ? up : zs);
            const float4 zm = make_float4(zh == 0 ? zs : dn, Pc.x, Pc.y, Pc.z);
            float4 off = f4add(Pp, Pm);
            off = f4add(off, f4add(f4mul(A.yp, df), f4mul(A.ym, df)));
            off = f4add(off, f4add(zp, zm));
            finish(i, march_value<MODE>(xc, off, A.b, dg4, iv4, w, wsor, one_minus_wsor, X0 + i + Y), A.b, xc);
            Pm = Pc;
            Pc = Pp;
            xc = xp;
            xp = xn;
            A = B;
        }
    } else {
        const uint64_t mw = L.mask[(long long)leaf * 8 + (q & 7)];
        const unsigned fx = nx.y >= 0 ? L.flags[nx.y] : ~0u, fy = ny.y >= 0 ? L.flags[ny.y] : ~0u,
                       fz = nz.y >= 0 ? L.flags[nz.y] : ~0u;
        const float4 df4 = f4splat(df);
        const long long at = l0 + 64 * X0 + 4 * q;
        auto coef = [&](const E* a, bool trimmed, float dv, int i) { return trimmed ? f4splat(dv) : P::q(a + at + 64 * i); };
        const bool tx = fl & TRIM_X, ty = fl & TRIM_Y, tz = fl & TRIM_Z, td = fl & TRIM_DIAG;
        const bool tyn = (Y < 7 ? fl : fy) & TRIM_Y, txn = (X0 + NP < 8 ? fl : fx) & TRIM_X;
        const E* pcyp = Y < 7 ? L.cy + at + 8 : L.cy + (long long)(ny.y >= 0 ? ny.y : leaf) * UAAMG_LEAF + 64 * X0 + 4 * zh;
        const E* pcxp = X0 + NP < 8 ? L.cx + at + 64 * NP : L.cx + (long long)(nx.y >= 0 ? nx.y : leaf) * UAAMG_LEAF + 4 * q;
        const E* pczp = L.cz + (long long)(nz.y >= 0 ? nz.y : leaf) * UAAMG_LEAF + 64 * X0 + 8 * Y;
        float4 cxm = coef(L.cx, tx, df, 0);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            float4 xn = xp;
            MarchPlane B = A;
            if (i + 1 < NP) {
                xn = i + 2 < NP ? P::q(px + 64 * (i + 2)) : P::q(pxp);
                B = plane(i + 1);
            }
            const float4 cxp = i + 1 < NP ? coef(L.cx, tx, df, i + 1) : (txn ? df4 : P::q(pcxp));
            const float4 cym = coef(L.cy, ty, df, i), cyp = tyn ? df4 : P::q(pcyp + 64 * i);
            const float4 czo = coef(L.cz, tz, df, i);
            const float cznb = (fz & TRIM_Z) ? df : P::v(pczp + 64 * i);
            float4 dg = f4zero(), iv = f4zero();
            if (MODE != M_RED && MODE != M_BLACK) dg = coef(L.diag, td, ddg, i);
            if (MODE == M_RED || MODE == M_BLACK || MODE == M_JACOBI) iv = coef(L.invdiag, td, div, i);
            if constexpr (MODE == M_SPAI0) iv = coef(T::spai0(L), fl & TRIM_SPAI0, div, i);
            const float up = __shfl_xor_sync(FULLMASK, xc.x, 1), dn = __shfl_xor_sync(FULLMASK, xc.w, 1);
            const float cup = __shfl_xor_sync(FULLMASK, czo.x, 1);
            const float4 zp = make_float4(xc.y, xc.z, xc.w, zh == 0 ? up : A.z);
            const float4 zm = make_float4(zh == 0 ? A.z : dn, xc.x, xc.y, xc.z);
            const float4 czp = make_float4(czo.y, czo.z, czo.w, zh == 0 ? cup : cznb);
            float4 off = f4add(f4mul(xp, cxp), f4mul(xm, cxm));
            off = f4add(off, f4add(f4mul(A.yp, cyp), f4mul(A.ym, cym)));
            off = f4add(off, f4add(f4mul(zp, czp), f4mul(zm, czo)));
            float4 res = march_value<MODE>(xc, off, A.b, dg, iv, w, wsor, one_minus_wsor, X0 + i + Y);
            const uint64_t word = __shfl_sync(FULLMASK, mw, (lane & 16) + X0 + i);
            const unsigned m = (unsigned)(word >> (4 * q)) & 0xFu;
            if (!(m & 1)) res.x = 0.f;
            if (!(m & 2)) res.y = 0.f;
            if (!(m & 4)) res.z = 0.f;
            if (!(m & 8)) res.w = 0.f;
            finish(i, res, A.b, xc);
            cxm = cxp;
            xm = xc;
            xc = xp;
            xp = xn;
            A = B;
        }
    }
    return sum;
}

// The block's part of a dot product into slot `slot` of `count`; the last block updates the PCG's scalars.
template <int DOTK>
__device__ __forceinline__ void march_dot(double sum, const DotOut& dot, int slot, int count) {
    __shared__ double shd[MARCH_THREADS / 32];
    const double part = block_sum128(sum, shd);
    double tot = 0.0;
    constexpr int TK = DOTK == 1 ? 2 : 0;
    if (reduce_sum(part, dot.partials, &dot.st->ticket[TK], slot, count, tot) && threadIdx.x == 0) {
        PcgState* st = dot.st;
        if constexpr (DOTK == 1) {
            const float sigma = (float)tot;
            st->sigma = sigma;
            st->alpha = __fdiv_rn(st->rho, sigma);
            st->first = 0;
        } else {
            const float rho_new = (float)tot;
            st->rho_new = rho_new;
            st->beta = st->first ? 0.f : __fdiv_rn(rho_new, st->rho);
            st->rho = rho_new;
        }
        st->ticket[TK] = 0;
    }
}

// One pass over a level (march_leaf).  The dot products: rho and beta (PCG lines
// 13-15, DOTK 0), or sigma and alpha (lines 6-7, DOTK 1); a partial per CTA, in
// an order that depends on the level only (NP 1: a CTA is a leaf, its threads those of the one-leaf kernels).
template <int MODE, class LV, typename TOut, bool RESTRICT, int NP, int DOTK = 0>
__global__ void __launch_bounds__(MARCH_THREADS, MarchLv<LV>::SCALED ? MARCH_MINB16 : MARCH_MINB)
    k_march(LV L, const typename MarchLv<LV>::E* x, const typename MarchLv<LV>::E* b, TOut* out, float w, float wsor,
            float one_minus_wsor, DotOut dot, const float* zscale, float coarse_scale) {
    constexpr int SEG = 8 / NP;
    const long long item = (long long)blockIdx.x * (MARCH_THREADS / 16) + (threadIdx.x >> 4);
    const bool on = item < (long long)L.nl * SEG;
    const int leaf = on ? (int)(item / SEG) : L.nl - 1, X0 = (int)(item % SEG) * NP;
    const double sum = march_leaf<MODE, LV, TOut, RESTRICT, NP, DOTK>(L, leaf, X0, on, x, b, out, w, wsor, one_minus_wsor,
                                                                       dot, zscale, coarse_scale);
    if constexpr (!RESTRICT) {
        if (dot.r) march_dot<DOTK>(sum, dot, (int)blockIdx.x, (int)gridDim.x);
    }
}

}  // namespace uaamg
