// viscosity_march.cuh -- passes over one viscosity level that treat leaves of
// constant coefficients apart.
//
// The general applier reads fifteen coefficient values, one of b and up to
// fifteen of the three velocity channels for every voxel, through a
// neighbour table; a leaf per block, its issue slots and load latency bound it.  Most leaves of a large domain are plain: all
// voxels DOF of the channel, and every coefficient the channel's stencil
// reads there equal to one constant per array.  In those, sixteen lanes march
// through the leaf plane by plane (as poisson_march.cuh does): the constants
// sit in registers, what a voxel reads along x is carried from plane to plane,
// and the next plane's loads are issued before the current one is computed.
//
// A level's leaves are listed once when the hierarchy is built: general leaves
// with DOFs, leaves without, plain leaves; per channel, and for passes over
// all three channels at once (list 3: plain in all three).  A pass is one
// launch of a few CTAs per SM that take the general leaves first, a leaf per
// CTA, then the plain ones, four or two planes per half-warp.  Values are
// those of vapply_value_k bit for bit.
//
// 240^3 level 0 (15,056 leaves, 8,048 to 8,328 of them plain, 4,300 general): a
// colour of a channel 75-85 -> 48-55 us (154 MB of vectors and 120 MB of
// the general leaves' coefficients at least), A p 261 -> 116, residual +
// restriction 357 -> 189, the first residual 657 -> 129.  128^3 (2,774 leaves,
// 992 plain): 15-17 -> 13-14, 42 -> 28, 54 -> 44, 105 -> 35.  General leaves
// bound it: their coefficients' bytes, and the latency of a leaf (table,
// loads, sum) over the CTAs' rounds.
#pragma once
#include "poisson_march.cuh"
#include "viscosity_kernels.cuh"

namespace uaamg {

struct VPlain {
    const int* list;  // [4][nl]: general leaves with DOFs, leaves without, plain leaves
    const int* cnt;   // [4][4]: how many of each
    const float* K;   // [27] the constants of a plain leaf
};

// ---------------------------------------------------------------------------
// lists
enum { VP_GENERAL = 0, VP_EMPTY = 1, VP_PLAIN = 2 };
// An untrimmed level's constants are those of its first leaf whose voxels are
// DOF of all channels and whose 27 arrays are constant (cand).  A CTA per
// leaf; carr: which of its arrays are.
__global__ void __launch_bounds__(128) k_vconst(VLevel L, uint32_t* carr, int* cand) {
    griddep_wait();
    griddep_launch();
    const int leaf = blockIdx.x, t = threadIdx.x;
    const bool full = __syncthreads_and(t >= 24 || L.dof[((long long)(t >> 3) * L.nl + leaf) * 8 + (t & 7)] == ~0ull);
    uint32_t bits = 0;
#pragma unroll 3
    for (int a = 0; a < 3 * VNA; ++a) {
        const float* p = L.coef + ((long long)a * L.nl + leaf) * UAAMG_LEAF;
        const uint4 v = reinterpret_cast<const uint4*>(p)[t];
        const unsigned k = __float_as_uint(p[0]);
        if (__syncthreads_and(v.x == k && v.y == k && v.z == k && v.w == k)) bits |= 1u << a;
    }
    if (t) return;
    carr[leaf] = bits;
    if (full && bits == (1u << (3 * VNA)) - 1u) atomicMin(cand, leaf);
}
// Class of every leaf in the four lists; a warp per leaf.  Trimmed level 0
// (L.trim): the constants are the applier defaults, which trimmed arrays hold.
__global__ void __launch_bounds__(128) k_vclass(VLevel L, const uint32_t* carr, const int* cand, unsigned char* cls,
                                                float* K) {
    griddep_wait();
    griddep_launch();
    const int lane = threadIdx.x & 31, leaf = (int)(blockIdx.x * 4 + (threadIdx.x >> 5));
    if (leaf >= L.nl) return;
    const int first = L.trim ? 0 : *cand;
    const bool known = first < L.nl;
    const long long as = (long long)L.nl * UAAMG_LEAF;
    const int* nb = L.nb + (long long)leaf * 27;
    auto constant = [&](int a) { return L.trim ? L.app[a] : L.coef[a * as + (long long)first * UAAMG_LEAF]; };
    // the leaf's own arrays that hold their constant
    bool same = false;
    if (known && lane < 3 * VNA) {
        if (L.trim) same = L.trim[leaf] >> lane & 1u;
        else same = (carr[leaf] >> lane & 1u) && __float_as_uint(L.coef[lane * as + (long long)leaf * UAAMG_LEAF]) == __float_as_uint(constant(lane));
        if (leaf == 0) K[lane] = constant(lane);
    }
    const unsigned own = __ballot_sync(FULLMASK, same);
    uint64_t w = 0;
    if (lane < 24) w = L.dof[((long long)(lane >> 3) * L.nl + leaf) * 8 + (lane & 7)];
    const unsigned full = __ballot_sync(FULLMASK, w == ~0ull), any = __ballot_sync(FULLMASK, w != 0ull);
    // whether array a holds its constant in the layer of a face neighbour that touches this leaf
    auto layer = [&](int a, int axis, bool plus) {
        const int step = axis == 0 ? 9 : axis == 1 ? 3 : 1, n = nb[13 + (plus ? step : -step)];
        const unsigned k = __float_as_uint(constant(a));
        bool ok = true;
        if (n < 0) {
            ok = __float_as_uint(L.app[a]) == k;
        } else if (!(L.trim && (L.trim[n] >> a & 1u))) {
            const float* p = L.coef + a * as + (long long)n * UAAMG_LEAF;
            const int at = plus ? 0 : 7;
#pragma unroll
            for (int i = lane; i < 64; i += 32) {
                const int u = i >> 3, v = i & 7;
                ok &= __float_as_uint(p[axis == 0 ? voff3(at, u, v) : axis == 1 ? voff3(u, at, v) : voff3(u, v, at)]) == k;
            }
        }
        return (bool)__all_sync(FULLMASK, ok);
    };
    unsigned plain = 0;
    for (int c = 0; c < 3; ++c) {
        const int d1 = (c + 1) % 3, d2 = (c + 2) % 3;
        const unsigned need = 0x1Fu << (c * VNA) | 0xFu << (d1 * VNA + VA_T00) | 0xFu << (d2 * VNA + VA_T00);
        if ((own & need) != need || (full >> (8 * c) & 0xFFu) != 0xFFu) continue;
        bool ok = true;
        for (int ax = 0; ax < 3 && ok; ++ax) ok = layer(c * VNA + VA_NEGX + ax, ax, true);
        ok = ok && layer(d2 * VNA + VA_T10, c, false) && layer(d2 * VNA + VA_T11, c, false) &&
             layer(d1 * VNA + VA_T01, c, false) && layer(d1 * VNA + VA_T11, c, false);
        if (ok) plain |= 1u << c;
    }
    if (lane < 4) {
        const unsigned ch = lane < 3 ? 0xFFu << (8 * lane) : 0xFFFFFFu, pl = lane < 3 ? 1u << lane : 7u;
        cls[(long long)lane * L.nl + leaf] = (plain & pl) == pl ? VP_PLAIN : (any & ch) ? VP_GENERAL : VP_EMPTY;
    }
}
// The lists in leaf order within each class; a CTA of 1024 threads per list.
__global__ void __launch_bounds__(1024) k_vlist(int nl, const unsigned char* cls, int* list, int* cnt) {
    griddep_wait();
    griddep_launch();
    __shared__ int wsum[3][32];
    __shared__ int base[3];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    cls += (long long)blockIdx.x * nl;
    list += (long long)blockIdx.x * nl;
    int n[3] = {0, 0, 0};
    for (int i = t; i < nl; i += 1024)
#pragma unroll
        for (int k = 0; k < 3; ++k) n[k] += cls[i] == k;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int s = __reduce_add_sync(FULLMASK, n[k]);
        if (lane == 0) wsum[k][warp] = s;
    }
    __syncthreads();
    if (warp == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            n[k] = __reduce_add_sync(FULLMASK, wsum[k][lane]);
            if (lane == 0) cnt[blockIdx.x * 4 + k] = n[k];
        }
    if (t == 0) {
        base[0] = 0;
        base[1] = n[0];
        base[2] = n[0] + n[1];
    }
    for (int at = 0; at < nl; at += 1024) {
        const int i = at + t, k = i < nl ? cls[i] : 3;
        unsigned m[3];
        __syncthreads();  // base set, wsum read
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            m[q] = __ballot_sync(FULLMASK, k == q);
            if (lane == 0) wsum[q][warp] = __popc(m[q]);
        }
        __syncthreads();
        if (k < 3) {
            int o = base[k] + __popc(m[k] & ((1u << lane) - 1u));
            for (int v = 0; v < warp; ++v) o += wsum[k][v];
            list[o] = i;
        }
        __syncthreads();
        if (t < 3) {
            int s = 0;
            for (int v = 0; v < 32; ++v) s += wsum[t][v];
            base[t] += s;
        }
    }
}

// ---------------------------------------------------------------------------
// plain leaves
__device__ __forceinline__ float4 f4up(float4 a, float n) { return make_float4(a.y, a.z, a.w, n); }    // at z + 1
__device__ __forceinline__ float4 f4down(float4 a, float n) { return make_float4(n, a.x, a.y, a.z); }  // at z - 1
// address of voxel (X, Y, Z), coordinates -1..8, of a [nl][512] vector near a leaf (its row of L.nb); zeros if missing
__device__ __forceinline__ const float* vnear(const float* v, const float* zp, const int* nb, int X, int Y, int Z) {
    const int lf = nb[vnb_index(X, Y, Z)];
    return (lf >= 0 ? v + (long long)lf * UAAMG_LEAF : zp) + voff3(X, Y, Z);
}
__device__ __forceinline__ float4 vq(const float* p) { return *reinterpret_cast<const float4*>(p); }

// a plane of what channel c's stencil reads of the other two channels (see vmarch_leaf)
struct VCross {
    float4 g1, h1, g2, h2;
    float s1, t1, s2, t2;
};
// NP planes from X0 on of a plain leaf, channel c, by the 16 lanes q of a half-warp; xc, x1, x2 the channels c, c+1,
// c+2 of x, b the channel of b; finish(i, value at plane X0 + i).
template <int MODE, int c, int NP, class Finish>
__device__ __forceinline__ void vmarch_leaf(const VLevel& L, const float* K, int leaf, int X0, int q,
                                            const float* xv, const float* x1, const float* x2, const float* b,
                                            float w, Finish&& finish) {
    constexpr int d1 = (c + 1) % 3, d2 = (c + 2) % 3;
    constexpr int PM = MODE == VM_RED ? M_RED : MODE == VM_BLACK ? M_BLACK : MODE == VM_NORMAL ? M_LAPLACIAN : M_RESIDUAL;
    const int Y = q >> 1, Z0 = (q & 1) * 4;
    const int* nb = L.nb + (long long)leaf * 27;
    const float* zp = L.zpage;
    auto at = [&](const float* v, int X, int dy, int Z) { return vnear(v, zp, nb, X, Y + dy, Z); };
    const float W0 = K[c * VNA + VA_NEGX], W1 = K[c * VNA + VA_NEGY], W2 = K[c * VNA + VA_NEGZ];
    const float a00 = K[d2 * VNA + VA_T00], a01 = K[d2 * VNA + VA_T01], a10 = K[d2 * VNA + VA_T10], a11 = K[d2 * VNA + VA_T11];
    const float b00 = K[d1 * VNA + VA_T00], b01 = K[d1 * VNA + VA_T01], b10 = K[d1 * VNA + VA_T10], b11 = K[d1 * VNA + VA_T11];
    const float4 dg = f4splat(K[c * VNA + VA_DIAG]), iv = f4splat(K[c * VNA + VA_INV]);
    // own channel
    const float* px = xv + (long long)leaf * UAAMG_LEAF + 64 * X0 + 4 * q;
    const float* pxp = at(xv, X0 + NP, 0, Z0);
    const float* pyp = at(xv, X0, 1, Z0);
    const float* pym = at(xv, X0, -1, Z0);
    const float* pz = at(xv, X0, 0, Z0 ? 8 : -1);
    const float* pb = MODE == VM_NORMAL ? zp : b + (long long)leaf * UAAMG_LEAF + 64 * X0 + 4 * q;
    // The other channels' rows and z edges:
    //   c 0: u1 = y, rows Y, Y+1; u2 = z, row Y and its z+1 edge; each also one plane back
    //   c 1: u1 = z, rows Y, Y-1 and their z+1 edges; u2 = x, rows Y, Y-1, also one plane on
    //   c 2: u1 = x, row Y and its z-1 edge, also one plane on; u2 = y, rows Y, Y+1 and their z-1 edges
    const int Ze = c == 2 ? Z0 - 1 : Z0 + 4, XE = c == 0 ? X0 - 1 : X0 + NP;
    constexpr int hy = c == 1 ? -1 : 1;
    const float* g1 = at(x1, X0, 0, Z0);
    const float* g2 = at(x2, X0, 0, Z0);
    const float* h1 = c != 2 ? at(x1, X0, hy, Z0) : zp;
    const float* h2 = c != 0 ? at(x2, X0, hy, Z0) : zp;
    const float* s1 = c != 0 ? at(x1, X0, 0, Ze) : zp;
    const float* t1 = c == 1 ? at(x1, X0, hy, Ze) : zp;
    const float* s2 = c != 1 ? at(x2, X0, 0, Ze) : zp;
    const float* t2 = c == 2 ? at(x2, X0, hy, Ze) : zp;
    auto cross = [&](int i) {
        VCross r;
        r.g1 = vq(g1 + 64 * i);
        r.g2 = vq(g2 + 64 * i);
        if (c != 2) r.h1 = vq(h1 + 64 * i);
        if (c != 0) r.h2 = vq(h2 + 64 * i);
        if (c != 0) r.s1 = s1[64 * i];
        if (c == 1) r.t1 = t1[64 * i];
        if (c != 1) r.s2 = s2[64 * i];
        if (c == 2) r.t2 = t2[64 * i];
        return r;
    };
    VCross E{};  // the plane before the first (c 0) or after the last (c 1, 2)
    if (c == 0) {
        E.g1 = vq(at(x1, XE, 0, Z0));
        E.h1 = vq(at(x1, XE, 1, Z0));
        E.g2 = vq(at(x2, XE, 0, Z0));
        E.s2 = *at(x2, XE, 0, Ze);
    } else if (c == 1) {
        E.g2 = vq(at(x2, XE, 0, Z0));
        E.h2 = vq(at(x2, XE, -1, Z0));
    } else {
        E.g1 = vq(at(x1, XE, 0, Z0));
        E.s1 = *at(x1, XE, 0, Ze);
    }
    auto plane = [&](int i) {
        MarchPlane r;
        r.yp = vq(pyp + 64 * i);
        r.ym = vq(pym + 64 * i);
        r.z = pz[64 * i];
        r.b = MODE == VM_NORMAL ? f4zero() : vq(pb + 64 * i);
        return r;
    };
    float4 xc = vq(px), xp = NP > 1 ? vq(px + 64) : vq(pxp);
    MarchPlane A = plane(0);
    VCross C = cross(0), P = E;  // P: the plane before (c 0)
    float4 Qm = f4mul(vq(at(xv, X0 - 1, 0, Z0)), W0), Qc = f4mul(xc, W0);  // the x products of this and the last plane
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        float4 xn = xp;
        MarchPlane B = A;
        VCross N = E;
        if (i + 1 < NP) {
            xn = i + 2 < NP ? vq(px + 64 * (i + 2)) : vq(pxp);
            B = plane(i + 1);
            N = cross(i + 1);
        }
        const float4 Qp = f4mul(xp, W0);
        const float4 zc = f4mul(xc, W2);
        const float up = __shfl_xor_sync(FULLMASK, zc.x, 1), dn = __shfl_xor_sync(FULLMASK, zc.w, 1);
        const float ze = __fmul_rn(A.z, W2);
        float4 off = f4add(Qp, Qm);
        off = f4add(off, f4add(f4mul(A.yp, W1), f4mul(A.ym, W1)));
        off = f4add(off, f4add(f4up(zc, Z0 ? ze : up), f4down(zc, Z0 ? dn : ze)));
        float4 u1p, u1m, u1mp, u2m, u2p, u2mp;
        if (c == 0) {
            u1p = C.h1;
            u1m = P.g1;
            u1mp = P.h1;
            u2m = P.g2;
            u2p = f4up(C.g2, C.s2);
            u2mp = f4up(P.g2, P.s2);
        } else if (c == 1) {
            u1p = f4up(C.g1, C.s1);
            u1m = C.h1;
            u1mp = f4up(C.h1, C.t1);
            u2m = C.h2;
            u2p = N.g2;
            u2mp = N.h2;
        } else {
            u1p = N.g1;
            u1m = f4down(C.g1, C.s1);
            u1mp = f4down(N.g1, N.s1);
            u2m = f4down(C.g2, C.s2);
            u2p = C.h2;
            u2mp = f4down(C.h2, C.t2);
        }
        const float4 td2 = f4add(f4add(f4mul(C.g1, a00), f4mul(u1p, a01)), f4add(f4mul(u1m, a10), f4mul(u1mp, a11)));
        const float4 td1 = f4add(f4add(f4mul(C.g2, b00), f4mul(u2m, b01)), f4add(f4mul(u2p, b10), f4mul(u2mp, b11)));
        off = f4add(f4add(off, td2), td1);
        finish(i, march_value<PM>(xc, off, A.b, dg, iv, w, w, __fsub_rn(1.0f, w), X0 + i + Y));
        Qm = Qc;
        Qc = Qp;
        xc = xp;
        xp = xn;
        A = B;
        P = C;
        C = N;
    }
}

// CTAs of the passes below: as many as are resident.  Per SM (240^3 level 0, a colour, and A p): 55-58 and 120 us at 3,
// 49-54 and 116 at 4, 50-52 and 121 at 5 (which spills in the restriction).
constexpr int VMARCH_THREADS = 128;
constexpr int VMARCH_MINB = 4;
constexpr int VMARCH_PER_CTA = VMARCH_THREADS / 16;  // plain items (NP planes of a leaf) at once
// this CTA's first group of plain items: the CTAs that had one general leaf fewer start first
__device__ __forceinline__ int vmarch_start(int ngen) {
    const int G = (int)gridDim.x;
    return ((int)blockIdx.x + G - ngen % G) % G;
}

// RED / BLACK of channel c, x updated in place (as k_vapply_seq).
template <int MODE, int c>
__global__ void __launch_bounds__(VMARCH_THREADS, VMARCH_MINB) k_vmarch(VLevel L, VPlain S, float* x, const float* b,
                                                                        float w) {
    __shared__ VNbSh sh[2];
    const int t = threadIdx.x;
    const int* list = S.list + (long long)c * L.nl;
    const int ngen = S.cnt[4 * c], nempty = S.cnt[4 * c + 1], nplain = S.cnt[4 * c + 2];
    const long long cs = (long long)L.nl * UAAMG_LEAF;
    // general leaves; the next leaf's table entries load while this one computes
    int i = blockIdx.x, leaf = i < ngen ? list[i] : -1;
    int next = i + (int)gridDim.x < ngen ? list[i + gridDim.x] : -1;
    unsigned m = 0;
    if (leaf >= 0) {
        if (t < 27) {
            const int v = L.nb[(long long)leaf * 27 + t];
            sh[0].nb[t] = v;
            sh[0].cnb[t] = L.cnb ? L.cnb[(long long)leaf * 27 + t] : v;
        }
        m = vmask4(L, c, leaf, t);
    }
    __syncthreads();
    griddep_wait();
    griddep_launch();
    for (int it = 0; leaf >= 0; ++it) {
        const VNbSh& cur = sh[it & 1];
        int nb_n = -1, cnb_n = -1;
        unsigned m_n = 0;
        i += gridDim.x;
        const int next2 = i + (int)gridDim.x < ngen ? list[i + gridDim.x] : -1;
        if (next >= 0) {
            if (t < 27) {
                nb_n = L.nb[(long long)next * 27 + t];
                cnb_n = L.cnb ? L.cnb[(long long)next * 27 + t] : nb_n;
            }
            m_n = vmask4(L, c, next, t);
        }
        vapply_tab<MODE, c, false>(L, cur, leaf, m, x, b, x, w);
        if (t < 27) {
            sh[(it + 1) & 1].nb[t] = nb_n;
            sh[(it + 1) & 1].cnb[t] = cnb_n;
        }
        m = m_n;
        leaf = next;
        next = next2;
        __syncthreads();
    }
    // plain leaves
    constexpr int NP = 4, SEG = 8 / NP;
    const int items = nplain * SEG, q = t & 15;
    list += ngen + nempty;
    float* xo = x + c * cs;
    const float* x1 = x + ((c + 1) % 3) * cs;
    const float* x2 = x + ((c + 2) % 3) * cs;
    for (int g = vmarch_start(ngen) * VMARCH_PER_CTA; g < items; g += (int)gridDim.x * VMARCH_PER_CTA) {
        const int item = g + (t >> 4);
        const bool on = item < items;
        const int lf = list[(on ? item : items - 1) / SEG], X0 = (on ? item : items - 1) % SEG * NP;
        float* po = xo + (long long)lf * UAAMG_LEAF + 64 * X0 + 4 * q;
        vmarch_leaf<MODE, c, NP>(L, S.K, lf, X0, q, xo, x1, x2, b + c * cs, w, [&](int k, float4 v) {
            if (on) *reinterpret_cast<float4*>(po + 64 * k) = v;
        });
    }
}

// Passes over the three channels: q = A x (VM_NORMAL), r = b - A x with |r|_inf
// and the start of the PCG (VM_RESIDUAL; lines 2-3), and the residual restricted
// into C's rhs (VM_RESTRICT; coarse_lhs is zeroed as by k_vresrestrict).  List 3:
// a plain leaf is plain in every channel, so what the channels share is read once.
enum { VM_RESTRICT = 16 };
struct VMarchOut {
    float* out;         // q, r or the coarse rhs
    float* coarse_lhs;  // or null
    double* partials;
    PcgState* st;
    cudaGraphConditionalHandle cond;
    int use_cond;
    int pad;  // (the recorder of the solve-graph cache compares argument bytes)
};
template <int OP, int c, int NP>
__device__ __forceinline__ void vmarch3_leaf(const VLevel& F, const VLevel& C, const VPlain& S, int leaf, int X0, int q,
                                             bool on, const float* x, const float* b, const VMarchOut& O, float& a) {
    constexpr int MODE = OP == VM_NORMAL ? VM_NORMAL : VM_RESIDUAL;
    const long long cs = (long long)F.nl * UAAMG_LEAF;
    const float* xv = x + c * cs;
    const float* x1 = x + ((c + 1) % 3) * cs;
    const float* x2 = x + ((c + 2) % 3) * cs;
    if constexpr (OP == VM_RESTRICT) {
        const int P = F.parent[leaf], oc = F.octant[leaf], Y = q >> 1;
        const int cx = ((oc >> 2) & 1) * 4 + (X0 >> 1), cy = ((oc >> 1) & 1) * 4 + (Y >> 1), cz = (oc & 1) * 4 + 2 * (q & 1);
        const long long co = ((long long)c * C.nl + (P < 0 ? 0 : P)) * UAAMG_LEAF + voff3(cx, cy, cz);
        const uint64_t* cm = C.dof + ((long long)c * C.nl + (P < 0 ? 0 : P)) * 8;
        float4 keep = f4zero();
        vmarch_leaf<MODE, c, NP>(F, S.K, leaf, X0, q, xv, x1, x2, b + c * cs, 1.f, [&](int k, float4 v) {
            if ((k & 1) == 0) {
                keep = v;
                return;
            }
            float4 up0, up1;  // the row above, both planes (even rows use it)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                f4set(up0, j, __shfl_down_sync(FULLMASK, f4get(keep, j), 2));
                f4set(up1, j, __shfl_down_sync(FULLMASK, f4get(v, j), 2));
            }
            const unsigned bits = (unsigned)(cm[cx + (k >> 1)] >> (8 * cy + cz)) & 3u;
            float r[2];
#pragma unroll
            for (int z = 0; z < 2; ++z) {  // the order of k_vrestrict
                float s = __fadd_rn(0.f, f4get(keep, 2 * z));
                s = __fadd_rn(s, f4get(keep, 2 * z + 1));
                s = __fadd_rn(s, f4get(up0, 2 * z));
                s = __fadd_rn(s, f4get(up0, 2 * z + 1));
                s = __fadd_rn(s, f4get(v, 2 * z));
                s = __fadd_rn(s, f4get(v, 2 * z + 1));
                s = __fadd_rn(s, f4get(up1, 2 * z));
                s = __fadd_rn(s, f4get(up1, 2 * z + 1));
                r[z] = (bits >> z & 1u) ? __fmul_rn(__fmul_rn(__fmul_rn(s, 0.125f), 0.5f), 2.0f) : 0.f;
            }
            if (on && P >= 0 && (Y & 1) == 0) {
                *reinterpret_cast<float2*>(O.out + co + 64 * (k >> 1)) = make_float2(r[0], r[1]);
                if (O.coarse_lhs) *reinterpret_cast<float2*>(O.coarse_lhs + co + 64 * (k >> 1)) = make_float2(0.f, 0.f);
            }
        });
    } else {
        float* po = O.out + c * cs + (long long)leaf * UAAMG_LEAF + 64 * X0 + 4 * q;
        vmarch_leaf<MODE, c, NP>(F, S.K, leaf, X0, q, xv, x1, x2, b + c * cs, 1.f, [&](int k, float4 v) {
            if (!on) return;
            *reinterpret_cast<float4*>(po + 64 * k) = v;
            if (OP == VM_RESIDUAL) a = nanmax(a, vabs4(v, 0xFu));
        });
    }
}
template <int OP, int c>
__device__ __forceinline__ void vmarch3_general(const VLevel& F, const VLevel& C, const VNbSh& sh, float* rs, int leaf,
                                                unsigned m, const float* x, const float* b, const VMarchOut& O, float& a) {
    if constexpr (OP == VM_RESTRICT) {
        vresrestrict_tab<c, false>(F, C, sh, rs, leaf, m, x, b, O.out, O.coarse_lhs);
    } else {
        const float4 v = vapply_tab<OP == VM_NORMAL ? VM_NORMAL : VM_RESIDUAL, c, false>(F, sh, leaf, m, x, b, O.out, 1.f);
        if (OP == VM_RESIDUAL) a = nanmax(a, vabs4(v, 0xFu));
    }
}
template <int OP>
__global__ void __launch_bounds__(VMARCH_THREADS, VMARCH_MINB) k_vmarch3(VLevel F, VLevel C, VPlain S, const float* x,
                                                                         const float* b, VMarchOut O) {
    __shared__ VNbSh sh[2];
    __shared__ __align__(16) float rs[OP == VM_RESTRICT ? UAAMG_LEAF : 4];
    const int t = threadIdx.x;
    const int* list = S.list + 3LL * F.nl;
    const int nplain = S.cnt[14], ngen = S.cnt[12];
    float a = 0.f;
    // general leaves, a channel at a time (the coarse voxels of leaves without DOFs hold none: they stay zero); the next
    // item's table entries load while this one computes
    const int n3 = 3 * ngen, step = (int)gridDim.x;
    auto leaf_of = [&](int i) { return i < n3 ? list[i / 3] : -1; };
    auto table = [&](int leaf, int c, int& nb, int& cnb, unsigned& m) {
        if (leaf < 0) return;
        if (t < 27) {
            nb = F.nb[(long long)leaf * 27 + t];
            cnb = F.cnb ? F.cnb[(long long)leaf * 27 + t] : nb;
        }
        m = vmask4(F, c, leaf, t);
    };
    int i = blockIdx.x, leaf = leaf_of(i), next = leaf_of(i + step);
    int nb = -1, cnb = -1;
    unsigned m = 0;
    table(leaf, i % 3, nb, cnb, m);
    griddep_wait();
    griddep_launch();
#pragma unroll 1
    for (int it = 0; leaf >= 0; ++it) {
        VNbSh& cur = sh[it & 1];
        if (t < 27) {
            cur.nb[t] = nb;
            cur.cnb[t] = cnb;
        }
        __syncthreads();
        const int c = i % 3, here = leaf;
        const unsigned mh = m;
        i += step;
        table(next, i % 3, nb, cnb, m);
        leaf = next;
        next = leaf_of(i + step);
        if (c == 0) vmarch3_general<OP, 0>(F, C, cur, rs, here, mh, x, b, O, a);
        else if (c == 1) vmarch3_general<OP, 1>(F, C, cur, rs, here, mh, x, b, O, a);
        else vmarch3_general<OP, 2>(F, C, cur, rs, here, mh, x, b, O, a);
    }
    constexpr int NP = 2, SEG = 8 / NP;
    const int items = nplain * SEG, q = t & 15;
    list += S.cnt[12] + S.cnt[13];
#pragma unroll 1
    for (int g = vmarch_start(3 * ngen) * VMARCH_PER_CTA; g < items; g += (int)gridDim.x * VMARCH_PER_CTA) {
        const int item = g + (t >> 4);
        const bool on = item < items;
        const int leaf = list[(on ? item : items - 1) / SEG], X0 = (on ? item : items - 1) % SEG * NP;
        asm volatile("" ::: "memory");  // no loads of the next channel ahead of this one's: they would spill
        vmarch3_leaf<OP, 0, NP>(F, C, S, leaf, X0, q, on, x, b, O, a);
        asm volatile("" ::: "memory");
        vmarch3_leaf<OP, 1, NP>(F, C, S, leaf, X0, q, on, x, b, O, a);
        asm volatile("" ::: "memory");
        vmarch3_leaf<OP, 2, NP>(F, C, S, leaf, X0, q, on, x, b, O, a);
    }
    if constexpr (OP == VM_RESIDUAL) {
        __shared__ float shf[4];
        __shared__ bool last;
        const float part = block_max128(a, shf);
        if (vpublish((double)part, O.partials, &O.st->ticket[1], &last)) {
            const float nu = vgather_max(O.partials, shf);
            if (t == 0) vpcg_start(O.st, nu, O.cond, O.use_cond);
        }
    }
}

}  // namespace uaamg
