// Adjoint-method gradients of <H> for parameterised circuits.
//
// No reference counterpart: BraketSimulator.jl declares AdjointGradient
// (src/results.jl:90-159) but rejects it at parse time (src/pragmas.jl:67-68).
// Algorithm (Jones & Gacon, arXiv:2009.02823): forward |psi_L>, |lambda> = H|psi_L>,
// then for l = L..1: gradient of gate l from <lambda| dU_l |psi_{l-1}>, and
// psi <- U_l^dag psi, lambda <- U_l^dag lambda.  Gates exp(-i theta G/2) with a
// Pauli-string generator G give dE/dtheta = Im <lambda|G|psi_l>; PhaseShift gives
// -2 Im <lambda|P1|psi_l>.
//
// Both backward states are swept together: one tile sweep loads the same tile of
// psi and lambda, applies the daggered gates of a run to both, and accumulates
// the inner products of the run's parameterised gates before applying them.
//
// Checkpoints: the forward pass runs in S segments and keeps psi after each of the
// first S-1; the backward pass, entering a segment, replaces the uncomputed psi by
// that checkpoint, so the rounding drift of uncomputation never spans more than
// one segment.  S comes from the handle's tuning (BS_TUNE_ADJ_SEGMENTS) or, by
// default, from the parameterised gate count and a quarter of the free device
// memory; when memory binds (an allocation fails) S is halved down to 1, pure
// uncomputation.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>
#include "bs_internal.h"
#include "bs_ff.cuh"

namespace {

constexpr int kAThreads = 256;

struct PauliTerm {
    uint64_t xm, zm;     // endian masks
    int ph;              // nY mod 4
    float ch, cl;        // coefficient as float-float
};

__device__ __forceinline__ cff f4c(float4 v) { return {v.x, v.y, v.z, v.w}; }
__device__ __forceinline__ float4 c4f(const cff& c) { return make_float4(c.rh, c.rl, c.ih, c.il); }

// lambda_i = sum_t c_t (-i)^ph_t (-1)^popc(i & zm_t) psi_{i ^ xm_t}
// C64: complex64 storage; the arithmetic and the sums stay float-float either way.
template <bool C64>
__global__ void __launch_bounds__(kAThreads) k_pauli_sum(const typename Elem<C64>::T* __restrict__ psi,
                                                         typename Elem<C64>::T* __restrict__ lam, int64_t n,
                                                         const PauliTerm* __restrict__ terms, int nt) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        ffacc ar{0.f, 0.f}, ai{0.f, 0.f};
        for (int t = 0; t < nt; t++) {
            PauliTerm p = terms[t];
            cff x = Elem<C64>::load(psi[i ^ (int64_t)p.xm]);
            int ph = p.ph + ((__popcll((unsigned long long)i & p.zm) & 1) ? 2 : 0);
            // (-i)^ph: multiply x by i^(4-ph)
            x = cmul_ipow(x, (4 - (ph & 3)) & 3);
            acc_add(ar, p.ch, p.cl, x.rh, x.rl);
            acc_add(ai, p.ch, p.cl, x.ih, x.il);
        }
        lam[i] = Elem<C64>::store(cdone(ar, ai));
    }
}

__device__ void block_sum2(double a, double b, double* out2) {
    __shared__ double ra[kAThreads / 32], rb[kAThreads / 32];
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) { ra[w] = a; rb[w] = b; }
    __syncthreads();
    if (w == 0) {
        a = (l < (int)(blockDim.x >> 5)) ? ra[l] : 0.0;
        b = (l < (int)(blockDim.x >> 5)) ? rb[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_down_sync(0xffffffffu, a, o);
            b += __shfl_down_sync(0xffffffffu, b, o);
        }
        if (l == 0) { atomicAdd(out2, a); atomicAdd(out2 + 1, b); }
    }
}

// <a|b> (complex) into out2[0..1]
template <bool C64>
__global__ void __launch_bounds__(kAThreads) k_inner(const typename Elem<C64>::T* __restrict__ a,
                                                     const typename Elem<C64>::T* __restrict__ b, int64_t n,
                                                     double* __restrict__ out2) {
    ffsum sr{0.f, 0.f}, si{0.f, 0.f};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        cff x = Elem<C64>::load(a[i]), y = Elem<C64>::load(b[i]);
        ffacc r, m;
        acc_first(r, x.rh, x.rl, y.rh, y.rl);
        acc_add(r, x.ih, x.il, y.ih, y.il);
        acc_first(m, x.rh, x.rl, y.ih, y.il);
        acc_add(m, -x.ih, -x.il, y.rh, y.rl);
        ff rr = acc_done(r), mm = acc_done(m);
        fsum_add(sr, rr.h, rr.l);
        fsum_add(si, mm.h, mm.l);
    }
    block_sum2(ff2d(sr.h, sr.l), ff2d(si.h, si.l), out2);
}

// ---------------------------------------------------------------- backward sweep of both states
// One sweep loads the same tile of psi and lambda, applies a run of daggered gates to both, and
// accumulates the inner products of the run's parameterised gates on the way.  Items:
//   kind 0 dense / 1 diagonal / 2 monomial: applied to both tiles;
//   kind 3 marker: grad[slot] += w * Im <lambda|G|psi> over the tile, G a Pauli string that flips
//          bits (xm on tile-local bits, zm on global bits, phase ph);
//   kind 6 a 1-target dense gate whose marker (generator X or Y on the same bit) comes right before
//          it: one pass over the pairs takes the inner product and applies the gate;
//   kind 7 a diagonal phase: every diagonal gate and every diagonal-generator marker that the order
//          of the run lets stand at this point.  Diagonal unitaries leave conj(lambda_i) psi_i as it
//          is, so all these markers are sign sums of one vector v_i = Im conj(lambda_i) psi_i, formed
//          once; the gates are folded on the host (FP64) into tables over up to 8 bits.
// The markers of a phase: the 3 tile bits above the thread index are transformed in registers
// (Walsh-Hadamard, 3 stages), the 8 x 512 partial sums go to shared memory, and each marker is then
// one warp's signed sum of 512 of them, instead of a pass over both tiles with a block reduction
// each (an ansatz layer has two diagonal parameters for every rotation).
// What bounds it: FP32/INT issue.  512 threads: the complex128 tiles (128 KiB) allow one CTA per SM,
// which at 256 threads left 8 warps to hide every latency.
struct AdjGate {
    TileGate g;          // kinds 0 and 6: npar = matrix class (0 complex, 1 real, 2 real diagonal and imaginary off-diagonal)
    uint32_t xm_local;   // kind 7: first table
    int32_t ph;          // kind 6: 0 generator X, 1 generator Y; kind 7: number of markers
    uint64_t zm;
    int32_t slot;        // kind 7: first marker
    int32_t n_tabs;      // kind 7: number of tables
    double weight;
};
struct AdjTab {          // a folded diagonal: index bit q is tile bit pos[q], or global bit gbit[q] when pos[q] < 0
    int32_t k, mat_off;
    int8_t pos[8], gbit[8];
};
struct AdjMark {         // grad[slot] += weight * sum_i (-1)^popc(i & z) v_i; z split into tile and outer bits
    uint64_t z_out;
    uint32_t z_tile;
    int32_t slot;
    double weight;
};

constexpr int kSweepThreads = 512, kSweepLog = 9, kSweepPer = 4096 >> kSweepLog;   // values per thread of a 2^12 tile
constexpr int kRotMax = 32;      // kind 6 / kind 3 sums kept per CTA before they are added to the result
constexpr int kTabsPerPass = 4;

// The two storages: complex128 tiles hold float-float values (float4: re hi, re lo, im hi, im lo) and
// gates run in float-float; complex64 tiles hold float2 and gates run in FP32.  Inner products are
// float-float sums of exact products in both.
template <bool C64> struct Tile;
template <> struct Tile<false> {
    using S = float4;
    using A = cff;
    using G = double2;
    static __device__ __forceinline__ A ld(const S& v) { return f4c(v); }
    static __device__ __forceinline__ S st(const A& v) { return c4f(v); }
    static __device__ __forceinline__ S from(const G& v) { return c4f(load_c128(v)); }
    static __device__ __forceinline__ G to(const S& v) { return store_c128(f4c(v)); }
    static __device__ __forceinline__ A mul(const float4& m, const A& x) { return cmul(f4c(m), x); }
    static __device__ __forceinline__ A ipow(const A& x, int p) { return cmul_ipow(x, p); }
    // a x + b y; CLS 1: a, b real; 2: a real, b imaginary (the dropped products are zeros)
    template <int CLS>
    static __device__ __forceinline__ A lin2(const float4& a, const A& x, const float4& b, const A& y) {
        ffacc r, i;
        if (CLS == 0) {
            cmac_first(r, i, f4c(a), x);
            cmac(r, i, f4c(b), y);
        } else {
            acc_first(r, a.x, a.y, x.rh, x.rl);
            acc_first(i, a.x, a.y, x.ih, x.il);
            if (CLS == 1) {
                acc_add(r, b.x, b.y, y.rh, y.rl);
                acc_add(i, b.x, b.y, y.ih, y.il);
            } else {
                acc_add(r, -b.z, -b.w, y.ih, y.il);
                acc_add(i, b.z, b.w, y.rh, y.rl);
            }
        }
        return cdone(r, i);
    }
    static __device__ __forceinline__ ff im_conj(const A& l, const A& x) {
        ffacc m;
        acc_first(m, l.rh, l.rl, x.ih, x.il);
        acc_add(m, -l.ih, -l.il, x.rh, x.rl);
        return acc_done(m);
    }
    static __device__ __forceinline__ ff re_conj(const A& l, const A& x) {
        ffacc m;
        acc_first(m, l.rh, l.rl, x.rh, x.rl);
        acc_add(m, l.ih, l.il, x.ih, x.il);
        return acc_done(m);
    }
};
template <> struct Tile<true> {
    using S = float2;
    using A = float2;
    using G = float2;
    static __device__ __forceinline__ A ld(const S& v) { return v; }
    static __device__ __forceinline__ S st(const A& v) { return v; }
    static __device__ __forceinline__ S from(const G& v) { return v; }
    static __device__ __forceinline__ G to(const S& v) { return v; }
    static __device__ __forceinline__ A mul(const float4& m, const A& x) {
        return make_float2(__fmaf_rn(m.x, x.x, -m.z * x.y), __fmaf_rn(m.x, x.y, m.z * x.x));
    }
    static __device__ __forceinline__ A ipow(const A& x, int p) {
        switch (p & 3) {
            case 0: return x;
            case 1: return make_float2(-x.y, x.x);
            case 2: return make_float2(-x.x, -x.y);
            default: return make_float2(x.y, -x.x);
        }
    }
    template <int CLS>
    static __device__ __forceinline__ A lin2(const float4& a, const A& x, const float4& b, const A& y) {
        if (CLS == 0) {
            const float2 u = make_float2(__fmaf_rn(a.x, x.x, -a.z * x.y), __fmaf_rn(a.x, x.y, a.z * x.x));
            return make_float2(__fmaf_rn(b.x, y.x, __fmaf_rn(-b.z, y.y, u.x)), __fmaf_rn(b.x, y.y, __fmaf_rn(b.z, y.x, u.y)));
        }
        if (CLS == 1) return make_float2(__fmaf_rn(b.x, y.x, a.x * x.x), __fmaf_rn(b.x, y.y, a.x * x.y));
        return make_float2(__fmaf_rn(-b.z, y.y, a.x * x.x), __fmaf_rn(b.z, y.x, a.x * x.y));
    }
    static __device__ __forceinline__ ff im_conj(const A& l, const A& x) {
        ffacc m;
        acc_first(m, l.x, 0.f, x.y, 0.f);
        acc_add(m, -l.y, 0.f, x.x, 0.f);
        return acc_done(m);
    }
    static __device__ __forceinline__ ff re_conj(const A& l, const A& x) {
        ffacc m;
        acc_first(m, l.x, 0.f, x.x, 0.f);
        acc_add(m, l.y, 0.f, x.y, 0.f);
        return acc_done(m);
    }
};

__device__ __forceinline__ int insert_zero(int x, int bit) { return ((x >> bit) << (bit + 1)) | (x & ((1 << bit) - 1)); }

// float-float sum over a warp, by shuffles (an FP64 shuffle sum would cost 16 cycles of the SM's FP64
// pipe per step and warp)
__device__ __forceinline__ void warp_fsum(ffsum& a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float h = __shfl_xor_sync(0xffffffffu, a.h, o), l = __shfl_xor_sync(0xffffffffu, a.l, o);
        fsum_add(a, h, l);
    }
}

// A 1-target dense gate on both tiles.  ROT: 0 no marker, 1 generator X, 2 generator Y on the same bit;
// the return value is then this thread's part of Im <lambda|G|psi> (before the gate).
template <bool C64, int CLS, int ROT>
__device__ __forceinline__ ffsum adj_1q(typename Tile<C64>::S* sa, typename Tile<C64>::S* sb, int T, const TileGate& g,
                                        const float4* __restrict__ mats) {
    using P = Tile<C64>;
    const int t = g.tbit[0], b = 1 << t, ngroups = 1 << (T - 1);
    const float4* m = mats + g.mat_off;
    const float4 m00 = __ldg(m), m01 = __ldg(m + 1), m10 = __ldg(m + 2), m11 = __ldg(m + 3);
    const int lcm = (int)g.lc_mask, lcv = (int)g.lc_val;
    ffsum acc{0.f, 0.f};
    for (int gr = threadIdx.x; gr < ngroups; gr += kSweepThreads) {
        const int j0 = insert_zero(gr, t), j1 = j0 | b;
        if (ROT == 0 && (j0 & lcm) != lcv) continue;
        const auto x0 = P::ld(sa[j0]), x1 = P::ld(sa[j1]), y0 = P::ld(sb[j0]), y1 = P::ld(sb[j1]);
        if (ROT == 1) {          // X: Im (conj(l0) x1 + conj(l1) x0)
            const ff u = P::im_conj(y0, x1), v = P::im_conj(y1, x0);
            fsum_add(acc, u.h, u.l);
            fsum_add(acc, v.h, v.l);
        } else if (ROT == 2) {   // Y: Im (-i conj(l0) x1 + i conj(l1) x0)
            const ff u = P::re_conj(y0, x1), v = P::re_conj(y1, x0);
            fsum_add(acc, -u.h, -u.l);
            fsum_add(acc, v.h, v.l);
        }
        sa[j0] = P::st(P::template lin2<CLS>(m00, x0, m01, x1));
        sa[j1] = CLS == 2 ? P::st(P::template lin2<CLS>(m11, x1, m10, x0)) : P::st(P::template lin2<CLS>(m10, x0, m11, x1));
        sb[j0] = P::st(P::template lin2<CLS>(m00, y0, m01, y1));
        sb[j1] = CLS == 2 ? P::st(P::template lin2<CLS>(m11, y1, m10, y0)) : P::st(P::template lin2<CLS>(m10, y0, m11, y1));
    }
    return acc;
}
template <bool C64, int ROT>
__device__ __forceinline__ ffsum adj_1q_cls(typename Tile<C64>::S* sa, typename Tile<C64>::S* sb, int T, const TileGate& g,
                                            const float4* __restrict__ mats) {
    if (g.npar == 1) return adj_1q<C64, 1, ROT>(sa, sb, T, g, mats);
    if (g.npar == 2) return adj_1q<C64, 2, ROT>(sa, sb, T, g, mats);
    return adj_1q<C64, 0, ROT>(sa, sb, T, g, mats);
}

// 2- to 4-target dense gates, one tile at a time
template <int K>
__device__ void adj_dense(float4* sm, int T, const TileGate& g, const float4* __restrict__ mats) {
    constexpr int D = 1 << K;
    int pos[K];
    for (int q = 0; q < K; q++) pos[q] = g.tbit[q];
    for (int a = 0; a < K; a++)
        for (int b = a + 1; b < K; b++)
            if (pos[b] < pos[a]) { int t = pos[a]; pos[a] = pos[b]; pos[b] = t; }
    const float4* m = mats + g.mat_off;
    for (int gr = threadIdx.x; gr < (1 << (T - K)); gr += blockDim.x) {
        int jb = gr;
        for (int q = 0; q < K; q++) jb = insert_zero(jb, pos[q]);
        if ((jb & (int)g.lc_mask) != (int)g.lc_val) continue;
        cff x[D];
        int idx[D];
#pragma unroll
        for (int c = 0; c < D; c++) {
            int j = jb;
            for (int q = 0; q < K; q++) if ((c >> q) & 1) j |= 1 << g.tbit[q];
            idx[c] = j;
            x[c] = f4c(sm[j]);
        }
#pragma unroll
        for (int r = 0; r < D; r++) {
            ffacc ar, ai;
            cmac_first(ar, ai, f4c(__ldg(m + r * D)), x[0]);
#pragma unroll
            for (int c = 1; c < D; c++) cmac(ar, ai, f4c(__ldg(m + r * D + c)), x[c]);
            sm[idx[r]] = c4f(cdone(ar, ai));
        }
    }
}
template <int K>
__device__ void adj_dense(float2* sm, int T, const TileGate& g, const float4* __restrict__ mats) {
    constexpr int D = 1 << K;
    int pos[K];
    for (int q = 0; q < K; q++) pos[q] = g.tbit[q];
    for (int a = 0; a < K; a++)
        for (int b = a + 1; b < K; b++)
            if (pos[b] < pos[a]) { int t = pos[a]; pos[a] = pos[b]; pos[b] = t; }
    const float4* m = mats + g.mat_off;
    for (int gr = threadIdx.x; gr < (1 << (T - K)); gr += blockDim.x) {
        int jb = gr;
        for (int q = 0; q < K; q++) jb = insert_zero(jb, pos[q]);
        if ((jb & (int)g.lc_mask) != (int)g.lc_val) continue;
        float2 x[D];
        int idx[D];
#pragma unroll
        for (int c = 0; c < D; c++) {
            int j = jb;
            for (int q = 0; q < K; q++) if ((c >> q) & 1) j |= 1 << g.tbit[q];
            idx[c] = j;
            x[c] = sm[j];
        }
#pragma unroll
        for (int r = 0; r < D; r++) {
            float2 u = make_float2(0.f, 0.f);
#pragma unroll
            for (int c = 0; c < D; c++) {
                const float4 mc = __ldg(m + r * D + c);
                u.x = __fmaf_rn(mc.x, x[c].x, __fmaf_rn(-mc.z, x[c].y, u.x));
                u.y = __fmaf_rn(mc.x, x[c].y, __fmaf_rn(mc.z, x[c].x, u.y));
            }
            sm[idx[r]] = u;
        }
    }
}
template <bool C64>
__device__ void adj_monomial(typename Tile<C64>::S* sm, int T, const TileGate& g, const int32_t* __restrict__ perms) {
    using P = Tile<C64>;
    const int D = 1 << g.k;
    int pos[BS_TILE_MAXK];
    for (int q = 0; q < g.k; q++) pos[q] = g.tbit[q];
    for (int a = 0; a < g.k; a++)
        for (int b = a + 1; b < g.k; b++)
            if (pos[b] < pos[a]) { int t = pos[a]; pos[a] = pos[b]; pos[b] = t; }
    const int32_t* p = perms + g.perm_off;
    for (int gr = threadIdx.x; gr < (1 << (T - g.k)); gr += blockDim.x) {
        int jb = gr;
        for (int q = 0; q < g.k; q++) jb = insert_zero(jb, pos[q]);
        if ((jb & (int)g.lc_mask) != (int)g.lc_val) continue;
        typename P::S x[16];
        int idx[16];
        for (int c = 0; c < D; c++) {
            int j = jb;
            for (int q = 0; q < g.k; q++) if ((c >> q) & 1) j |= 1 << g.tbit[q];
            idx[c] = j;
            x[c] = sm[j];
        }
        for (int c = 0; c < D; c++) sm[idx[__ldg(p + 2 * c)]] = P::st(P::ipow(P::ld(x[c]), __ldg(p + 2 * c + 1)));
    }
}

// index part of a folded diagonal's table from tile position j (bits outside the tile left out)
__device__ __forceinline__ int tab_index(const AdjTab& t, int j) {
    int di = 0;
#pragma unroll
    for (int q = 0; q < 8; q++)
        if (q < t.k && t.pos[q] >= 0) di |= ((j >> t.pos[q]) & 1) << q;
    return di;
}
__device__ __forceinline__ int tab_const(const AdjTab& t, int64_t base) {
    int di = 0;
#pragma unroll
    for (int q = 0; q < 8; q++)
        if (q < t.k && t.pos[q] < 0) di |= (int)((base >> t.gbit[q]) & 1) << q;
    return di;
}

template <bool C64>
__global__ void __launch_bounds__(kSweepThreads, C64 ? 2 : 1)
    k_adjoint_sweep(typename Elem<C64>::T* __restrict__ psi, typename Elem<C64>::T* __restrict__ lam, SweepDesc d,
                    const AdjGate* __restrict__ ag, const AdjTab* __restrict__ tabs, const AdjMark* __restrict__ marks,
                    double* __restrict__ grad_acc, int64_t tile0) {
    using P = Tile<C64>;
    using S = typename P::S;
    extern __shared__ float4 smem[];
    const int T = d.T, L = d.L, H = T - L;
    const int nt = 1 << T;
    S* sp = reinterpret_cast<S*>(smem);
    S* sl = sp + nt;
    float2* vt = reinterpret_cast<float2*>(sl + nt);                        // kSweepPer x kSweepThreads
    int64_t* off_tab = reinterpret_cast<int64_t*>(vt + kSweepPer * kSweepThreads);
    __shared__ double red[kRotMax][kSweepThreads / 32];
    __shared__ double red_w[kRotMax];
    __shared__ int red_slot[kRotMax];
    const int64_t base = bs_tile_base(d, tile0 + (int64_t)blockIdx.x);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < (1 << H); i += kSweepThreads) {
        int64_t o = 0;
        for (int j = 0; j < H; j++) if ((i >> j) & 1) o |= 1LL << d.hi_bits[j];
        off_tab[i] = o;
    }
    __syncthreads();
    const int lowmask = (1 << L) - 1;
    // tile loads: four positions (eight loads) per thread in flight at a time (tiles <= 2^12)
#pragma unroll
    for (int r = 0; r < kSweepPer; r += 4) {
        typename Elem<C64>::T xp[4], xl[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int j = (r + i) * kSweepThreads + tid;
            if (j < nt) {
                const int64_t gidx = base | off_tab[j >> L] | (int64_t)(j & lowmask);
                xp[i] = psi[gidx];
                xl[i] = lam[gidx];
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int j = (r + i) * kSweepThreads + tid;
            if (j < nt) {
                sp[j] = P::from(xp[i]);
                sl[j] = P::from(xl[i]);
            }
        }
    }
    __syncthreads();
    int nred = 0;   // inner products waiting in red
    // add the waiting inner products to the result (all threads; the caller's barrier is before it)
    auto flush_red = [&]() {
        if (tid < nred) {
            double s = 0.0;
            for (int w = 0; w < kSweepThreads / 32; w++) s += red[tid][w];
            atomicAdd(grad_acc + red_slot[tid], s * red_w[tid]);
        }
        __syncthreads();
        nred = 0;
    };
    auto keep_red = [&](ffsum acc, int slot, double w) {
        warp_fsum(acc);
        if (lane == 0) red[nred][warp] = ff2d(acc.h, acc.l);
        if (tid == 0) { red_slot[nred] = slot; red_w[nred] = w; }
        nred++;
    };
    for (int gi = 0; gi < d.n_gates; gi++) {
        const AdjGate& a = ag[gi];   // fields read where used (a copy of the whole descriptor went to local memory)
        const int kind = a.g.kind;
        if (kind == 7) {
            const int nm = a.ph, ntab = a.n_tabs;
            const AdjTab* tb = tabs + a.xm_local;
            // The gates first, in a rolled loop (one unrolled loop over values and tables overflowed the
            // instruction cache), then v: the gates do not change it.
            for (int t0 = 0; t0 < ntab; t0 += kTabsPerPass) {
                const int nk = min(kTabsPerPass, ntab - t0);
                const float4* tm[kTabsPerPass];
#pragma unroll
                for (int u = 0; u < kTabsPerPass; u++)
                    if (u < nk) tm[u] = d.mats + tb[t0 + u].mat_off + (tab_index(tb[t0 + u], tid) | tab_const(tb[t0 + u], base));
#pragma unroll 1
                for (int j = tid; j < nt; j += kSweepThreads) {
                    auto x = P::ld(sp[j]), l = P::ld(sl[j]);
#pragma unroll
                    for (int u = 0; u < kTabsPerPass; u++)
                        if (u < nk) {
                            const float4 m = __ldg(tm[u] + tab_index(tb[t0 + u], j - tid));
                            x = P::mul(m, x);
                            l = P::mul(m, l);
                        }
                    sp[j] = P::st(x);
                    sl[j] = P::st(l);
                }
            }
            if (nm) {
                ffsum v[kSweepPer];
#pragma unroll
                for (int i = 0; i < kSweepPer; i++) {
                    const int j = i * kSweepThreads + tid;
                    v[i] = {0.f, 0.f};
                    if (j < nt) {
                        const ff f = P::im_conj(P::ld(sl[j]), P::ld(sp[j]));
                        v[i] = {f.h, f.l};
                    }
                }
                // Walsh-Hadamard over the tile bits above the thread index
#pragma unroll
                for (int o = 1; o < kSweepPer; o <<= 1)
#pragma unroll
                    for (int i = 0; i < kSweepPer; i++)
                        if (!(i & o)) {
                            ffsum s = v[i], t = v[i];
                            fsum_add(s, v[i | o].h, v[i | o].l);
                            fsum_add(t, -v[i | o].h, -v[i | o].l);
                            v[i] = s;
                            v[i | o] = t;
                        }
#pragma unroll
                for (int i = 0; i < kSweepPer; i++) vt[i * kSweepThreads + tid] = make_float2(v[i].h, v[i].l);
                __syncthreads();
                for (int m = warp; m < nm; m += kSweepThreads / 32) {
                    const AdjMark& k = marks[a.slot + m];
                    const uint32_t z = k.z_tile;
                    const float2* row = vt + (z >> kSweepLog) * kSweepThreads;
                    const uint32_t neg0 = (uint32_t)__popcll((unsigned long long)base & k.z_out) + (uint32_t)__popc((uint32_t)lane & z);
                    ffsum s{0.f, 0.f};
#pragma unroll
                    for (int u = 0; u < kSweepThreads / 32; u++) {
                        const float2 w = row[32 * u + lane];
                        const uint32_t sg = (neg0 + (uint32_t)__popc((uint32_t)(32 * u) & z)) << 31;
                        fsum_add(s, __uint_as_float(__float_as_uint(w.x) ^ sg), __uint_as_float(__float_as_uint(w.y) ^ sg));
                    }
                    warp_fsum(s);
                    if (lane == 0) atomicAdd(grad_acc + k.slot, ff2d(s.h, s.l) * k.weight);
                }
            }
            __syncthreads();
            continue;
        }
        if (kind == 3) {
            // Im <lambda| G |psi> over the tile, G flipping bits
            ffsum acc{0.f, 0.f};
            for (int j = tid; j < nt; j += kSweepThreads) {
                const int64_t gidx = base | off_tab[j >> L] | (int64_t)(j & lowmask);
                const int ph = a.ph + ((__popcll((unsigned long long)gidx & a.zm) & 1) ? 2 : 0);
                const ff v = P::im_conj(P::ld(sl[j]), P::ipow(P::ld(sp[j ^ (int)a.xm_local]), (4 - (ph & 3)) & 3));
                fsum_add(acc, v.h, v.l);
            }
            keep_red(acc, a.slot, a.weight);
            __syncthreads();
            if (nred == kRotMax) flush_red();
            continue;
        }
        if (kind == 6) {
            const ffsum acc = a.ph ? adj_1q_cls<C64, 2>(sp, sl, T, a.g, d.mats) : adj_1q_cls<C64, 1>(sp, sl, T, a.g, d.mats);
            keep_red(acc, a.slot, a.weight);
            __syncthreads();
            if (nred == kRotMax) flush_red();
            continue;
        }
        if ((base & (int64_t)a.g.gc_mask) != (int64_t)a.g.gc_val) continue;
        if (kind == 1) {
            const float4* m = d.mats + a.g.mat_off;
            for (int j = tid; j < nt; j += kSweepThreads) {
                if ((j & (int)a.g.lc_mask) != (int)a.g.lc_val) continue;
                const int64_t gidx = base | off_tab[j >> L] | (int64_t)(j & lowmask);
                int di = 0;
                for (int q = 0; q < a.g.k; q++) di |= (int)((gidx >> a.g.gbit[q]) & 1) << q;
                const float4 dv = __ldg(m + di);
                sp[j] = P::st(P::mul(dv, P::ld(sp[j])));
                sl[j] = P::st(P::mul(dv, P::ld(sl[j])));
            }
        } else if (kind == 0) {
            switch (a.g.k) {
                case 1: adj_1q_cls<C64, 0>(sp, sl, T, a.g, d.mats); break;
                case 2: adj_dense<2>(sp, T, a.g, d.mats); adj_dense<2>(sl, T, a.g, d.mats); break;
                case 3: adj_dense<3>(sp, T, a.g, d.mats); adj_dense<3>(sl, T, a.g, d.mats); break;
                default: adj_dense<4>(sp, T, a.g, d.mats); adj_dense<4>(sl, T, a.g, d.mats); break;
            }
        } else {
            adj_monomial<C64>(sp, T, a.g, d.perms);
            adj_monomial<C64>(sl, T, a.g, d.perms);
        }
        __syncthreads();
    }
    if (nred) flush_red();
    for (int j = tid; j < nt; j += kSweepThreads) {
        const int64_t gidx = base | off_tab[j >> L] | (int64_t)(j & lowmask);
        psi[gidx] = P::to(sp[j]);
        lam[gidx] = P::to(sl[j]);
    }
}

inline float4 to_cff(double re, double im) {
    float4 v;
    v.x = (float)re; v.y = (float)(re - (double)v.x);
    v.z = (float)im; v.w = (float)(im - (double)v.z);
    return v;
}

struct BwdItem {          // one element of the reversed gate list
    HostGate g;
    bool marker = false;
    int slot = 0;
    int projector = 0;
    uint64_t xm = 0, zm = 0;   // endian masks of the generator
    int ph = 0;
    double weight = 1.0;
    bool unitary_diag = false;    // kind 1 with entries of modulus 1

    uint64_t touch() const {
        uint64_t m = g.cmask | zm | xm;
        for (int q = 0; q < g.k; q++) m |= 1ULL << g.ebit[q];
        return m;
    }
    // leaves conj(lambda_i) psi_i alone and reads nothing else: commutes with its like on any bits
    bool diag() const { return marker ? xm == 0 : unitary_diag; }
};

// Diagonal gates of one phase folded into tables over at most 8 bits each (they commute).
constexpr int kTabBits = 8;
struct FoldTab {
    std::vector<int> eb;                      // endian bits, table index bit q <-> eb[q]
    std::vector<std::complex<double>> d;
};
uint64_t tab_bits(const FoldTab& t) {
    uint64_t m = 0;
    for (int e : t.eb) m |= 1ULL << e;
    return m;
}
// t <- t * h, over the union of their bits
void fold_diag(FoldTab& t, const HostGate& h) {
    uint64_t nb = tab_bits(t) | h.cmask;
    for (int q = 0; q < h.k; q++) nb |= 1ULL << h.ebit[q];
    std::vector<int> eb;
    for (int e = 0; e < 64; e++) if ((nb >> e) & 1ULL) eb.push_back(e);
    std::vector<std::complex<double>> d((size_t)1 << eb.size());
    for (size_t x = 0; x < d.size(); x++) {
        uint64_t g = 0;
        for (size_t q = 0; q < eb.size(); q++) if ((x >> q) & 1) g |= 1ULL << eb[q];
        std::complex<double> v(1.0, 0.0);
        if (!t.d.empty()) {
            size_t xi = 0;
            for (size_t q = 0; q < t.eb.size(); q++) xi |= (size_t)((g >> t.eb[q]) & 1ULL) << q;
            v = t.d[xi];
        }
        if ((g & h.cmask) == h.cval) {
            int hi = 0;
            for (int q = 0; q < h.k; q++) hi |= (int)((g >> h.ebit[q]) & 1ULL) << q;
            v *= std::complex<double>(h.mat[2 * hi], h.mat[2 * hi + 1]);
        }
        d[x] = v;
    }
    t.eb = eb;
    t.d = d;
}
// Fold a run of diagonal gates (each on at most kTabBits bits): each joins the table it widens least.
void fold_diags(const std::vector<const HostGate*>& gates, std::vector<FoldTab>& tabs) {
    for (const HostGate* h : gates) {
        uint64_t hb = h->cmask;
        for (int q = 0; q < h->k; q++) hb |= 1ULL << h->ebit[q];
        int best = -1, added = 0;
        for (size_t t = 0; t < tabs.size(); t++) {
            const uint64_t tb = tab_bits(tabs[t]);
            const int add = __builtin_popcountll(hb & ~tb);
            if (__builtin_popcountll(tb | hb) <= kTabBits && (best < 0 || add < added)) { best = (int)t; added = add; }
        }
        if (best < 0) {
            best = (int)tabs.size();
            tabs.emplace_back();
        }
        fold_diag(tabs[(size_t)best], *h);
    }
}
bool unit_modulus(const HostGate& h) {
    for (int i = 0; i < (1 << h.k); i++) {
        const double m = h.mat[2 * i] * h.mat[2 * i] + h.mat[2 * i + 1] * h.mat[2 * i + 1];
        if (std::fabs(m - 1.0) > 4e-15) return false;
    }
    return true;
}
// U^dagger of a lowered gate (same targets and controls)
HostGate dagger(const HostGate& h) {
    HostGate d = h;
    const int D = 1 << h.k;
    if (h.kind == 1) {
        for (int i = 0; i < D; i++) d.mat[2 * i + 1] = -h.mat[2 * i + 1];
    } else if (h.kind == 0) {
        for (int r = 0; r < D; r++)
            for (int c = 0; c < D; c++) {
                d.mat[2 * (r * D + c)] = h.mat[2 * (c * D + r)];
                d.mat[2 * (r * D + c) + 1] = -h.mat[2 * (c * D + r) + 1];
            }
    } else {
        // column c -> row r with phase p  ==>  column r -> row c with phase -p
        for (int c = 0; c < D; c++) {
            int r = h.perm[2 * c], p = h.perm[2 * c + 1];
            d.perm[2 * r] = c;
            d.perm[2 * r + 1] = (4 - p) & 3;
        }
    }
    return d;
}

}  // namespace

extern "C" int bs_adjoint_gradient(bs_sim* s, const bs_op* ops, int64_t n_ops, const int32_t* param_index,
                                   const int32_t* gen_kind, const uint64_t* gen_xmask, const uint64_t* gen_zmask,
                                   int n_params, int n_terms, const uint64_t* xmask, const uint64_t* zmask,
                                   const double* coeffs, double* energy_out, double* grad_out) {
    if (!s) return BS_ERR_INVALID_ARG;
    if (s->kind != BS_KIND_SV) return bs_fail(s, BS_ERR_UNSUPPORTED, "adjoint gradients need a state-vector simulator");
    const bool c64 = s->precision == BS_PREC_C64;
    const size_t esz = c64 ? 8 : 16;
    if (n_ops < 0 || (n_ops && (!ops || !param_index || !gen_kind || !gen_xmask || !gen_zmask)) || n_params < 0 ||
        n_terms < 1 || !xmask || !zmask || !coeffs || !energy_out || (n_params && !grad_out))
        return bs_fail(s, BS_ERR_INVALID_ARG, "bad adjoint arguments");
    const int n = s->n;
    const int64_t len = s->len;
    auto to_endian = [n](uint64_t m) {
        uint64_t e = 0;
        for (int q = 0; q < n; q++) if ((m >> q) & 1ULL) e |= 1ULL << (n - 1 - q);
        return e;
    };
    // 0. segments and checkpoint buffers
    int n_param_gates = 0;
    for (int64_t i = 0; i < n_ops; i++) n_param_gates += (ops[i].kind == 0 && param_index[i] >= 0) ? 1 : 0;
    int S = s->tune.adj_segments;
    const size_t state_bytes = (size_t)len * esz;
    if (S < 0) {
        size_t fr = 0, tot = 0;
        cudaMemGetInfo(&fr, &tot);
        fr += bs_kept_bytes();   // freed where they are in the way
        const int by_mem = (int)std::min<size_t>(64, fr / 4 / std::max<size_t>(state_bytes, 1));
        S = std::min(std::min(16, 1 + n_param_gates / 16), by_mem + 1);
    }
    S = std::max(1, std::min<int>(S, (int)std::max<int64_t>(1, n_ops)));
    // One allocation for the checkpoints and lambda.  Up to kKeepBytes it stays with the handle for the next
    // gradient (15 allocations and frees a call were 1.2 ms, a fifth of a 20-qubit gradient); larger ones
    // are given back at the end of the call.
    const size_t slot = (state_bytes + 255) & ~(size_t)255;
    size_t work_bytes = 0;
    char* work = nullptr;
    for (;;) {
        const size_t need = slot * (size_t)S;   // S - 1 checkpoints, lambda
        work = (char*)bs_keep_take(s, need, &work_bytes);
        if (work) break;
        work_bytes = need;
        if (bs_malloc((void**)&work, need) == cudaSuccess) break;
        if (S == 1) return bs_fail(s, BS_ERR_ALLOC, "lambda allocation: out of memory");
        S = std::max(1, S / 2);   // memory binds: fewer checkpoints, more uncomputation
    }
    auto free_ckpt = [&]() {
        if (work_bytes <= kKeepBytes) bs_keep(s, work, work_bytes);
        else cudaFree(work);   // synchronises with the stream's work
    };
    // segment j covers ops [seg[j], seg[j+1]), split evenly by gate count
    std::vector<int64_t> seg(1, 0);
    {
        int64_t n_gates = 0;
        for (int64_t i = 0; i < n_ops; i++) n_gates += ops[i].kind == 0;
        int64_t cnt = 0;
        for (int64_t i = 0; i < n_ops && (int)seg.size() < S; i++) {
            cnt += ops[i].kind == 0;
            if (cnt * S >= n_gates * (int64_t)seg.size() && i + 1 < n_ops) seg.push_back(i + 1);
        }
        seg.push_back(n_ops);
        S = (int)seg.size() - 1;
    }
    // 1. forward pass, keeping psi after every segment but the last
    bs_stats fwd{};
    int rc = BS_OK;
    // segments are queued back to back: the host plans segment j+1 while the GPU runs segment j
    cudaEventRecord(s->ev0, s->stream);
    s->tc_events_used = 0;
    s->defer_sync = true;
    for (int j = 0; j < S && !rc; j++) {
        rc = bs_evolve(s, ops + seg[(size_t)j], seg[(size_t)j + 1] - seg[(size_t)j], 0);
        if (rc) break;
        fwd.sweeps += s->stats.sweeps;
        fwd.kernel_launches += s->stats.kernel_launches;
        fwd.gates += s->stats.gates;
        fwd.bytes_moved += s->stats.bytes_moved;
        fwd.tc_gates += s->stats.tc_gates;
        fwd.tc_launches += s->stats.tc_launches;
        if (j + 1 < S) rc = bs_cuda_check(s, cudaMemcpyAsync(work + slot * (size_t)(j + 1), s->state, state_bytes, cudaMemcpyDeviceToDevice, s->stream), "checkpoint");
    }
    s->defer_sync = false;
    if (rc) { cudaStreamSynchronize(s->stream); free_ckpt(); return rc; }
    s->stats = fwd;
    // 2. lambda = H psi
    void* lam = work;
    auto ckpt = [&](int j) { return (void*)(work + slot * (size_t)(j + 1)); };
    std::vector<PauliTerm> terms((size_t)n_terms);
    for (int t = 0; t < n_terms; t++) {
        uint64_t x = xmask[t], z = zmask[t];
        int ny = __builtin_popcountll(x & z);
        terms[(size_t)t].xm = to_endian(x);
        terms[(size_t)t].zm = to_endian(z);
        terms[(size_t)t].ph = ny & 3;
        terms[(size_t)t].ch = (float)coeffs[t];
        terms[(size_t)t].cl = (float)(coeffs[t] - (double)terms[(size_t)t].ch);
    }
    rc = bs_ensure_scratch(s, (int64_t)n_terms * (int64_t)sizeof(PauliTerm) + (int64_t)(n_params + 2) * 8 + 256);
    if (rc) { free_ckpt(); return rc; }
    PauliTerm* d_terms = (PauliTerm*)s->scratch;
    double* d_acc = (double*)((char*)s->scratch + (((int64_t)n_terms * (int64_t)sizeof(PauliTerm) + 255) & ~255LL));
    cudaMemcpyAsync(d_terms, terms.data(), terms.size() * sizeof(PauliTerm), cudaMemcpyHostToDevice, s->stream);
    cudaMemsetAsync(d_acc, 0, (size_t)(n_params + 2) * 8, s->stream);
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((len + kAThreads - 1) / kAThreads, 152 * 8));
    if (c64) {
        k_pauli_sum<true><<<blocks, kAThreads, 0, s->stream>>>((const float2*)s->state, (float2*)lam, len, d_terms, n_terms);
        k_inner<true><<<blocks, kAThreads, 0, s->stream>>>((const float2*)s->state, (const float2*)lam, len, d_acc + n_params);
    } else {
        k_pauli_sum<false><<<blocks, kAThreads, 0, s->stream>>>((const double2*)s->state, (double2*)lam, len, d_terms,
                                                                 n_terms);
        k_inner<false><<<blocks, kAThreads, 0, s->stream>>>((const double2*)s->state, (const double2*)lam, len,
                                                             d_acc + n_params);
    }
    // 3. backward: reversed, daggered gate list with gradient markers before each parameterised gate
    std::vector<BwdItem> items;
    std::vector<size_t> seg_item(1, 0);   // items of segment S-1-r start at seg_item[r]
    int cur_seg = S - 1;
    for (int64_t i = n_ops - 1; i >= 0; i--) {
        while (cur_seg > 0 && i < seg[(size_t)cur_seg]) {
            cur_seg--;
            seg_item.push_back(items.size());
        }
        const bs_op& op = ops[i];
        if (op.kind != 0) continue;
        std::vector<HostGate> hg;
        rc = bs_lower_gate(s, op.matrix, op.n_targets, op.targets, op.n_controls, op.controls, op.control_values,
                           op.flags, false, hg);
        if (rc) { free_ckpt(); return rc; }
        if (param_index[i] >= 0) {
            if (param_index[i] >= n_params) { free_ckpt(); return bs_fail(s, BS_ERR_INVALID_ARG, "parameter index out of range"); }
            BwdItem m;
            m.marker = true;
            m.slot = param_index[i];
            m.projector = gen_kind[i] == 1;
            if (m.projector) {
                // PhaseShift on its target: weight -2, projector on the target's endian bit
                m.g.k = 1;
                m.g.ebit[0] = n - 1 - op.targets[0];
                m.weight = -2.0;
            } else {
                m.xm = to_endian(gen_xmask[i]);
                m.zm = to_endian(gen_zmask[i]);
                m.ph = __builtin_popcountll(gen_xmask[i] & gen_zmask[i]) & 3;
                m.g.k = 0;
                for (int q = 0; q < n; q++)
                    if ((m.xm >> q) & 1ULL) m.g.ebit[m.g.k++] = q;
                m.weight = 1.0;
            }
            m.g.kind = 3;
            items.push_back(m);
        }
        for (const HostGate& h : hg) {
            BwdItem it;
            it.g = dagger(h);
            it.unitary_diag = it.g.kind == 1 && unit_modulus(it.g);
            items.push_back(it);
        }
    }
    while ((int)seg_item.size() < S) seg_item.push_back(items.size());
    seg_item.push_back(items.size());
    // plan sweeps segment by segment: markers need their flip bits in the tile, and they must not
    // move past a gate sharing bits (they read the current psi and lambda); diagonal gates and
    // diagonal-generator markers move past one another freely
    const int n_bits = n;
    const int T = std::min(BS_TILE_MAX_BITS, n_bits);
    // Four low bits leave 8 to choose in a tile of 2^12, for rows of 256 bytes (128 in complex64); with five there
    // were more sweeps: 21 qubits, 4 layers 5.55 -> 5.20 ms (three: 5.22), complex64 3.53 -> 3.42 (3.39)
    const int L = std::min(4, T);
    const int cap = T - L;
    std::vector<std::vector<int>> sweeps_items;
    std::vector<std::vector<int>> sweeps_hi;
    std::vector<int> sweep_restore;   // checkpoint to restore psi from before the sweep, -1 if none
    for (int r = 0; r < S; r++) {
        const size_t G = seg_item[(size_t)r + 1];
        std::vector<char> done(G, 0);
        size_t remaining = G - seg_item[(size_t)r], first = seg_item[(size_t)r];
        bool seg_first = true;
        auto need = [&](const BwdItem& it) -> uint64_t {
            uint64_t m = 0;
            if (!it.marker && it.g.kind == 1) return m;
            if (it.marker) return it.xm & ~(((uint64_t)1 << L) - 1);
            for (int q = 0; q < it.g.k; q++) if (it.g.ebit[q] >= L) m |= 1ULL << it.g.ebit[q];
            return m;
        };
        while (remaining) {
            std::vector<int> idx;
            uint64_t chosen = 0, blocked = 0, blocked_diag = 0;   // bits of items left behind: any, diagonal
            int nch = 0;
            for (size_t i = first; i < G; i++) {
                if (done[i]) continue;
                uint64_t t = items[i].touch();
                const bool dg = items[i].diag();
                if (t & (dg ? blocked : blocked | blocked_diag)) { (dg ? blocked_diag : blocked) |= t; continue; }
                uint64_t nb = need(items[i]) & ~chosen;
                int add = __builtin_popcountll(nb);
                bool too_big = !items[i].marker && items[i].g.kind != 1 &&
                               (items[i].g.k > BS_TILE_MAXK || __builtin_popcountll(need(items[i])) > cap);
                if (too_big || (items[i].marker && __builtin_popcountll(need(items[i])) > cap)) {
                    free_ckpt();
                    return bs_fail(s, BS_ERR_UNSUPPORTED, "adjoint gate too wide for a tile");
                }
                if (nch + add <= cap) {
                    chosen |= nb;
                    nch += add;
                    idx.push_back((int)i);
                    done[i] = 1;
                    remaining--;
                } else {
                    blocked |= t;
                }
            }
            while (first < G && done[first]) first++;
            std::vector<int> hi;
            for (int b = L; b < n_bits; b++) if ((chosen >> b) & 1ULL) hi.push_back(b);
            for (int b = L; b < n_bits && (int)hi.size() < cap; b++) if (!((chosen >> b) & 1ULL)) hi.push_back(b);
            std::sort(hi.begin(), hi.end());
            sweeps_items.push_back(idx);
            sweeps_hi.push_back(hi);
            // entering segment S-1-r (r > 0): psi is its end state, kept by the forward pass
            sweep_restore.push_back(seg_first && r > 0 ? S - 1 - r : -1);
            seg_first = false;
        }
    }
    // pack device data.  The items of a sweep are taken in alternating phases that keep the order of
    // items which share a bit and do not both stand on the diagonal: all diagonal items that nothing
    // holds back (one kind 7), then all others that nothing holds back.
    std::vector<AdjGate> ag;
    std::vector<AdjTab> tabs;
    std::vector<AdjMark> marks;
    std::vector<float4> mats;
    std::vector<int32_t> perms;
    std::vector<int64_t> sweep_first;
    for (size_t sw = 0; sw < sweeps_items.size(); sw++) {
        int local[64];
        for (int b = 0; b < 64; b++) local[b] = -1;
        for (int b = 0; b < L; b++) local[b] = b;
        for (size_t i = 0; i < sweeps_hi[sw].size(); i++) local[sweeps_hi[sw][i]] = L + (int)i;
        sweep_first.push_back((int64_t)ag.size());
        auto emit_gate = [&](const HostGate& hg) {
            AdjGate a{};
            a.g.kind = hg.kind;
            a.g.k = hg.k;
            uint64_t gcm = 0, gcv = 0;
            uint32_t lcm = 0, lcv = 0;
            for (int b = 0; b < n_bits; b++) {
                if (!((hg.cmask >> b) & 1ULL)) continue;
                uint64_t v = (hg.cval >> b) & 1ULL;
                if (local[b] >= 0) { lcm |= 1u << local[b]; lcv |= (uint32_t)v << local[b]; }
                else { gcm |= 1ULL << b; gcv |= v << b; }
            }
            a.g.lc_mask = lcm; a.g.lc_val = lcv; a.g.gc_mask = gcm; a.g.gc_val = gcv;
            for (int q = 0; q < hg.k; q++) {
                a.g.gbit[q] = hg.ebit[q];
                if (q < BS_TILE_MAXK) a.g.tbit[q] = local[hg.ebit[q]];
            }
            a.g.mat_off = (int32_t)mats.size();
            a.g.perm_off = (int32_t)perms.size();
            if (hg.kind == 0) for (int e = 0; e < (1 << (2 * hg.k)); e++) mats.push_back(to_cff(hg.mat[2 * e], hg.mat[2 * e + 1]));
            else if (hg.kind == 1) for (int e = 0; e < (1 << hg.k); e++) mats.push_back(to_cff(hg.mat[2 * e], hg.mat[2 * e + 1]));
            else perms.insert(perms.end(), hg.perm.begin(), hg.perm.end());
            if (hg.kind == 0 && hg.k == 1) a.g.npar = bs_class_2x2(hg);
            ag.push_back(a);
        };
        auto add_mark = [&](uint64_t zm, int slot, double w) {
            AdjMark m{};
            for (int b = 0; b < n_bits; b++) {
                if (!((zm >> b) & 1ULL)) continue;
                if (local[b] >= 0) m.z_tile |= 1u << local[b];
                else m.z_out |= 1ULL << b;
            }
            m.slot = slot;
            m.weight = w;
            marks.push_back(m);
        };
        std::vector<int> left = sweeps_items[sw], rest;
        while (!left.empty()) {
            // diagonal phase: nothing but an earlier non-diagonal item on the same bits holds one back
            std::vector<const HostGate*> folds;
            AdjGate ph{};
            ph.g.kind = 7;
            ph.slot = (int32_t)marks.size();
            uint64_t held = 0;
            rest.clear();
            std::vector<const HostGate*> wide;
            for (int ii : left) {
                const BwdItem& it = items[(size_t)ii];
                const uint64_t t = it.touch();
                if (!it.diag()) { held |= t; rest.push_back(ii); continue; }
                if (t & held) { rest.push_back(ii); continue; }
                if (!it.marker) {
                    (__builtin_popcountll(t) <= kTabBits ? folds : wide).push_back(&it.g);
                } else if (it.projector) {
                    // P1 = (1 - Z) / 2
                    add_mark(0, it.slot, 0.5 * it.weight);
                    add_mark(1ULL << it.g.ebit[0], it.slot, -0.5 * it.weight);
                } else {
                    add_mark(it.zm, it.slot, it.weight);   // the phase (-i)^0: no Y in a generator that flips nothing
                }
            }
            left.swap(rest);
            ph.ph = (int32_t)marks.size() - ph.slot;
            std::vector<FoldTab> ft;
            fold_diags(folds, ft);
            ph.xm_local = (uint32_t)tabs.size();
            ph.n_tabs = (int32_t)ft.size();
            for (const FoldTab& f : ft) {
                AdjTab t{};
                t.k = (int32_t)f.eb.size();
                t.mat_off = (int32_t)mats.size();
                for (size_t q = 0; q < f.eb.size(); q++) {
                    t.gbit[q] = (int8_t)f.eb[q];
                    t.pos[q] = (int8_t)local[f.eb[q]];
                }
                for (const std::complex<double>& v : f.d) mats.push_back(to_cff(v.real(), v.imag()));
                tabs.push_back(t);
            }
            if (ph.ph || ph.n_tabs) ag.push_back(ph);
            for (const HostGate* h : wide) emit_gate(*h);
            // the others: anything earlier on the same bits holds one back
            held = 0;
            rest.clear();
            for (size_t i = 0; i < left.size(); i++) {
                const BwdItem& it = items[(size_t)left[i]];
                const uint64_t t = it.touch();
                if (it.diag() || (t & held)) { held |= t; rest.push_back(left[i]); continue; }
                if (!it.marker) { emit_gate(it.g); continue; }
                // a marker whose gate comes next, one dense target and a generator X or Y on it: one pass
                if (i + 1 < left.size() && left[i + 1] == left[i] + 1) {
                    const BwdItem& nx = items[(size_t)left[i + 1]];
                    if (!nx.marker && nx.g.kind == 0 && nx.g.k == 1 && nx.g.cmask == 0 && it.xm == (1ULL << nx.g.ebit[0]) &&
                        (it.zm == 0 || it.zm == it.xm)) {
                        emit_gate(nx.g);
                        AdjGate& a = ag.back();
                        a.g.kind = 6;
                        a.ph = it.zm ? 1 : 0;
                        a.slot = it.slot;
                        a.weight = it.weight;
                        i++;
                        continue;
                    }
                }
                AdjGate a{};
                a.g.kind = 3;
                a.slot = it.slot;
                a.weight = it.weight;
                a.zm = it.zm;
                a.ph = it.ph;
                for (int b = 0; b < n_bits; b++) if ((it.xm >> b) & 1ULL) a.xm_local |= 1u << local[b];
                ag.push_back(a);
            }
            left.swap(rest);
        }
    }
    sweep_first.push_back((int64_t)ag.size());
    auto al = [](int64_t x) { return (x + 255) & ~(int64_t)255; };
    const int64_t b_ag = al((int64_t)ag.size() * (int64_t)sizeof(AdjGate));
    const int64_t b_m = al((int64_t)mats.size() * (int64_t)sizeof(float4));
    const int64_t b_p = al((int64_t)(perms.size() + 1) * 4);
    const int64_t b_t = al((int64_t)(tabs.size() + 1) * (int64_t)sizeof(AdjTab));
    const int64_t b_k = al((int64_t)(marks.size() + 1) * (int64_t)sizeof(AdjMark));
    rc = bs_ensure_plan(s, b_ag + b_m + b_p + b_t + b_k);
    if (rc) { free_ckpt(); return rc; }
    std::vector<char> host((size_t)(b_ag + b_m + b_p + b_t + b_k), 0);
    if (!ag.empty()) std::memcpy(host.data(), ag.data(), ag.size() * sizeof(AdjGate));
    if (!mats.empty()) std::memcpy(host.data() + b_ag, mats.data(), mats.size() * sizeof(float4));
    if (!perms.empty()) std::memcpy(host.data() + b_ag + b_m, perms.data(), perms.size() * 4);
    if (!tabs.empty()) std::memcpy(host.data() + b_ag + b_m + b_p, tabs.data(), tabs.size() * sizeof(AdjTab));
    if (!marks.empty()) std::memcpy(host.data() + b_ag + b_m + b_p + b_t, marks.data(), marks.size() * sizeof(AdjMark));
    cudaMemcpyAsync(s->plan_buf, host.data(), host.size(), cudaMemcpyHostToDevice, s->stream);
    const AdjGate* d_ag = (const AdjGate*)s->plan_buf;
    const float4* d_m = (const float4*)((char*)s->plan_buf + b_ag);
    const int32_t* d_p = (const int32_t*)((char*)s->plan_buf + b_ag + b_m);
    const AdjTab* d_t = (const AdjTab*)((char*)s->plan_buf + b_ag + b_m + b_p);
    const AdjMark* d_k = (const AdjMark*)((char*)s->plan_buf + b_ag + b_m + b_p + b_t);
    const int H = T - L;
    const size_t extra = (size_t)kSweepPer * kSweepThreads * sizeof(float2) + ((size_t)1 << H) * sizeof(int64_t);
    const size_t smem = (size_t)2 * ((size_t)1 << T) * sizeof(float4) + extra;
    const size_t smem64 = (size_t)2 * ((size_t)1 << T) * sizeof(float2) + extra;
    cudaFuncSetAttribute(k_adjoint_sweep<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(k_adjoint_sweep<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    const int64_t ntiles = (int64_t)1 << (n_bits - T);
    for (size_t sw = 0; sw < sweeps_items.size(); sw++) {
        if (sweep_restore[sw] >= 0)
            cudaMemcpyAsync(s->state, ckpt(sweep_restore[sw]), state_bytes, cudaMemcpyDeviceToDevice, s->stream);
        SweepDesc d{};
        bs_tile_geometry(d, n_bits, L, sweeps_hi[sw]);
        d.n_gates = (int)(sweep_first[sw + 1] - sweep_first[sw]);
        d.mats = d_m;
        d.perms = d_p;
        for (int64_t t0 = 0; t0 < ntiles; t0 += (1LL << 30)) {
            int64_t nb = std::min<int64_t>(ntiles - t0, 1LL << 30);
            if (c64)
                k_adjoint_sweep<true><<<(unsigned)nb, kSweepThreads, smem64, s->stream>>>((float2*)s->state, (float2*)lam, d,
                                                                                          d_ag + sweep_first[sw], d_t, d_k, d_acc, t0);
            else
                k_adjoint_sweep<false><<<(unsigned)nb, kSweepThreads, smem, s->stream>>>((double2*)s->state, (double2*)lam, d,
                                                                                         d_ag + sweep_first[sw], d_t, d_k, d_acc, t0);
        }
        s->stats.kernel_launches++;
        s->stats.sweeps++;
        s->stats.bytes_moved += 4.0 * (double)esz * (double)len;
    }
    std::vector<double> res((size_t)n_params + 2);
    cudaMemcpyAsync(res.data(), d_acc, res.size() * 8, cudaMemcpyDeviceToHost, s->stream);
    cudaEventRecord(s->ev1, s->stream);
    rc = bs_cuda_check(s, cudaStreamSynchronize(s->stream), "adjoint");
    free_ckpt();
    if (rc) return rc;
    float ms = 0;
    cudaEventElapsedTime(&ms, s->ev0, s->ev1);
    s->stats.gpu_ms = ms;   // forward and backward
    bs_collect_tc_time(s);
    rc = bs_check_device_flag(s);
    if (rc) return rc;
    *energy_out = res[(size_t)n_params];
    for (int p = 0; p < n_params; p++) grad_out[p] = res[(size_t)p];
    return BS_OK;
}
