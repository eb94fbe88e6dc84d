// Tile sweeps: one CTA owns 2^T amplitudes of the state (the L lowest endian bits
// plus T-L chosen higher bits, all other bits fixed by the CTA index), converts
// them once to float-float in shared memory, applies every gate of the sweep
// whose targets lie inside the tile, and writes them back.  A sweep therefore
// reads and writes the state once however many gates it carries.
//
// Reference kernels replaced (src/gate_kernels.jl): 1q :489-537, 2q :540-576,
// controlled :579-670, generic k-target :753-775, custom diagonal/excitation
// kernels src/custom_gates.jl:364-416; the density-matrix gate of
// src/dm_simulator.jl:130-140 is two tile gates (column bits U, row bits conj U).
#include <algorithm>
#include <atomic>
#include <cooperative_groups.h>
#include <cmath>
#include <complex>
#include <cstring>
#include "bs_internal.h"
#include "bs_ff.cuh"
#include "bs_tc.cuh"
#include "bs_cdf.cuh"

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ int insert0(int x, int bit) {
    int low = x & ((1 << bit) - 1);
    return ((x >> bit) << (bit + 1)) | low;
}
// shared-memory index of tile element j: swizzled (tensor-core sweep) or plain
template <bool SW>
__device__ __forceinline__ int sx(int j) { return SW ? tc::sw(j) : j; }
// Tile amplitudes in shared memory are float4 (re hi, im hi, re lo, im lo): the two high words and
// the two low words each form an aligned register pair for the packed f32x2 arithmetic of the
// tensor-core sweep.  Matrix entries in global memory are float4 (re hi, re lo, im hi, im lo).
// Gate descriptors of a sweep are staged in shared memory in chunks (one coalesced copy per chunk
// instead of dependent global loads of every field by every thread at every gate).
constexpr int kGateChunk = 32;
__device__ __forceinline__ void stage_words(void* dst, const void* __restrict__ src, int words) {
    const int* s = reinterpret_cast<const int*>(src);
    int* t = reinterpret_cast<int*>(dst);
    for (int w = threadIdx.x; w < words; w += blockDim.x) t[w] = __ldg(s + w);
}
__device__ __forceinline__ void stage_gates(TileGate* dst, const TileGate* __restrict__ src, int ng) {
    __syncthreads();   // the previous chunk is no longer read
    stage_words(dst, src, ng * (int)(sizeof(TileGate) / 4));
    __syncthreads();
}

__device__ __forceinline__ cff f4c(float4 v) { return {v.x, v.z, v.y, v.w}; }
__device__ __forceinline__ float4 c4f(const cff& c) { return make_float4(c.rh, c.ih, c.rl, c.il); }
__device__ __forceinline__ cff f4m(float4 v) { return {v.x, v.y, v.z, v.w}; }
// read-only operand load: through the non-coherent cache from global memory, or plainly from shared
// memory (operands staged there)
template <bool S, typename V>
__device__ __forceinline__ V ldro(const V* p) {
    if constexpr (S) return *p;
    else return __ldg(p);
}

// 2x2 gate on tile bit t, the matrix in registers.  CLS (TileGate.npar): 0 complex, 1 all real (Ry, H),
// 2 real diagonal and imaginary off-diagonal (Rx): the products with the entries' zero parts, which are
// half of the float-float work (86 -> 38 instructions an amplitude), are left out; the sums do not
// change by them.
template <int CLS, bool SW, bool SM>
__device__ __forceinline__ void tile_1q(float4* sm, int ngroups, int t, uint32_t lcm, uint32_t lcv, const float4* m) {
    const cff m00 = f4m(ldro<SM>(m)), m01 = f4m(ldro<SM>(m + 1)), m10 = f4m(ldro<SM>(m + 2)), m11 = f4m(ldro<SM>(m + 3));
    const int b0 = 1 << t;
#pragma unroll 2
    for (int gr = threadIdx.x; gr < ngroups; gr += blockDim.x) {
        const int jb = insert0(gr, t);
        if ((jb & (int)lcm) != (int)lcv) continue;
        const int ia = sx<SW>(jb), ib = sx<SW>(jb | b0);
        const cff a = f4c(sm[ia]), b = f4c(sm[ib]);
        ffacc ar, ai, br, bi;
        if (CLS == 0) {
            cmac_first(ar, ai, m00, a);
            cmac(ar, ai, m01, b);
            cmac_first(br, bi, m10, a);
            cmac(br, bi, m11, b);
        } else if (CLS == 1) {
            acc_first(ar, m00.rh, m00.rl, a.rh, a.rl);
            acc_first(ai, m00.rh, m00.rl, a.ih, a.il);
            acc_add(ar, m01.rh, m01.rl, b.rh, b.rl);
            acc_add(ai, m01.rh, m01.rl, b.ih, b.il);
            acc_first(br, m10.rh, m10.rl, a.rh, a.rl);
            acc_first(bi, m10.rh, m10.rl, a.ih, a.il);
            acc_add(br, m11.rh, m11.rl, b.rh, b.rl);
            acc_add(bi, m11.rh, m11.rl, b.ih, b.il);
        } else {
            acc_first(ar, m00.rh, m00.rl, a.rh, a.rl);
            acc_first(ai, m00.rh, m00.rl, a.ih, a.il);
            acc_add(ar, -m01.ih, -m01.il, b.ih, b.il);
            acc_add(ai, m01.ih, m01.il, b.rh, b.rl);
            acc_first(br, -m10.ih, -m10.il, a.ih, a.il);
            acc_first(bi, m10.ih, m10.il, a.rh, a.rl);
            acc_add(br, m11.rh, m11.rl, b.rh, b.rl);
            acc_add(bi, m11.rh, m11.rl, b.ih, b.il);
        }
        sm[ia] = c4f(cdone(ar, ai));
        sm[ib] = c4f(cdone(br, bi));
    }
}

template <int K, bool SW = false, bool SM = false>
__device__ void tile_dense(float4* sm, int T, const TileGate& g, const float4* __restrict__ mats) {
    constexpr int D = 1 << K;
    int pos[K];
#pragma unroll
    for (int q = 0; q < K; q++) pos[q] = g.tbit[q];
    // ascending order for padding
#pragma unroll
    for (int a = 0; a < K; a++)
#pragma unroll
        for (int b = a + 1; b < K; b++)
            if (pos[b] < pos[a]) { int t = pos[a]; pos[a] = pos[b]; pos[b] = t; }
    const int ngroups = 1 << (T - K);
    const float4* m = mats + g.mat_off;
    const uint32_t lcm = g.lc_mask, lcv = g.lc_val;
    int tb[K];
#pragma unroll
    for (int q = 0; q < K; q++) tb[q] = g.tbit[q];
    if (K == 1) {
        if (g.npar == 1) tile_1q<1, SW, SM>(sm, ngroups, pos[0], lcm, lcv, m);
        else if (g.npar == 2) tile_1q<2, SW, SM>(sm, ngroups, pos[0], lcm, lcv, m);
        else tile_1q<0, SW, SM>(sm, ngroups, pos[0], lcm, lcv, m);
        return;
    }
    for (int gr = threadIdx.x; gr < ngroups; gr += blockDim.x) {
        int jb = gr;
#pragma unroll
        for (int q = 0; q < K; q++) jb = insert0(jb, pos[q]);
        if ((jb & (int)lcm) != (int)lcv) continue;
        cff x[D];
        int idx[D];
#pragma unroll
        for (int c = 0; c < D; c++) {
            int j = jb;
#pragma unroll
            for (int q = 0; q < K; q++) if ((c >> q) & 1) j |= 1 << tb[q];
            idx[c] = sx<SW>(j);
            x[c] = f4c(sm[idx[c]]);
        }
#pragma unroll
        for (int r = 0; r < D; r++) {
            ffacc ar, ai;
            cmac_first(ar, ai, f4m(ldro<SM>(m + r * D)), x[0]);
#pragma unroll
            for (int c = 1; c < D; c++) cmac(ar, ai, f4m(ldro<SM>(m + r * D + c)), x[c]);
            sm[idx[r]] = c4f(cdone(ar, ai));
        }
    }
}

// X on tile bit t under NC in-tile controls (CNOT, CCNOT; TileGate.npar 1 of kind 2): the pairs that meet
// the controls are enumerated directly and change places.  The general monomial pass walks all pairs,
// skips half of its lanes at a control and looks up rows and phases (1400 SM cycles a pass of a full
// tile against 600).
template <int NC, bool SW>
__device__ __forceinline__ void tile_cx(float4* sm, int T, const TileGate& g) {
    int pos[NC + 1];
    uint32_t m = g.lc_mask;
    pos[0] = g.tbit[0];
#pragma unroll
    for (int q = 1; q <= NC; q++) {
        pos[q] = __ffs((int)m) - 1;
        m &= m - 1;
    }
#pragma unroll
    for (int a = 0; a <= NC; a++)
#pragma unroll
        for (int b = a + 1; b <= NC; b++)
            if (pos[b] < pos[a]) { int t = pos[a]; pos[a] = pos[b]; pos[b] = t; }
    const int bt = 1 << g.tbit[0], on = (int)g.lc_val, n = 1 << (T - 1 - NC);
#pragma unroll 4
    for (int gr = threadIdx.x; gr < n; gr += blockDim.x) {
        int j = gr;
#pragma unroll
        for (int q = 0; q <= NC; q++) j = insert0(j, pos[q]);
        const int ia = sx<SW>(j | on), ib = sx<SW>(j | on | bt);
        const float4 a = sm[ia], b = sm[ib];
        sm[ia] = b;
        sm[ib] = a;
    }
}

// monomial gate: column c goes to row perm[2c] with phase i^perm[2c+1]
template <int K, bool SW = false, bool SM = false>
__device__ void tile_monomial(float4* sm, int T, const TileGate& g, const int32_t* __restrict__ perms) {
    if (K == 1 && g.npar == 1) {   // uniform
        switch (__popc(g.lc_mask)) {
            case 0: tile_cx<0, SW>(sm, T, g); return;
            case 1: tile_cx<1, SW>(sm, T, g); return;
            case 2: tile_cx<2, SW>(sm, T, g); return;
            default: break;
        }
    }
    constexpr int D = 1 << K;
    int pos[K];
#pragma unroll
    for (int q = 0; q < K; q++) pos[q] = g.tbit[q];
#pragma unroll
    for (int a = 0; a < K; a++)
#pragma unroll
        for (int b = a + 1; b < K; b++)
            if (pos[b] < pos[a]) { int t = pos[a]; pos[a] = pos[b]; pos[b] = t; }
    const int ngroups = 1 << (T - K);
    const int32_t* p = perms + g.perm_off;
    for (int gr = threadIdx.x; gr < ngroups; gr += blockDim.x) {
        int jb = gr;
#pragma unroll
        for (int q = 0; q < K; q++) jb = insert0(jb, pos[q]);
        if ((jb & (int)g.lc_mask) != (int)g.lc_val) continue;
        float4 x[D];
        int idx[D];
#pragma unroll
        for (int c = 0; c < D; c++) {
            int j = jb;
#pragma unroll
            for (int q = 0; q < K; q++) if ((c >> q) & 1) j |= 1 << g.tbit[q];
            idx[c] = sx<SW>(j);
            x[c] = sm[idx[c]];
        }
#pragma unroll
        for (int c = 0; c < D; c++) {
            const int r = ldro<SM>(p + 2 * c), ph = ldro<SM>(p + 2 * c + 1);
            int j = jb;
#pragma unroll
            for (int q = 0; q < K; q++) if ((r >> q) & 1) j |= 1 << g.tbit[q];
            sm[sx<SW>(j)] = c4f(cmul_ipow(f4c(x[c]), ph));
        }
    }
}

// phase of a merged run of CZ gates at global index gi: odd parity -> -1
__device__ __forceinline__ bool parity_odd(const TileGate& g, int64_t gi) {
    int par = 0;
    for (int q = 0; q < g.npar; q++)
        par ^= __popcll((unsigned long long)(gi & (gi >> g.pshift[q])) & g.pmask[q]);
    return par & 1;
}

// off_tab[h] << osh: global offset of the tile's high-bit pattern h
template <typename OT, bool SW = false, bool SM = false>
__device__ void tile_diag(float4* sm, int T, int L, const TileGate& g, const float4* __restrict__ mats,
                          int64_t base, OT off_tab, int osh) {
    const int nt = 1 << T, lowmask = (1 << L) - 1;
    const float4* m = mats + g.mat_off;
    // pattern bit q: tile bit tbit[q] (32-bit), or a CTA constant for a bit outside the tile;
    // gates with more than BS_TILE_MAXK bits take the pattern from the 64-bit global index.  The number of
    // threads is a power of two.
    auto apply = [&](int js, int di) {
        const float4 d = ldro<SM>(m + di);
        if (d.y == 0.f && d.w == 0.f) {
            if (d.z == 0.f && d.x == 1.f) return;
            if (d.z == 0.f && d.x == -1.f) { sm[js] = c4f(cmul_ipow(f4c(sm[js]), 2)); return; }
            if (d.x == 0.f && d.z == 1.f) { sm[js] = c4f(cmul_ipow(f4c(sm[js]), 1)); return; }
            if (d.x == 0.f && d.z == -1.f) { sm[js] = c4f(cmul_ipow(f4c(sm[js]), 3)); return; }
        }
        sm[js] = c4f(cmul(f4m(d), f4c(sm[js])));
    };
    const uint32_t lcm = g.lc_mask, lcv = g.lc_val;
    if (g.k <= BS_TILE_MAXK) {
        int cst = 0;
        uint32_t enc = 0;   // per in-tile pattern bit: tile position (5 bits) | q << 5, one byte each
        int nk = 0;
        for (int q = 0; q < g.k; q++) {
            if (g.tbit[q] >= 0) enc |= (uint32_t)(g.tbit[q] | (q << 5)) << (8 * nk++);
            else cst |= (int)((base >> g.gbit[q]) & 1) << q;
        }
        auto pattern = [&](int j) {
            int di = 0;
            for (int u = 0; u < nk; u++) {
                const uint32_t b = (enc >> (8 * u)) & 255u;
                di |= ((j >> (b & 31u)) & 1) << (b >> 5);
            }
            return di;
        };
        // the pattern of a thread's positions: its own bits once, the bits above them (uniform) each time
        const int mine = cst | pattern((int)threadIdx.x);
        for (int j0 = 0; j0 < nt; j0 += blockDim.x) {
            const int j = j0 | (int)threadIdx.x;
            if (j >= nt || (j & (int)lcm) != (int)lcv) continue;
            apply(sx<SW>(j), mine | pattern(j0));
        }
    } else {
        for (int j = threadIdx.x; j < nt; j += blockDim.x) {
            if ((j & (int)lcm) != (int)lcv) continue;
            const int64_t gi = base | ((int64_t)off_tab[j >> L] << osh) | (int64_t)(j & lowmask);
            int di = 0;
            for (int q = 0; q < g.k; q++) di |= (int)((gi >> g.gbit[q]) & 1) << q;
            apply(sx<SW>(j), di);
        }
    }
}

// Kraus channel on K <= 2 targets in the reference's update rule (src/noise_kernels.jl:105-168): the
// stored matrix S gets B <- sum_q K_q B K_q^dagger on every D x D block B whose row and column agree on
// all non-target bits (vec(S) index = row + column 2^n); other elements are left alone.  tbit[0..K-1]:
// tile positions of the row target bits (matrix bit j <-> tbit[j]), tbit[K..2K-1]: of the column
// target bits; pmask[0]: row-index mask of the non-target bits; pmask[1]: the non-target bits whose
// row and column bits both lie outside the tile (so that part of the test is uniform in the CTA).
// The channel comes as its superoperator on the block, a D^2 x D^2 matrix at mat_off (row and column
// index r + D c), formed on the host in FP64: one product per pair of elements.  With the Kraus
// matrices themselves a 2-target depolarizing channel was a chain of 16 x 4 x 5 complex products per
// element, 60 k cycles in the few tiles that hold such blocks (13 qubits, 3 layers: 31.8 -> 27.4 ms).
// Candidate blocks are tested and the ones that pass the row/column test collected (all candidates
// tested in one pass), then one thread per output element of a collected block; all reads of the
// collected blocks finish before any of their outputs is written.  s_act: 32 ints of shared scratch.
template <int K, bool SW, typename OT>
__device__ void tile_kraus_ref_lr(float4* sm, int T, int L, const TileGate& g, const float4* __restrict__ mats,
                                  int64_t base, OT off_tab, int osh, int n, int* s_act, int* s_cnt) {
    constexpr int D = 1 << K, DD = D * D, kChunkG = 32;   // capacity of s_act: at most this many blocks pass
    const int64_t rmask = ((int64_t)1 << n) - 1;
    if ((((base & rmask) ^ (base >> n)) & (int64_t)g.pmask[1]) != 0) return;   // uniform in the CTA
    int pos[2 * K];
#pragma unroll
    for (int q = 0; q < 2 * K; q++) pos[q] = g.tbit[q];
#pragma unroll
    for (int a = 0; a < 2 * K; a++)
#pragma unroll
        for (int b = a + 1; b < 2 * K; b++)
            if (pos[b] < pos[a]) { int t = pos[a]; pos[a] = pos[b]; pos[b] = t; }
    const int lowmask = (1 << L) - 1, ngroups = 1 << (T - 2 * K);
    const float4* km = mats + g.mat_off;
    // Every candidate block is tested in one pass by all threads.  A block passes when, for every
    // non-target qubit, its row and column bits agree; each non-target tile bit belongs to a qubit
    // whose other bit is either in the tile (one constraint per pair) or constant in the CTA (one per
    // bit), so at most 2^((T - 2K) / 2) <= 32 blocks pass (T <= 12): s_act holds them all.
    if (threadIdx.x == 0) *s_cnt = 0;
    __syncthreads();
    for (int b = (int)threadIdx.x; b < ngroups; b += (int)blockDim.x) {
        int j0 = b;
#pragma unroll
        for (int q = 0; q < 2 * K; q++) j0 = insert0(j0, pos[q]);
        const int64_t gi = base | ((int64_t)off_tab[j0 >> L] << osh) | (int64_t)(j0 & lowmask);
        if (((((gi & rmask) ^ (gi >> n)) & (int64_t)g.pmask[0]) == 0)) {
            const int slot = atomicAdd(s_cnt, 1);
            if (slot < kChunkG) s_act[slot] = j0;
        }
    }
    __syncthreads();
    const int nact = min(*s_cnt, kChunkG);
    const int items = nact * DD;
    for (int it0 = 0; it0 < items; it0 += blockDim.x) {
        const int it = it0 + (int)threadIdx.x;
        float4 outv = make_float4(0.f, 0.f, 0.f, 0.f);
        int dst = -1;
        if (it < items) {
            const int j0 = s_act[it / DD], e = it % DD, i = e / D, jj = e % D;
            auto at = [&](int r, int c) {
                int j = j0;
#pragma unroll
                for (int q = 0; q < K; q++) {
                    if ((r >> q) & 1) j |= 1 << g.tbit[q];
                    if ((c >> q) & 1) j |= 1 << g.tbit[K + q];
                }
                return sx<SW>(j);
            };
            const float4* row = km + (i + D * jj) * DD;
            ffacc ar, ai;
            cmac_first(ar, ai, f4m(__ldg(row)), f4c(sm[at(0, 0)]));
#pragma unroll 3
            for (int f = 1; f < DD; f++) cmac(ar, ai, f4m(__ldg(row + f)), f4c(sm[at(f % D, f / D)]));
            outv = c4f(cdone(ar, ai));
            dst = at(i, jj);
        }
        __syncthreads();   // every read of the collected blocks is done
        if (dst >= 0) sm[dst] = outv;
        __syncthreads();
    }
}

// KMAX: widest dense/monomial gate of the sweep (2 or 4); narrow sweeps get a
// kernel with fewer live registers and therefore more resident warps.  At 256 threads three or (wide) two
// CTAs share an SM; without the bound the wide kernel took 186 registers and an SM to itself (one 4-target
// gate at 21 qubits 140 -> 222 us).
template <int KMAX, int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? (KMAX == 2 ? 3 : 2) : 1) k_tile_sweep(double2* __restrict__ psi, SweepDesc d, int64_t tile0) {
    extern __shared__ float4 smem[];
    const int T = d.T, L = d.L, H = T - L;
    const int nt = 1 << T;
    int64_t* off_tab = reinterpret_cast<int64_t*>(smem + nt);
    const int64_t base = bs_tile_base(d, tile0 + (int64_t)blockIdx.x);
    for (int i = threadIdx.x; i < (1 << H); i += blockDim.x) {
        int64_t o = 0;
        for (int j = 0; j < H; j++) if ((i >> j) & 1) o |= 1LL << d.hi_bits[j];
        off_tab[i] = o;
    }
    __syncthreads();
    const int lowmask = (1 << L) - 1;
    // tile load: all of a thread's loads in flight (tiles are at most 2^12 amplitudes)
    {
        double2 x[4096 / NT];
#pragma unroll
        for (int i = 0; i < 4096 / NT; i++) {
            const int j = i * NT + (int)threadIdx.x;
            if (j < nt) x[i] = __ldcs(psi + (base | off_tab[j >> L] | (int64_t)(j & lowmask)));
        }
#pragma unroll
        for (int i = 0; i < 4096 / NT; i++) {
            const int j = i * NT + (int)threadIdx.x;
            if (j < nt) smem[j] = c4f(load_c128(x[i]));
        }
    }
    __syncthreads();
    __shared__ TileGate s_gates[kGateChunk];
    __shared__ int s_act[32], s_cnt;   // kind 5: blocks passing the row/column test
    for (int g0 = 0; g0 < d.n_gates; g0 += kGateChunk) {
    const int ng = min(kGateChunk, d.n_gates - g0);
    stage_gates(s_gates, d.gates + g0, ng);
    for (int gl = 0; gl < ng; gl++) {
        const TileGate& g = s_gates[gl];
        if ((base & (int64_t)g.gc_mask) != (int64_t)g.gc_val) continue;   // uniform in the CTA
        const int kind = g.kind, k = g.k;
        if (kind == 3) {
            for (int j = threadIdx.x; j < nt; j += blockDim.x) {
                const int64_t gi = base | off_tab[j >> L] | (int64_t)(j & lowmask);
                if (parity_odd(g, gi)) { float4 v = smem[j]; smem[j] = make_float4(-v.x, -v.y, -v.z, -v.w); }
            }
        } else if (kind == 1) {
            tile_diag(smem, T, L, g, d.mats, base, off_tab, 0);
        } else if (kind == 5) {
            if (k == 1) tile_kraus_ref_lr<1, false>(smem, T, L, g, d.mats, base, off_tab, 0, d.n_bits / 2, s_act, &s_cnt);
            else tile_kraus_ref_lr<2, false>(smem, T, L, g, d.mats, base, off_tab, 0, d.n_bits / 2, s_act, &s_cnt);
        } else if (kind == 0) {
            if (k == 1) tile_dense<1>(smem, T, g, d.mats);
            else if (k == 2 || KMAX == 2) tile_dense<2>(smem, T, g, d.mats);
            else if (KMAX > 2 && k == 3) tile_dense<3>(smem, T, g, d.mats);
            else if (KMAX > 2) tile_dense<4>(smem, T, g, d.mats);
        } else {
            if (k == 1) tile_monomial<1>(smem, T, g, d.perms);
            else if (k == 2 || KMAX == 2) tile_monomial<2>(smem, T, g, d.perms);
            else if (KMAX > 2 && k == 3) tile_monomial<3>(smem, T, g, d.perms);
            else if (KMAX > 2) tile_monomial<4>(smem, T, g, d.perms);
        }
        __syncthreads();
    }
    }
    for (int j = threadIdx.x; j < nt; j += blockDim.x) {
        int64_t gidx = base | off_tab[j >> L] | (int64_t)(j & lowmask);
        __stcs(psi + gidx, store_c128(f4c(smem[j])));
    }
}

// Sweep with fused 5-bit unitaries on the tensor cores (gate kind 4), T = 12, L = 3 to 5.
// Dynamic shared memory: 48 KiB matrix digit slices | 64 KiB tile (static: split offset tables, the
// per-warp exponents, kind-5 scratch), so that two CTAs fit on an SM; each holds 256 of the SM's 512
// TMEM columns, so one CTA's MMAs overlap the other's CUDA-core work.  The tile is stored with the
// bank swizzle tc::sw.
#ifndef BS_TC_THREADS
#define BS_TC_THREADS 256
#endif
constexpr int kTcThreads = BS_TC_THREADS;   // 256 (128 registers) or 512 (64 registers, spills; measured slower)
constexpr int kTcSmem = 49152 + 65536;

// Global offset (>> L) of the tile's high-bit pattern i (12 - L bits) from two small tables:
// a[i & 15] | b[i >> 4].
struct HiOff {
    const uint32_t* a;
    const uint32_t* b;
    __device__ __forceinline__ uint32_t operator[](int i) const { return a[i & 15] | b[i >> 4]; }
};

// Persistent: two CTAs per SM take tiles in turn, so that barriers, offset tables and TMEM are set up once.
// Without any gate a sweep of 28 qubits takes 1.8 ms (2.4 with a CTA per tile; HBM allows 1.26), with the
// gates of the 12-qubit density matrix 7.3 ms instead of 7.7.  The next tile's loads issued before this
// one's stores (64 registers of them) were slower, 62 against 59 ms at 28 qubits.
template <int L>
__global__ void __launch_bounds__(kTcThreads, 2) k_tile_sweep_tc(double2* __restrict__ psi, SweepDesc d, int64_t tile0,
                                                                 int64_t tile_end) {
    // 128-byte alignment: each 128-byte core matrix of the matrix operand sits in one shared-memory line
    extern __shared__ __align__(128) unsigned char dsm[];
    uint16_t* sB = reinterpret_cast<uint16_t*>(dsm);
    float4* smem = reinterpret_cast<float4*>(dsm + 49152);
    __shared__ __align__(8) uint64_t bars[7];   // digit copy, MMAs into D0 / D1, D0 / D1 read, D1 free, D2
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    __shared__ uint32_t s_offa[16], s_offb[1 << (8 - L)];
    __shared__ uint32_t s_wmax[kTcThreads / 32];   // per-warp largest high-word exponent field
    __shared__ int s_act[32], s_cnt;                 // kind 5: blocks passing the row/column test
    __shared__ int s_tcq[16], s_ntc;                 // the tile's first 16 fused gates, in order
    __shared__ const uint16_t* s_nsrc;
    const HiOff off32{s_offa, s_offb};
    constexpr int T = 12, H = T - L, nt = 1 << T, lowmask = (1 << L) - 1, NL = nt / kTcThreads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        s_fail = 0;
        tc::mbar_init(tc::su32(&bars[0]));
        tc::mbar_init(tc::su32(&bars[1]));
        tc::mbar_init(tc::su32(&bars[2]));
        tc::mbar_init_n(tc::su32(&bars[3]), kTcThreads / 32);
        tc::mbar_init_n(tc::su32(&bars[4]), kTcThreads / 32);
        tc::mbar_init(tc::su32(&bars[5]));
        tc::mbar_init(tc::su32(&bars[6]));
    }
    if (threadIdx.x < 16 + (1 << (H - 4))) {
        const int i = threadIdx.x < 16 ? threadIdx.x : (threadIdx.x - 16) << 4;
        int64_t o = 0;
        for (int j = 0; j < H; j++) if ((i >> j) & 1) o |= 1LL << d.hi_bits[j];
        if (threadIdx.x < 16) s_offa[threadIdx.x] = (uint32_t)(o >> L);
        else s_offb[threadIdx.x - 16] = (uint32_t)(o >> L);
    }
    if (warp == 0) tc::tmem_alloc(tc::su32(&s_tmem));
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    tc::State st{s_tmem, tc::su32(&bars[0]), 0u, false};
    double2 x[NL];   // the next tile's amplitudes, coalesced 512 B rows, all loads issued together
    auto load = [&](int64_t b) {
#pragma unroll
        for (int i = 0; i < NL; i++) {
            const int j = i * kTcThreads + (int)threadIdx.x;
            x[i] = __ldcs(psi + (b | ((int64_t)off32[j >> L] << L) | (int64_t)(j & lowmask)));
        }
    };
    int64_t tile = tile0 + (int64_t)blockIdx.x;
    int64_t base = bs_tile_base(d, tile);
    load(base);
    for (;;) {
        if (warp == kTcThreads / 32 - 1) {
            // while the loads are in flight: the fused gates this tile runs (those whose controls its
            // base satisfies), and the copy of the first one's digit slices
            int cnt = 0, first = -1;
            for (int c0 = 0; c0 < d.n_gates; c0 += 32) {
                const int gi = c0 + lane;
                bool f = false;
                if (gi < d.n_gates) {
                    const TileGate& g = d.gates[gi];
                    f = g.kind == 4 && (base & (int64_t)g.gc_mask) == (int64_t)g.gc_val;
                }
                const unsigned bal = __ballot_sync(0xffffffffu, f);
                if (f) {
                    const int pos = cnt + __popc(bal & ((1u << lane) - 1u));
                    if (pos < 16) s_tcq[pos] = gi;
                }
                if (first < 0 && bal) first = c0 + __ffs((int)bal) - 1;
                cnt += __popc(bal);
            }
            if (lane == 0) {
                s_ntc = cnt < 16 ? cnt : 16;
                if (first >= 0) tc::copy_slices(tc::su32(sB), tc::slice_src(d.gates[first], d.tc_pool, base), tc::su32(&bars[0]));
            }
        }
        // float-float at the swizzled positions
        {
            uint32_t eb = 0;
#pragma unroll
            for (int i = 0; i < NL; i++) {
                const float4 v = c4f(load_c128(x[i]));
                smem[tc::sw(i * kTcThreads + (int)threadIdx.x)] = v;
                eb = max(eb, max(__float_as_uint(v.x) & 0x7F800000u, __float_as_uint(v.y) & 0x7F800000u));
            }
            eb = __reduce_max_sync(0xffffffffu, eb);
            if (lane == 0) s_wmax[warp] = eb;
        }
        __syncthreads();
        st.pref = s_ntc > 0;
        int q = 0;             // fused gates run so far
        bool emax_ok = true;   // s_wmax holds the tile's largest exponent (no magnitude-changing gate since)
        for (int gi = 0; gi < d.n_gates; gi++) {
            const TileGate& g = d.gates[gi];
            if ((base & (int64_t)g.gc_mask) != (int64_t)g.gc_val) continue;
            const int kind = g.kind, k = g.k;
            if (kind == 0 || kind == 1 || kind == 5) emax_ok = false;   // these may change magnitudes
            if (kind == 4) {
                if (s_fail) continue;
                const TileGate* gn = q + 1 < s_ntc ? d.gates + s_tcq[q + 1] : nullptr;
                tc::apply<kTcThreads>(smem, g, gn, d.tc_pool, reinterpret_cast<const uint16_t*>(d.perms + g.perm_off), sB,
                                      st, base, s_wmax, emax_ok, &s_nsrc, &s_fail,
                                      d.err);
                q++;
                emax_ok = true;
            } else if (kind == 3) {
                for (int j = threadIdx.x; j < nt; j += blockDim.x) {
                    const int64_t gg = base | ((int64_t)off32[j >> L] << L) | (int64_t)(j & lowmask);
                    if (parity_odd(g, gg)) {
                        const int js = tc::sw(j);
                        float4 v = smem[js];
                        smem[js] = make_float4(-v.x, -v.y, -v.z, -v.w);
                    }
                }
            } else if (kind == 1) {
                tile_diag<HiOff, true>(smem, T, L, g, d.mats, base, off32, L);
            } else if (kind == 5) {
                if (k == 1) tile_kraus_ref_lr<1, true, HiOff>(smem, T, L, g, d.mats, base, off32, L, d.n_bits / 2, s_act, &s_cnt);
                else tile_kraus_ref_lr<2, true, HiOff>(smem, T, L, g, d.mats, base, off32, L, d.n_bits / 2, s_act, &s_cnt);
            } else if (kind == 0) {   // the planner routes sweeps with unfused 3- or 4-target gates elsewhere
                if (k == 1) tile_dense<1, true>(smem, T, g, d.mats);
                else tile_dense<2, true>(smem, T, g, d.mats);
            } else {
                if (k == 1) tile_monomial<1, true>(smem, T, g, d.perms);
                else tile_monomial<2, true>(smem, T, g, d.perms);
            }
            __syncthreads();
        }
        const int64_t here = base;
        tile += gridDim.x;
        const bool more = tile < tile_end && !s_fail;   // uniform: s_fail is written before a barrier of the loop above
        // tile store: streaming stores, nothing waits for them
#pragma unroll 4
        for (int i = 0; i < NL; i++) {
            const int j = i * kTcThreads + (int)threadIdx.x;
            __stcs(psi + (here | ((int64_t)off32[j >> L] << L) | (int64_t)(j & lowmask)), store_c128(f4c(smem[tc::sw(j)])));
        }
        if (!more) break;
        base = bs_tile_base(d, tile);
        load(base);
        __syncthreads();   // every thread has read the tile (and s_ntc) before the next one is written
    }
    // a wait gave up: give the copies and MMAs in flight a bounded time to land before releasing TMEM
    if (threadIdx.x == 0 && s_fail) {
        tc::mbar_wait(st.bar, st.ph & 1u);
        tc::mbar_wait(st.bar + 8u, (st.ph >> 1) & 1u);
        tc::mbar_wait(st.bar + 16u, (st.ph >> 2) & 1u);
        tc::mbar_wait(st.bar + 48u, (st.ph >> 6) & 1u);
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(st.tmem);
}

// The matrices of the fused unitaries, complex 32x32 row-major FP64 per variant, as the product of their gates.
// A CTA forms 8 columns of one variant (columns are independent), a thread one entry of each product; the
// entries that are still zero (the product starts from the identity) are skipped.  largest: per fused unitary
// the bits of its largest |re| or |im|.  Bound by the FP64 units (2 products a clock per SM): 30 to 60 us a list.
// On the host, in up to 8 threads, the products and their copies kept the GPU waiting: 22 qubits, 30 layers of a
// gate mix 3.14 -> 1.89 ms, 25 qubits 17.8 -> 16.1, 28-qubit dense circuit 59.7 -> 56.8, 12-qubit density matrix with
// channels 8.5 -> 7.6.
__global__ void __launch_bounds__(256) k_tc_build(const TcBlock* __restrict__ blocks, const int32_t* __restrict__ var_block,
                                                  const TcPart* __restrict__ parts, const double2* __restrict__ pool,
                                                  const int32_t* __restrict__ perms, double2* __restrict__ mats,
                                                  unsigned long long* __restrict__ largest) {
    __shared__ double2 U[2][32][8];
    const int v = blockIdx.x >> 2, row = threadIdx.x >> 3, col = threadIdx.x & 7, gcol = (blockIdx.x & 3) * 8 + col;
    const int bi = var_block[v];
    const TcBlock b = blocks[bi];
    const int var = v - b.var0;
    double2 x = make_double2(row == gcol ? 1.0 : 0.0, 0.0);
    int cur = 0;
    U[0][row][col] = x;
    __syncthreads();
    for (int i = 0; i < b.n_parts; i++) {
        const TcPart p = parts[b.part0 + i];
        if ((var & p.umask) != p.uval) continue;   // uniform
        const int k = p.k;
        if (p.kind == 1) {
            int d = 0;
            for (int q = 0; q < k; q++) d |= (p.pos[q] < 8 ? (row >> p.pos[q]) & 1 : (var >> (p.pos[q] - 8)) & 1) << q;
            if ((row & p.cmask) == p.cval) {
                const double2 m = pool[p.off + d];
                x = make_double2(m.x * x.x - m.y * x.y, m.x * x.y + m.y * x.x);
            }
        } else {
            int t = 0, base = row;
            for (int q = 0; q < k; q++) {
                t |= ((row >> p.pos[q]) & 1) << q;
                base &= ~(1 << p.pos[q]);
            }
            if ((row & p.cmask) == p.cval) {
                double2 y = make_double2(0.0, 0.0);
                for (int c = 0; c < (1 << k); c++) {
                    int src = base;
                    for (int q = 0; q < k; q++) src |= ((c >> q) & 1) << p.pos[q];
                    if (p.kind == 0) {
                        const double2 u = U[cur][src][col];
                        if (u.x == 0.0 && u.y == 0.0) continue;
                        const double2 m = pool[p.off + (t << k) + c];
                        y.x += m.x * u.x - m.y * u.y;
                        y.y += m.x * u.y + m.y * u.x;
                    } else if (perms[p.off + 2 * c] == t) {
                        const double2 u = U[cur][src][col];
                        const int ph = perms[p.off + 2 * c + 1] & 3;
                        y = ph == 0 ? u : ph == 1 ? make_double2(-u.y, u.x) : ph == 2 ? make_double2(-u.x, -u.y) : make_double2(u.y, -u.x);
                    }
                }
                x = y;
            }
        }
        cur ^= 1;          // the other buffer's readers are behind the previous barrier
        U[cur][row][col] = x;
        __syncthreads();
    }
    mats[(size_t)v * 1024 + row * 32 + gcol] = x;
    unsigned long long mx = (unsigned long long)__double_as_longlong(fmax(fabs(x.x), fabs(x.y)));
    for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) atomicMax(largest + bi, mx);
}

// Digit slices of the fused matrices for the tensor-core sweep, one CTA per matrix variant.
// mats: complex 32x32 row-major FP64 per variant; largest: bits of the largest entry of the fused unitary,
// which gives its tc_eu (entries below 2^tc_eu), written to its TileGate.
// Entry (n, k) of the real 64x64 embedding (n = 2t'+c' output re/im, k = 2t+c input re/im) is split
// into six balanced digits d_i in [-256, 256] (u 2^(8-eu), rounded to a multiple of 2^-45, = sum_i d_i 2^(-9i);
// taken from the 54-bit integer, the FP64 units would make it 30 us instead of 8), digit i stored as the bf16 of d_i 2^(-9i) at its place in the K-major no-swizzle
// operand layout (per digit and k-step a 2 KiB block of 8x8 core matrices: row group n/8 at 256 B,
// K half at 128 B, row n%8 at 16 B).
__global__ void __launch_bounds__(256) k_tc_digits(const double* __restrict__ mats, const TcBlock* __restrict__ blocks,
                                                   const int32_t* __restrict__ var_block,
                                                   const unsigned long long* __restrict__ largest,
                                                   TileGate* __restrict__ gates, uint16_t* __restrict__ pool) {
    const int v = blockIdx.x, bi = var_block[v];
    const double* m = mats + (size_t)v * 2048;
    uint16_t* dst = pool + (size_t)v * tc::kPoolBlock;
    const unsigned long long lb = largest[bi];
    const int eu = lb ? max((int)(lb >> 52) - 1022, -60) : 0;
    if (threadIdx.x == 0 && v == blocks[bi].var0) gates[blocks[bi].gate].tc_eu = eu;
    const double sc = __longlong_as_double((long long)(1023 + 53 - eu) << 52);   // 2^(53 - eu): the entry as a multiple of 2^(eu-53)
    for (int e = threadIdx.x; e < 64 * 64; e += blockDim.x) {
        const int n = e >> 6, k = e & 63;
        const int tp = n >> 1, cp = n & 1, t = k >> 1, c = k & 1;
        const double re = m[2 * (tp * 32 + t)], im = m[2 * (tp * 32 + t) + 1];
        const double u = (cp == c) ? re : (cp == 0 ? -im : im);
        const int s = k >> 4, kc = (k >> 3) & 1, rg = n >> 3, r = n & 7, el = k & 7;
        const int pos = rg * 128 + kc * 64 + r * 8 + el;
        long long x = __double2ll_rn(u * sc);
#pragma unroll
        for (int i = 5; i >= 0; i--) {
            const int d = i ? (int)((x + 256) & 511) - 256 : (int)x;
            x = (x - d) >> 9;
            const float f = (float)d * __int_as_float((127 - 9 * i) << 23);   // exact: |d| <= 256
            dst[(size_t)(i * 4 + s) * 1024 + pos] = (uint16_t)(__float_as_uint(f) >> 16);
        }
    }
}

// Dense gate with more targets than a tile holds: one CTA per group of 2^k
// amplitudes, gathered into shared memory, rows computed by the CTA's threads.
__global__ void __launch_bounds__(kThreads) k_dense_big(double2* __restrict__ psi, int n_bits, int k,
                                                        const int* __restrict__ ebits, uint64_t cmask,
                                                        uint64_t cval, const float4* __restrict__ mat,
                                                        int64_t group0) {
    extern __shared__ float4 smem[];
    const int D = 1 << k;
    __shared__ int64_t s_base;
    __shared__ int s_skip;
    if (threadIdx.x == 0) {
        // insert zeros at the sorted target bits
        int ord[BS_MAX_TARGETS];
        for (int q = 0; q < k; q++) ord[q] = ebits[q];
        for (int a = 0; a < k; a++)
            for (int b = a + 1; b < k; b++)
                if (ord[b] < ord[a]) { int t = ord[a]; ord[a] = ord[b]; ord[b] = t; }
        int64_t x = group0 + (int64_t)blockIdx.x;
        for (int q = 0; q < k; q++) {
            int64_t low = x & ((1LL << ord[q]) - 1);
            x = ((x >> ord[q]) << (ord[q] + 1)) | low;
        }
        s_base = x;
        s_skip = ((uint64_t)x & cmask) != cval;
    }
    __syncthreads();
    if (s_skip) return;
    const int64_t base = s_base;
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
        int64_t gi = base;
        for (int q = 0; q < k; q++) if ((c >> q) & 1) gi |= 1LL << ebits[q];
        smem[c] = c4f(load_c128(psi[gi]));
    }
    __syncthreads();
    float4* outv = smem + D;
    for (int r = threadIdx.x; r < D; r += blockDim.x) {
        ffacc ar, ai;
        cmac_first(ar, ai, f4m(mat[(int64_t)r * D]), f4c(smem[0]));
        for (int c = 1; c < D; c++) cmac(ar, ai, f4m(mat[(int64_t)r * D + c]), f4c(smem[c]));
        outv[r] = c4f(cdone(ar, ai));
    }
    __syncthreads();
    for (int r = threadIdx.x; r < D; r += blockDim.x) {
        int64_t gi = base;
        for (int q = 0; q < k; q++) if ((r >> q) & 1) gi |= 1LL << ebits[q];
        psi[gi] = store_c128(f4c(outv[r]));
    }
}

inline void split_d(double x, float& h, float& l) {
    h = (float)x;
    l = (float)(x - (double)h);
}
// ---------------------------------------------------------------------------
// complex64 states: the same tiles and gate tables, FP32 complex arithmetic
// (the matrix entries are the FP32-rounded hi parts of the float-float table).
__device__ __forceinline__ float2 c64_mul(float4 m, float2 x) {
    return make_float2(fmaf(m.x, x.x, -m.z * x.y), fmaf(m.x, x.y, m.z * x.x));
}
__device__ __forceinline__ float2 c64_ipow(float2 x, int p) {
    switch (p & 3) {
        case 0: return x;
        case 1: return make_float2(-x.y, x.x);
        case 2: return make_float2(-x.x, -x.y);
        default: return make_float2(x.y, -x.x);
    }
}

template <int K>
__device__ void tile_dense_c64(float2* sm, int T, const TileGate& g, const float4* __restrict__ mats) {
    constexpr int D = 1 << K;
    int pos[K], tb[K];
#pragma unroll
    for (int q = 0; q < K; q++) pos[q] = tb[q] = g.tbit[q];
#pragma unroll
    for (int a = 0; a < K; a++)
#pragma unroll
        for (int b = a + 1; b < K; b++)
            if (pos[b] < pos[a]) { int t = pos[a]; pos[a] = pos[b]; pos[b] = t; }
    const int ngroups = 1 << (T - K);
    const float4* m = mats + g.mat_off;
    const uint32_t lcm = g.lc_mask, lcv = g.lc_val;
    // 1- and 2-target matrices are held in registers across the thread's groups
    constexpr int MR = K <= 2 ? D * D : 1;
    float mre[MR], mim[MR];
    if (K <= 2) {
#pragma unroll
        for (int e = 0; e < MR; e++) {
            const float4 mv = __ldg(m + e);
            mre[e] = mv.x;
            mim[e] = mv.z;
        }
    }
    for (int gr = threadIdx.x; gr < ngroups; gr += blockDim.x) {
        int jb = gr;
#pragma unroll
        for (int q = 0; q < K; q++) jb = insert0(jb, pos[q]);
        if ((jb & (int)lcm) != (int)lcv) continue;
        float2 x[D];
        int idx[D];
#pragma unroll
        for (int c = 0; c < D; c++) {
            int j = jb;
#pragma unroll
            for (int q = 0; q < K; q++) if ((c >> q) & 1) j |= 1 << tb[q];
            idx[c] = j;
            x[c] = sm[j];
        }
#pragma unroll
        for (int r = 0; r < D; r++) {
            float re = 0.f, im = 0.f;
#pragma unroll
            for (int c = 0; c < D; c++) {
                float ar, ai;
                if (K <= 2) { ar = mre[(r * D + c) % MR]; ai = mim[(r * D + c) % MR]; }
                else { const float4 mv = __ldg(m + r * D + c); ar = mv.x; ai = mv.z; }
                re = fmaf(ar, x[c].x, fmaf(-ai, x[c].y, re));
                im = fmaf(ar, x[c].y, fmaf(ai, x[c].x, im));
            }
            sm[idx[r]] = make_float2(re, im);
        }
    }
}

template <int K>
__device__ void tile_mono_c64(float2* sm, int T, const TileGate& g, const int32_t* __restrict__ perms) {
    constexpr int D = 1 << K;
    int pos[K], tb[K];
#pragma unroll
    for (int q = 0; q < K; q++) pos[q] = tb[q] = g.tbit[q];
#pragma unroll
    for (int a = 0; a < K; a++)
#pragma unroll
        for (int b = a + 1; b < K; b++)
            if (pos[b] < pos[a]) { int t = pos[a]; pos[a] = pos[b]; pos[b] = t; }
    const int32_t* p = perms + g.perm_off;
    for (int gr = threadIdx.x; gr < (1 << (T - K)); gr += blockDim.x) {
        int jb = gr;
#pragma unroll
        for (int q = 0; q < K; q++) jb = insert0(jb, pos[q]);
        if ((jb & (int)g.lc_mask) != (int)g.lc_val) continue;
        float2 x[D];
        int idx[D];
#pragma unroll
        for (int c = 0; c < D; c++) {
            int j = jb;
#pragma unroll
            for (int q = 0; q < K; q++) if ((c >> q) & 1) j |= 1 << tb[q];
            idx[c] = j;
            x[c] = sm[j];
        }
#pragma unroll
        for (int c = 0; c < D; c++) {
            const int r = __ldg(p + 2 * c);
            int j = jb;
#pragma unroll
            for (int q = 0; q < K; q++) if ((r >> q) & 1) j |= 1 << tb[q];
            sm[j] = c64_ipow(x[c], __ldg(p + 2 * c + 1));
        }
    }
}

__device__ void tile_diag_c64(float2* sm, int T, int L, const TileGate& g, const float4* __restrict__ mats, int64_t base,
                              const int64_t* off_tab) {
    const int nt = 1 << T, lowmask = (1 << L) - 1;
    const float4* m = mats + g.mat_off;
    if (g.k <= BS_TILE_MAXK) {
        // bit q of the pattern: tile bit tbit[q], or a constant of the CTA when the bit is outside the tile
        int cst = 0, nk = 0;
        uint32_t enc = 0;   // per in-tile pattern bit: tile position (5 bits) | q << 5, one byte each
        for (int q = 0; q < g.k; q++) {
            if (g.tbit[q] >= 0) enc |= (uint32_t)(g.tbit[q] | (q << 5)) << (8 * nk++);
            else cst |= (int)((base >> g.gbit[q]) & 1) << q;
        }
        for (int j = threadIdx.x; j < nt; j += blockDim.x) {
            if ((j & (int)g.lc_mask) != (int)g.lc_val) continue;
            int di = cst;
            for (int u = 0; u < nk; u++) {
                const uint32_t b = (enc >> (8 * u)) & 255u;
                di |= ((j >> (b & 31u)) & 1) << (b >> 5);
            }
            const float4 d = __ldg(m + di);
            if (d.z == 0.f && d.x == 1.f && d.y == 0.f) continue;
            sm[j] = c64_mul(d, sm[j]);
        }
        return;
    }
    for (int j = threadIdx.x; j < nt; j += blockDim.x) {
        if ((j & (int)g.lc_mask) != (int)g.lc_val) continue;
        const int64_t gi = base | off_tab[j >> L] | (int64_t)(j & lowmask);
        int di = 0;
        for (int q = 0; q < g.k; q++) di |= (int)((gi >> g.gbit[q]) & 1) << q;
        const float4 d = __ldg(m + di);
        if (d.z == 0.f && d.x == 1.f && d.y == 0.f) continue;
        sm[j] = c64_mul(d, sm[j]);
    }
}


// FULL: tiles of 2^12 with 5 low bits (vectors of 12 bits and more): a thread's 16 loads are all in flight, at
// one pointer plus uniform offsets; smaller tiles take eight at a time.
template <int KMAX, bool FULL>
__global__ void __launch_bounds__(kThreads, KMAX == 2 ? 4 : 3) k_tile_sweep_c64(float2* __restrict__ psi, SweepDesc d, int64_t tile0) {
    extern __shared__ float4 smem4[];
    float2* smem = reinterpret_cast<float2*>(smem4);
    const int T = FULL ? 12 : d.T, L = FULL ? 5 : d.L, H = T - L;
    const int nt = 1 << T;
    int64_t* off_tab = reinterpret_cast<int64_t*>(smem + nt);
    const int64_t base = bs_tile_base(d, tile0 + (int64_t)blockIdx.x);
    const int tid = threadIdx.x;
    for (int i = tid; i < (1 << H); i += kThreads) {
        int64_t o = 0;
        for (int j = 0; j < H; j++) if ((i >> j) & 1) o |= 1LL << d.hi_bits[j];
        off_tab[i] = o;
    }
    __syncthreads();
    const int lowmask = (1 << L) - 1;
    // the offset of a tile position is linear over XOR of its bits: position i * kThreads + tid of a full tile
    // lies at rows + off_tab[8 i]
    float2* rows = FULL ? psi + (base | off_tab[tid >> 5] | (int64_t)(tid & 31)) : psi;
    if (FULL) {
        float2 x[4096 / kThreads];
#pragma unroll
        for (int i = 0; i < 4096 / kThreads; i++) x[i] = __ldcs(rows + off_tab[(kThreads >> 5) * i]);
#pragma unroll
        for (int i = 0; i < 4096 / kThreads; i++) smem[i * kThreads + tid] = x[i];
    } else {
#pragma unroll
        for (int r = 0; r < 4096 / kThreads; r += 8) {
            float2 x[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int j = (r + i) * kThreads + tid;
                if (j < nt) x[i] = __ldcs(psi + (base | off_tab[j >> L] | (int64_t)(j & lowmask)));
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int j = (r + i) * kThreads + tid;
                if (j < nt) smem[j] = x[i];
            }
        }
    }
    __syncthreads();
    __shared__ TileGate s_gates[kGateChunk];
    for (int g0 = 0; g0 < d.n_gates; g0 += kGateChunk) {
    const int ng = min(kGateChunk, d.n_gates - g0);
    stage_gates(s_gates, d.gates + g0, ng);
    for (int gl = 0; gl < ng; gl++) {
        const TileGate& g = s_gates[gl];
        if ((base & (int64_t)g.gc_mask) != (int64_t)g.gc_val) continue;
        const int kind = g.kind, k = g.k;
        if (kind == 3) {
            for (int j = tid; j < nt; j += kThreads) {
                const int64_t gi = base | off_tab[j >> L] | (int64_t)(j & lowmask);
                if (parity_odd(g, gi)) { float2 v = smem[j]; smem[j] = make_float2(-v.x, -v.y); }
            }
        } else if (kind == 1) {
            tile_diag_c64(smem, T, L, g, d.mats, base, off_tab);
        } else if (kind == 0) {
            if (k == 1) tile_dense_c64<1>(smem, T, g, d.mats);
            else if (k == 2 || KMAX == 2) tile_dense_c64<2>(smem, T, g, d.mats);
            else if (KMAX > 2 && k == 3) tile_dense_c64<3>(smem, T, g, d.mats);
            else if (KMAX > 2) tile_dense_c64<4>(smem, T, g, d.mats);
        } else {
            if (k == 1) tile_mono_c64<1>(smem, T, g, d.perms);
            else if (k == 2 || KMAX == 2) tile_mono_c64<2>(smem, T, g, d.perms);
            else if (KMAX > 2 && k == 3) tile_mono_c64<3>(smem, T, g, d.perms);
            else if (KMAX > 2) tile_mono_c64<4>(smem, T, g, d.perms);
        }
        __syncthreads();
    }
    }
    if (FULL) {
#pragma unroll
        for (int i = 0; i < 4096 / kThreads; i++) __stcs(rows + off_tab[(kThreads >> 5) * i], smem[i * kThreads + tid]);
    } else {
        for (int j = tid; j < nt; j += kThreads)
            __stcs(psi + (base | off_tab[j >> L] | (int64_t)(j & lowmask)), smem[j]);
    }
}

__global__ void __launch_bounds__(kThreads) k_dense_big_c64(float2* __restrict__ psi, int n_bits, int k,
                                                            const int* __restrict__ ebits, uint64_t cmask, uint64_t cval,
                                                            const float4* __restrict__ mat, int64_t group0) {
    extern __shared__ float4 smem4[];
    float2* smem = reinterpret_cast<float2*>(smem4);
    const int D = 1 << k;
    __shared__ int64_t s_base;
    __shared__ int s_skip;
    if (threadIdx.x == 0) {
        int ord[BS_MAX_TARGETS];
        for (int q = 0; q < k; q++) ord[q] = ebits[q];
        for (int a = 0; a < k; a++)
            for (int b = a + 1; b < k; b++)
                if (ord[b] < ord[a]) { int t = ord[a]; ord[a] = ord[b]; ord[b] = t; }
        int64_t x = group0 + (int64_t)blockIdx.x;
        for (int q = 0; q < k; q++) {
            int64_t low = x & ((1LL << ord[q]) - 1);
            x = ((x >> ord[q]) << (ord[q] + 1)) | low;
        }
        s_base = x;
        s_skip = ((uint64_t)x & cmask) != cval;
    }
    __syncthreads();
    if (s_skip) return;
    const int64_t base = s_base;
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
        int64_t gi = base;
        for (int q = 0; q < k; q++) if ((c >> q) & 1) gi |= 1LL << ebits[q];
        smem[c] = psi[gi];
    }
    __syncthreads();
    float2* outv = smem + D;
    for (int r = threadIdx.x; r < D; r += blockDim.x) {
        float re = 0.f, im = 0.f;
        for (int c = 0; c < D; c++) {
            const float4 mv = mat[(int64_t)r * D + c];
            re = fmaf(mv.x, smem[c].x, fmaf(-mv.z, smem[c].y, re));
            im = fmaf(mv.x, smem[c].y, fmaf(mv.z, smem[c].x, im));
        }
        outv[r] = make_float2(re, im);
    }
    __syncthreads();
    for (int r = threadIdx.x; r < D; r += blockDim.x) {
        int64_t gi = base;
        for (int q = 0; q < k; q++) if ((r >> q) & 1) gi |= 1LL << ebits[q];
        psi[gi] = outv[r];
    }
}


inline float4 to_cff(double re, double im) {
    float4 v;
    split_d(re, v.x, v.y);
    split_d(im, v.z, v.w);
    return v;
}

}  // namespace

namespace {

bool plain_x(const HostGate& h) {
    return h.kind == 2 && h.k == 1 && h.perm.size() == 4 && h.perm[0] == 1 && h.perm[1] == 0 && h.perm[2] == 0 && h.perm[3] == 0;
}

bool plain_cz(const HostGate& h) {
    return h.kind == 1 && h.k == 1 && h.mat.size() == 4 && h.mat[0] == 1.0 && h.mat[1] == 0.0 && h.mat[2] == -1.0 &&
           h.mat[3] == 0.0 && __builtin_popcountll(h.cmask) == 1 && h.cval == h.cmask;
}

uint64_t gate_bits(const HostGate& h) {
    uint64_t m = h.cmask;
    if (h.kind == 5) return ~0ULL;
    for (int q = 0; q < h.k; q++) m |= 1ULL << h.ebit[q];
    return m;
}

// Diagonal gates (other than CZ, which merge into parity phases when packed) are folded into one
// diagonal table over the union of their bits, up to kMaxMergedDiag bits.  The open table floats
// forward past gates it commutes with (diagonal ones, and any gate on other bits), and is emitted
// before the first non-diagonal gate that touches one of its bits.  One pass over the tile then
// replaces a pass per gate.
constexpr int kMaxMergedDiag = BS_TILE_MAXK;

struct DiagTable {
    uint64_t bits = 0;                 // endian bits, ascending in ebit order
    std::vector<int> eb;
    std::vector<std::complex<double>> d;
};

void diag_absorb(DiagTable& t, const HostGate& h) {
    const uint64_t nb = t.bits | gate_bits(h);
    std::vector<int> eb;
    for (int e = 0; e < 64; e++) if ((nb >> e) & 1ULL) eb.push_back(e);
    const int k = (int)eb.size();
    std::vector<std::complex<double>> d((size_t)1 << k);
    for (int x = 0; x < (1 << k); x++) {
        uint64_t g = 0;   // the assignment x on the endian bits
        for (int q = 0; q < k; q++) if ((x >> q) & 1) g |= 1ULL << eb[(size_t)q];
        std::complex<double> v(1.0, 0.0);
        if (!t.eb.empty() || t.bits == 0) {
            int xi = 0;
            for (size_t q = 0; q < t.eb.size(); q++) xi |= (int)((g >> t.eb[q]) & 1ULL) << q;
            if (!t.d.empty()) v = t.d[(size_t)xi];
        }
        if ((g & h.cmask) == h.cval) {
            int hi = 0;
            for (int q = 0; q < h.k; q++) hi |= (int)((g >> h.ebit[q]) & 1ULL) << q;
            v *= std::complex<double>(h.mat[2 * hi], h.mat[2 * hi + 1]);
        }
        d[(size_t)x] = v;
    }
    t.bits = nb;
    t.eb = eb;
    t.d = d;
}

void merge_diagonals(const std::vector<HostGate>& in, std::vector<HostGate>& out) {
    out.clear();
    DiagTable open;
    int n_open = 0;
    const HostGate* first = nullptr;
    // CZ gates float forward the same way and are emitted together sorted by the distance of their
    // two bits, so that the packer folds each distance into one parity-phase term
    std::vector<const HostGate*> czs;
    uint64_t cz_bits = 0;
    auto cz_dist = [](const HostGate* h) {
        const int c = 63 - __builtin_clzll(h->cmask), t = h->ebit[0];
        return c > t ? c - t : t - c;
    };
    auto flush_cz = [&]() {
        std::stable_sort(czs.begin(), czs.end(), [&](const HostGate* a, const HostGate* b) { return cz_dist(a) < cz_dist(b); });
        for (const HostGate* h : czs) out.push_back(*h);
        czs.clear();
        cz_bits = 0;
    };
    auto flush = [&]() {
        if (n_open == 1) {
            out.push_back(*first);   // a single gate keeps its own form
        } else if (n_open > 1) {
            HostGate m;
            m.kind = 1;
            m.k = (int)open.eb.size();
            for (int q = 0; q < m.k; q++) m.ebit[q] = open.eb[(size_t)q];
            m.mat.resize(2 * open.d.size());
            for (size_t x = 0; x < open.d.size(); x++) {
                m.mat[2 * x] = open.d[x].real();
                m.mat[2 * x + 1] = open.d[x].imag();
            }
            out.push_back(std::move(m));
        }
        open = DiagTable{};
        n_open = 0;
        first = nullptr;
    };
    for (const HostGate& h : in) {
        if (plain_cz(h)) {
            czs.push_back(&h);
            cz_bits |= gate_bits(h);
            continue;
        }
        const bool mergeable = h.kind == 1 && __builtin_popcountll(gate_bits(h)) <= kMaxMergedDiag;
        if (mergeable) {
            if (n_open && __builtin_popcountll(open.bits | gate_bits(h)) > kMaxMergedDiag) flush();
            if (n_open == 0) first = &h;
            diag_absorb(open, h);
            n_open++;
            continue;
        }
        if (h.kind != 1) {
            if (n_open && (gate_bits(h) & open.bits)) flush();
            if (!czs.empty() && (gate_bits(h) & cz_bits)) flush_cz();
        }
        out.push_back(h);
    }
    flush();
    flush_cz();
}

}  // namespace

namespace {
// The tensor-core sweep's offsets of a fused gate on tile bits tb[0..4], in its bank-swizzled tile
// (tc::sw, restated here for the host): 56 uint16 packed two per int32 — sw of the deposit of a
// column index's bits 0..3 and 4..6 into the 7 other tile bits (ascending), then sw of each of the 32
// target patterns.  The swizzle is linear over XOR, so sw(column) = table[m & 15] ^ table[16 + (m >> 4)].
int host_sw(int j) { return j ^ (((j >> 3) ^ (j >> 6) ^ (j >> 9)) & 7); }
void tc_offset_tables(const int32_t* tb, std::vector<int32_t>& out) {
    uint32_t tmask = 0;
    for (int q = 0; q < 5; q++) tmask |= 1u << tb[q];
    int nb[7], k = 0;
    for (int b = 0; b < 12; b++)
        if (!((tmask >> b) & 1u)) nb[k++] = b;
    uint16_t v[56];
    for (int i = 0; i < 16; i++) {
        int p = 0;
        for (int j = 0; j < 4; j++) if ((i >> j) & 1) p |= 1 << nb[j];
        v[i] = (uint16_t)host_sw(p);
    }
    for (int i = 0; i < 8; i++) {
        int p = 0;
        for (int j = 0; j < 3; j++) if ((i >> j) & 1) p |= 1 << nb[4 + j];
        v[16 + i] = (uint16_t)host_sw(p);
    }
    for (int t = 0; t < 32; t++) {
        int p = 0;
        for (int q = 0; q < 5; q++) if ((t >> q) & 1) p |= 1 << tb[q];
        v[24 + t] = (uint16_t)host_sw(p);
    }
    for (int i = 0; i < 28; i++) out.push_back((int32_t)((uint32_t)v[2 * i] | ((uint32_t)v[2 * i + 1] << 16)));
}
}  // namespace

int bs_run_sweeps(bs_sim* s, const std::vector<Sweep>& sweeps) {
    if (sweeps.empty()) return BS_OK;
    const int n_bits = bs_vec_bits(s);
    const int T = sweeps.front().tile;   // of one plan: all sweeps the same
    // pack: per sweep [TileGate...], then one float4 pool, then one int pool
    std::vector<TileGate> tg;
    std::vector<float4> mats;
    std::vector<int32_t> perms;
    struct Launch {
        int64_t gate0; int n_gates; std::vector<int> hi; int low; bool big; int big_gate; int kmax = 1;
        int n_tc = 0;
    };
    std::vector<Launch> launches;
    std::vector<int32_t> big_bits;
    std::vector<double> tc_pool;             // the fused gates' own matrices (complex), then read by k_tc_build
    std::vector<TcPart> tc_parts;
    std::vector<TcBlock> tc_blocks;
    std::vector<int32_t> tc_var;             // fused unitary of each variant
    int64_t n_var = 0;
    const bool c64 = s->precision == BS_PREC_C64;
    const bool use_tc = sweeps.front().tc;
    const double tc_threshold = bs_tc_cost(s);
    // A sweep keeps its plain gate list, on the float-float kernel, where it is left with unfused 3/4-target gates
    // (the tensor-core sweep carries float-float paths for 1- and 2-target gates only) and where a fused matrix would
    // reach 2^12, beyond its digits' range (gates far from unitary; the float-float values have FP32's exponents).
    // Below 16 bits only the environment or a handle's tuning brings a list here; asked by BS_TC_MIN_BITS for
    // tensor-core sweeps of such a size, one that has no digits is refused, not run elsewhere.
    const bool refuse = n_bits < 16 && s->tune.tc_min_bits < 0;
    std::vector<HostGate> fused;
    bool out_of_range = false;
    auto fuse = [&](const Sweep& sw, const int* local) {
        if (!use_tc || (int)sw.hi_bits.size() != T - sw.low) return false;
        std::vector<const HostGate*> in;
        for (const HostGate& g : sw.gates) in.push_back(&g);
        bs_fuse_tc(in, local, T, tc_threshold, &fused);
        for (const HostGate& hg : fused) {
            if (hg.kind != 1 && hg.kind != 4 && hg.kind != 5 && hg.k >= 3) return false;
            if (hg.kind == 4 && !bs_tc_in_range(hg, sw.gates)) {
                out_of_range = true;
                return false;
            }
        }
        return true;
    };
    for (const Sweep& sw : sweeps) {
        Launch ln;
        ln.gate0 = (int64_t)tg.size();
        ln.n_gates = 0;
        ln.hi = sw.hi_bits;
        const int L = sw.low;
        ln.low = L;
        ln.big = false;
        ln.big_gate = -1;
        // tile-local position of each endian bit
        int local[64];
        for (int b = 0; b < 64; b++) local[b] = -1;
        for (int b = 0; b < L; b++) local[b] = b;
        for (size_t i = 0; i < sw.hi_bits.size(); i++) local[sw.hi_bits[i]] = L + (int)i;
        std::vector<HostGate> merged, small;
        const bool tc = fuse(sw, local);
        if (out_of_range && refuse) return bs_fail(s, BS_ERR_INVALID_ARG, "fused gate matrix out of range");
        if (tc) {
            merge_diagonals(fused, merged);
        } else if (c64) {
            // complex64 sweep: 1- and 2-bit runs fused into dense 2-bit gates where that saves passes (a
            // pass of the complex64 kernel costs about four 1-qubit gates' arithmetic; batch of 512
            // circuits 1.79 -> 1.48 s on the device).  The float-float kernel is bound by its
            // arithmetic: fusing there measured slower (18 qubits: 7.7 -> 9.2 ms).  The products are formed in
            // FP64, so matrix and state are rounded once per run; 32 amplitudes in a thread's registers and
            // an operation per gate (25 qubits, 415 gates 9.9 -> 6.0 ms) rounded the state once per gate, up
            // to 1.6 times the error on lists of generic matrices, and is not used
            bs_fuse_small(sw.gates, local, 4.0, 2, small);
            merge_diagonals(small, merged);
        } else {
            merge_diagonals(sw.gates, merged);
        }
        const std::vector<HostGate>* glist = &merged;
        for (const HostGate& hg : *glist) {
            if (hg.kind == 5) {
                // reference-rule channel: its row and column target bits are tile bits (the planner needs them)
                TileGate t{};
                t.kind = 5;
                t.k = hg.k;
                const int nq = n_bits / 2;
                uint64_t rt = 0;
                for (int q = 0; q < 2 * hg.k; q++) t.tbit[q] = local[hg.ebit[q]];
                for (int q = 0; q < hg.k; q++) rt |= 1ULL << hg.ebit[q];
                const uint64_t nt = (((uint64_t)1 << nq) - 1) & ~rt;
                uint64_t unif = 0;
                for (int b = 0; b < nq; b++)
                    if (((nt >> b) & 1ULL) && local[b] < 0 && local[b + nq] < 0) unif |= 1ULL << b;
                t.pmask[0] = nt;
                t.pmask[1] = unif;
                t.mat_off = (int32_t)mats.size();
                for (size_t e = 0; e + 1 < hg.mat.size(); e += 2) mats.push_back(to_cff(hg.mat[e], hg.mat[e + 1]));
                tg.push_back(t);
                ln.n_gates++;
                continue;
            }
            if (hg.kind == 4) {
                TileGate t{};
                t.kind = 4;
                t.k = 5;
                for (int q = 0; q < 5; q++) t.gbit[q] = local[hg.ebit[q]];
                t.perm_off = (int32_t)perms.size();
                tc_offset_tables(t.gbit, perms);
                const int nvar = 1 << hg.ubits.size();
                t.tc_nu = (int32_t)hg.ubits.size();
                for (size_t i = 0; i < hg.ubits.size(); i++) t.tc_ub[i] = hg.ubits[i];
                t.tc_off = (int32_t)n_var;
                int where[64];           // block or variant bit of an endian bit
                for (int b = 0; b < 64; b++) where[b] = -1;
                for (int q = 0; q < 5; q++) where[hg.ebit[q]] = q;
                for (size_t i = 0; i < hg.ubits.size(); i++) where[hg.ubits[i]] = 8 + (int)i;
                tc_blocks.push_back({(int32_t)tc_parts.size(), (int32_t)hg.perm.size(), (int32_t)n_var, (int32_t)tg.size()});
                for (int gi : hg.perm) {
                    const HostGate& g = sw.gates[(size_t)gi];
                    TcPart p{};
                    p.kind = (uint8_t)g.kind;
                    p.k = (uint8_t)g.k;
                    for (int q = 0; q < g.k; q++) p.pos[q] = (uint8_t)where[g.ebit[q]];
                    for (uint64_t r = g.cmask; r; r &= r - 1) {
                        const int e = __builtin_ctzll(r), w = where[e], v = (int)((g.cval >> e) & 1);
                        if (w < 8) { p.cmask |= (uint8_t)(1 << w); p.cval |= (uint8_t)(v << w); }
                        else { p.umask |= (uint8_t)(1 << (w - 8)); p.uval |= (uint8_t)(v << (w - 8)); }
                    }
                    if (g.kind == 2) {
                        p.off = (int32_t)perms.size();
                        perms.insert(perms.end(), g.perm.begin(), g.perm.end());
                    } else {
                        p.off = (int32_t)(tc_pool.size() / 2);
                        tc_pool.insert(tc_pool.end(), g.mat.begin(), g.mat.begin() + ((size_t)2 << (g.kind == 0 ? 2 * g.k : g.k)));
                    }
                    tc_parts.push_back(p);
                }
                tc_var.insert(tc_var.end(), (size_t)nvar, (int32_t)tc_blocks.size() - 1);
                n_var += nvar;
                ln.n_tc++;
                tg.push_back(t);
                ln.n_gates++;
                continue;
            }
            // consecutive CZ gates (Z on one bit, one control at value 1) merge into one parity-phase gate
            if (hg.kind == 1 && hg.k == 1 && hg.mat.size() == 4 && hg.mat[0] == 1.0 && hg.mat[1] == 0.0 &&
                hg.mat[2] == -1.0 && hg.mat[3] == 0.0 && __builtin_popcountll(hg.cmask) == 1 && hg.cval == hg.cmask) {
                const int c = 63 - __builtin_clzll(hg.cmask), t = hg.ebit[0];
                const int lo = std::min(c, t), dd = std::max(c, t) - lo;
                auto add_pair = [&](TileGate& g) {
                    for (int q = 0; q < g.npar; q++)
                        if (g.pshift[q] == dd) { g.pmask[q] ^= 1ULL << lo; return true; }   // CZ twice = identity
                    if (g.npar == 4) return false;
                    g.pshift[g.npar] = dd;
                    g.pmask[g.npar] = 1ULL << lo;
                    g.npar++;
                    return true;
                };
                if (!(ln.n_gates > 0 && tg.back().kind == 3 && add_pair(tg.back()))) {
                    TileGate t3{};
                    t3.kind = 3;
                    add_pair(t3);
                    tg.push_back(t3);
                    ln.n_gates++;
                }
                continue;
            }
            bool big = hg.kind != 1 && hg.k > BS_TILE_MAXK;
            if (!big && hg.kind != 1)
                for (int q = 0; q < hg.k; q++) if (local[hg.ebit[q]] < 0) big = true;
            if (big) {
                // runs alone: sweeps hold a single out-of-tile gate
                ln.big = true;
                ln.big_gate = (int)tg.size();
                TileGate t{};
                t.kind = hg.kind;
                t.k = hg.k;
                t.gc_mask = hg.cmask;
                t.gc_val = hg.cval;
                t.mat_off = (int32_t)mats.size();
                t.perm_off = (int32_t)big_bits.size();
                for (int q = 0; q < hg.k; q++) big_bits.push_back(hg.ebit[q]);
                if (hg.kind == 0) {
                    for (int i = 0; i < (1 << (2 * hg.k)); i++) mats.push_back(to_cff(hg.mat[2 * i], hg.mat[2 * i + 1]));
                } else {
                    // monomial given as dense
                    int D = 1 << hg.k;
                    std::vector<float4> dense((size_t)D * D, make_float4(0, 0, 0, 0));
                    for (int c = 0; c < D; c++) {
                        int r = hg.perm[2 * c], p = hg.perm[2 * c + 1] & 3;
                        double re = (p == 0) ? 1 : (p == 2 ? -1 : 0), im = (p == 1) ? 1 : (p == 3 ? -1 : 0);
                        dense[(size_t)r * D + c] = to_cff(re, im);
                    }
                    t.kind = 0;
                    mats.insert(mats.end(), dense.begin(), dense.end());
                }
                tg.push_back(t);
                ln.n_gates++;
                continue;
            }
            TileGate t{};
            t.kind = hg.kind;
            t.k = hg.k;
            uint64_t gcm = 0, gcv = 0;
            uint32_t lcm = 0, lcv = 0;
            for (int b = 0; b < n_bits; b++) {
                if (!((hg.cmask >> b) & 1ULL)) continue;
                uint64_t v = (hg.cval >> b) & 1ULL;
                if (local[b] >= 0) { lcm |= 1u << local[b]; lcv |= (uint32_t)v << local[b]; }
                else { gcm |= 1ULL << b; gcv |= v << b; }
            }
            t.lc_mask = lcm; t.lc_val = lcv; t.gc_mask = gcm; t.gc_val = gcv;
            for (int q = 0; q < hg.k; q++) {
                t.gbit[q] = hg.ebit[q];
                if (q < BS_TILE_MAXK) t.tbit[q] = local[hg.ebit[q]];
            }
            t.mat_off = (int32_t)mats.size();
            t.perm_off = (int32_t)perms.size();
            if (hg.kind == 0) {
                for (int i = 0; i < (1 << (2 * hg.k)); i++) mats.push_back(to_cff(hg.mat[2 * i], hg.mat[2 * i + 1]));
            } else if (hg.kind == 1) {
                for (int i = 0; i < (1 << hg.k); i++) mats.push_back(to_cff(hg.mat[2 * i], hg.mat[2 * i + 1]));
            } else {
                perms.insert(perms.end(), hg.perm.begin(), hg.perm.end());
                if (plain_x(hg)) t.npar = 1;
            }
            if (hg.kind != 1) ln.kmax = std::max(ln.kmax, hg.k);
            if (hg.kind == 0 && hg.k == 1) t.npar = bs_class_2x2(hg);
            tg.push_back(t);
            ln.n_gates++;
        }
        launches.push_back(std::move(ln));
    }
    // upload
    auto al = [](int64_t x) { return (x + 255) & ~(int64_t)255; };
    int64_t b_tg = al((int64_t)tg.size() * (int64_t)sizeof(TileGate));
    int64_t b_m = al((int64_t)mats.size() * (int64_t)sizeof(float4));
    int64_t b_p = al((int64_t)(perms.size() + big_bits.size() + 1) * (int64_t)sizeof(int32_t));
    const int64_t b_fm = al((int64_t)tc_pool.size() * (int64_t)sizeof(double)), b_fp = al((int64_t)tc_parts.size() * (int64_t)sizeof(TcPart));
    const int64_t b_fb = al((int64_t)tc_blocks.size() * (int64_t)sizeof(TcBlock)), b_fv = al(n_var * (int64_t)sizeof(int32_t));
    const int64_t b_fx = al((int64_t)tc_blocks.size() * (int64_t)sizeof(unsigned long long));   // largest entries, from 0
    const int64_t o_fm = b_tg + b_m + b_p, o_fp = o_fm + b_fm, o_fb = o_fp + b_fp, o_fv = o_fb + b_fb;
    const int64_t o_fx = o_fv + b_fv, o_up = o_fx + b_fx;                       // uploaded up to here
    const int64_t o_tm = o_up, b_tm = al(n_var * 2048 * (int64_t)sizeof(double));   // written on the device:
    const int64_t o_tc = o_tm + b_tm, b_tc = al(n_var * tc::kPoolBlock * (int64_t)sizeof(uint16_t));
    int rc = bs_ensure_plan(s, o_tc + b_tc);
    if (rc) return rc;
    char* host = bs_stage(s, (size_t)o_up);
    if (!host) return bs_fail(s, BS_ERR_ALLOC, "pinned staging allocation");
    std::memset(host, 0, (size_t)o_up);
    if (n_var) {
        std::memcpy(host + o_fm, tc_pool.data(), tc_pool.size() * sizeof(double));
        std::memcpy(host + o_fp, tc_parts.data(), tc_parts.size() * sizeof(TcPart));
        std::memcpy(host + o_fb, tc_blocks.data(), tc_blocks.size() * sizeof(TcBlock));
        std::memcpy(host + o_fv, tc_var.data(), tc_var.size() * sizeof(int32_t));
    }
    if (!tg.empty()) std::memcpy(host, tg.data(), tg.size() * sizeof(TileGate));
    if (!mats.empty()) std::memcpy(host + b_tg, mats.data(), mats.size() * sizeof(float4));
    if (!perms.empty()) std::memcpy(host + b_tg + b_m, perms.data(), perms.size() * sizeof(int32_t));
    if (!big_bits.empty())
        std::memcpy(host + b_tg + b_m + perms.size() * sizeof(int32_t), big_bits.data(), big_bits.size() * sizeof(int32_t));
    char* dev = (char*)s->plan_buf;
    rc = bs_cuda_check(s, cudaMemcpyAsync(dev, host, (size_t)o_up, cudaMemcpyHostToDevice, s->stream), "plan upload");
    bs_stage_done(s);
    if (rc) return rc;
    const TileGate* d_tg = (const TileGate*)dev;
    const float4* d_m = (const float4*)(dev + b_tg);
    const int32_t* d_p = (const int32_t*)(dev + b_tg + b_m);
    const int32_t* d_big = d_p + perms.size();

    static bool attr_set[64] = {false};
    if (!attr_set[s->device & 63]) {
        // largest carveout: three 65 KiB tiles per SM instead of two
        auto attrs = [](const void* f) {
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
            cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        };
        attrs((const void*)k_tile_sweep<2, 256>);
        attrs((const void*)k_tile_sweep<4, 256>);
        attrs((const void*)k_tile_sweep<2, 512>);
        attrs((const void*)k_tile_sweep<4, 512>);
        attrs((const void*)k_tile_sweep_c64<2, false>);
        attrs((const void*)k_tile_sweep_c64<4, false>);
        attrs((const void*)k_tile_sweep_c64<2, true>);
        attrs((const void*)k_tile_sweep_c64<4, true>);
        cudaFuncSetAttribute(k_dense_big_c64, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        cudaFuncSetAttribute(k_dense_big, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        for (auto f : {k_tile_sweep_tc<3>, k_tile_sweep_tc<4>, k_tile_sweep_tc<5>}) {
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
            cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        }
        attr_set[s->device & 63] = true;
    }
    double2* psi = (double2*)s->state;
    uint16_t* d_tc = (uint16_t*)(dev + o_tc);
    if (n_var) {
        const TcBlock* d_fb = (const TcBlock*)(dev + o_fb);
        const int32_t* d_fv = (const int32_t*)(dev + o_fv);
        unsigned long long* d_fx = (unsigned long long*)(dev + o_fx);
        k_tc_build<<<(unsigned)(4 * n_var), 256, 0, s->stream>>>(d_fb, d_fv, (const TcPart*)(dev + o_fp), (const double2*)(dev + o_fm),
                                                                 d_p, (double2*)(dev + o_tm), d_fx);
        k_tc_digits<<<(unsigned)n_var, 256, 0, s->stream>>>((const double*)(dev + o_tm), d_fb, d_fv, d_fx, (TileGate*)dev, d_tc);
        s->stats.kernel_launches += 2;
        if (!s->dev_flag) {
            rc = bs_cuda_check(s, bs_malloc((void**)&s->dev_flag, 256), "flag alloc");
            if (rc) return rc;
        }
        if (!s->flag_armed) {
            rc = bs_cuda_check(s, cudaMemsetAsync(s->dev_flag, 0, sizeof(int), s->stream), "flag reset");
            if (rc) return rc;
            s->flag_armed = true;
        }
    }
    const double esz = c64 ? 8.0 : 16.0;          // bytes per stored amplitude
    const int64_t ntiles = (int64_t)1 << (n_bits - T);
    for (size_t li = 0; li < launches.size(); li++) {
        const Launch& ln = launches[li];
        if (ln.big) {
            const TileGate& t = tg[(size_t)ln.big_gate];
            int64_t groups = (int64_t)1 << (n_bits - t.k);
            size_t bsm = ((size_t)2 << t.k) * sizeof(float4);
            if (bsm > 100 * 1024) return bs_fail(s, BS_ERR_UNSUPPORTED, "gate has too many targets");
            for (int64_t g0 = 0; g0 < groups; g0 += 1LL << 30) {
                int64_t ng = std::min<int64_t>(groups - g0, 1LL << 30);
                if (c64)
                    k_dense_big_c64<<<(unsigned)ng, kThreads, bsm, s->stream>>>((float2*)s->state, n_bits, t.k,
                                                                              d_big + t.perm_off, t.gc_mask, t.gc_val,
                                                                              d_m + t.mat_off, g0);
                else
                    k_dense_big<<<(unsigned)ng, kThreads, bsm, s->stream>>>(psi, n_bits, t.k, d_big + t.perm_off,
                                                                            t.gc_mask, t.gc_val, d_m + t.mat_off, g0);
            }
            s->stats.kernel_launches++;
            s->stats.sweeps++;
            s->stats.gates++;
            s->stats.bytes_moved += 2.0 * esz * (double)s->len;
            continue;
        }
        SweepDesc d{};
        const int L = ln.low, H = T - L;
        const size_t smem = ((size_t)1 << T) * sizeof(float4) + ((size_t)1 << H) * sizeof(int64_t);
        auto ktc = L == 5 ? k_tile_sweep_tc<5> : L == 4 ? k_tile_sweep_tc<4> : k_tile_sweep_tc<3>;
        bs_tile_geometry(d, n_bits, L, ln.hi);
        d.n_gates = ln.n_gates;
        d.gates = d_tg + ln.gate0;
        d.mats = d_m;
        d.perms = d_p;
        d.tc_pool = d_tc;
        d.err = s->dev_flag;
        for (int64_t t0 = 0; t0 < ntiles; t0 += (1LL << 30)) {
            int64_t nb = std::min<int64_t>(ntiles - t0, 1LL << 30);
            if (ln.n_tc > 0 && s->capturing) {
                ktc<<<(unsigned)std::min<int64_t>(nb, 2 * 152), kTcThreads, kTcSmem, s->stream>>>(psi, d, t0, t0 + nb);
                s->stats.tc_launches++;
            } else if (ln.n_tc > 0) {
                const size_t pe = 2 * s->tc_events_used;
                while (s->tc_events.size() < pe + 2) {
                    cudaEvent_t e;
                    rc = bs_cuda_check(s, cudaEventCreate(&e), "event");
                    if (rc) return rc;
                    s->tc_events.push_back(e);
                }
                cudaEventRecord(s->tc_events[pe], s->stream);
                ktc<<<(unsigned)std::min<int64_t>(nb, 2 * 152), kTcThreads, kTcSmem, s->stream>>>(psi, d, t0, t0 + nb);
                cudaEventRecord(s->tc_events[pe + 1], s->stream);
                s->tc_events_used++;
                s->stats.tc_launches++;
            } else if (c64) {
                const size_t sm64 = ((size_t)1 << T) * sizeof(float2) + ((size_t)1 << H) * sizeof(int64_t);
                const bool full = T == 12 && L == 5;
                auto kern = ln.kmax <= 2 ? (full ? k_tile_sweep_c64<2, true> : k_tile_sweep_c64<2, false>)
                                         : (full ? k_tile_sweep_c64<4, true> : k_tile_sweep_c64<4, false>);
                kern<<<(unsigned)nb, kThreads, sm64, s->stream>>>((float2*)s->state, d, t0);
            } else if (bs_sweep_threads(s, ntiles) == 512) {
                if (ln.kmax <= 2) k_tile_sweep<2, 512><<<(unsigned)nb, 512, smem, s->stream>>>(psi, d, t0);
                else k_tile_sweep<4, 512><<<(unsigned)nb, 512, smem, s->stream>>>(psi, d, t0);
            } else {
                if (ln.kmax <= 2) k_tile_sweep<2, 256><<<(unsigned)nb, 256, smem, s->stream>>>(psi, d, t0);
                else k_tile_sweep<4, 256><<<(unsigned)nb, 256, smem, s->stream>>>(psi, d, t0);
            }
        }
        s->stats.kernel_launches++;
        s->stats.sweeps++;
        s->stats.gates += ln.n_gates;
        s->stats.tc_gates += ln.n_tc;
        s->stats.bytes_moved += 2.0 * esz * (double)s->len;
    }
    return bs_cuda_check(s, cudaGetLastError(), "tile sweep launch");
}

void bs_collect_tc_time(bs_sim* s) {
    for (size_t i = 0; i < s->tc_events_used; i++) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, s->tc_events[2 * i], s->tc_events[2 * i + 1]) == cudaSuccess)
            s->stats.tc_ms += ms;
    }
    s->tc_events_used = 0;
}

namespace {
// Waits that nothing completes, in the form of the tensor-core sweep: two issuing threads wait on a fresh mbarrier (no
// arrival, no copy and no MMA in flight) with its bounded wait, give up after `limit` cycles, their warps take no
// further warp-wide step, and all threads meet at a barrier.  Raises the device flag, as a sweep whose copy or MMA
// never landed would, where exactly those two warps left, each as a whole.
__global__ void __launch_bounds__(kTcThreads) k_wait_selftest(int* __restrict__ err, long long limit) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) tc::mbar_init(tc::su32(&bar));
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0 || threadIdx.x == 128) ok = tc::mbar_wait_for(tc::su32(&bar), 0u, limit);
    ok = tc::warp_ok(ok);
    if (ok) ok = __shfl_sync(0xffffffffu, 1, 0) != 0;
    if (__syncthreads_count(!ok) == 64 && threadIdx.x == 0) atomicExch(err, 1);
}
}  // namespace

extern "C" int bs_selftest_wait_timeout(bs_sim* s, double seconds) {
    if (!s) return BS_ERR_INVALID_ARG;
    if (!(seconds > 0.0) || seconds > 1.0) return bs_fail(s, BS_ERR_INVALID_ARG, "wait limit must be in (0, 1] s");
    if (s->capturing) return bs_fail(s, BS_ERR_STATE, "not during graph capture");
    int rc = BS_OK;
    if (!s->dev_flag) {
        rc = bs_cuda_check(s, bs_malloc((void**)&s->dev_flag, 256), "flag alloc");
        if (rc) return rc;
    }
    rc = bs_cuda_check(s, cudaMemsetAsync(s->dev_flag, 0, sizeof(int), s->stream), "flag reset");
    if (rc) return rc;
    s->flag_armed = true;
    k_wait_selftest<<<1, kTcThreads, 0, s->stream>>>(s->dev_flag, (long long)(seconds * 2.0e9));
    rc = bs_cuda_check(s, cudaGetLastError(), "self-test launch");
    if (rc) return rc;
    rc = bs_check_device_flag(s);
    if (rc == BS_ERR_TIMEOUT) return bs_fail(s, BS_ERR_TIMEOUT, "self-test: the bounded wait gave up and raised the device flag");
    if (rc == BS_OK) return bs_fail(s, BS_ERR_STATE, "self-test: the wait completed");
    return rc;
}

int bs_check_device_flag(bs_sim* s) {
    if (!s->flag_armed) return BS_OK;
    s->flag_armed = false;
    int flag = 0;
    const int rc = bs_copy_out(s, &flag, s->dev_flag, sizeof(int), "flag read");
    if (rc) return rc;
    if (flag) return bs_fail(s, BS_ERR_TIMEOUT, "a tensor-core sweep gave up waiting for its copies or MMAs");
    return BS_OK;
}

// ---------------------------------------------------------------------------
// Whole small state vectors in one CTA (bs_run_small): the reference's simulate of a small circuit
// (src/BraketSimulator.jl:307-322: reinit!, evolve!, then results) as one launch.  The CTA builds
// |0...0> in shared memory, applies every gate of the planned sweeps in order with the tile kernels'
// float-float gates (the whole state is the tile, so sweep boundaries cost nothing), writes the state
// back and the probabilities, computed from the stored complex128 values exactly as bs_probabilities
// computes them.
namespace {

struct NoOff {
    __device__ __forceinline__ int64_t operator[](int) const { return 0; }
};

__device__ __forceinline__ int64_t globaltimer_ns() {
    int64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The end of a small run, for a host that polls instead of synchronising: the kernel's end time, then
// every thread's writes are made visible to the system, then one thread writes the call's ticket into
// the host-mapped word.
__device__ __forceinline__ void small_run_done(volatile int64_t* done, int64_t ticket, int64_t* times) {
    if (!done) return;
    if (times && threadIdx.x == 0) times[1] = globaltimer_ns();
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) *done = ticket;
}

// The shots sh0, sh0 + step, ... as bs_sample draws them for a state of one CDF block (k_sample_small):
// the same chunk sums and chunk prefix sums, the same in-chunk running sums (a warp's shuffle scan, kept
// here per element), the same uniforms and comparisons, so the same indices; one thread per shot.
// sprob: the nt probabilities; scan: room for two arrays of whole chunks.
struct SmallCdf {
    float ch[kCpb], cl[kCpb];
    double cinc[kCpb], total;
    long long ckey[kCpb];
};
__device__ __forceinline__ void small_shots(const double* sprob, int nt, double* scan, SmallCdf& c, int64_t sh0, int64_t step,
                                            int64_t shots, uint64_t seed, int64_t* __restrict__ samples) {
    const int nc32 = (nt + kChunk - 1) / kChunk * kChunk;
    block_chunk_sums_p(sprob, nt, 0, c.ch, c.cl, &c.total, c.cinc);
    // per element: the largest value, as an integer key, of (chunk base + running sum) over the chunk
    // up to it, so that a binary search finds the first element whose own value reaches the target
    long long* fkey = reinterpret_cast<long long*>(scan + nc32);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int q = warp; q * kChunk < nt; q += nw) {
        const int i = q * kChunk + lane;
        double p = (i < nt) ? sprob[i] : 0.0;
        const double cb = q == 0 ? 0.0 : c.cinc[q - 1];   // 0.0 + cb is cb: the sums are non-negative
        if (__ballot_sync(0xffffffffu, p != 0.0) == 0u) {
            // a chunk of zeros: every running sum is 0, every compared value the chunk base
            scan[i] = 0.0;
            fkey[i] = __double_as_longlong(cb);
            continue;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, p, o);
            if (lane >= o) p += v;
        }
        scan[i] = p;
        long long key = __double_as_longlong(cb + p);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long v = __shfl_up_sync(0xffffffffu, key, o);
            if (lane >= o) key = max(key, v);
        }
        fkey[i] = key;
    }
    for (int q = threadIdx.x; q < kCpb; q += blockDim.x) c.ckey[q] = __double_as_longlong(0.0 + c.cinc[q]);
    __syncthreads();
    // Every value compared below is a sum of probabilities, so non-negative: its order is the order of
    // its bit pattern as an integer, which keeps the comparisons off the FP64 pipe (2 per clock per SM).
    const double total = 0.0 + c.total;
    // u * total with u = (r >> 11) 2^-53: the scaling by 2^-53 is exact on either factor, so
    // (r >> 11) * (total 2^-53) rounds the same real product once, as the samplers' u * total does
    const double tscale = total * 0x1.0p-53;
    for (int64_t sh = sh0; sh < shots; sh += step) {
        const uint64_t r = splitmix64(seed ^ splitmix64((uint64_t)sh));
        const double t = (double)(r >> 11) * tscale;
        const long long tb = __double_as_longlong(t);
        int clo = 0, chi = kCpb - 1;
        while (clo < chi) {
            const int mid = (clo + chi) >> 1;
            if (c.ckey[mid] >= tb) chi = mid; else clo = mid + 1;
        }
        const int c0 = clo * kChunk;
        int lo = 0, hi = kChunk;   // first element of the chunk whose value reaches the target
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (fkey[c0 + mid] >= tb) hi = mid; else lo = mid + 1;
        }
        int64_t out = nt - 1;
        bool found = lo < kChunk && c0 + lo < nt;
        if (found) out = c0 + lo;
        if (!found && c0 < nt) {
            // the chunk's own running sum fell short of its prefix sum by rounding: go on as the
            // one-block sampler does, with the running sum carried from chunk to chunk
            double cw = (0.0 + (clo == 0 ? 0.0 : c.cinc[clo - 1])) + scan[c0 + kChunk - 1];
            for (int q = c0 + kChunk; q < nt && !found; q += kChunk) {
                for (int l = 0; l < kChunk; l++) {
                    const int i = q + l;
                    if (i < nt && cw + scan[i] >= t) { out = i; found = true; break; }
                }
                cw += scan[q + kChunk - 1];
            }
        }
        samples[sh] = out;
    }
}

// STAGED: gates, matrices and permutations are copied into shared memory first, in one go (one round
// trip to the plan, which may live in host-mapped memory), instead of being read at every gate.
template <int KMAX, bool STAGED>
__device__ __forceinline__ void small_run(double2* __restrict__ psi, int n, const TileGate* gates, int ng, const float4* mats,
                                          int n_mats, const int32_t* perms, int n_perms, double* __restrict__ probs,
                                          int64_t shots, uint64_t seed, int64_t* __restrict__ samples, volatile int64_t* done,
                                          int64_t ticket, int64_t* times) {
    if (times && threadIdx.x == 0) times[0] = globaltimer_ns();
    extern __shared__ float4 smem[];
    __shared__ TileGate s_gates[STAGED ? 1 : kGateChunk];
    const int nt = 1 << n, nc32 = (nt + kChunk - 1) / kChunk * kChunk;
    // the probabilities, after the tile (or after the sampler's two arrays, which replace the tile),
    // then the staged plan
    double* sprob = reinterpret_cast<double*>(reinterpret_cast<char*>(smem) + max(nt * 16, 2 * nc32 * 8));
    float4* ms = reinterpret_cast<float4*>(sprob + (nt + 1) / 2 * 2);
    TileGate* gs = reinterpret_cast<TileGate*>(ms + n_mats);
    int32_t* ps = reinterpret_cast<int32_t*>(gs + ng);
    if (STAGED) {
        for (int j = threadIdx.x; j < n_mats; j += blockDim.x) ms[j] = mats[j];
        const int* gw = reinterpret_cast<const int*>(gates);
        for (int j = threadIdx.x; j < ng * (int)(sizeof(TileGate) / 4); j += blockDim.x) reinterpret_cast<int*>(gs)[j] = gw[j];
        for (int j = threadIdx.x; j < n_perms; j += blockDim.x) ps[j] = perms[j];
    }
    const float4* m_op = STAGED ? ms : mats;
    const int32_t* p_op = STAGED ? ps : perms;
    for (int j = threadIdx.x; j < nt; j += blockDim.x) smem[j] = make_float4(j == 0 ? 1.f : 0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    for (int gi = 0; gi < ng; gi++) {
        if (!STAGED && gi % kGateChunk == 0) stage_gates(s_gates, gates + gi, min(kGateChunk, ng - gi));   // one latency per 32 gates
        const TileGate& g = STAGED ? gs[gi] : s_gates[gi % kGateChunk];
        const int kind = g.kind, k = g.k;
        if (kind == 0) {
            if (k == 1) tile_dense<1, false, STAGED>(smem, n, g, m_op);
            else if (k == 2) tile_dense<2, false, STAGED>(smem, n, g, m_op);
            else if (KMAX == 4 && k == 3) tile_dense<3, false, STAGED>(smem, n, g, m_op);
            else if (KMAX == 4) tile_dense<4, false, STAGED>(smem, n, g, m_op);
        } else if (kind == 1) {
            tile_diag<NoOff, false, STAGED>(smem, n, n, g, m_op, 0, NoOff{}, 0);
        } else {
            if (k == 1) tile_monomial<1, false, STAGED>(smem, n, g, p_op);
            else if (k == 2) tile_monomial<2, false, STAGED>(smem, n, g, p_op);
            else if (KMAX == 4 && k == 3) tile_monomial<3, false, STAGED>(smem, n, g, p_op);
            else if (KMAX == 4) tile_monomial<4, false, STAGED>(smem, n, g, p_op);
        }
        __syncthreads();
    }
    for (int j = threadIdx.x; j < nt; j += blockDim.x) {
        const double2 v = store_c128(f4c(smem[j]));
        psi[j] = v;
        const cff x = load_c128(v);
        ffacc a;
        acc_first(a, x.rh, x.rl, x.rh, x.rl);
        acc_add(a, x.ih, x.il, x.ih, x.il);
        const ff r = acc_done(a);
        const double pj = ff2d(r.h, r.l);   // prob_at's value for this amplitude
        probs[j] = pj;
        sprob[j] = pj;
    }
    __syncthreads();
    if (shots <= 0) {
        small_run_done(done, ticket, times);
        return;
    }
    __shared__ SmallCdf s_cdf;
    small_shots(sprob, nt, reinterpret_cast<double*>(smem) /* the tile is no longer needed */, s_cdf, threadIdx.x, blockDim.x, shots,
                seed, samples);
    small_run_done(done, ticket, times);
}

template <int KMAX, bool STAGED>
__global__ void __launch_bounds__(512) k_small_run(double2* __restrict__ psi, int n, const TileGate* __restrict__ gates,
                                                   int ng, const float4* __restrict__ mats, int n_mats,
                                                   const int32_t* __restrict__ perms, int n_perms,
                                                   double* __restrict__ probs, int64_t shots, uint64_t seed,
                                                   int64_t* __restrict__ samples, volatile int64_t* done, int64_t ticket,
                                                   int64_t* times) {
    small_run<KMAX, STAGED>(psi, n, gates, ng, mats, n_mats, perms, n_perms, probs, shots, seed, samples, done, ticket, times);
}

// A short plan (a GHZ circuit on 10 qubits takes 2.6 KB) travels in the kernel's parameters, which saves
// the round trip to host memory.
struct alignas(16) SmallInline {
    char bytes[3584];   // gates, matrices, permutations
};
template <int KMAX>
__global__ void __launch_bounds__(512) k_small_run_inline(double2* __restrict__ psi, int n, const __grid_constant__ SmallInline plan,
                                                          int ng, int n_mats, int n_perms, double* __restrict__ probs,
                                                          int64_t shots, uint64_t seed, int64_t* __restrict__ samples,
                                                          volatile int64_t* done, int64_t ticket, int64_t* times) {
    const char* p = plan.bytes;
    const TileGate* gates = reinterpret_cast<const TileGate*>(p);
    const float4* mats = reinterpret_cast<const float4*>(p + (size_t)ng * sizeof(TileGate));
    const int32_t* perms = reinterpret_cast<const int32_t*>(mats + n_mats);
    small_run<KMAX, true>(psi, n, gates, ng, mats, n_mats, perms, n_perms, probs, shots, seed, samples, done, ticket, times);
}

// The same for states of 2^11 and 2^12: a cluster of 4 or 8 CTAs holds 2^9 amplitudes each, so that the
// gates' float-float arithmetic, which bounds the one-CTA kernel (1.6 us a gate at 12 qubits), runs on
// as many SMs.  The plan is the sweeps bs_evolve would run for tiles of 2^9; between sweeps every CTA
// gathers its next tile from the others' shared memory (two tiles by turns, one cluster barrier a
// sweep).  At the end every CTA gets all probabilities and draws its share of the shots.
template <int KMAX, bool STAGED>
__global__ void __launch_bounds__(256) k_small_cluster(double2* __restrict__ psi, int n, const SmallSweep* __restrict__ sweeps,
                                                       int ns, const TileGate* __restrict__ gates, int ng,
                                                       const float4* __restrict__ mats, int n_mats,
                                                       const int32_t* __restrict__ perms, int n_perms,
                                                       double* __restrict__ probs, int64_t shots, uint64_t seed,
                                                       int64_t* __restrict__ samples, volatile int64_t* done, int64_t ticket,
                                                       int64_t* times) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr int T = kSmallTileBits, L = 5, nt = 1 << T;
    const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks(), rb = n - T, dim = 1 << n;
    const int tid = threadIdx.x;
    if (times && rank == 0 && tid == 0) times[0] = globaltimer_ns();
    extern __shared__ float4 smem[];
    __shared__ int64_t s_off[1 << (T - L)];
    __shared__ SmallCdf s_cdf;
    float4* tile0 = smem;                                         // two tiles, taken by turns
    double* sprob = reinterpret_cast<double*>(smem + 2 * nt);     // all probabilities
    double* scan = sprob + dim;                                   // two arrays for the sampler
    float4* ms = reinterpret_cast<float4*>(scan + 2 * dim);
    TileGate* gs = reinterpret_cast<TileGate*>(ms + (STAGED ? n_mats : 0));
    int32_t* ps = reinterpret_cast<int32_t*>(gs + (STAGED ? ng : 0));
    SmallSweep* ss = reinterpret_cast<SmallSweep*>(ps + (STAGED ? (n_perms + 3) / 4 * 4 : 0));
    if (STAGED) {
        // the plan may live in host-mapped memory: one round trip for all of it
        for (int j = tid; j < n_mats; j += blockDim.x) ms[j] = mats[j];
        stage_words(gs, gates, ng * (int)(sizeof(TileGate) / 4));
        for (int j = tid; j < n_perms; j += blockDim.x) ps[j] = perms[j];
        stage_words(ss, sweeps, ns * (int)(sizeof(SmallSweep) / 4));
    }
    const float4* m_op = STAGED ? ms : mats;
    const int32_t* p_op = STAGED ? ps : perms;
    const TileGate* g_op = STAGED ? gs : gates;
    const SmallSweep* w_op = STAGED ? ss : sweeps;
    cluster.sync();   // every CTA runs before another touches its shared memory; also orders the staging
    int64_t base = 0;
    for (int w = 0; w < ns; w++) {
        const SmallSweep sw = w_op[w];
        float4* cur = tile0 + (w & 1) * nt;
        base = 0;
        for (int q = 0; q < rb; q++) base |= (int64_t)((rank >> q) & 1) << sw.out[q];
        if (tid < (1 << (T - L))) {
            int64_t o = 0;
            for (int q = 0; q < T - L; q++) o |= (int64_t)((tid >> q) & 1) << sw.hi[q];
            s_off[tid] = o;
        }
        if (w == 0) {
            for (int j = tid; j < nt; j += blockDim.x)
                cur[j] = make_float4(j == 0 && base == 0 ? 1.f : 0.f, 0.f, 0.f, 0.f);
            __syncthreads();
        } else {
            const SmallSweep pv = w_op[w - 1];
            cluster.sync();   // the previous sweep is done everywhere; also orders s_off
            for (int j = tid; j < nt; j += blockDim.x) {
                const int64_t g = base | s_off[j >> L];
                int pj = j & ((1 << L) - 1), pr = 0;
                for (int q = 0; q < T - L; q++) pj |= (int)((g >> pv.hi[q]) & 1) << (L + q);
                for (int q = 0; q < rb; q++) pr |= (int)((g >> pv.out[q]) & 1) << q;
                // through complex128, as a sweep's store and the next one's load: the same values
                cur[j] = c4f(load_c128(store_c128(f4c(cluster.map_shared_rank(tile0 + ((w - 1) & 1) * nt, pr)[pj]))));
            }
            __syncthreads();
        }
        for (int gi = sw.g0; gi < sw.g0 + sw.ng; gi++) {
            const TileGate& g = g_op[gi];
            if ((base & (int64_t)g.gc_mask) != (int64_t)g.gc_val) continue;   // uniform in the CTA
            const int kind = g.kind, k = g.k;
            if (kind == 0) {
                if (k == 1) tile_dense<1, false, STAGED>(cur, T, g, m_op);
                else if (k == 2) tile_dense<2, false, STAGED>(cur, T, g, m_op);
                else if (KMAX == 4 && k == 3) tile_dense<3, false, STAGED>(cur, T, g, m_op);
                else if (KMAX == 4) tile_dense<4, false, STAGED>(cur, T, g, m_op);
            } else if (kind == 1) {
                tile_diag<const int64_t*, false, STAGED>(cur, T, L, g, m_op, base, s_off, 0);
            } else {
                if (k == 1) tile_monomial<1, false, STAGED>(cur, T, g, p_op);
                else if (k == 2) tile_monomial<2, false, STAGED>(cur, T, g, p_op);
                else if (KMAX == 4 && k == 3) tile_monomial<3, false, STAGED>(cur, T, g, p_op);
                else if (KMAX == 4) tile_monomial<4, false, STAGED>(cur, T, g, p_op);
            }
            __syncthreads();
        }
    }
    // the state and its probabilities, these to every CTA
    const float4* cur = tile0 + ((ns - 1) & 1) * nt;
    for (int j = tid; j < nt; j += blockDim.x) {
        const int64_t i = base | s_off[j >> L] | (int64_t)(j & ((1 << L) - 1));
        const double2 v = store_c128(f4c(cur[j]));
        psi[i] = v;
        const cff x = load_c128(v);
        ffacc a;
        acc_first(a, x.rh, x.rl, x.rh, x.rl);
        acc_add(a, x.ih, x.il, x.ih, x.il);
        const ff r = acc_done(a);
        const double pj = ff2d(r.h, r.l);   // prob_at's value for this amplitude
        probs[i] = pj;
        if (shots > 0)
            for (int r2 = 0; r2 < ranks; r2++) cluster.map_shared_rank(sprob, r2)[i] = pj;
    }
    cluster.sync();   // no CTA's shared memory is touched by another from here on
    if (shots > 0)
        small_shots(sprob, dim, scan, s_cdf, (int64_t)rank * blockDim.x + tid, (int64_t)ranks * blockDim.x, shots, seed, samples);
    if (!done) return;
    __threadfence_system();
    cluster.sync();   // every CTA's results are visible to the host
    if (rank == 0 && tid == 0) {
        if (times) times[1] = globaltimer_ns();
        __threadfence_system();
        *done = ticket;
    }
}

}  // namespace

int bs_small_pack(const bs_sim* s, const std::vector<Sweep>& sweeps, SmallPlan& out) {
    const int n = s->n;
    if (s->kind != BS_KIND_SV || s->precision != BS_PREC_C128 || n > 12) return BS_ERR_UNSUPPORTED;
    const int T = std::min(bs_sweep_tile_bits(s), n), L = BS_TILE_LOW_BITS;
    // One CTA has the whole state as its tile, whatever the sweeps.  Its launch is 3 to 4 us cheaper than a cluster's, which
    // takes 0.5 to 1 us less for a gate (11 qubits, a call of 1 gate 26 and 31 us, of 5 gates 35 both); only lists of one
    // sweep may take it, since a value is rounded to complex128 between two.
    const bool cluster = T == kSmallTileBits && n > T && (sweeps.size() > 1 || (!sweeps.empty() && sweeps[0].gates.size() > 4));
    std::vector<TileGate>& tg = out.tg;
    std::vector<float4>& mats = out.mats;
    std::vector<int32_t>& perms = out.perms;
    out.sweeps.clear();
    tg.clear();
    mats.clear();
    perms.clear();
    int kmax = 1;
    std::vector<HostGate> merged;
    for (const Sweep& sw : sweeps) {
        int local[64];           // tile position of an endian bit: its own, or (cluster) as in the sweep
        for (int b = 0; b < 64; b++) local[b] = cluster ? -1 : b;
        if (cluster) {
            if ((int)sw.hi_bits.size() != T - L) return BS_ERR_UNSUPPORTED;   // a gate no tile holds
            SmallSweep w{};
            for (int b = 0; b < L; b++) local[b] = b;
            for (int q = 0; q < T - L; q++) {
                local[sw.hi_bits[(size_t)q]] = L + q;
                w.hi[q] = (int8_t)sw.hi_bits[(size_t)q];
            }
            int r = 0;
            for (int b = L; b < n; b++) if (local[b] < 0) w.out[r++] = (int8_t)b;
            w.g0 = (int32_t)tg.size();
            out.sweeps.push_back(w);
        }
        merge_diagonals(sw.gates, merged);
        for (const HostGate& hg : merged) {
            if (hg.kind != 0 && hg.kind != 1 && hg.kind != 2) return BS_ERR_UNSUPPORTED;
            if (hg.kind != 1 && hg.k > BS_TILE_MAXK) return BS_ERR_UNSUPPORTED;
            TileGate t{};
            t.kind = hg.kind;
            t.k = hg.k;
            for (int b = 0; b < n; b++) {
                if (!((hg.cmask >> b) & 1ULL)) continue;
                const uint64_t v = (hg.cval >> b) & 1ULL;
                if (local[b] >= 0) { t.lc_mask |= 1u << local[b]; t.lc_val |= (uint32_t)v << local[b]; }
                else { t.gc_mask |= 1ULL << b; t.gc_val |= v << b; }
            }
            for (int q = 0; q < hg.k; q++) {
                t.gbit[q] = hg.ebit[q];
                if (q < BS_TILE_MAXK) t.tbit[q] = local[hg.ebit[q]];
                if (hg.kind != 1 && local[hg.ebit[q]] < 0) return BS_ERR_UNSUPPORTED;
            }
            t.mat_off = (int32_t)mats.size();
            t.perm_off = (int32_t)perms.size();
            if (hg.kind == 0) {
                for (int i = 0; i < (1 << (2 * hg.k)); i++) mats.push_back(to_cff(hg.mat[2 * i], hg.mat[2 * i + 1]));
                kmax = std::max(kmax, hg.k);
                if (hg.k == 1) t.npar = bs_class_2x2(hg);
            } else if (hg.kind == 1) {
                for (int i = 0; i < (1 << hg.k); i++) mats.push_back(to_cff(hg.mat[2 * i], hg.mat[2 * i + 1]));
            } else {
                perms.insert(perms.end(), hg.perm.begin(), hg.perm.end());
                kmax = std::max(kmax, hg.k);
                if (plain_x(hg)) t.npar = 1;
            }
            tg.push_back(t);
        }
        if (cluster) out.sweeps.back().ng = (int32_t)tg.size() - out.sweeps.back().g0;
    }
    out.kmax = kmax;
    return BS_OK;
}

int bs_small_launch(bs_sim* s, const SmallPlan& plan, double* dprobs, int64_t shots, uint64_t seed,
                    int64_t* dsamples, int64_t* done, int64_t ticket, const SmallIO* io) {
    const int n = s->n;
    const std::vector<TileGate>& tg = plan.tg;
    const std::vector<float4>& mats = plan.mats;
    const std::vector<int32_t>& perms = plan.perms;
    const int kmax = plan.kmax;
    auto al = [](int64_t x) { return (x + 255) & ~(int64_t)255; };
    const int64_t b_tg = al((int64_t)(tg.size() + 1) * (int64_t)sizeof(TileGate));
    const int64_t b_m = al((int64_t)(mats.size() + 1) * (int64_t)sizeof(float4));
    const int64_t b_p = al((int64_t)(perms.size() + 1) * (int64_t)sizeof(int32_t));
    const int64_t b_w = al((int64_t)(plan.sweeps.size() + 1) * (int64_t)sizeof(SmallSweep));
    const int64_t b_all = b_tg + b_m + b_p + b_w;
    char* dev = nullptr;
    int rc;
    const size_t b_inline = tg.size() * sizeof(TileGate) + mats.size() * sizeof(float4) + perms.size() * sizeof(int32_t);
    const bool inl = plan.sweeps.empty() && b_inline <= sizeof(SmallInline);
    auto write = [&](char* host) {
        if (!tg.empty()) std::memcpy(host, tg.data(), tg.size() * sizeof(TileGate));
        if (!mats.empty()) std::memcpy(host + b_tg, mats.data(), mats.size() * sizeof(float4));
        if (!perms.empty()) std::memcpy(host + b_tg + b_m, perms.data(), perms.size() * sizeof(int32_t));
        if (!plan.sweeps.empty()) std::memcpy(host + b_tg + b_m + b_p, plan.sweeps.data(), plan.sweeps.size() * sizeof(SmallSweep));
    };
    if (inl) {
        // in the kernel's parameters
    } else if (io && b_all <= (int64_t)io->plan_cap) {
        // the plan goes straight into host-mapped memory, which the kernel reads (the previous run on
        // this thread has completed, so nothing reads it any more); the launch orders these writes
        // before the kernel's reads
        write(io->hplan);
        std::atomic_thread_fence(std::memory_order_release);
        dev = io->dplan;
    } else {
        rc = bs_ensure_plan(s, b_all);
        if (rc) return rc;
        char* host = bs_stage(s, (size_t)b_all);
        if (!host) return bs_fail(s, BS_ERR_ALLOC, "pinned staging allocation");
        write(host);
        dev = (char*)s->plan_buf;
        rc = bs_cuda_check(s, cudaMemcpyAsync(dev, host, (size_t)b_all, cudaMemcpyHostToDevice, s->stream), "plan upload");
        bs_stage_done(s);
        if (rc) return rc;
    }
    if (!plan.sweeps.empty()) {
        const int dim = 1 << n;
        const size_t base = (size_t)2 * sizeof(float4) * ((size_t)1 << kSmallTileBits) + (size_t)3 * dim * sizeof(double);
        const size_t stage = mats.size() * sizeof(float4) + tg.size() * sizeof(TileGate) +
                             (perms.size() + 3) / 4 * 4 * sizeof(int32_t) + plan.sweeps.size() * sizeof(SmallSweep);
        constexpr size_t kClusterCap = 216 * 1024;
        const bool staged = base + stage <= kClusterCap;
        auto kern = kmax <= 2 ? (staged ? k_small_cluster<2, true> : k_small_cluster<2, false>)
                              : (staged ? k_small_cluster<4, true> : k_small_cluster<4, false>);
        static bool attr_set[64] = {false};
        if (!attr_set[s->device & 63]) {
            cudaFuncSetAttribute(k_small_cluster<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterCap);
            cudaFuncSetAttribute(k_small_cluster<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterCap);
            cudaFuncSetAttribute(k_small_cluster<4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterCap);
            cudaFuncSetAttribute(k_small_cluster<4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterCap);
            attr_set[s->device & 63] = true;
        }
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 1u << (n - kSmallTileBits);
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1u << (n - kSmallTileBits));
        cfg.blockDim = dim3(256);
        cfg.dynamicSmemBytes = staged ? base + stage : base;
        cfg.stream = s->stream;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, (double2*)s->state, n, (const SmallSweep*)(dev + b_tg + b_m + b_p),
                                                 (int)plan.sweeps.size(), (const TileGate*)dev, (int)tg.size(),
                                                 (const float4*)(dev + b_tg), (int)mats.size(), (const int32_t*)(dev + b_tg + b_m),
                                                 (int)perms.size(), dprobs, shots, seed, dsamples, (volatile int64_t*)done, ticket,
                                                 io ? io->dtimes : (int64_t*)nullptr);
        rc = bs_cuda_check(s, e, "small run");
        if (rc) return rc;
        s->stats.kernel_launches++;
        s->stats.sweeps++;
        s->stats.gates += (int64_t)tg.size();
        s->stats.bytes_moved += 16.0 * (double)dim;
        return bs_cuda_check(s, cudaGetLastError(), "small run");
    }
    // the tile (afterwards two arrays of the sampler, whole 32-element chunks), then the probabilities,
    // then (staged) the matrices and permutations
    const size_t base = std::max(((size_t)1 << n) * sizeof(float4), (size_t)2 * (((1 << n) + 31) / 32 * 32) * sizeof(double)) +
                        ((size_t)1 << n) * sizeof(double);
    const size_t stage = mats.size() * sizeof(float4) + tg.size() * sizeof(TileGate) + perms.size() * sizeof(int32_t) + 16;
    constexpr size_t kSmemCap = 160 * 1024;
    const bool staged = base + stage <= kSmemCap;
    const size_t smem = staged ? base + stage : base;
    const TileGate* d_tg = (const TileGate*)dev;
    const float4* d_m = (const float4*)(dev + b_tg);
    const int32_t* d_p = (const int32_t*)(dev + b_tg + b_m);
    static bool attr_set[64] = {false};
    if (!attr_set[s->device & 63]) {
        cudaFuncSetAttribute(k_small_run<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
        cudaFuncSetAttribute(k_small_run<4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
        cudaFuncSetAttribute(k_small_run<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
        cudaFuncSetAttribute(k_small_run<4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
        cudaFuncSetAttribute(k_small_run_inline<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
        cudaFuncSetAttribute(k_small_run_inline<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
        attr_set[s->device & 63] = true;
    }
    const int threads = std::min(512, std::max(128, (1 << n) / 2));
    if (inl) {
        SmallInline blob;
        char* p = blob.bytes;
        if (!tg.empty()) std::memcpy(p, tg.data(), tg.size() * sizeof(TileGate));
        p += tg.size() * sizeof(TileGate);
        if (!mats.empty()) std::memcpy(p, mats.data(), mats.size() * sizeof(float4));
        p += mats.size() * sizeof(float4);
        if (!perms.empty()) std::memcpy(p, perms.data(), perms.size() * sizeof(int32_t));
        auto k = kmax <= 2 ? k_small_run_inline<2> : k_small_run_inline<4>;
        k<<<1, threads, base + stage, s->stream>>>((double2*)s->state, n, blob, (int)tg.size(), (int)mats.size(), (int)perms.size(),
                                                   dprobs, shots, seed, dsamples, done, ticket, io ? io->dtimes : nullptr);
    } else {
    auto kern = kmax <= 2 ? (staged ? k_small_run<2, true> : k_small_run<2, false>)
                          : (staged ? k_small_run<4, true> : k_small_run<4, false>);
    kern<<<1, threads, smem, s->stream>>>((double2*)s->state, n, d_tg, (int)tg.size(), d_m, (int)mats.size(), d_p,
                                          (int)perms.size(), dprobs, shots, seed, dsamples, done, ticket,
                                          io ? io->dtimes : nullptr);
    }
    s->stats.kernel_launches++;
    s->stats.sweeps++;
    s->stats.gates += (int64_t)tg.size();
    s->stats.bytes_moved += 16.0 * (double)((int64_t)1 << n);
    return bs_cuda_check(s, cudaGetLastError(), "small run");
}
