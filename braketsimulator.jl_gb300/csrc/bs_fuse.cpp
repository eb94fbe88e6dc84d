// Gate fusion for the tensor-core tile path.
//
// Inside one tile sweep, runs of gates are folded into dense unitaries on 5
// tile bits.  A gate can join a block when its dense targets lie in the tile and
// its tile bits fit the block; bits outside the tile (controls, and target bits
// of diagonal gates) are constant within a CTA, so the block is built once per
// assignment of those "uniform" bits (at most 3 of them) and each CTA picks its
// variant.  The products are formed on the device in FP64 (k_tc_build) and applied to
// the tile as real 64x64 GEMMs on tcgen05 tensor cores, with both operands split
// into exact 8-bit bf16 digits (an Ozaki-style split) so that the result keeps
// float-float accuracy.  This replaces, for those gates, the per-gate amplitude
// loops of the reference (src/gate_kernels.jl:489-775, src/custom_gates.jl:364-416);
// the fused product itself has no counterpart there.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdlib>
#include <cstring>
#include "bs_internal.h"

namespace {

using cd = std::complex<double>;
constexpr int kMaxUniform = 3;

// cost of a gate on the float-float path, in units of one dense 1-qubit gate
double ff_cost(const HostGate& g) {
    if (g.kind == 0) return (double)(1 << g.k) / 2.0;
    if (g.kind == 2) return 0.25;
    return 0.3;
}

bool is_plain_cz(const HostGate& g) {
    return g.kind == 1 && g.k == 1 && g.mat.size() == 4 && g.mat[0] == 1.0 && g.mat[1] == 0.0 && g.mat[2] == -1.0 &&
           g.mat[3] == 0.0 && __builtin_popcountll(g.cmask) == 1 && g.cval == g.cmask;
}

// Left-multiply the 32x32 block matrix U (row r, column c at U[r * 32 + c]) by a canonical gate.
// pos[e]: block bit of endian bit e, or -1 for a uniform bit whose value is (uval >> e) & 1.
void apply_block(const HostGate& g, const int* pos, uint64_t uval, cd* U) {
    // controls: in-block ones become a row-index condition, uniform ones decide whether the gate acts
    uint32_t cm = 0, cv = 0;
    uint64_t rest = g.cmask;
    while (rest) {
        const int e = __builtin_ctzll(rest);
        rest &= rest - 1;
        const uint64_t want = (g.cval >> e) & 1ULL;
        if (pos[e] < 0) {
            if (((uval >> e) & 1ULL) != want) return;
        } else {
            cm |= 1u << pos[e];
            cv |= (uint32_t)want << pos[e];
        }
    }
    const int D = 1 << g.k;
    if (g.kind == 1) {
        // diagonal: target bits may be uniform (constant over the block); row r scales by d[index(r)]
        for (uint32_t r = 0; r < 32; r++) {
            if ((r & cm) != cv) continue;
            int di = 0;
            for (int q = 0; q < g.k; q++) {
                const int e = g.ebit[q];
                const int bit = pos[e] >= 0 ? (int)((r >> pos[e]) & 1u) : (int)((uval >> e) & 1ULL);
                di |= bit << q;
            }
            const double dr = g.mat[2 * di], dim = g.mat[2 * di + 1];
            for (int c = 0; c < 32; c++) {
                const double ur = U[r * 32 + c].real(), ui = U[r * 32 + c].imag();
                U[r * 32 + c] = cd(dr * ur - dim * ui, dr * ui + dim * ur);
            }
        }
        return;
    }
    uint32_t off[32];
    uint32_t tmask = 0;
    for (int q = 0; q < g.k; q++) tmask |= 1u << pos[g.ebit[q]];
    for (int c = 0; c < D; c++) {
        uint32_t j = 0;
        for (int q = 0; q < g.k; q++) if ((c >> q) & 1) j |= 1u << pos[g.ebit[q]];
        off[c] = j;
    }
    static const cd ipow[4] = {cd(1, 0), cd(0, 1), cd(-1, 0), cd(0, -1)};
    cd x[32], y[32];
    for (uint32_t i = 0; i < 32; i++) {
        if (i & tmask) continue;
        if ((i & cm) != cv) continue;
        for (int col = 0; col < 32; col++) {
            for (int c = 0; c < D; c++) x[c] = U[(i | off[c]) * 32 + col];
            if (g.kind == 0) {
                // plain real arithmetic (std::complex products go through a NaN-checking library call)
                for (int r = 0; r < D; r++) {
                    double sr = 0, si = 0;
                    const double* mr = g.mat.data() + 2 * r * D;
                    for (int c = 0; c < D; c++) {
                        const double ar = mr[2 * c], ai = mr[2 * c + 1], xr = x[c].real(), xi = x[c].imag();
                        sr += ar * xr - ai * xi;
                        si += ar * xi + ai * xr;
                    }
                    y[r] = cd(sr, si);
                }
            } else {
                for (int c = 0; c < D; c++) y[g.perm[2 * c]] = ipow[g.perm[2 * c + 1] & 3] * x[c];
            }
            for (int r = 0; r < D; r++) U[(i | off[r]) * 32 + col] = y[r];
        }
    }
}

// What the tensor-core fusion needs to know of a gate.
struct FuseGate {
    uint64_t bits = 0;    // tile bits it touches
    uint64_t ub = 0;      // bits outside the tile it depends on (constant in a CTA)
    uint64_t hard = 0;    // bits it moves amplitudes along
    double cost = 0;
    bool fusable = false;
    bool wide = false;    // 3 or more moved bits: no float-float path in the tensor-core sweep
};

}  // namespace

// Greedy over the gates in order.  A block starts at the first gate left and grows bit by bit: of all
// bit sets that add the bits of one more gate, the one whose block takes the most work (gates that
// commute with everything they leave behind, out-of-tile bits at most kMaxUniform).  Blocks of one layer
// of single-qubit gates therefore fill up with gates on other bits, and follow the light cone into the
// next layers; fusing only blocks that share a bit left 18 single dense gates beside 30 fused unitaries
// in the 28-qubit dense circuit, each of which costs 3/4 of a fused unitary (evolve 84.6 -> 60.1 ms).  Returns that cost in fused unitaries.
double bs_fuse_tc(const std::vector<const HostGate*>& in, const int* local, int T, double threshold, std::vector<HostGate>* out) {
    if (out) out->clear();
    double total = 0;
    const size_t G = in.size();
    std::vector<FuseGate> info(G);
    for (size_t i = 0; i < G; i++) {
        const HostGate& g = *in[i];
        FuseGate& f = info[i];
        if (g.kind == 5) continue;
        f.fusable = g.kind <= 2 && g.k <= 5;
        for (int q = 0; q < g.k; q++) {
            const int e = g.ebit[q];
            if (g.kind != 1) f.hard |= 1ULL << e;
            if (local[e] >= 0) f.bits |= 1ULL << e;
            else if (g.kind == 1) f.ub |= 1ULL << e;
            else f.fusable = false;
        }
        for (uint64_t r = g.cmask; r; r &= r - 1) {
            const int e = __builtin_ctzll(r);
            (local[e] >= 0 ? f.bits : f.ub) |= 1ULL << e;
        }
        if (__builtin_popcountll(f.bits) > 5 || __builtin_popcountll(f.ub) > kMaxUniform || f.bits == 0) f.fusable = false;
        f.wide = g.kind != 1 && g.k >= 3;
        // real and real/imaginary 2x2 matrices take half the products on the float-float path
        f.cost = is_plain_cz(g) ? 0.1 : (g.kind == 0 && g.k == 1 && bs_class_2x2(g)) ? 0.6 : ff_cost(g);
    }
    auto emit = [&](uint64_t bits, uint64_t ubits, const std::vector<int>& idx, double cost) {
        int ndense = 0;
        bool wide = false;   // 3- and 4-target gates always fuse: the tensor-core sweep has no float-float path for them
        for (int i : idx) {
            ndense += in[(size_t)i]->kind == 0;
            wide = wide || info[(size_t)i].wide;
        }
        if (!wide && (cost <= threshold || ndense == 0)) {
            if (out) for (int i : idx) out->push_back(*in[(size_t)i]);
            total += 0.75 * cost;
            return;
        }
        total += 1;
        if (!out) return;
        // block bits ascending by tile position, padded to 5 with other tile bits (high ones first, so that
        // the low contiguous bits stay column bits of the GEMM where possible)
        std::vector<int> eb;
        for (int e = 0; e < 64; e++) if ((bits >> e) & 1ULL) eb.push_back(e);
        std::vector<int> tile_e(T, -1);
        for (int e = 0; e < 64; e++) if (local[e] >= 0 && local[e] < T) tile_e[local[e]] = e;
        for (int p = T - 1; p >= 0 && (int)eb.size() < 5; p--) {
            int e = tile_e[p];
            if (e >= 0 && !((bits >> e) & 1ULL)) eb.push_back(e);
        }
        std::sort(eb.begin(), eb.end(), [&](int a, int c) { return local[a] < local[c]; });
        HostGate f;
        f.kind = 4;
        f.k = 5;
        for (int q = 0; q < 5; q++) f.ebit[q] = eb[(size_t)q];
        for (int e = 0; e < 64; e++) if ((ubits >> e) & 1ULL) f.ubits.push_back(e);
        f.perm = idx;
        out->push_back(std::move(f));
    };
    std::vector<char> done(G, 0);
    std::vector<int> left, take;
    std::vector<uint64_t> tried;
    for (size_t s0 = 0; s0 < G;) {
        if (in[s0]->kind == 5) {   // commutes with nothing
            if (out) out->push_back(*in[s0]);
            s0++;
            continue;
        }
        size_t s1 = s0;
        while (s1 < G && in[s1]->kind != 5) s1++;
        size_t first = s0;
        while (true) {
            while (first < s1 && done[first]) first++;
            if (first == s1) break;
            if (!info[first].fusable) {
                if (out) out->push_back(*in[first]);
                total += 0.75 * info[first].cost;
                done[first] = 1;
                continue;
            }
            left.clear();   // the gates a block may draw from
            for (size_t i = first; i < s1 && left.size() < 96; i++) if (!done[i]) left.push_back((int)i);
            // the work a block on these bits takes, its gates into `take` when asked for
            auto scan = [&](uint64_t bits, uint64_t* ubits, bool collect) {
                uint64_t left_hard = 0, left_any = 0, u = 0;
                double cost = 0;
                for (int i : left) {
                    const FuseGate& f = info[(size_t)i];
                    const uint64_t all = f.bits | f.ub | f.hard;
                    if (f.fusable && !(f.bits & ~bits) && !(f.hard & left_any) && !(all & left_hard) &&
                        __builtin_popcountll(u | f.ub) <= kMaxUniform) {
                        u |= f.ub;
                        cost += f.cost;
                        if (collect) take.push_back(i);
                    } else {
                        left_hard |= f.hard;
                        left_any |= all;
                        if (!(bits & ~left_hard)) break;   // every block bit is held back
                    }
                }
                if (ubits) *ubits = u;
                return cost;
            };
            uint64_t bits = info[first].bits;
            while (__builtin_popcountll(bits) < 5) {
                tried.clear();
                uint64_t best = 0;
                double best_cost = -1;
                for (int i : left) {
                    const FuseGate& f = info[(size_t)i];
                    const uint64_t nb = bits | f.bits;
                    if (!f.fusable || nb == bits || __builtin_popcountll(nb) > 5) continue;
                    if (std::find(tried.begin(), tried.end(), nb) != tried.end()) continue;
                    tried.push_back(nb);
                    const double c = scan(nb, nullptr, false) / (double)__builtin_popcountll(nb);   // work per bit
                    if (c > best_cost + 1e-9) { best_cost = c; best = nb; }
                }
                if (!best) break;
                bits = best;
            }
            take.clear();
            uint64_t ubits = 0;
            const double cost = scan(bits, &ubits, true);
            for (int i : take) done[(size_t)i] = 1;
            emit(bits, ubits, take, cost);
        }
        s0 = s1;
    }
    return total;
}

// Fusion for the sweeps that run on the CUDA cores (float-float and complex64 tile kernels): runs of
// gates whose tile bits (targets and controls) fit in maxk bits become one dense maxk-bit gate when
// that is cheaper, counting one shared-memory pass of the tile (pass, in units of a dense 1-qubit
// gate's arithmetic) per gate applied.  The kernels apply every gate as one pass, so fusing two
// 1-qubit gates on different bits into a 4x4 keeps the arithmetic and halves the passes.  Gates with
// bits outside the tile, 3+-bit gates and channels stay as they are and close the blocks they touch.
void bs_fuse_small(const std::vector<HostGate>& in, const int* local, double pass, int maxk, std::vector<HostGate>& out) {
    out.clear();
    struct SBlock {
        uint64_t bits = 0;
        std::vector<int> idx;
        double cost = 0;
    };
    std::vector<SBlock> open;
    auto gate_bits = [&](const HostGate& g, bool& in_tile) {
        uint64_t b = g.cmask;
        for (int q = 0; q < g.k; q++) b |= 1ULL << g.ebit[q];
        in_tile = true;
        for (uint64_t r = b; r; r &= r - 1)
            if (local[__builtin_ctzll(r)] < 0) in_tile = false;
        return b;
    };
    auto emit = [&](SBlock& b) {
        const int k = __builtin_popcountll(b.bits);
        if (b.idx.size() < 2 || pass + (double)(1 << k) / 2.0 >= b.cost) {
            for (int i : b.idx) out.push_back(in[(size_t)i]);
            return;
        }
        // the block's bits take block positions 0..k-1; the 32x32 product then holds U (x) I
        int pos[64];
        for (int e = 0; e < 64; e++) pos[e] = -1;
        HostGate f;
        f.kind = 0;
        f.k = k;
        int q = 0;
        for (int e = 0; e < 64; e++)
            if ((b.bits >> e) & 1ULL) { pos[e] = q; f.ebit[q] = e; q++; }
        std::vector<cd> U(32 * 32, cd(0, 0));
        for (int r = 0; r < 32; r++) U[(size_t)r * 33] = 1;
        for (int i : b.idx) apply_block(in[(size_t)i], pos, 0, U.data());
        const int D = 1 << k;
        f.mat.assign((size_t)2 * D * D, 0.0);
        for (int r = 0; r < D; r++)
            for (int c = 0; c < D; c++) {
                f.mat[(size_t)2 * (r * D + c)] = U[(size_t)r * 32 + c].real();
                f.mat[(size_t)2 * (r * D + c) + 1] = U[(size_t)r * 32 + c].imag();
            }
        out.push_back(std::move(f));
    };
    auto close_touching = [&](uint64_t bits) {
        for (size_t j = 0; j < open.size();) {
            if (open[j].bits & bits) {
                emit(open[j]);
                open.erase(open.begin() + (long)j);
            } else {
                j++;
            }
        }
    };
    for (size_t i = 0; i < in.size(); i++) {
        const HostGate& g = in[i];
        if (g.kind == 5) {   // a reference-rule channel commutes with nothing
            for (SBlock& b : open) emit(b);
            open.clear();
            out.push_back(g);
            continue;
        }
        bool in_tile = false;
        const uint64_t bits = gate_bits(g, in_tile);
        const bool fusable = g.kind <= 2 && in_tile && bits && __builtin_popcountll(bits) <= maxk;
        if (!fusable) {
            close_touching(bits);
            out.push_back(g);
            continue;
        }
        uint64_t uni = bits;
        for (const SBlock& b : open) if (b.bits & bits) uni |= b.bits;
        if (__builtin_popcountll(uni) > maxk) {
            close_touching(bits);
            uni = bits;
        }
        SBlock nb;
        nb.bits = uni;
        // merge the intersecting blocks (pairwise disjoint, so their gates commute), then the gate
        for (size_t j = 0; j < open.size();) {
            if (open[j].bits & bits) {
                nb.idx.insert(nb.idx.end(), open[j].idx.begin(), open[j].idx.end());
                nb.cost += open[j].cost;
                open.erase(open.begin() + (long)j);
            } else {
                j++;
            }
        }
        std::sort(nb.idx.begin(), nb.idx.end());
        nb.idx.push_back((int)i);
        nb.cost += is_plain_cz(g) ? 0.1 : pass + ff_cost(g);   // CZs share one parity pass anyway
        open.push_back(std::move(nb));
    }
    for (SBlock& b : open) emit(b);
}

namespace {

// What a register block needs to know of a gate.
struct RegGate {
    enum Kind { kOneBit, kSwap, kDiag, kOther } kind = kOther;
    uint64_t hard = 0;    // bits it moves amplitudes along: must be block bits
    uint64_t soft = 0;    // controls and diagonal bits: read from the index anywhere
};

bool plain_swap(const HostGate& g) {
    return g.kind == 2 && g.k == 2 && g.cmask == 0 && g.perm.size() == 8 && g.perm[0] == 0 && g.perm[1] == 0 &&
           g.perm[2] == 2 && g.perm[3] == 0 && g.perm[4] == 1 && g.perm[5] == 0 && g.perm[6] == 3 && g.perm[7] == 0;
}
bool sign_only(const HostGate& g) {   // Z on one bit, any controls
    return g.kind == 1 && g.k == 1 && g.mat[0] == 1.0 && g.mat[1] == 0.0 && g.mat[2] == -1.0 && g.mat[3] == 0.0;
}

RegGate reg_gate(const HostGate& g) {
    RegGate r;
    uint64_t t = 0;
    for (int q = 0; q < g.k; q++) t |= 1ULL << g.ebit[q];
    if (g.kind == 1) {
        const int nb = __builtin_popcountll(t | g.cmask);
        if (nb <= 2 || sign_only(g)) {
            r.kind = RegGate::kDiag;
            r.soft = t | g.cmask;
        } else {
            r.soft = t | g.cmask;
        }
    } else {
        r.hard = t;
        r.soft = g.cmask;
        if (g.kind <= 2 && g.k == 1) r.kind = RegGate::kOneBit;
        else if (plain_swap(g)) r.kind = RegGate::kSwap;
    }
    return r;
}

void matrix_2x2(const HostGate& g, cd* m) {
    for (int i = 0; i < 4; i++) m[i] = 0;
    if (g.kind == 0) {
        for (int i = 0; i < 4; i++) m[i] = cd(g.mat[2 * i], g.mat[2 * i + 1]);
    } else if (g.kind == 1) {
        m[0] = cd(g.mat[0], g.mat[1]);
        m[3] = cd(g.mat[2], g.mat[3]);
    } else {
        static const cd ipow[4] = {cd(1, 0), cd(0, 1), cd(-1, 0), cd(0, -1)};
        for (int c = 0; c < 2; c++) m[g.perm[2 * c] * 2 + c] = ipow[g.perm[2 * c + 1] & 3];
    }
}

bool complex_2x2(const cd* m) {
    const bool dr = m[0].imag() == 0.0 && m[3].imag() == 0.0;
    return !(dr && m[1].imag() == 0.0 && m[2].imag() == 0.0) && !(dr && m[1].real() == 0.0 && m[2].real() == 0.0) &&
           !(m[1] == 0.0 && m[2] == 0.0);
}

// The gates of one block in order, turned into operations.  One-bit gates without controls that meet on
// the same bit are multiplied out in FP64 where that saves work; diagonal gates fold into one table while they commute back
// to it; signs with the same outside controls fold into one mask.
struct BlockBuilder {
    int pos[64];                      // block bit of an endian bit, or -1
    const int* local;
    std::vector<RegOp> ops;
    std::vector<std::vector<cd>> tab; // per op (type 5): its table, variant-major
    std::vector<cd> mats;             // per op (types 0..4): 2x2 in FP64
    std::vector<uint64_t> hard, soft; // per op, endian bits

    void push(const RegOp& o, const cd* m, std::vector<cd> t, uint64_t h, uint64_t s) {
        ops.push_back(o);
        for (int i = 0; i < 4; i++) mats.push_back(m ? m[i] : cd(0, 0));
        tab.push_back(std::move(t));
        hard.push_back(h);
        soft.push_back(s);
    }
    void outside_controls(RegOp& o, uint64_t cmask, uint64_t cval) const {
        for (uint64_t r = cmask; r; r &= r - 1) {
            const int e = __builtin_ctzll(r);
            if (pos[e] >= 0) continue;
            const uint32_t v = (uint32_t)((cval >> e) & 1ULL);
            if (local[e] >= 0) { o.lc_mask |= (uint16_t)(1u << local[e]); o.lc_val |= (uint16_t)(v << local[e]); }
            else { o.gc_mask |= 1ULL << e; o.gc_val |= (uint64_t)v << e; }
        }
    }
    // pairs of block bit b whose pattern meets the controls inside the block
    uint32_t pair_mask(int b, uint64_t cmask, uint64_t cval) const {
        uint32_t m = 0;
        for (uint32_t p = 0; p < 16; p++) {
            const uint32_t c = ((p >> b) << (b + 1)) | (p & ((1u << b) - 1u));
            bool ok = true;
            for (uint64_t r = cmask; r; r &= r - 1) {
                const int e = __builtin_ctzll(r);
                if (pos[e] >= 0 && ((c >> pos[e]) & 1u) != (uint32_t)((cval >> e) & 1ULL)) ok = false;
            }
            if (ok) m |= 1u << p;
        }
        return m;
    }
    void one_bit(const HostGate& g) {
        const int e = g.ebit[0], b = pos[e];
        const uint64_t h = 1ULL << e;
        cd m[4];
        matrix_2x2(g, m);
        if (!g.cmask) {
            // the last operation on this bit, if it is a one-bit gate without controls
            for (int i = (int)ops.size() - 1; i >= 0; i--) {
                if (!((hard[(size_t)i] | soft[(size_t)i]) & h)) continue;
                if (hard[(size_t)i] == h && soft[(size_t)i] == 0 && ops[(size_t)i].type <= 3) {
                    cd* a = &mats[4 * (size_t)i];
                    const cd r[4] = {m[0] * a[0] + m[1] * a[2], m[0] * a[1] + m[1] * a[3], m[2] * a[0] + m[3] * a[2],
                                     m[2] * a[1] + m[3] * a[3]};
                    // two gates of the cheap classes stay two where their product is a full complex matrix
                    // (as many instructions, and their shape can be kept)
                    if (complex_2x2(r) && !complex_2x2(a) && !complex_2x2(m)) break;
                    for (int q = 0; q < 4; q++) a[q] = r[q];
                    return;
                }
                break;
            }
        }
        RegOp o{};
        o.bit = (uint8_t)b;
        o.mask = pair_mask(b, g.cmask, g.cval);
        outside_controls(o, g.cmask, g.cval);
        push(o, m, {}, h, g.cmask);
    }
    void diag(const HostGate& g) {
        uint64_t bits = g.cmask;
        for (int q = 0; q < g.k; q++) bits |= 1ULL << g.ebit[q];
        if (sign_only(g)) {
            uint32_t mask = 0;
            for (uint32_t c = 0; c < 32; c++) {
                bool ok = true;
                for (uint64_t r = bits; r; r &= r - 1) {
                    const int e = __builtin_ctzll(r);
                    const uint32_t want = ((g.cmask >> e) & 1ULL) ? (uint32_t)((g.cval >> e) & 1ULL) : 1u;
                    if (pos[e] >= 0 && ((c >> pos[e]) & 1u) != want) ok = false;
                }
                if (ok) mask |= 1u << c;
            }
            RegOp o{};
            o.type = 6;
            o.mask = mask;
            outside_controls(o, bits, g.cval | (bits & ~g.cmask));
            for (int i = (int)ops.size() - 1; i >= 0 && !(hard[(size_t)i] & bits); i--) {
                RegOp& p = ops[(size_t)i];
                if (p.type == 6 && p.lc_mask == o.lc_mask && p.lc_val == o.lc_val && p.gc_mask == o.gc_mask && p.gc_val == o.gc_val) {
                    p.mask ^= mask;
                    soft[(size_t)i] |= bits;
                    return;
                }
            }
            push(o, nullptr, {}, 0, bits);
            return;
        }
        uint64_t out = 0;
        for (uint64_t r = bits; r; r &= r - 1) if (pos[__builtin_ctzll(r)] < 0) out |= r & (0 - r);
        // back to a table this gate commutes with, if the bits outside the block stay at most two
        int at = -1;
        for (int i = (int)ops.size() - 1; i >= 0 && !(hard[(size_t)i] & bits); i--)
            if (ops[(size_t)i].type == 5 && __builtin_popcountll(outside(i) | out) <= 2) { at = i; break; }
        if (at < 0 && g.k == 1 && !g.cmask && pos[g.ebit[0]] >= 0) {   // Rz, S, T, ... on a block bit
            one_bit(g);
            return;
        }
        if (at < 0) {
            RegOp o{};
            o.type = 5;
            push(o, nullptr, std::vector<cd>(32, cd(1, 0)), 0, 0);
            at = (int)ops.size() - 1;
        }
        widen(at, out);
        RegOp& o = ops[(size_t)at];
        soft[(size_t)at] |= bits;
        for (int v = 0; v < (1 << o.nu); v++)
            for (uint32_t c = 0; c < 32; c++) {
                auto bit_of = [&](int e) -> int {
                    if (pos[e] >= 0) return (int)((c >> pos[e]) & 1u);
                    for (int u = 0; u < o.nu; u++) if (o.ub[u] == code(e)) return (v >> u) & 1;
                    return 0;
                };
                bool ok = true;
                for (uint64_t r = g.cmask; r; r &= r - 1) {
                    const int e = __builtin_ctzll(r);
                    if (bit_of(e) != (int)((g.cval >> e) & 1ULL)) ok = false;
                }
                if (!ok) continue;
                int di = 0;
                for (int q = 0; q < g.k; q++) di |= bit_of(g.ebit[q]) << q;
                tab[(size_t)at][(size_t)v * 32 + c] *= cd(g.mat[2 * di], g.mat[2 * di + 1]);
            }
    }
    int code(int e) const { return local[e] >= 0 ? local[e] : 64 + e; }
    uint64_t outside(int i) const {
        uint64_t m = 0;
        for (int e = 0; e < 64; e++)
            for (int u = 0; u < ops[(size_t)i].nu; u++) if (pos[e] < 0 && code(e) == ops[(size_t)i].ub[u]) m |= 1ULL << e;
        return m;
    }
    void widen(int i, uint64_t out) {
        for (uint64_t r = out & ~outside(i); r; r &= r - 1) {
            RegOp& o = ops[(size_t)i];
            o.ub[o.nu] = (int16_t)code(__builtin_ctzll(r));
            std::vector<cd>& t = tab[(size_t)i];
            t.insert(t.end(), t.begin(), t.begin() + (long)(32 << o.nu));
            o.nu++;
        }
    }
    // FP32 matrix entries are off by up to 2^-25, equal gates (every H) by the same amount, and after a few
    // hundred gates that is the larger part of a complex64 state's error (18 qubits, 30 layers: 1e-6 of
    // the expectation values from rounded matrices, 2e-7 from rounded states).  So a common factor near
    // 1 is chosen whose rounded entries keep the matrix's shape, which works where few entries differ
    // (real, real/imaginary and diagonal matrices); the size error that leaves (`drift`) goes into the
    // next factor, so it does not add up.  A table's 32 entries have no such factor and carry low words
    // (22-qubit gradient, 30 inputs: error of the energy 7.0e-8 -> 5.5e-8 of the Hamiltonian's norm, of the
    // gradient 4.7e-7 -> 4.0e-7, before register blocks 6.7e-8 and 5.7e-7; 6.84 -> 7.29 ms).
    void finish(RegBlock& b, std::vector<float4>& tabs, double& drift) {
        for (size_t i = 0; i < ops.size(); i++) {
            RegOp o = ops[i];
            const cd* m = &mats[4 * i];
            const bool whole = !o.lc_mask && !o.gc_mask && o.mask == 0xffffu;
            if (o.type == 5) {
                o.tab = (int32_t)tabs.size();
                for (const cd& e : tab[i]) {
                    const float re = (float)e.real(), im = (float)e.imag();
                    tabs.push_back(make_float4(re, re, -im, im));
                    const float rl = (float)(e.real() - (double)re), il = (float)(e.imag() - (double)im);
                    tabs.push_back(make_float4(rl, rl, -il, il));
                }
            } else if (o.type != 6) {
                double e[8], n2 = 0;
                for (int q = 0; q < 4; q++) { e[2 * q] = m[q].real(); e[2 * q + 1] = m[q].imag(); }
                for (double x : e) n2 += x * x;
                const bool x = m[0] == 0.0 && m[3] == 0.0 && m[1] == 1.0 && m[2] == 1.0;
                const bool dr = e[1] == 0.0 && e[7] == 0.0;
                if (x) o.type = 3;
                else if (o.mask != 0xffffu) o.type = 4;
                else if (dr && e[3] == 0.0 && e[5] == 0.0) o.type = 1;
                else if (dr && e[2] == 0.0 && e[4] == 0.0) o.type = 2;
                else if (e[2] == 0.0 && e[3] == 0.0 && e[4] == 0.0 && e[5] == 0.0) o.type = 7;
                else o.type = 0;
                double fix = 1.0;
                if (whole && !x && n2 > 0) {
                    double best = 0, best_fix = 1.0, best_drift = drift;
                    const double f0 = 1.0 / (1.0 + drift);
                    for (int k = -8; k <= 8; k++) {
                        const double f = f0 * (1.0 + k * 0x1p-26);
                        // R = rounded entries; its size against e, and its distance from e at that size
                        double r2 = 0, re = 0;
                        for (double v : e) { const double d = (double)(float)(v * f) - v; r2 += d * d; re += d * v; }
                        const double rel = re / n2;                          // size error, to first order
                        const double dn = drift + rel;
                        const double cost = r2 / n2 - rel * rel + dn * dn / 16.0;   // shape, and the size error carried on
                        if (k == -8 || cost < best) { best = cost; best_fix = f; best_drift = dn; }
                    }
                    fix = best_fix;
                    drift = best_drift;
                }
                for (int q = 0; q < 8; q++) o.m[q] = (float)(e[q] * fix);
            }
            b.ops.push_back(o);
        }
    }
};

}  // namespace

// Greedy, as the sweep planner: a block takes every gate, in order, that commutes with all the gates it
// leaves behind and whose moved bits fit into 5 block bits; diagonal gates and controls need no block bit.
void bs_block_c64(const std::vector<HostGate>& in, const int* local, int T, std::vector<RegItem>& items,
                  std::vector<RegBlock>& blocks, std::vector<float4>& tabs, double& drift) {
    const size_t G = in.size();
    std::vector<RegGate> info(G);
    for (size_t i = 0; i < G; i++) info[i] = reg_gate(in[i]);
    std::vector<char> done(G, 0);
    int tile_e[16];
    for (int p = 0; p < 16; p++) tile_e[p] = -1;
    for (int e = 0; e < 64; e++) if (local[e] >= 0 && local[e] < T) tile_e[local[e]] = e;
    for (size_t first = 0; first < G;) {
        if (done[first]) { first++; continue; }
        if (info[first].kind == RegGate::kOther) {
            RegItem it;
            it.gate = (int)first;
            items.push_back(it);
            done[first] = 1;
            continue;
        }
        uint64_t bits = 0, left_hard = 0, left_any = 0, wish = 0;
        std::vector<size_t> take;
        for (size_t i = first; i < G; i++) {
            if (done[i]) continue;
            const RegGate& r = info[i];
            const bool ok = r.kind != RegGate::kOther && !(r.hard & left_any) && !(r.soft & left_hard) &&
                            __builtin_popcountll(bits | r.hard) <= 5;
            if (!ok) {
                left_hard |= r.hard;
                left_any |= r.hard | r.soft;
                continue;
            }
            bits |= r.hard;
            wish |= r.soft;
            take.push_back(i);
            done[i] = 1;
        }
        // fill up with tile bits the gates read (as block bits they need no outside control), then others
        for (int e = 0; e < 64 && __builtin_popcountll(bits) < 5; e++)
            if (((wish >> e) & 1ULL) && local[e] >= 0) bits |= 1ULL << e;
        for (int p = T - 1; p >= 0 && __builtin_popcountll(bits) < 5; p--)
            if (tile_e[p] >= 0) bits |= 1ULL << tile_e[p];
        RegBlock b;
        BlockBuilder bb;
        bb.local = local;
        for (int e = 0; e < 64; e++) bb.pos[e] = -1;
        int nb = 0;
        for (int p = 0; p < T && nb < 5; p++)
            if (tile_e[p] >= 0 && ((bits >> tile_e[p]) & 1ULL)) { bb.pos[tile_e[p]] = nb; b.bits[nb++] = p; }
        for (size_t i : take) {
            const HostGate& g = in[i];
            if (info[i].kind == RegGate::kDiag) {
                bb.diag(g);
            } else if (info[i].kind == RegGate::kSwap) {
                // three controlled X
                for (int s = 0; s < 3; s++) {
                    HostGate x;
                    x.kind = 2;
                    x.k = 1;
                    x.perm = {1, 0, 0, 0};
                    x.ebit[0] = g.ebit[s & 1];
                    x.cmask = x.cval = 1ULL << g.ebit[1 - (s & 1)];
                    bb.one_bit(x);
                }
            } else {
                bb.one_bit(g);
            }
        }
        bb.finish(b, tabs, drift);
        RegItem it;
        it.block = (int)blocks.size();
        blocks.push_back(std::move(b));
        items.push_back(it);
    }
}

namespace {
// Upper bound of the largest singular value of a gate's matrix (sqrt(|A^H A|_inf) up to 4x4, which is 1 for a
// unitary one; else the smaller of the Frobenius norm and sqrt(|A|_1 |A|_inf)); infinite if an entry is not finite.
double norm_bound(const HostGate& g) {
    if (g.kind == 2) return 1;
    for (double v : g.mat) if (!std::isfinite(v)) return INFINITY;
    const int D = 1 << g.k;
    const double* m = g.mat.data();
    if (g.kind == 1) {
        double mx = 0;
        for (int i = 0; i < D; i++) mx = std::max(mx, std::hypot(m[2 * i], m[2 * i + 1]));
        return std::max(mx, 1.0);
    }
    double b = 0;
    if (D <= 4) {
        for (int i = 0; i < D; i++) {
            double sum = 0;
            for (int j = 0; j < D; j++) {
                double re = 0, im = 0;
                for (int r = 0; r < D; r++) {
                    const double *x = m + 2 * (r * D + i), *y = m + 2 * (r * D + j);
                    re += x[0] * y[0] + x[1] * y[1];
                    im += x[0] * y[1] - x[1] * y[0];
                }
                sum += std::fabs(re) + std::fabs(im);
            }
            b = std::max(b, sum);
        }
    } else {
        double fro = 0, rmax = 0, cmax = 0, col[32] = {0};
        for (int r = 0; r < D; r++) {
            double row = 0;
            for (int c = 0; c < D; c++) {
                const double a2 = m[2 * (r * D + c)] * m[2 * (r * D + c)] + m[2 * (r * D + c) + 1] * m[2 * (r * D + c) + 1];
                const double a = std::sqrt(a2);
                fro += a2;
                row += a;
                col[c] += a;
            }
            rmax = std::max(rmax, row);
        }
        for (int c = 0; c < D; c++) cmax = std::max(cmax, col[c]);
        b = std::min(fro, rmax * cmax);
    }
    return g.cmask ? std::max(std::sqrt(b), 1.0) : std::sqrt(b);
}
}  // namespace

// Whether every entry of a fused unitary (all variants) is below 2^12.  The device forms the products; here a
// bound from the gates' norms decides, and only where it does not (many gates far from unitary, or entries that
// are not finite) are the products formed to look at them.
bool bs_tc_in_range(const HostGate& f, const std::vector<HostGate>& in) {
    double bound = 1;
    for (int i : f.perm) bound *= norm_bound(in[(size_t)i]);
    if (bound < 4000.0) return true;
    int pos[64];
    for (int e = 0; e < 64; e++) pos[e] = -1;
    for (int q = 0; q < 5; q++) pos[f.ebit[q]] = q;
    std::vector<cd> U(32 * 32);
    for (int var = 0; var < (1 << f.ubits.size()); var++) {
        uint64_t uval = 0;
        for (size_t i = 0; i < f.ubits.size(); i++) if ((var >> i) & 1) uval |= 1ULL << f.ubits[i];
        std::fill(U.begin(), U.end(), cd(0, 0));
        for (int r = 0; r < 32; r++) U[(size_t)r * 33] = 1;
        for (int i : f.perm) apply_block(in[(size_t)i], pos, uval, U.data());
        for (const cd& u : U)
            if (!(std::fabs(u.real()) < 4096.0) || !(std::fabs(u.imag()) < 4096.0)) return false;
    }
    return true;
}
