// Gate fusion for the tensor-core tile path.
//
// Inside one tile sweep, runs of gates are folded into dense unitaries on 5
// tile bits.  A gate can join a block when its dense targets lie in the tile and
// its tile bits fit the block; bits outside the tile (controls, and target bits
// of diagonal gates) are constant within a CTA, so the block is built once per
// assignment of those "uniform" bits (at most 3 of them) and each CTA picks its
// variant.  The products are formed on the device in FP64 (k_tc_build) and applied to
// the tile as real 64x64 GEMMs on tcgen05 tensor cores, with both operands split
// into exact 9-bit digits carried in bf16 (an Ozaki-style split) so that the result keeps
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
