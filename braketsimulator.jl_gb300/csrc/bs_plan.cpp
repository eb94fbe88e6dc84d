// Host side of gate application: lowering of a reference-convention gate or
// channel into canonical gates on endian bits, and the fusion planner that packs
// consecutive gates into tile sweeps.
//
// Reference conventions mapped here (src/gate_kernels.jl):
//   1- and 2-target kernels: matrix bit j <-> targets[j]            (:489-576)
//   >= 3 targets: matrix bit j <-> j-th smallest endian bit         (:753-775)
//   density-matrix gate: U on the column bits of vec(S), conj(U) on the row bits
//   (src/dm_simulator.jl:130-140).
#include <algorithm>
#include <cmath>
#include <complex>
#include "bs_internal.h"

namespace {

using cd = std::complex<double>;

bool valid_qubits(int n, int k, const int* t, int nc, const int* c, const int* cv, std::string& why) {
    uint64_t seen = 0;
    for (int i = 0; i < k; i++) {
        if (t[i] < 0 || t[i] >= n) { why = "target qubit out of range"; return false; }
        if ((seen >> t[i]) & 1ULL) { why = "repeated qubit"; return false; }
        seen |= 1ULL << t[i];
    }
    for (int i = 0; i < nc; i++) {
        if (c[i] < 0 || c[i] >= n) { why = "control qubit out of range"; return false; }
        if ((seen >> c[i]) & 1ULL) { why = "repeated qubit"; return false; }
        seen |= 1ULL << c[i];
        if (cv && cv[i] != 0 && cv[i] != 1) { why = "control value must be 0 or 1"; return false; }
    }
    return true;
}

// canonical target order: bit j <-> ct[j]
void canonical_targets(int k, const int* targets, unsigned flags, int* ct) {
    for (int j = 0; j < k; j++) ct[j] = targets[j];
    if (flags & BS_GATE_SORTED_TARGETS) {
        std::sort(ct, ct + k, [](int a, int b) { return a > b; });   // largest qubit = smallest endian bit
    } else if (flags & BS_GATE_MSB_FIRST) {
        for (int j = 0; j < k; j++) ct[j] = targets[k - 1 - j];
    }
}

void classify(HostGate& g) {
    const int D = 1 << g.k;
    if (g.kind == 1) return;
    bool diag = true;
    for (int r = 0; r < D && diag; r++)
        for (int c = 0; c < D; c++)
            if (r != c && (g.mat[2 * (r * D + c)] != 0.0 || g.mat[2 * (r * D + c) + 1] != 0.0)) { diag = false; break; }
    if (diag) {
        std::vector<double> d(2 * D);
        for (int i = 0; i < D; i++) { d[2 * i] = g.mat[2 * (i * D + i)]; d[2 * i + 1] = g.mat[2 * (i * D + i) + 1]; }
        g.mat.swap(d);
        g.kind = 1;
        return;
    }
    // monomial with unit phases (X, Y, CNOT, SWAP, ISWAP, CCNOT, ...)
    std::vector<int> perm(2 * D, -1);
    std::vector<int> rows_used(D, 0);
    for (int c = 0; c < D; c++) {
        int nz = 0, row = -1, ph = -1;
        for (int r = 0; r < D; r++) {
            double re = g.mat[2 * (r * D + c)], im = g.mat[2 * (r * D + c) + 1];
            if (re == 0.0 && im == 0.0) continue;
            nz++;
            row = r;
            if (im == 0.0 && re == 1.0) ph = 0;
            else if (re == 0.0 && im == 1.0) ph = 1;
            else if (im == 0.0 && re == -1.0) ph = 2;
            else if (re == 0.0 && im == -1.0) ph = 3;
        }
        if (nz != 1 || ph < 0 || rows_used[row]) return;
        rows_used[row] = 1;
        perm[2 * c] = row;
        perm[2 * c + 1] = ph;
    }
    g.perm = perm;
    g.kind = 2;
}

}  // namespace

int bs_lower_gate(bs_sim* s, const double* matrix, int k, const int* targets, int nc, const int* controls,
                  const int* cvals, unsigned flags, bool dm_superop, std::vector<HostGate>& out) {
    const int nvec = bs_vec_bits(s);
    const int nq = dm_superop ? s->n : nvec;   // qubit range of the arguments
    if (k < 1 || k > BS_MAX_TARGETS) return bs_fail(s, BS_ERR_INVALID_ARG, "gate needs 1..10 targets");
    if (nc < 0 || nc > BS_MAX_CONTROLS) return bs_fail(s, BS_ERR_INVALID_ARG, "too many controls");
    if (!matrix) return bs_fail(s, BS_ERR_INVALID_ARG, "null matrix");
    std::string why;
    if (!valid_qubits(nq, k, targets, nc, controls, cvals, why)) return bs_fail(s, BS_ERR_INVALID_ARG, why);
    const int D = 1 << k;
    int ct[BS_MAX_TARGETS];
    canonical_targets(k, targets, flags, ct);
    HostGate g;
    g.k = k;
    const bool diag = (flags & BS_GATE_DIAGONAL) != 0;
    g.kind = diag ? 1 : 0;
    const int ne = diag ? D : D * D;
    g.mat.assign(matrix, matrix + 2 * ne);
    if (flags & BS_GATE_CONJ)
        for (int i = 0; i < ne; i++) g.mat[2 * i + 1] = -g.mat[2 * i + 1];
    for (double v : g.mat)
        if (!std::isfinite(v)) return bs_fail(s, BS_ERR_INVALID_ARG, "matrix has non-finite entries");
    classify(g);
    auto put = [&](int offset, bool conj, bool last) {
        HostGate h = last ? std::move(g) : g;
        for (int j = 0; j < k; j++) h.ebit[j] = offset + (nq - 1 - ct[j]);
        h.cmask = 0;
        h.cval = 0;
        for (int i = 0; i < nc; i++) {
            int e = offset + (nq - 1 - controls[i]);
            h.cmask |= 1ULL << e;
            if (!cvals || cvals[i]) h.cval |= 1ULL << e;
        }
        if (conj) {
            if (h.kind == 2) {
                for (int c = 0; c < D; c++) h.perm[2 * c + 1] = (4 - h.perm[2 * c + 1]) & 3;
            } else {
                for (size_t i = 1; i < h.mat.size(); i += 2) h.mat[i] = -h.mat[i];
            }
        }
        out.push_back(std::move(h));
    };
    if (dm_superop) {
        put(s->n, false, false);   // column bits: U
        put(0, true, true);        // row bits: conj(U)
    } else {
        put(0, false, true);
    }
    return BS_OK;
}

// Full channel on the stored matrix: S <- sum_q conj(K_q) S K_q^T, as one dense
// gate on (row bits, column bits) of vec(S).
int bs_lower_kraus_physical(bs_sim* s, const double* kraus, int nk, int k, const int* targets, unsigned flags,
                            std::vector<HostGate>& out) {
    if (s->kind != BS_KIND_DM) return bs_fail(s, BS_ERR_STATE, "noise needs a density-matrix simulator");
    if (k < 1 || 2 * k > BS_MAX_TARGETS) return bs_fail(s, BS_ERR_UNSUPPORTED, "physical channel supports 1..5 targets");
    if (nk < 1) return bs_fail(s, BS_ERR_INVALID_ARG, "no Kraus matrices");
    std::string why;
    if (!valid_qubits(s->n, k, targets, 0, nullptr, nullptr, why)) return bs_fail(s, BS_ERR_INVALID_ARG, why);
    const int D = 1 << k, D2 = D * D;
    int ct[BS_MAX_TARGETS];
    canonical_targets(k, targets, flags, ct);
    HostGate g;
    g.kind = 0;
    g.k = 2 * k;
    for (int j = 0; j < k; j++) {
        g.ebit[j] = s->n - 1 - ct[j];           // row bits
        g.ebit[k + j] = 2 * s->n - 1 - ct[j];   // column bits
    }
    g.mat.assign((size_t)2 * D2 * D2, 0.0);
    for (int q = 0; q < nk; q++) {
        const double* K = kraus + (size_t)q * 2 * D2;
        for (double* p = (double*)K; p < K + 2 * D2; p++)
            if (!std::isfinite(*p)) return bs_fail(s, BS_ERR_INVALID_ARG, "Kraus matrix has non-finite entries");
        for (int br = 0; br < D; br++)
            for (int bc = 0; bc < D; bc++)
                for (int ar = 0; ar < D; ar++)
                    for (int ac = 0; ac < D; ac++) {
                        cd kr(K[2 * (br * D + ar)], -K[2 * (br * D + ar) + 1]);   // conj(K)[br, ar]
                        cd kc(K[2 * (bc * D + ac)], K[2 * (bc * D + ac) + 1]);    // K[bc, ac]
                        cd v = kr * kc;
                        size_t row = (size_t)(br | (bc << k)), col = (size_t)(ar | (ac << k));
                        g.mat[2 * (row * D2 + col)] += v.real();
                        g.mat[2 * (row * D2 + col) + 1] += v.imag();
                    }
    }
    classify(g);
    out.push_back(std::move(g));
    return BS_OK;
}

int bs_class_2x2(const HostGate& h) {
    if (h.mat[1] != 0.0 || h.mat[7] != 0.0) return 0;
    if (h.mat[3] == 0.0 && h.mat[5] == 0.0) return 1;
    if (h.mat[2] == 0.0 && h.mat[4] == 0.0) return 2;
    return 0;
}

int bs_tile_bits(const bs_sim* s) {
    int b = s ? s->tune.tile_bits : -1;
    if (b < 0) {
        const char* e = getenv("BS_TILE_BITS");
        b = e ? atoi(e) : BS_TILE_MAX_BITS;
    }
    return (b >= 10 && b <= BS_TILE_MAX_BITS) ? b : BS_TILE_MAX_BITS;
}

// Complex128 vectors of 11 to 18 bits take smaller tiles where nothing sets the tile bits (the
// tensor-core sweeps have tiles of 2^12): 128 tiles at 16 to 18 bits, 4 to 64 of
// 2^9 below, for 152 SMs.  A gate's pass over a tile takes its time per amplitude, which outweighs the
// launches of the extra sweeps: 17 qubits, 8 ansatz layers, 15 sweeps of 32 tiles (2^12) 0.90 ms, 22 of
// 128 (2^10) 0.33 ms, with 16 warps a tile and half the products of the real rotations.
int bs_sweep_tile_bits(const bs_sim* s) {
    const int n = bs_vec_bits(s), b = bs_tile_bits(s);
    if (s->tune.tile_bits >= 0 || getenv("BS_TILE_BITS") || s->precision != BS_PREC_C128) return b;
    if (n <= 10 || n >= 19) return b;
    return std::max(kSmallTileBits, n - 7);
}

int bs_tile_threads(const bs_sim* s) {
    int t = s ? s->tune.tile_threads : -1;
    if (t < 0) {
        const char* e = getenv("BS_TILE_THREADS");
        t = e ? atoi(e) : 256;
    }
    return (t == 512) ? 512 : 256;
}

// With one tile per SM at most, 16 warps on it instead of 8, where nothing sets the threads.
int bs_sweep_threads(const bs_sim* s, int64_t ntiles) {
    if (s->tune.tile_threads < 0 && !getenv("BS_TILE_THREADS") && ntiles <= 152) return 512;
    return bs_tile_threads(s);
}

// Handles (one stream each) that run the larger circuits of a batch side by side (BS_BATCH_STREAMS, at most 64; else 4,
// or 8 for a batch run at once whose lists have 8192 instructions or more).  Replays of a captured batch do not depend
// on it (4, 16 and 32 took the same time on 512 circuits of up to 26 qubits: the largest circuits' sweeps fill the
// GPU on their own).  A batch run at once plans each handle's next circuit on its own thread, but a handle takes
// 0.25 ms to set up and give back: 48 circuits of 12 to 22 qubits, 14 thousand instructions, 18.7 ms on 4, 17.2 on
// 8, 19.1 on 16; 14 circuits of 12 to 16 qubits, 4 thousand, 5.2 on 4 and 6.1 on 8.  Each handle holds a state, so
// eight are taken only where theirs are 8 GiB together: larger ones fill the GPU from four.
int bs_batch_handles(size_t n_large, int64_t n_ops, double eight_bytes) {
    const char* v = getenv("BS_BATCH_STREAMS");
    const int set = v ? std::max(1, std::min(64, atoi(v))) : 0;
    return (int)std::min<size_t>(n_large, (size_t)(set ? set : n_ops >= 8192 && eight_bytes <= 8.0 * (1 << 30) ? 8 : 4));
}

bool bs_tc_enabled(const bs_sim* s) {
    if (s && s->tune.tc >= 0) return s->tune.tc != 0;
    const char* v = getenv("BS_TC");   // read on every call, so a process can compare both paths
    return !(v && v[0] == '0');
}

int bs_tc_min_bits(const bs_sim* s) {
    if (s && s->tune.tc_min_bits >= 0) return s->tune.tc_min_bits;
    const char* v = getenv("BS_TC_MIN_BITS");
    return v ? atoi(v) : 22;   // some lists from 16 (use_tc)
}

double bs_tc_cost(const bs_sim* s) {
    if (s && s->tune.tc_cost >= 0) return s->tune.tc_cost;
    const char* v = getenv("BS_TC_COST");
    return v ? atof(v) : 2.0;
}

namespace {
struct SweepIdx {
    std::vector<int> hi_bits, gates;   // gates: indices into the list
};

// Greedy sweep planner.  A gate may move ahead of gates it does not share a bit
// with; a dense or monomial gate needs its target bits inside the tile, a
// diagonal gate or a control never does (their bits are read from the index).
void plan_greedy(const std::vector<HostGate>& gates, int n_bits, int T, int L, std::vector<SweepIdx>& out) {
    const int cap = T - L;
    const size_t G = gates.size();
    out.clear();
    // what a gate touches, and the bits above L it needs in the tile.  kind 5 (reference-rule channel) acts on
    // the elements whose row and column agree on every other bit: it commutes with nothing, so it touches
    // every bit, and it needs its row and column bits
    std::vector<uint64_t> touch(G), need(G);
    for (size_t i = 0; i < G; i++) {
        const HostGate& g = gates[i];
        uint64_t m = g.cmask, nd = 0;
        for (int q = 0; q < g.k; q++) m |= 1ULL << g.ebit[q];
        if (g.kind != 1)
            for (int q = 0; q < (g.kind == 5 ? 2 * g.k : g.k); q++) if (g.ebit[q] >= L) nd |= 1ULL << g.ebit[q];
        touch[i] = g.kind == 5 ? ~(uint64_t)0 : m;
        need[i] = nd;
    }
    std::vector<char> done(G, 0);
    size_t remaining = G, first = 0;
    while (remaining) {
        SweepIdx sw;
        uint64_t chosen = 0, blocked = 0;
        int nchosen = 0;
        bool big_alone = false;
        for (size_t i = first; i < G; i++) {
            if (done[i]) continue;
            const HostGate& g = gates[i];
            const uint64_t t = touch[i];
            if (t & blocked) { blocked |= t; continue; }
            const uint64_t nb = need[i] & ~chosen;
            const int add = __builtin_popcountll(nb);
            const bool too_big = (g.kind != 1) && (g.k > BS_TILE_MAXK || __builtin_popcountll(need[i]) > cap);
            if (too_big) {
                // a gate no tile can hold runs in a sweep of its own
                if (sw.gates.empty()) { sw.gates.push_back((int)i); done[i] = 1; remaining--; big_alone = true; }
                blocked |= t;
                break;
            }
            if (nchosen + add <= cap) {
                chosen |= nb;
                nchosen += add;
                sw.gates.push_back((int)i);
                done[i] = 1;
                remaining--;
            } else {
                blocked |= t;
            }
        }
        while (first < G && done[first]) first++;
        if (!big_alone) {
            for (int b = L; b < n_bits; b++) if ((chosen >> b) & 1ULL) sw.hi_bits.push_back(b);
            for (int b = L; b < n_bits && (int)sw.hi_bits.size() < cap; b++)
                if (!((chosen >> b) & 1ULL)) sw.hi_bits.push_back(b);
            std::sort(sw.hi_bits.begin(), sw.hi_bits.end());
        }
        out.push_back(std::move(sw));
    }
}

// Time of a plan with tensor-core sweeps, in fused unitaries (1.45 ms of 2^28 amplitudes; a sweep's read and
// write is 1.3 of them, with rows of 128 bytes 1.4).  Given up once it is above `most`.
double tc_plan_cost(const bs_sim* s, const std::vector<HostGate>& gates, int T, int L, const std::vector<SweepIdx>& sweeps,
                    double most) {
    double cost = (L == 3 ? 1.4 : 1.3) * (double)sweeps.size();
    std::vector<const HostGate*> in;
    for (const SweepIdx& sw : sweeps) {
        if (cost > most) break;
        int local[64];
        for (int b = 0; b < 64; b++) local[b] = b < L ? b : -1;
        for (size_t q = 0; q < sw.hi_bits.size(); q++) local[sw.hi_bits[q]] = L + (int)q;
        in.clear();
        for (int i : sw.gates) in.push_back(&gates[(size_t)i]);
        cost += bs_fuse_tc(in, local, T, bs_tc_cost(s), nullptr);
    }
    return cost;
}

// Whether a list runs in tensor-core sweeps: from bs_tc_min_bits vector bits; and, where nothing sets those, below
// the default of 22 for the lists the float-float path is slowest at, counted in its time for a dense 1-qubit gate.
// Gates on 4 targets (the two-qubit channels of a density matrix among them) from 16 bits: 8-qubit density
// matrix with channels, 1 layer 0.42 -> 0.21 ms, 10 qubits, 4 layers 5.05 -> 0.87; three gates 0.18 -> 0.15 at 17
// qubits.  Gates on 3 targets lose there (17 qubits, 6 of them 0.13 -> 0.19, 40 even) and count as generic ones.
// Generic complex matrices from 20 bits: 6 dense layers of 20 qubits 0.64 -> 0.29 ms, 2 layers 0.23 -> 0.15; at 19
// bits with 2 layers they lose what the matrices' forming takes (0.14 both).  Of those lists the norm-wise error
// against FP64 is lower too (1.6e-14 for 2.7e-14 at 20 qubits; 0.7e-14 for 2.0e-14 of an 8-qubit density matrix); single
// elements far below a tile's largest lose a digit or two (there, relative, 7e-12 for 2e-13).  Real rotations and H, which cost the float-float path half, stay there: 21 qubits of
// them would gain time, but the error grows by up to a fifth.
bool use_tc(const bs_sim* s, const std::vector<HostGate>& gates, int n_bits) {
    if (!bs_tc_enabled(s) || s->precision != BS_PREC_C128 || bs_tile_bits(s) != BS_TILE_MAX_BITS || n_bits < BS_TILE_MAX_BITS)
        return false;
    if (n_bits >= bs_tc_min_bits(s)) return true;
    if (n_bits < 16 || s->tune.tc_min_bits >= 0 || getenv("BS_TC_MIN_BITS")) return false;
    double generic = 0, wide = 0;
    for (const HostGate& g : gates) {
        if (g.kind != 0 || (g.k == 1 && bs_class_2x2(g))) continue;
        const double cost = (double)(1 << g.k) / 2.0;
        generic += cost;
        if (g.k >= 4) wide += cost;
    }
    return wide >= 24 || (n_bits >= 20 && generic >= 40);
}
}  // namespace

// Low contiguous bits of the tiles.  Fewer of them leave more bits to choose, which saves sweeps (each reads and
// writes the state once), for shorter rows of memory: 512, 256 or 128 bytes of complex128.  At 26 bits the sweeps
// of a 13-qubit density matrix cost the same with rows of 256 bytes and 5% more with 128 (24 sweeps 24.0 ms, 19
// sweeps 21.7 and 22.2).  Complex128 vectors of 19 bits and more take 4 low bits (20 bits 0.85 -> 0.82 ms), as do
// the tensor-core sweeps; from 24 bits these take the best of 3, 4 and 5, since how the sweeps' gates group into
// fused unitaries differs (28-qubit dense circuit: 24 unitaries in 9 sweeps 56.9 ms with 5, 22 in 7 48.4 with 4; 25
// qubits: 11 in 5 3.67 with 5, 14 in 5 4.12 with 4).  The other two plans cost 0.05 to 0.1 ms, too much below.
// The gates are moved into the sweeps.
void bs_plan_sweeps(const bs_sim* s, std::vector<HostGate>& gates, std::vector<Sweep>& out) {
    const int n_bits = bs_vec_bits(s);
    const bool tc = !s->collect && use_tc(s, gates, n_bits);   // not where the plan is for a small run
    const int T = std::min(tc ? BS_TILE_MAX_BITS : bs_sweep_tile_bits(s), n_bits);
    std::vector<SweepIdx> best, other;
    int low = std::min(BS_TILE_LOW_BITS, T);
    if (s->precision == BS_PREC_C128 && T == BS_TILE_MAX_BITS && (tc || n_bits >= 19)) low = 4;
    plan_greedy(gates, n_bits, T, low, best);
    if (tc && n_bits >= 24) {
        double cost = tc_plan_cost(s, gates, T, low, best, 1e300);
        for (int L : {5, 3}) {
            plan_greedy(gates, n_bits, T, L, other);
            if (L == 3 && other.size() >= best.size()) continue;
            const double c = tc_plan_cost(s, gates, T, L, other, cost);
            if (c < cost) { cost = c; low = L; best.swap(other); }
        }
    }
    for (SweepIdx& b : best) {
        Sweep sw;
        sw.tile = T;
        sw.low = low;
        sw.tc = tc;
        sw.hi_bits = std::move(b.hi_bits);
        for (int i : b.gates) sw.gates.push_back(std::move(gates[(size_t)i]));
        out.push_back(std::move(sw));
    }
}
