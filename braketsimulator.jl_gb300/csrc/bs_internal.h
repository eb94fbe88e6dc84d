// Internal structures shared by the translation units of libbraket_gb300.so.
#pragma once
#include <cstdint>
#include <string>
#include <vector>
#include <cuda_runtime.h>
#include "../../include/braket_gb300.h"

#define BS_TILE_MAX_BITS 12      // 2^12 complex float-float values = 64 KiB of shared memory
#define BS_TILE_LOW_BITS 5       // low endian bits always in a tile, 32 contiguous amplitudes, but for complex128
                                 // vectors of 19 bits and more (bs_plan_sweeps)
#define BS_TILE_MAXK 4           // dense targets per tile gate (16x16 superoperators for 2q noise)

// One gate inside a tile sweep.
//   kind 0: dense 2^k x 2^k on tile-local bits tbit[0..k-1] (matrix bit j <-> tbit[j]); k = 1: npar is
//           the matrix class (bs_class_2x2)
//   kind 1: diagonal 2^k entries selected by global bits gbit[0..k-1]
//   kind 2: monomial (one unit-modulus phase i^p per column) on tile-local bits; npar 1: X
//   kind 3: a run of CZ gates applied as one parity phase (npar, pshift, pmask)
//   kind 4: fused dense unitary on 5 tile-local bits gbit[0..4] (matrix bit j <-> gbit[j]),
//           applied on the tensor cores from the bf16 digit slices at tc_off (48 KiB blocks)
//   kind 5: Kraus channel on k <= 2 targets in the reference's block-diagonal update rule
//           (density matrix): tbit[0..2k-1] row then column target bits, pmask[0..1], its superoperator
//           at mat_off
// Controls: (tile_index & lc_mask) == lc_val for in-tile controls,
//           (global_base & gc_mask) == gc_val for controls outside the tile.
struct TileGate {
    int32_t kind;
    int32_t k;
    int32_t tbit[BS_TILE_MAXK];
    int32_t gbit[BS_MAX_TARGETS];
    uint32_t lc_mask, lc_val;
    uint64_t gc_mask, gc_val;
    int32_t mat_off;            // offset (in cff units) into the sweep's matrix pool
    int32_t perm_off;           // monomial: offset into the permutation pool (int32 pairs)
    // kind 3: a run of CZ gates as one phase (-1)^(sum_q popc(i & (i >> pshift[q]) & pmask[q]))
    int32_t npar;
    int32_t pshift[4];
    uint64_t pmask[4];
    int32_t tc_off;             // kind 4: index of the digit-slice block in the sweep's pool
    int32_t tc_eu;              // kind 4: matrix entries are below 2^tc_eu
    int32_t tc_nu;              // kind 4: the CTA's base bits tc_ub[0..tc_nu-1] select the variant block
    int32_t tc_ub[3];
};

// One gate of a fused unitary, for the kernel that forms its matrices.  Block bit q: 0..4; variant bit i: 8 + i.
struct TcPart {
    uint8_t kind, k;            // as TileGate kinds 0..2
    uint8_t pos[5];             // target j: its block bit, or (diagonal) variant bit
    uint8_t cmask, cval;        // controls in the block: (row & cmask) == cval
    uint8_t umask, uval;        // controls among the variant bits
    int32_t off;                // matrix (complex) or permutation (int pairs) in the pool
};
// One fused unitary: its gates, its first matrix variant and its TileGate.
struct TcBlock {
    int32_t part0, n_parts, var0, gate;
};

struct SweepDesc {
    int32_t n_bits;             // endian bits of the vector (n for SV, 2n for DM)
    int32_t T;                  // tile bits
    int32_t L;                  // low contiguous bits
    int32_t n_gates;
    int32_t hi_bits[BS_TILE_MAX_BITS];
    uint64_t tile_mask;
    int8_t out_bits[32];        // the endian bits outside the tile, ascending: the tile number's bits (63: none)
    const TileGate* gates;      // device
    const float4* mats;         // device, complex float-float entries (rh, rl, ih, il)
    const int32_t* perms;       // device
    const uint16_t* tc_pool;    // device, kind-4 digit slices (24576 bf16 per gate)
    int* err;                   // device flag: a bounded tensor-core wait gave up
};

// Fills hi_bits, tile_mask and out_bits of a sweep over n_bits with L low tile bits and the bits hi above.
inline void bs_tile_geometry(SweepDesc& d, int n_bits, int L, const std::vector<int>& hi) {
    d.n_bits = n_bits;
    d.L = L;
    d.T = L + (int)hi.size();
    d.tile_mask = (1ULL << L) - 1;
    for (size_t i = 0; i < hi.size(); i++) { d.hi_bits[i] = hi[i]; d.tile_mask |= 1ULL << hi[i]; }
    int k = 0;
    for (int b = 0; b < n_bits && k < 32; b++) if (!((d.tile_mask >> b) & 1ULL)) d.out_bits[k++] = (int8_t)b;
    while (k < 32) d.out_bits[k++] = 63;
}

struct HostGate {                // a gate after lowering to the canonical convention
    int kind;                    // 0 dense, 1 diagonal, 2 monomial, 4 fused 5-bit unitary,
                                 // 5 reference-rule Kraus channel (ebit: k row bits, then k column bits;
                                 // mat: its superoperator on a block, index row + 2^k column)
    int k;
    int ebit[BS_MAX_TARGETS];    // endian bit of target j (matrix bit j)
    std::vector<double> mat;     // interleaved complex; dense 4^k*2, diag 2^k*2
    uint64_t cmask = 0, cval = 0;// controls on endian bits
    std::vector<int> perm;       // monomial: column c -> (row, i-power); kind 4: its gates in order, indices
                                 // into the list that was fused
    std::vector<int> ubits;      // kind 4: out-of-tile bits the fused matrix depends on: 2^|ubits|
                                 // matrices, variant v for bit values v_i at ubits[i]
};

struct Sweep {
    int tile = 0;                // bits of the tile
    int low = BS_TILE_LOW_BITS;  // the low contiguous ones
    bool tc = false;             // gates may be fused for the tensor cores
    std::vector<int> hi_bits;    // tile bits above them
    std::vector<HostGate> gates;
};

// Per-handle tuning (bs_set_tuning); a negative value means "environment variable, else the
// built-in default" (BS_TILE_BITS 12, BS_TILE_THREADS 256, BS_TC 1, BS_TC_MIN_BITS 22, BS_TC_COST 2).
struct BsTuning {
    int tile_bits = -1;      // tile bits of the sweep kernels, 10..12
    int tile_threads = -1;   // threads per CTA of the float-float sweep kernel, 256 or 512
    int tc = -1;             // fused tensor-core sweeps on (1) or off (0)
    int tc_min_bits = -1;    // vector bits from which fused tensor-core sweeps are used
    double tc_cost = -1;     // float-float cost (dense 1-qubit gates) above which a block is fused
    int adj_segments = -1;   // adjoint gradients: forward segments (checkpoints + 1); -1 = from memory
};

// The packed plan of one small-circuit run (bs_run_small): the whole state is one tile, so the plan is
// the gate table, its matrices and permutations, and the largest dense or monomial target count.
// States above 2^10 run in a cluster of CTAs that hold 2^9 amplitudes each, sweep by sweep: `sweeps` then
// lists the sweeps (else it is empty).
constexpr int kSmallTileBits = 9;
struct SmallSweep {
    int32_t g0, ng;             // its gates
    int8_t hi[4];               // tile bits 5..8: endian bits
    int8_t out[4];              // the endian bits outside the tile, ascending: the CTA's rank
};
struct SmallPlan {
    std::vector<SmallSweep> sweeps;
    std::vector<TileGate> tg;
    std::vector<float4> mats;
    std::vector<int32_t> perms;
    int kmax = 1;
};

struct bs_sim {
    int kind = BS_KIND_SV;
    int n = 0;                    // qubits
    int precision = BS_PREC_C128;
    int device = 0;
    cudaStream_t stream = nullptr;
    void* state = nullptr;        // complex128: double2[len]
    int64_t len = 0;              // elements of the state vector / vec(S)
    int64_t cap_bytes = 0;
    // scratch for reductions and sampling
    void* scratch = nullptr;
    int64_t scratch_bytes = 0;
    double* alias_ap = nullptr;
    int64_t* alias_ix = nullptr;
    int64_t alias_len = 0;
    bool alias_valid = false;
    // plan upload buffer
    void* plan_buf = nullptr;
    int64_t plan_bytes = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int* dev_flag = nullptr;      // device error flag of the tensor-core sweeps
    bool flag_armed = false;
    std::vector<cudaEvent_t> tc_events;   // pool: an event pair around each tensor-core launch
    size_t tc_events_used = 0;            // pairs recorded since the last bs_collect_tc_time
    bs_stats stats{};
    BsTuning tune{};
    std::string err;
    // Host staging of uploads: pinned, reused once the previous upload has landed (hstage_ev).
    char* hstage = nullptr;
    size_t hstage_cap = 0;
    cudaEvent_t hstage_ev = nullptr;
    bool hstage_pending = false;
    // While the handle's stream is captured into a CUDA graph: no host synchronisation, no device
    // buffer growth, and staging comes from an append-only pinned arena that lives as long as the
    // graph (the graph's copy nodes read it on every replay).
    bool capturing = false;
    bool defer_sync = false;   // bs_evolve returns without synchronising (an internal caller syncs later)
    bool stats_pending = false;   // an evolve returned before its end event (ev1) completed
    std::vector<std::pair<char*, size_t>> arena;   // chunks (pointer, capacity)
    size_t arena_used = 0;                          // bytes used in the last chunk
    std::vector<Sweep>* collect = nullptr;          // bs_evolve plans into this list instead of launching
    // bs_run_small: the plan of the last instruction list, kept with the list's exact bytes (op structs
    // without their matrix pointers, the matrix values, the qubit count and tile setting) so that the
    // same list again skips the planning
    std::vector<char> small_key;
    SmallPlan small_plan;
    bool small_valid = false;
};

// ---- helpers implemented in bs_api.cu
int bs_fail(bs_sim* s, int code, const std::string& msg);
int bs_cuda_check(bs_sim* s, cudaError_t e, const char* what);
// Device-to-host copy of a result, stream synchronised; small ones land in a pinned per-thread
// buffer first (a pageable copy takes a staged driver path).  During graph capture: enqueue only.
int bs_copy_out(bs_sim* s, void* host, const void* dev, size_t bytes, const char* what);
// This thread's pinned host memory mapped into the device's address space, for a result of up to `bytes`
// that a kernel writes and a ticket it writes after it (null: not available, or too large).  One result
// at a time: the call that takes it waits for its ticket (bs_wait_ticket) before it returns.
struct MapSlot {
    char* h = nullptr;           // result, host and device address
    char* d = nullptr;
    volatile int64_t* word = nullptr;   // ticket word, host address
    int64_t* dword = nullptr;           // and device address
    int64_t ticket = 0;
};
MapSlot bs_map_slot(size_t bytes);
// Called by a thread that lives for one call: its results take the copy, since mapping memory for it costs more.
void bs_thread_without_map();
// Polls for the slot's ticket; after 2 s (a failed or very long kernel) synchronises the stream, which
// reports the error.  A stream that ended without the ticket is an error too.
int bs_wait_ticket(bs_sim* s, const MapSlot& m, const char* what);
// Device allocation (cudaMalloc's status).  The blocks that handles keep between calls (bs_keep.h: the checkpoints and
// lambda of adjoint gradients, up to 1 GiB a handle and 4 GiB over all) are freed before it fails.
cudaError_t bs_malloc(void** p, size_t bytes);
constexpr size_t kKeepBytes = (size_t)1 << 30, kKeepAll = 4 * kKeepBytes;
void* bs_keep_take(const bs_sim* s, size_t bytes, size_t* got);   // the handle's kept block, if it is large enough
void bs_keep(const bs_sim* s, void* p, size_t bytes);              // for its next call
size_t bs_kept_bytes();
void bs_free_kept();
int bs_ensure_scratch(bs_sim* s, int64_t bytes);
int bs_ensure_plan(bs_sim* s, int64_t bytes);
// The counter with which the last block of an expectation is found (zero between calls), behind the scratch buffer
// (after bs_ensure_scratch).
unsigned* bs_scratch_counter(const bs_sim* s);
// Pinned host region for one upload of `bytes`; call bs_stage_done after queuing the copy.
char* bs_stage(bs_sim* s, size_t bytes);
void bs_stage_done(bs_sim* s);
// Release the capture arena (the graph that read it is gone).
void bs_arena_release(bs_sim* s);
int bs_vec_bits(const bs_sim* s);

#ifdef __CUDACC__
// Base index of a tile, by a whole warp (the same value in every lane): lane i places the tile number's
// bit i.  (One thread walking the vector's bits held up the whole CTA for 600 cycles at its start.)
__device__ __forceinline__ int64_t bs_tile_base(const SweepDesc& d, int64_t tile) {
    const int lane = threadIdx.x & 31, b = d.out_bits[lane];
    const uint64_t v = (b < 63 && ((tile >> lane) & 1)) ? 1ULL << b : 0ULL;
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)v), hi = __reduce_or_sync(0xffffffffu, (uint32_t)(v >> 32));
    return (int64_t)(((uint64_t)hi << 32) | lo);
}
#endif

// ---- lowering (bs_plan.cpp)
// Convert a gate (reference convention flags) into canonical HostGate(s) on the
// vector's endian bits.  For DM, returns the column-side U and row-side conj(U).
int bs_lower_gate(bs_sim* s, const double* matrix, int k, const int* targets, int nc,
                  const int* controls, const int* cvals, unsigned flags, bool dm_superop,
                  std::vector<HostGate>& out);
int bs_lower_kraus_physical(bs_sim* s, const double* kraus, int nk, int k, const int* targets,
                            unsigned flags, std::vector<HostGate>& out);
// The gates are moved into the sweeps (the input is left with moved-from gates).
void bs_plan_sweeps(const bs_sim* s, std::vector<HostGate>& gates, std::vector<Sweep>& out);
// Matrix class of a 2x2 gate: 1 all real, 2 real diagonal and imaginary off-diagonal, else 0 (TileGate.npar).
int bs_class_2x2(const HostGate& h);
// Tuned values of a handle (its setting, else the environment, else the default)
int bs_tile_bits(const bs_sim* s);
int bs_sweep_tile_bits(const bs_sim* s);   // tile bits the sweeps use for the handle's size
int bs_tile_threads(const bs_sim* s);
int bs_batch_handles(size_t n_large, int64_t n_ops, double eight_bytes);   // handles of a batch
int bs_sweep_threads(const bs_sim* s, int64_t ntiles);   // threads of a float-float sweep over that many tiles
bool bs_tc_enabled(const bs_sim* s);
int bs_tc_min_bits(const bs_sim* s);
double bs_tc_cost(const bs_sim* s);

// ---- tensor-core fusion (bs_fuse.cpp)
// Fold runs of in-tile gates into kind-4 HostGates (5 endian bits and the gates' indices) where that is cheaper
// (float-float cost above `threshold`).  local[e]: tile position of endian bit e or -1.
double bs_fuse_tc(const std::vector<const HostGate*>& in, const int* local, int T, double threshold,
                  std::vector<HostGate>* out);   // out null: only the list's cost, in fused unitaries
void bs_fuse_small(const std::vector<HostGate>& in, const int* local, double pass, int maxk, std::vector<HostGate>& out);
// Whether every entry of a fused gate's matrices is finite and below 2^12 (in: the list that was fused).
bool bs_tc_in_range(const HostGate& f, const std::vector<HostGate>& in);

// ---- execution (bs_tile.cu)
int bs_run_sweeps(bs_sim* s, const std::vector<Sweep>& sweeps);
// BS_ERR_TIMEOUT if a tensor-core sweep since the last check gave up on a bounded wait
int bs_check_device_flag(bs_sim* s);
// After the stream has synchronised: add the device time of the recorded tensor-core launches to stats.tc_ms
void bs_collect_tc_time(bs_sim* s);

// ---- reference-compat Kraus (bs_dm.cu)
int bs_kraus_reference(bs_sim* s, const double* kraus, int nk, int k, const int* targets,
                       unsigned flags);
// The same channel (1 or 2 targets) as a kind-5 HostGate applied inside a sweep.
int bs_lower_kraus_reference(bs_sim* s, const double* kraus, int nk, int k, const int* targets, unsigned flags,
                             std::vector<HostGate>& out);

// ---- parallel alias table (bs_alias_par.cu)
int64_t bs_alias_parallel_scratch(int64_t n);
int bs_alias_parallel(bs_sim* s, const double* dprobs, int64_t n, double wsum, double* ap, int64_t* alias, void* work);

// ---- small state vectors in one CTA (bs_tile.cu, bs_sample.cu)
// bs_small_launch: |0...0>, the packed plan's gates, the state written back, its probabilities into
// dprobs and `shots` draws of bs_sample's generator with `seed` into dsamples, in one launch (dprobs
// and dsamples: device addresses, mapped host memory included); at its end the kernel writes `ticket`
// into *done (a host-mapped word, may be null) once every result is visible to the host.  io (may be
// null): host-mapped memory for the plan (written at hplan, read by the kernel at dplan, when it fits
// in plan_cap bytes; otherwise the plan is uploaded) and for the kernel's start and end times
// (globaltimer nanoseconds, at dtimes[0] and dtimes[1]).
struct SmallIO {
    char* hplan;
    char* dplan;
    size_t plan_cap;
    int64_t* dtimes;
};
// Pack the planned sweeps of a small run; BS_ERR_UNSUPPORTED (nothing packed) when a gate has no in-tile
// kernel or the state is not a complex128 state vector of at most 12 qubits.
int bs_small_pack(const bs_sim* s, const std::vector<Sweep>& sweeps, SmallPlan& out);
int bs_small_launch(bs_sim* s, const SmallPlan& plan, double* dprobs, int64_t shots, uint64_t seed,
                    int64_t* dsamples, int64_t* done, int64_t ticket, const SmallIO* io);
