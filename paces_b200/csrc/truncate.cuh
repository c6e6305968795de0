// Amplitude-ranked truncation to `maxstates` states.
//
// Reference (paces/core/time_evolution.py:833-910): stable ascending argsort of |psi|,
// keep the last `maxstates` entries (among equal values the highest indices), lexsort
// the kept rows.  With shuffle_seed set and a tie at the cut, the tied states at the
// cut are drawn at random.
//
// B200 design: no sort.  The weights |psi| are non-negative doubles, so their bit
// patterns order like the values; a radix select (4096 bins a pass, shared-memory
// histograms) finds the threshold value v* and the number of states equal to v* that
// must be kept.  Because the basis is already sorted, keeping the selected states in
// index order *is* the lexsorted result: one order-preserving compaction writes the
// new basis (keys and block offsets).  Tie rule as in the reference: the states equal
// to v* with the highest indices; with shuffling, the tied states whose 64-bit hash of
// (seed, step, index) is smallest -- a uniformly random subset, like the reference's
// random permutation, but not the same stream (parity unpinned for that branch).
#pragma once

#include "common.cuh"

namespace paces {

struct TruncWs {
    unsigned* hist;              // [3][4096] radix histograms in rotation
    unsigned* barrier;           // behind them: the grid barrier and the counters below
    unsigned long long* cand;    // [cap] candidate weight bits (or hashes)
    int* cand_idx;               // [cap]
    long long* sel;              // selection state, see truncate.cu
    unsigned long long* block_sum;   // [1024] the selection's blocks: counts of their chunks
    unsigned long long* chunk;       // [trunc_chunks_cap(cap)] counts, then prefixes of the chunks
    int64_t cap;
    uint64_t wait_ns;            // grid-barrier wait limit (kWaitLimitNs unless a test shortens it)
    int skip_block;              // test hook: this block skips its first grid-barrier arrival (-1: none)
};
// words of TruncWs.barrier
constexpr int kTruncListed = 1;  // states listed for the last bin
constexpr int kTruncDone = 2;    // blocks of the compaction done
constexpr int kTruncGaveUp = 3;  // a block of the selection gave up waiting
constexpr size_t kTruncHistBytes = (3 * 4096 + 16) * 4;  // histograms and counters, zeroed per truncation

constexpr int kTruncChunk = 256;  // states a warp of the compaction takes at a time

inline int64_t trunc_chunks_cap(int64_t cap) { return cap / kTruncChunk + 2; }

// Bits below this one are zero in every weight of a kind (0 complex128 |psi|, 1 complex64
// |psi|, 2 precomputed fp64 weights): a complex64 weight is an fp32 value widened to a double.
inline int weight_low_bit(int wk) { return wk == 1 ? 29 : 0; }
// Kernels one truncation enqueues.
inline int trunc_launches(bool shuffle) { return 2 + (shuffle ? 16 : 0); }

// weights (optional, one non-negative double per state): rank by these instead of |psi|
// (the look-ahead weighting, lookahead.cu).
// scratch (optional, without weights: 4 bytes per state for complex64, 8 for complex128):
// the selection's first pass stores |psi| there and the later passes read it instead of the
// amplitudes, so |psi| is computed once per state.
// out_w (optional, out_cap + 1 floats): the ranked weight (|psi|) of every kept state in the
// new basis' order, and at out_w[out_cap] the cut -- the weight of the smallest kept state, 0
// when nothing was dropped.
// sel_sms: SMs that the launch whose blocks wait for one another may take; truncations that may
// run at the same time on this GPU take no more than all of them together.
// cleared: the caller's last kernel has zeroed ws.hist (kTruncHistBytes)
int launch_truncate(int nw, bool c64, const ModelDev& m, const uint64_t* x_keys, const int* x_blk,
                    const void* psi, const double* weights, void* scratch, int64_t maxstates, int shuffle, uint64_t seed,
                    uint64_t step, const TruncWs& ws, uint64_t* out_keys, int* out_blk, int64_t out_cap, float* out_w,
                    int* n_tied_out, int* n_kept_out, int* status, int num_sms, int sel_sms, cudaStream_t st,
                    bool cleared = false);

}  // namespace paces
