// Amplitude-ranked truncation (see truncate.cuh).
#include <type_traits>

#include "grid.cuh"
#include "truncate.cuh"

namespace paces {

namespace {

// selection state words (TruncWs.sel)
enum : int {
    SEL_S = 0,        // number of input states
    SEL_ALL = 1,      // 1: keep everything (S <= maxstates)
    SEL_W = 2,        // weight select: [2] prefix [3] mask [4] need [5] active
    SEL_H = 6,        // hash select:   [6] prefix [7] mask [8] need [9] active
    SEL_CAND = 10,    // candidate count
    SEL_TIES = 11,    // states equal to the threshold
    SEL_SHUFFLE = 12, // 1: ties at the cut are shuffled
    SEL_WORDS = 16
};

constexpr int kRounds = 6;
__host__ __device__ constexpr int round_shift(int r) { return r < 5 ? 52 - 12 * r : 0; }
__host__ __device__ constexpr int round_bits(int r) { return r < 5 ? 12 : 4; }

// The ranked weight of state i: WK 0 = |psi| of complex128 amplitudes, 1 = |psi| of
// complex64 amplitudes, 2 = precomputed non-negative fp64 weights (the look-ahead
// weighting, or |psi| of complex128 amplitudes stored by the first pass), 3 = |psi|
// of complex64 amplitudes stored as fp32 by the first round (exact: hypotf's result,
// widened like WK 1 widens it).  Non-negative doubles order like their bit patterns.  The
// load and the conversion are separate so that loops can issue several loads before the
// first use.
template <int WK>
using RawW = typename std::conditional<
    WK == 0, double2,
    typename std::conditional<WK == 1, float2, typename std::conditional<WK == 2, double, float>::type>::type>::type;

// the kind the first round stores for later passes (WK 0 -> 2, WK 1 -> 3)
__host__ __device__ constexpr int stored_kind(int wk) { return wk == 1 ? 3 : 2; }

template <int WK>
__device__ __forceinline__ RawW<WK> load_raw(const void* psi, int64_t i) {
    return __ldcs(reinterpret_cast<const RawW<WK>*>(psi) + i);
}

template <int WK>
__device__ __forceinline__ unsigned long long raw_bits(const RawW<WK>& z, int* status) {
    double w;
    if constexpr (WK == 1) w = double(hypotf(z.x, z.y));
    else if constexpr (WK == 0) w = hypot(z.x, z.y);
    else w = double(z);
    if (!(w <= 1.7976931348623157e308)) raise_status(status, PACES_ERR_NONFINITE);
    return (unsigned long long)__double_as_longlong(w);
}

template <int WK>
__device__ __forceinline__ unsigned long long weight_bits(const void* psi, int64_t i, int* status) {
    return raw_bits<WK>(load_raw<WK>(psi, i), status);
}

// splitmix64 finaliser applied to (index + stream offset): a bijection of the index, so
// hashes of distinct states never collide.
__device__ __forceinline__ unsigned long long tie_hash(uint64_t seed, uint64_t step, int64_t i) {
    unsigned long long z = (unsigned long long)i + seed * 0x9E3779B97F4A7C15ull + step * 0xD1B54A32D192ED03ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    return ~z;  // keep the largest ~hash == the smallest hash
}

// One radix round of the tie shuffle: find the digit holding the need-th largest hash and
// narrow the prefix.
__global__ void __launch_bounds__(1024) trunc_select_kernel(TruncWs ws, int base, int round) {
    __shared__ long long s_warp[32];
    __shared__ int s_bin;
    __shared__ long long s_above;
    if (!ws.sel[base + 3]) return;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int bits = round_bits(round), shift = round_shift(round);
    const int nb = 1 << bits;
    const int per = (nb + 1023) / 1024;  // 4 or 1
    const long long need = ws.sel[base + 2];
    long long mine = 0;
    for (int q = 0; q < per; ++q) {
        const int b = tid * per + q;
        if (b < nb) mine += ws.hist[b];
    }
    // suffix sums: threads above me
    long long incl = mine;  // inclusive suffix within the warp (lanes >= lane)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long v = __shfl_down_sync(0xffffffffu, incl, o);
        if (lane + o < 32) incl += v;
    }
    if (lane == 0) s_warp[wid] = incl;
    if (tid == 0) s_bin = -1;
    __syncthreads();
    long long warps_above = 0;
    for (int w = wid + 1; w < 32; ++w) warps_above += s_warp[w];
    const long long above_me = warps_above + (incl - mine);  // sum of bins above my range
    if (mine > 0 && above_me < need && need <= above_me + mine) {
        long long acc = above_me;
        for (int q = per - 1; q >= 0; --q) {
            const int b = tid * per + q;
            if (b >= nb) continue;
            const long long hb = ws.hist[b];
            if (acc < need && need <= acc + hb) {
                s_bin = b;
                s_above = acc;
                break;
            }
            acc += hb;
        }
    }
    __syncthreads();
    if (tid == 0 && s_bin >= 0) {
        const int b = s_bin;
        ws.sel[base + 2] = need - s_above;
        ws.sel[base + 0] |= (long long)((unsigned long long)b << shift);
        ws.sel[base + 1] |= (long long)((unsigned long long)(nb - 1) << shift);
    }
    __syncthreads();
    for (int b = tid; b < 4096; b += blockDim.x) ws.hist[b] = 0;
}

constexpr int kSelThreads = 1024;
constexpr int kSelWarps = kSelThreads / 32;
constexpr int kU = kTruncChunk / 32;  // states per lane of a chunk, their loads in flight together
constexpr int kSelCand = 2048;        // a bin this small is settled from a list of its weights
// the first pass's bins: 2^-63 .. 2 in steps of 2^-6 of a binade
constexpr int kFirstShift = 46;
constexpr unsigned long long kFirstBase = (unsigned long long)(1023 - 63) << 52;

// Calls f(chunk, weight bits, existing states' bits) for chunks [c0, c1) of kTruncChunk states,
// `warps` warps of which this is number w: lane l holds states 32 u + l of the chunk.
template <int K, class F>
__device__ __forceinline__ void for_chunks(const void* from, int64_t S, int64_t c0, int64_t c1, int w, int warps,
                                           int* status, F f) {
    const int lane = threadIdx.x & 31;
    for (int64_t c = c0 + w; c < c1; c += warps) {
        const int64_t i0 = c * kTruncChunk + lane;
        constexpr int kG = sizeof(RawW<K>) >= 16 ? kU / 2 : kU;  // loads in flight together
        unsigned ok = 0;
        unsigned long long k[kU];
#pragma unroll
        for (int g = 0; g < kU; g += kG) {
            RawW<K> z[kG];
#pragma unroll
            for (int u = 0; u < kG; ++u) {
                if (i0 + 32 * (g + u) < S) {
                    z[u] = load_raw<K>(from, i0 + 32 * (g + u));
                    ok |= 1u << (g + u);
                }
            }
#pragma unroll
            for (int u = 0; u < kG; ++u) k[g + u] = ok >> (g + u) & 1u ? raw_bits<K>(z[u], status) : 0ull;
        }
        f(c, k, ok);
    }
}

// Block-wide exclusive prefix of one value per thread; `total` gets the block's sum.  s_sum:
// one word per warp.
__device__ unsigned long long block_prefix(unsigned long long v, unsigned long long* s_sum, unsigned long long& total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    __syncthreads();
    if (lane == 31) s_sum[wid] = incl;
    __syncthreads();
    unsigned long long before = 0;
    total = 0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) {
        const unsigned long long x = s_sum[w];
        if (w < wid) before += x;
        total += x;
    }
    return before + incl - v;
}

// The need-th largest of a histogram's entries, by all threads of the block: thread t holds the
// counts hb[] of bins [t * PER, (t + 1) * PER).  s_pick: bin, entries above it, its count.
template <int PER>
__device__ __forceinline__ void pick_bin(const unsigned (&hb)[PER], long long need, long long* s_warp, long long* s_pick) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    long long mine = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) mine += hb[q];
    long long incl = mine;  // this thread's bins and those of the higher lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long v = __shfl_down_sync(0xffffffffu, incl, o);
        if (lane + o < 32) incl += v;
    }
    if (lane == 0) s_warp[wid] = incl;
    if (tid == 0) s_pick[0] = -1;
    __syncthreads();
    long long above = incl - mine;
    for (int w = wid + 1; w < int(blockDim.x >> 5); ++w) above += s_warp[w];
    if (mine > 0 && above < need && need <= above + mine) {
#pragma unroll
        for (int q = PER - 1; q >= 0; --q) {
            if (above < need && need <= above + hb[q]) {
                s_pick[0] = tid * PER + q;
                s_pick[1] = above;
                s_pick[2] = hb[q];
            }
            above += hb[q];
        }
    }
    __syncthreads();
}

// The selection in one cooperative launch, one block of 1024 threads per SM.
//  * The threshold's bits lie in [lo, lo + width): streaming passes, each into a shared-memory
//    histogram of 4096 bins over that range, a grid barrier, and every block picking the bin
//    from the grid's histogram itself.  The first pass bins 64 binades below 2 by 6 mantissa
//    bits (what lies below or above goes to its end bins): exponents alone put most states
//    into a few bins, whose atomics collide.
//    An end bin is no power of two wide, so the next pass's last bin may be cut short.
//  * Once the chosen bin holds at most kSelCand states (two passes leave a few of millions;
//    all bits take 5 passes, 7 from an end bin of the first), one more pass lists the bin's
//    states and every block settles the remaining bits among them.
//  * That pass also counts the states above the bin per chunk of the compaction; with the
//    listed states added and the blocks' totals exchanged, the counts become every chunk's
//    prefix (states above the threshold | tied states << 31), so the compaction's warps need
//    nothing from each other.
// A launch per pass and selection, and a counting and a scanning launch, took 85 us for 15K
// complex128 states, nearly all of it latency.
//
// STORE: the first round computes |psi| and writes it to `wout` in the stored kind, which the
// later passes read (each thread its own states).
template <int WK, bool STORE>
__global__ void __launch_bounds__(kSelThreads, 1)
trunc_threshold_kernel(int L, const int* __restrict__ x_blk, const void* __restrict__ psi, TruncWs ws,
                       int64_t maxstates, void* wout, int low, int* status) {
    constexpr int WS = STORE ? stored_kind(WK) : WK;  // the kind the passes after the first read
    __shared__ unsigned h[4096];
    __shared__ long long s_warp[kSelWarps], s_pick[3];
    __shared__ unsigned long long s_sum[kSelWarps], s_own;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t S = x_blk[L];
    const bool all = S <= maxstates;
    if (blockIdx.x == 0 && tid < SEL_WORDS) {
        // until the selection is known: nothing to write
        long long v = 0;
        if (tid == SEL_ALL) v = 1;
        if (all && tid == SEL_S) v = S;
        ws.sel[tid] = v;
    }
    if (all) return;
    const int64_t nch = (S + kTruncChunk - 1) / kTruncChunk;
    const int64_t c0 = nch * blockIdx.x / gridDim.x, c1 = nch * (blockIdx.x + 1) / gridDim.x;  // this block's chunks
    unsigned gen = 0;
    // A block whose wait runs out says so: the others may have gone on and finished, but without its
    // chunks' prefixes the compaction would place states wrongly, so it writes none.
    auto grid_wait = [&]() {
        const bool ok = grid_barrier(ws.barrier, gridDim.x, gen, status, ws.wait_ns, int(blockIdx.x) == ws.skip_block);
        if (!ok && tid == 0) ws.barrier[kTruncGaveUp] = 1u;
        return ok;
    };
    unsigned long long lo = 0, width = ~0ull;
    long long need = maxstates, count = S;
    const void* src = psi;
    // width - 1 takes this many bits; bits below `low` are zero in every weight
    auto bits_of = [](unsigned long long x) { return 64 - __clzll((long long)(x - 1)); };
    for (int round = 0;; ++round) {
        const int shift = round == 0 ? kFirstShift : max(bits_of(width) - 12, 0);
        for (int b = tid; b < 4096; b += kSelThreads) h[b] = 0;
        __syncthreads();
        if (round == 0) {
            for_chunks<WK>(src, S, c0, c1, wid, kSelWarps, status, [&](int64_t c, const unsigned long long (&k)[kU], unsigned ok) {
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    if (!(ok >> u & 1u)) continue;
                    if constexpr (STORE) {
                        const double wv = __longlong_as_double((long long)k[u]);
                        const int64_t i = c * kTruncChunk + 32 * u + lane;
                        if constexpr (WS == 3) reinterpret_cast<float*>(wout)[i] = float(wv);
                        else reinterpret_cast<double*>(wout)[i] = wv;
                    }
                    const long long b = (long long)(k[u] >> kFirstShift) - (long long)(kFirstBase >> kFirstShift);
                    atomicAdd(&h[int(min(max(b, 0ll), 4095ll))], 1u);
                }
            });
            if constexpr (STORE) src = wout;
        } else {
            for_chunks<WS>(src, S, c0, c1, wid, kSelWarps, status, [&](int64_t, const unsigned long long (&k)[kU], unsigned ok) {
#pragma unroll
                for (int u = 0; u < kU; ++u)
                    if ((ok >> u & 1u) && k[u] - lo < width) atomicAdd(&h[unsigned((k[u] - lo) >> shift)], 1u);
            });
        }
        __syncthreads();
        unsigned* gh = ws.hist + (round % 3) * 4096;
        for (int b = tid; b < 4096; b += kSelThreads)
            if (h[b]) atomicAdd(&gh[b], h[b]);
        if (!grid_wait()) return;
        constexpr int per = 4096 / kSelThreads;
        unsigned hb[per];
#pragma unroll
        for (int q = 0; q < per; ++q) hb[q] = __ldcg(gh + tid * per + q);
        if (blockIdx.x == 0)  // the histogram of the round after next
            for (int b = tid; b < 4096; b += kSelThreads) ws.hist[((round + 2) % 3) * 4096 + b] = 0;
        pick_bin<per>(hb, need, s_warp, s_pick);
        if (s_pick[0] < 0) {  // cannot happen: the states' count does not change between rounds
            if (blockIdx.x == 0 && tid == 0) raise_status(status, PACES_ERR_BADARG);
            return;
        }
        const unsigned long long bin = (unsigned long long)s_pick[0];
        if (round > 0) {
            // the last bin ends with the range: what lies past it was counted as above before
            width = min(1ull << shift, width - (bin << shift));
            lo += bin << shift;
        } else {
            lo = bin == 0 ? 0ull : kFirstBase + (bin << shift);
            width = bin == 0 ? kFirstBase + (1ull << shift) : (bin == 4095 ? 0ull - lo : 1ull << shift);
        }
        need -= s_pick[1];
        count = s_pick[2];
        if (width <= (1ull << low) || count <= kSelCand) break;
        __syncthreads();  // s_pick has been read
    }
    // the chunks' counts; the bin's states listed, or (every bit decided) counted as the tied ones
    const bool list = width > (1ull << low);
    if (tid == 0) s_own = 0;
    __syncthreads();
    for_chunks<WS>(src, S, c0, c1, wid, kSelWarps, status, [&](int64_t c, const unsigned long long (&k)[kU], unsigned ok) {
        unsigned na = 0, nt = 0;
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const bool v = (ok >> u & 1u) && k[u] >= lo, in = v && k[u] - lo < width;
            na += __popc(__ballot_sync(0xffffffffu, v && !in));
            if (list) {
                if (in) {
                    const unsigned slot = atomicAdd(ws.barrier + kTruncListed, 1u);
                    if (slot < kSelCand && slot < ws.cap) {
                        ws.cand[slot] = k[u];
                        ws.cand_idx[slot] = int(c * kTruncChunk + 32 * u + lane);
                    }
                }
            } else {
                nt += __popc(__ballot_sync(0xffffffffu, in));
            }
        }
        if (lane == 0) {
            const unsigned long long n = (unsigned long long)na | ((unsigned long long)nt << 31);
            ws.chunk[c] = n;
            atomicAdd(&s_own, n);
        }
    });
    long long ties = count;
    if (list) {
        if (!grid_wait()) return;
        // the need-th largest of the listed weights, 12 bits a round
        const int n = int(count);
        constexpr int kMine = kSelCand / kSelThreads, per = 4096 / kSelThreads;
        unsigned long long w[kMine];
        int wi[kMine];
#pragma unroll
        for (int q = 0; q < kMine; ++q) {
            const int i = tid + q * kSelThreads;
            const bool have = i < n && i < ws.cap;
            w[q] = have ? __ldcg(ws.cand + i) : 0ull;
            wi[q] = have ? __ldcg(ws.cand_idx + i) : -1;
        }
        while (width > (1ull << low)) {
            const int shift = max(bits_of(width) - 12, 0);
            __syncthreads();
            for (int b = tid; b < 4096; b += kSelThreads) h[b] = 0;
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kMine; ++q)
                if (wi[q] >= 0 && w[q] - lo < width) atomicAdd(&h[unsigned((w[q] - lo) >> shift)], 1u);
            __syncthreads();
            unsigned hb[per];
#pragma unroll
            for (int q = 0; q < per; ++q) hb[q] = h[tid * per + q];
            pick_bin<per>(hb, need, s_warp, s_pick);
            if (s_pick[0] < 0) {  // cannot happen, as above
                if (blockIdx.x == 0 && tid == 0) raise_status(status, PACES_ERR_BADARG);
                return;
            }
            const unsigned long long off = (unsigned long long)s_pick[0] << shift;
            width = min(1ull << shift, width - off);  // as above
            lo += off;
            need -= s_pick[1];
            ties = s_pick[2];
        }
        // this block's listed states join its chunks' counts
#pragma unroll
        for (int q = 0; q < kMine; ++q) {
            const int64_t c = wi[q] / kTruncChunk;
            if (wi[q] < 0 || c < c0 || c >= c1 || w[q] < lo) continue;
            const unsigned long long one = w[q] - lo >= width ? 1ull : 1ull << 31;
            atomicAdd(ws.chunk + c, one);
            atomicAdd(&s_own, one);
        }
    }
    // exclusive prefixes: the blocks' totals, then this block's chunks
    __syncthreads();
    if (tid == 0) ws.block_sum[blockIdx.x] = s_own;
    if (!grid_wait()) return;
    unsigned long long before, total;
    block_prefix(tid < blockIdx.x ? __ldcg(ws.block_sum + tid) : 0ull, s_sum, before);
    for (int64_t c = c0; c < c1; c += kSelThreads) {
        const unsigned long long v = c + tid < c1 ? __ldcg(ws.chunk + c + tid) : 0ull;
        const unsigned long long e = block_prefix(v, s_sum, total);
        if (c + tid < c1) ws.chunk[c + tid] = before + e;
        before += total;
    }
    if (blockIdx.x == 0 && tid == 0) {
        ws.sel[SEL_W + 0] = (long long)lo;
        ws.sel[SEL_W + 1] = -1;  // every bit decided
        ws.sel[SEL_W + 2] = need;
        ws.sel[SEL_W + 3] = 1;
        ws.sel[SEL_TIES] = ties;
        ws.sel[SEL_S] = S;
        ws.sel[SEL_ALL] = 0;
    }
}

__global__ void __launch_bounds__(256) trunc_hist_cand_kernel(TruncWs ws, int base, int round) {
    __shared__ unsigned h[4096];
    if (!ws.sel[base + 3]) return;
    const int bits = round_bits(round), shift = round_shift(round);
    const unsigned long long dm = (1ull << bits) - 1;
    for (int b = threadIdx.x; b < 4096; b += blockDim.x) h[b] = 0;
    __syncthreads();
    const long long nc = min(ws.sel[SEL_CAND], (long long)ws.cap);
    const unsigned long long pre = (unsigned long long)ws.sel[base + 0];
    const unsigned long long msk = (unsigned long long)ws.sel[base + 1];
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nc; c += (long long)gridDim.x * blockDim.x) {
        const unsigned long long k = ws.cand[c];
        if ((k & msk) == pre) atomicAdd(&h[(k >> shift) & dm], 1u);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < (1 << bits); b += blockDim.x)
        if (h[b]) atomicAdd(&ws.hist[b], h[b]);
}

// Decide whether the tie at the cut is shuffled; if so, collect the tied states' hashes.
__global__ void __launch_bounds__(1024) trunc_shuffle_prep_kernel(TruncWs ws, int* status) {
    for (int b = threadIdx.x; b < 4096; b += blockDim.x) ws.hist[b] = 0;
    if (threadIdx.x != 0) return;
    const long long ties = ws.sel[SEL_TIES];
    const long long need = ws.sel[SEL_W + 2];
    const bool active = ws.sel[SEL_W + 3] && ties > need;
    ws.sel[SEL_SHUFFLE] = active ? 1 : 0;
    if (active && double(ties) > 0.9 * double(ws.sel[SEL_S])) raise_status(status, PACES_ERR_SHUFFLE);
    ws.sel[SEL_H + 0] = 0;
    ws.sel[SEL_H + 1] = 0;
    ws.sel[SEL_H + 2] = need;
    ws.sel[SEL_H + 3] = active ? 1 : 0;
    ws.sel[SEL_CAND] = 0;
}

template <int WK>
__global__ void __launch_bounds__(256) trunc_collect_ties_kernel(const void* __restrict__ psi, TruncWs ws,
                                                                 uint64_t seed, uint64_t step, int* status) {
    if (!ws.sel[SEL_H + 3]) return;
    const int64_t S = ws.sel[SEL_S];
    const unsigned long long vstar = (unsigned long long)ws.sel[SEL_W + 0];
    const int lane = threadIdx.x & 31;
    for (int64_t i0 = blockIdx.x * int64_t(blockDim.x); i0 < S; i0 += int64_t(gridDim.x) * blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        bool take = false;
        if (i < S) take = weight_bits<WK>(psi, i, status) == vstar;
        const unsigned ballot = __ballot_sync(0xffffffffu, take);
        if (!ballot) continue;
        int basei = 0;
        if (lane == 0) basei = int(atomicAdd(reinterpret_cast<unsigned long long*>(&ws.sel[SEL_CAND]),
                                            (unsigned long long)__popc(ballot)));
        basei = __shfl_sync(0xffffffffu, basei, 0);
        if (take) {
            const int slot = basei + __popc(ballot & ((1u << lane) - 1));
            if (slot < ws.cap) {
                ws.cand[slot] = tie_hash(seed, step, i);
                ws.cand_idx[slot] = int(i);
            }
        }
    }
}

// With shuffled ties: the chunks' kept states (above the threshold, or tied and picked by the
// hash), then their prefixes.
template <int WK>
__global__ void __launch_bounds__(256) trunc_shuffle_count_kernel(const void* __restrict__ psi, TruncWs ws, uint64_t seed,
                                                                  uint64_t step, int* status) {
    if (ws.sel[SEL_ALL] || !ws.sel[SEL_SHUFFLE]) return;
    const int64_t S = ws.sel[SEL_S];
    const unsigned long long vstar = (unsigned long long)ws.sel[SEL_W + 0];
    const unsigned long long hstar = (unsigned long long)ws.sel[SEL_H + 0];
    const int lane = threadIdx.x & 31;
    for_chunks<WK>(psi, S, 0, (S + kTruncChunk - 1) / kTruncChunk, int(blockIdx.x * 8 + (threadIdx.x >> 5)), int(gridDim.x * 8),
                   status, [&](int64_t c, const unsigned long long (&k)[kU], unsigned ok) {
                       unsigned n = 0;
#pragma unroll
                       for (int u = 0; u < kU; ++u) {
                           const bool keep = (ok >> u & 1u) &&
                                             (k[u] > vstar || (k[u] == vstar &&
                                                               tie_hash(seed, step, c * kTruncChunk + 32 * u + lane) >= hstar));
                           n += __popc(__ballot_sync(0xffffffffu, keep));
                       }
                       if (lane == 0) ws.chunk[c] = n;
                   });
}

__global__ void __launch_bounds__(1024) trunc_shuffle_scan_kernel(TruncWs ws) {
    __shared__ unsigned long long s_sum[32];
    if (ws.sel[SEL_ALL] || !ws.sel[SEL_SHUFFLE]) return;
    const int64_t nch = (ws.sel[SEL_S] + kTruncChunk - 1) / kTruncChunk;
    unsigned long long before = 0, total;
    for (int64_t c = threadIdx.x; c - threadIdx.x < nch; c += blockDim.x) {
        const unsigned long long e = block_prefix(c < nch ? ws.chunk[c] : 0ull, s_sum, total);
        if (c < nch) ws.chunk[c] = before + e;
        before += total;
    }
}

// The compaction: a warp holds the weights of a chunk's 256 consecutive states in registers,
// ballots and the chunk's prefix give every kept state its rank among the kept ones.  Lanes
// read consecutive keys and the kept ones write consecutive outputs, so both sides coalesce,
// and no warp waits for another (a look-back over 1024-state tiles in place of the prefixes:
// 158 us at 15.2M states).
// The weights come from `wsrc` (kind WK); when every state is kept the selection rounds
// did not run, so the out_w weights come from `psi` (kind WKA).  The last block to finish
// writes the offsets of empty exciton blocks and the counts.
template <int NW, int WK, int WKA>
__global__ void __launch_bounds__(256, NW <= 2 ? 4 : (NW <= 4 ? 3 : 2)) trunc_write_kernel(ModelDev m, const uint64_t* __restrict__ x_keys,
                                                          const int* __restrict__ x_blk,
                                                          const void* __restrict__ wsrc,
                                                          const void* __restrict__ psi, TruncWs ws, int64_t maxstates,
                                                          uint64_t seed, uint64_t step,
                                                          uint64_t* __restrict__ out_keys,
                                                          int* __restrict__ out_blk, int64_t out_cap,
                                                          float* __restrict__ out_w, int* n_tied_out, int* n_kept_out,
                                                          int* status) {
    __shared__ int s_blk[kMaxSites + 1];
    const int L = m.L;
    for (int i = threadIdx.x; i <= L; i += blockDim.x) s_blk[i] = x_blk[i];
    __syncthreads();
    const bool gave_up = ws.barrier[kTruncGaveUp] != 0;  // nothing is written
    const int64_t S = gave_up ? 0 : ws.sel[SEL_S];
    const bool all = gave_up || ws.sel[SEL_ALL] != 0;
    const unsigned long long vstar = (unsigned long long)ws.sel[SEL_W + 0];
    const long long skip_ties = ws.sel[SEL_TIES] - ws.sel[SEL_W + 2];  // tied states dropped (the lowest indices)
    const bool shuf = ws.sel[SEL_SHUFFLE] != 0;
    const unsigned long long hstar = (unsigned long long)ws.sel[SEL_H + 0];
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    auto place = [&](int64_t c, const unsigned long long (&k)[kU], unsigned ok) {
        const int64_t q0 = c * kTruncChunk;
        const unsigned long long b = all ? (unsigned long long)q0 : __ldg(ws.chunk + c);
        long long T = (long long)(b >> 31);  // tied states before the chunk
        long long out = (long long)(b & 0x7fffffffull);
        if (!all && !shuf) out += max(0ll, T - skip_ties);
        const long long out0 = out;
        unsigned kept[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const bool v = ok >> u & 1u;
            const bool eq = v && !all && k[u] == vstar;
            bool keep = v && (all || k[u] > vstar);
            if (shuf) {
                keep |= eq && tie_hash(seed, step, q0 + 32 * u + lane) >= hstar;
            } else {
                const unsigned tie = __ballot_sync(0xffffffffu, eq);
                keep |= eq && T + __popc(tie & lt_mask) >= skip_ties;
                T += __popc(tie);
            }
            kept[u] = __ballot_sync(0xffffffffu, keep);
        }
        constexpr int kG = 4;  // keys in flight per lane
#pragma unroll
        for (int g = 0; g < kU; g += kG) {
            Key<NW> kk[kG];
#pragma unroll
            for (int u = 0; u < kG; ++u)
                if (kept[g + u] >> lane & 1u) kk[u] = load_key<NW>(x_keys, q0 + 32 * (g + u) + lane);
#pragma unroll
            for (int u = 0; u < kG; ++u) {
                if (kept[g + u] >> lane & 1u) {
                    const long long o = out + __popc(kept[g + u] & lt_mask);
                    if (o < out_cap) {
                        store_key<NW>(out_keys, o, kk[u]);
                        if (out_w) out_w[o] = float(__longlong_as_double((long long)k[g + u]));
                    } else {
                        raise_status(status, PACES_ERR_CAPACITY);
                    }
                }
                out += __popc(kept[g + u]);
            }
        }
        // exciton blocks that start among the chunk's states: the kept states before them
        for (int p = lane; p < L; p += 32) {
            const int64_t e = int64_t(s_blk[p]) - q0;
            if (e < 0 || e >= kTruncChunk || s_blk[p] >= s_blk[p + 1]) continue;
            long long o = out0;
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                if (u < int(e >> 5)) o += __popc(kept[u]);
                else if (u == int(e >> 5)) o += __popc(kept[u] & ((1u << (e & 31)) - 1u));
            }
            out_blk[p] = int(o);
        }
    };
    const int64_t nch = (S + kTruncChunk - 1) / kTruncChunk;
    const int w = int(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)), warps = int(gridDim.x * (blockDim.x >> 5));
    if (all) for_chunks<WKA>(psi, S, 0, nch, w, warps, status, place);
    else for_chunks<WK>(wsrc, S, 0, nch, w, warps, status, place);
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(ws.barrier + kTruncDone, 1u) != gridDim.x - 1) return;
    __threadfence();
    // the cut: |psi| of the smallest kept state when states were dropped, else 0
    if (out_w) out_w[out_cap] = all ? 0.f : float(__longlong_as_double((long long)vstar));
    long long total = all ? S : maxstates;
    if (total > out_cap) {
        raise_status(status, PACES_ERR_CAPACITY);
        total = out_cap;
    }
    if (ws.sel[SEL_CAND] > ws.cap) raise_status(status, PACES_ERR_CAPACITY);
    out_blk[L] = int(total);
    for (int p = L - 1; p >= 0; --p)  // (no states: every block is empty)
        if (S == 0 || s_blk[p] == s_blk[p + 1]) out_blk[p] = __ldcg(out_blk + p + 1);
    if (n_tied_out) *n_tied_out = int(all ? 0 : ws.sel[SEL_TIES]);
    if (n_kept_out) *n_kept_out = int(total);
}

// WK: the kind of `psi`.  WKS: the kind the passes after round 0 read from `src` -- WK
// itself reading `psi`, or the stored kind reading the weights round 0 wrote to scratch.
template <int NW, int WK, int WKS>
int launch_truncate_t(const ModelDev& m, const uint64_t* x_keys, const int* x_blk, const void* psi, void* scratch,
                      int64_t maxstates, int shuffle, uint64_t seed, uint64_t step, const TruncWs& ws,
                      uint64_t* out_keys, int* out_blk, int64_t out_cap, float* out_w, int* n_tied_out, int* n_kept_out,
                      int* status, int num_sms, int sel_sms, cudaStream_t st) {
    constexpr bool kStore = WKS != WK;
    const void* src = kStore ? scratch : psi;
    const int g = grid_for(ws.cap, 1024, num_sms * 4);  // streaming passes of the tie shuffle
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid_for(ws.cap, kSelThreads * 2, sel_sms));
        cfg.blockDim = dim3(kSelThreads);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, trunc_threshold_kernel<WK, kStore>, m.L, x_blk, psi, ws, maxstates, scratch,
                               weight_low_bit(WK), status) != cudaSuccess)
            return PACES_ERR_CUDA;
    }
    if (shuffle) {
        trunc_shuffle_prep_kernel<<<1, 1024, 0, st>>>(ws, status);
        trunc_collect_ties_kernel<WKS><<<g, 256, 0, st>>>(src, ws, seed, step, status);
        for (int r = 0; r < kRounds; ++r) {
            trunc_hist_cand_kernel<<<g, 256, 0, st>>>(ws, SEL_H, r);
            trunc_select_kernel<<<1, 1024, 0, st>>>(ws, SEL_H, r);
        }
        trunc_shuffle_count_kernel<WKS><<<g, 256, 0, st>>>(src, ws, seed, step, status);
        trunc_shuffle_scan_kernel<<<1, 1024, 0, st>>>(ws);
    }
    trunc_write_kernel<NW, WKS, WK><<<grid_for(ws.cap, 8 * kTruncChunk, num_sms * 8), 256, 0, st>>>(
        m, x_keys, x_blk, src, psi, ws, maxstates, seed, step, out_keys, out_blk, out_cap, out_w, n_tied_out, n_kept_out,
        status);
    return cudaGetLastError() == cudaSuccess ? PACES_OK : PACES_ERR_CUDA;
}

template <int NW>
int dispatch_prec(bool c64, const ModelDev& m, const uint64_t* x_keys, const int* x_blk,
                  const void* psi, const double* weights, void* scratch, int64_t maxstates, int shuffle, uint64_t seed,
                  uint64_t step, const TruncWs& ws, uint64_t* out_keys, int* out_blk, int64_t out_cap,
                  float* out_w, int* n_tied_out, int* n_kept_out, int* status, int num_sms, int sel_sms, cudaStream_t st) {
#define PACES_TRUNC_LAUNCH(WK, WKS, SRC)                                                                     \
    return launch_truncate_t<NW, WK, WKS>(m, x_keys, x_blk, SRC, scratch, maxstates, shuffle, seed, step, ws, \
                                          out_keys, out_blk, out_cap, out_w, n_tied_out, n_kept_out, status,  \
                                          num_sms, sel_sms, st)
    if (weights) PACES_TRUNC_LAUNCH(2, 2, weights);
    if (c64) {
        if (scratch) PACES_TRUNC_LAUNCH(1, stored_kind(1), psi);
        PACES_TRUNC_LAUNCH(1, 1, psi);
    }
    if (scratch) PACES_TRUNC_LAUNCH(0, stored_kind(0), psi);
    PACES_TRUNC_LAUNCH(0, 0, psi);
#undef PACES_TRUNC_LAUNCH
}

}  // namespace

int launch_truncate(int nw, bool c64, const ModelDev& m, const uint64_t* x_keys, const int* x_blk,
                    const void* psi, const double* weights, void* scratch, int64_t maxstates, int shuffle, uint64_t seed,
                    uint64_t step, const TruncWs& ws, uint64_t* out_keys, int* out_blk, int64_t out_cap, float* out_w,
                    int* n_tied_out, int* n_kept_out, int* status, int num_sms, int sel_sms, cudaStream_t st,
                    bool cleared) {
    if (!cleared && cudaMemsetAsync(ws.hist, 0, kTruncHistBytes, st) != cudaSuccess) return PACES_ERR_CUDA;
#define PACES_TRUNC_CASE(N)                                                                       \
    case N:                                                                                       \
        return dispatch_prec<N>(c64, m, x_keys, x_blk, psi, weights, scratch, maxstates, shuffle, seed, step, ws, \
                                out_keys, out_blk, out_cap, out_w, n_tied_out, n_kept_out, status, num_sms, sel_sms, st);
    switch (nw) {
        PACES_TRUNC_CASE(1)
        PACES_TRUNC_CASE(2)
        PACES_TRUNC_CASE(3)
        PACES_TRUNC_CASE(4)
        PACES_TRUNC_CASE(5)
        PACES_TRUNC_CASE(6)
        PACES_TRUNC_CASE(7)
        PACES_TRUNC_CASE(8)
        default: return PACES_ERR_BADARG;
    }
#undef PACES_TRUNC_CASE
}

}  // namespace paces
