// select.cu -- selection kernels.
//
//  * sample_threshold_kernel: per query, the K-th best approximate score of a doc sample, lowered by
//    the error bounds into a threshold that every true top-K doc is guaranteed to clear.
//  * select_topk_kernel: per query, from the candidate list: the K-th best approximate score, the
//    set of candidates that can still reach the top K, their exact FP32 rescoring in the ground
//    truth's order, and the final deterministic top K (score desc, doc id asc).
//  * aggregate_* kernels: stable compaction of (score, location) by the filter bitmap -- the
//    reference's Aggregator operator (kernel_aggregator.h:18-206) without the host count round trip.
//  * topk_op_kernel: exact top K of a compacted (score, location) list -- the reference's TOPK
//    operator (kernel_topk.h:27-419), which there is only a pivot pre-select followed by a host sort.
#include <cooperative_groups.h>

#include <atomic>

#include "hss_device.cuh"
#include "hss_kernels.h"

namespace cg = cooperative_groups;

namespace hss {
namespace {

// threads of a CTA: 1,024 in the TOPK operator, the threshold of a listed sample or pass, and, for batches of at most
// as many queries as SMs, the select step and the threshold of group maxima; else these two take 512
constexpr int kST = 1024;
constexpr int kSelT = 512;
constexpr int kBins = 4096;           // histogram bins: 12-bit digits
// candidate scores a CTA holds in shared memory: the usual select form (two CTAs of 512 threads per SM),
// the form for few queries or for lists that run long (large K; one CTA of 1,024), the threshold kernels
constexpr uint32_t kFast = 8192;
constexpr uint32_t kFastLarge = 32768;
constexpr uint32_t kFastSample = 20480;

struct HistSmem {
    __align__(16) uint32_t hist[kBins];
    uint32_t wsum[32], wmax[32];
    uint32_t bcast[4];
    uint32_t counter, total, lost;
};

struct SelectSmem : HistSmem {
    __align__(16) unsigned long long sortbuf[kMaxTopK];  // keys to sort
    uint32_t locs[kMaxTopK];  // select: locations of the first list entries; TOPK: a slice of the bins
};

// The next place of a list counted in shared memory, one addition per warp for its active lanes.
__device__ __forceinline__ uint32_t next_place(uint32_t* counter) {
    const uint32_t active = __activemask(), lane = threadIdx.x & 31;
    const uint32_t leader = __ffs(active) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, static_cast<uint32_t>(__popc(active)));
    return __shfl_sync(active, base, leader) + __popc(active & ((1u << lane) - 1u));
}

// Picks, from the top of a 4096-bin histogram, the bin holding the k-th largest key (blockDim.x == NT:
// thread t owns the 4096 / NT bins below 4096 (NT - t) / NT). Returns the bin; *krem becomes the rank
// inside it and *in_bin (if given) the keys it holds. The caller has synchronised after the last
// addition; a synchronisation lies between this and the next use of S.wsum and S.bcast.
template <int NT>
__device__ inline uint32_t pick_digit4096(const uint32_t* hist, uint32_t* krem, HistSmem& S,
                                          uint32_t* in_bin = nullptr) {
    constexpr int B = kBins / NT;
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t kr = *krem;
    uint32_t h[B], local = 0;  // h[j]: bin kBins - 1 - B t - j
#pragma unroll
    for (int j = 0; j < B; j += 4) {
        const uint4 x = *reinterpret_cast<const uint4*>(hist + kBins - B * t - j - 4);
        h[j] = x.w;
        h[j + 1] = x.z;
        h[j + 2] = x.y;
        h[j + 3] = x.x;
        local += x.x + x.y + x.z + x.w;
    }
    uint32_t x = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= static_cast<uint32_t>(o)) x += y;
    }
    if (lane == 31) S.wsum[warp] = x;
    __syncthreads();
    // every warp adds up the warps before it
    const uint32_t before = warp_sum(lane < warp ? S.wsum[lane] : 0u);
    const uint32_t incl = before + x, excl = incl - local;
    if (excl < kr && incl >= kr) {  // exactly one thread
        uint32_t cum = excl;
#pragma unroll
        for (int j = 0; j < B; ++j) {
            if (cum + h[j] >= kr) {
                S.bcast[0] = kBins - 1 - B * t - j;
                S.bcast[1] = kr - cum;
                S.bcast[2] = h[j];
                break;
            }
            cum += h[j];
        }
    }
    __syncthreads();
    *krem = S.bcast[1];
    if (in_bin) *in_bin = S.bcast[2];
    return S.bcast[0];
}

template <int NT>
__device__ __forceinline__ void clear_hist(HistSmem& S) {
    for (uint32_t i = threadIdx.x; i < kBins / 4; i += NT) reinterpret_cast<uint4*>(S.hist)[i] = make_uint4(0, 0, 0, 0);
}

// Adds digits to a histogram, each thread merging its runs of equal digits before it does (keys of one
// query cluster, so consecutive keys mostly share a digit). flush() before the histogram is read.
struct RunAdder {
    uint32_t* hist;
    uint32_t cur = 0, cnt = 0;
    __device__ __forceinline__ explicit RunAdder(uint32_t* h) : hist(h) {}
    __device__ __forceinline__ void add(uint32_t d) {
        if (d != cur) {
            if (cnt) atomicAdd(&hist[cur], cnt);
            cur = d;
            cnt = 0;
        }
        ++cnt;
    }
    __device__ __forceinline__ void flush() {
        if (cnt) atomicAdd(&hist[cur], cnt);
        cnt = 0;
    }
};

// Smallest and largest of the block's u32 keys (each thread's in lo, hi; none: lo > hi), in every
// thread afterwards. S.wsum and S.wmax are used, once between two synchronisations.
template <int NT>
__device__ __forceinline__ void block_minmax(uint32_t& lo, uint32_t& hi, HistSmem& S) {
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        S.wsum[warp] = lo;
        S.wmax[warp] = hi;
    }
    __syncthreads();
    lo = __reduce_min_sync(0xffffffffu, lane < NT / 32 ? S.wsum[lane] : 0xffffffffu);
    hi = __reduce_max_sync(0xffffffffu, lane < NT / 32 ? S.wmax[lane] : 0u);
}

// A lower bound of the k-th largest (1-based, k <= the number of keys) of the u32 keys that visit(fn)
// hands to fn, all of them in [lo, hi]: at least k keys are >= it -- all a proven threshold or a
// rescoring cut needs -- and it shares the k-th key's top 24 bits at least (as an order-preserving float
// key it is at most 2^-15, relatively, below). Two passes over a 4096-bin histogram: the bins of the first
// divide [lo, hi], those of the second the k-th key's bin. Digits of the keys themselves would crowd a few
// bins, whose shared-memory additions serialise: a query's scores share their exponents.
template <int NT, class Visit>
__device__ __forceinline__ uint32_t kth_lower_bound(Visit visit, uint32_t k, uint32_t lo, uint32_t hi, HistSmem& S) {
    uint32_t krem = k;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        const int bits = 32 - __clz(hi - lo);
        const int shift = bits > 12 ? bits - 12 : 0;
        __syncthreads();
        clear_hist<NT>(S);
        __syncthreads();
        RunAdder add(S.hist);
        visit([&](uint32_t v) {
            if (v - lo <= hi - lo) add.add((v - lo) >> shift);
        });
        add.flush();
        __syncthreads();
        lo += pick_digit4096<NT>(S.hist, &krem, S) << shift;
        hi = lo + ((1u << shift) - 1u);
        if (shift == 0) break;
    }
    return lo;
}

// A lower bound of the k-th largest (1-based) of the finite scores that visit(fn) hands to fn, all of them
// in [lo, hi], k <= their number: at least k of them are >= it. The 4096 bins divide [lo, hi] evenly (a
// monotone map, so a score in a higher bin is a higher score): scores of both signs, whose keys would
// crowd the bins of a few exponents, spread over them. The bound is the least score of the k-th's bin;
// where that bin is crowded (an outlier stretches the range, or many equal scores) it is refined by keys.
template <int NT, class Visit>
__device__ __forceinline__ float kth_score_bound(Visit visit, uint32_t k, float lo, float hi, HistSmem& S) {
    const float scale = 4096.0f / (hi - lo);
    uint32_t krem = k, in_bin = 0;
    uint32_t key_lo = float_key(lo), key_hi = float_key(hi);
    if (scale > 0.0f && scale < 1e30f) {  // else: equal scores, or a range past the floats
        auto bin = [&](float v) { return min(static_cast<uint32_t>((v - lo) * scale), 4095u); };
        __syncthreads();
        clear_hist<NT>(S);
        __syncthreads();
        visit([&](float v) { atomicAdd(&S.hist[bin(v)], 1u); });
        __syncthreads();
        const uint32_t d = pick_digit4096<NT>(S.hist, &krem, S, &in_bin);
        uint32_t a = 0xffffffffu, b = 0;
        visit([&](float v) {
            if (bin(v) == d) {
                a = min(a, float_key(v));
                b = max(b, float_key(v));
            }
        });
        block_minmax<NT>(a, b, S);
        if (in_bin <= 64u) return key_float(a);
        key_lo = a;
        key_hi = b;
    }
    return key_float(kth_lower_bound<NT>([&](auto fn) { visit([&](float v) { fn(float_key(v)); }); }, krem, key_lo,
                                         key_hi, S));
}

// A lower bound of the k-th largest of n u64 keys key(i) that at most kMaxTopK keys reach, where there is
// one (else the k-th largest itself).
template <int NT, class KeyFn>
__device__ __forceinline__ uint64_t kth_bound_u64(KeyFn key, uint32_t n, uint32_t k, HistSmem& S) {
    uint64_t prefix = 0, mask = 0;
    uint32_t krem = k, in_bin = 0;
    const int shifts[6] = {52, 40, 32, 20, 8, 0};
#pragma unroll 1
    for (int p = 0; p < 6; ++p) {
        const int shift = shifts[p];
        const uint64_t digit = p == 2 || p == 5 ? 255ull : 4095ull;
        __syncthreads();
        clear_hist<NT>(S);
        __syncthreads();
        RunAdder add(S.hist);
        for (uint32_t i = threadIdx.x; i < n; i += NT) {
            const uint64_t v = key(i);
            if ((v & mask) == prefix) add.add(static_cast<uint32_t>((v >> shift) & digit));
        }
        add.flush();
        __syncthreads();
        const uint64_t d = pick_digit4096<NT>(S.hist, &krem, S, &in_bin);
        prefix |= d << shift;
        mask |= digit << shift;
        if ((k - krem) + in_bin <= static_cast<uint32_t>(kMaxTopK)) break;
    }
    return prefix;
}

// Calls fn(index, valid, score) for every stored entry of a query's segmented list of scores src (counts:
// per-segment counts, seg_cap the most a segment stores), in no particular order. A warp takes up to 32
// segments at a time, a lane each, and walks their entries flattened: lane l's entry belongs to the last
// segment that starts at or before it, found by five shuffles, so the loads are coalesced within a
// segment, independent and eight per thread in flight, and no block-wide scan or barrier is needed. Every
// call is made by a full warp (valid = false past the end), so fn may use warp collectives; begin(m) is
// called by the full warp before a group's m entries. LONG: segments of 64 entries or more on average are
// walked one after the other, without the lookups (doc-sample lists hold about 110 a segment). Returns whether
// a segment of this lane lost entries.
template <int NT, bool LONG, class Begin, class Fn>
__device__ __forceinline__ bool walk_segments(const uint32_t* counts, uint32_t segs, uint32_t seg_cap, const float* src,
                                              Begin begin, Fn fn) {
    constexpr uint32_t U = 8, kLong = 4, kWarps = NT / 32;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // segments per warp and round: as even a share as 32 lanes allow
    const uint32_t rounds = (segs + 32 * kWarps - 1) / (32 * kWarps);
    const uint32_t per = (segs + kWarps * rounds - 1) / (kWarps * rounds);
    bool lost = false;
    for (uint32_t g0 = warp * per; g0 < segs; g0 += kWarps * per) {
        uint32_t c = lane < per && g0 + lane < segs ? counts[g0 + lane] : 0u;
        lost |= c > seg_cap;
        c = min(c, seg_cap);
        uint32_t x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= static_cast<uint32_t>(o)) x += y;
        }
        const uint32_t off = x - c, total = __shfl_sync(0xffffffffu, x, 31);
        if (total == 0) continue;
        if (LONG && total >= 64 * per) {
            for (uint32_t j = 0; j < per; ++j) {
                const uint32_t m = __shfl_sync(0xffffffffu, c, j);
                if (m == 0) continue;
                begin(m);
                const uint32_t first = (g0 + j) * seg_cap;
                for (uint32_t b = 0; b < m; b += 32 * kLong) {
                    float v[kLong];
#pragma unroll
                    for (uint32_t u = 0; u < kLong; ++u) {
                        const uint32_t idx = b + 32 * u + lane;
                        v[u] = idx < m ? src[first + idx] : 0.0f;
                    }
#pragma unroll
                    for (uint32_t u = 0; u < kLong; ++u) {
                        if (b + 32 * u >= m) break;  // warp-uniform
                        fn(first + b + 32 * u + lane, b + 32 * u + lane < m, v[u]);
                    }
                }
            }
            continue;
        }
        begin(total);
        for (uint32_t b = 0; b < total; b += 32 * U) {
            uint32_t at[U];
            float v[U];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t idx = b + 32 * u + lane;
                uint32_t lo = 0;
#pragma unroll
                for (uint32_t step = 16; step > 0; step >>= 1) {
                    const uint32_t o = __shfl_sync(0xffffffffu, off, lo + step);
                    if (o <= idx) lo += step;
                }
                at[u] = (g0 + lo) * seg_cap + idx - __shfl_sync(0xffffffffu, off, lo);
                v[u] = idx < total ? src[at[u]] : 0.0f;
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                if (b + 32 * u >= total) break;  // warp-uniform
                fn(at[u], b + 32 * u + lane < total, v[u]);
            }
        }
    }
    return lost;
}

// The first walk of a list: scores into `cache` (as many as fit), where locs is given the locations of the
// first kMaxTopK too, and the smallest and largest key. Returns the number of entries; *overflow = some
// segment lost entries. Synchronised at its end.
template <int NT, bool LONG>
__device__ __forceinline__ uint32_t load_list(HistSmem& S, const uint32_t* counts, uint32_t segs, uint32_t seg_cap,
                                              const float* src, const uint32_t* loc_src, float* cache, uint32_t cap,
                                              uint32_t* locs, bool* overflow, uint32_t* key_lo, uint32_t* key_hi) {
    if (threadIdx.x == 0) {
        S.counter = 0;
        S.lost = 0;
    }
    __syncthreads();
    uint32_t pos = 0, lo = 0xffffffffu, hi = 0;
    const uint32_t lane = threadIdx.x & 31;
    const bool lost = walk_segments<NT, LONG>(
        counts, segs, seg_cap, src,
        [&](uint32_t m) {
            if (lane == 0) pos = atomicAdd(&S.counter, m);
            pos = __shfl_sync(0xffffffffu, pos, 0) + lane;
        },
        [&](uint32_t at, bool ok, float v) {
            if (ok) {
                if (locs && pos < static_cast<uint32_t>(kMaxTopK)) locs[pos] = loc_src[at];
                if (pos < cap) cache[pos] = v;
                const uint32_t key = float_key(v);
                lo = min(lo, key);
                hi = max(hi, key);
            }
            pos += 32;
        });
    if (lost) S.lost = 1;
    block_minmax<NT>(lo, hi, S);
    *key_lo = lo;
    *key_hi = hi;
    *overflow = S.lost != 0;
    const uint32_t n = S.counter;
    __syncthreads();  // every thread has read the count: the caller may clear it at once
    return n;
}

// Sorts E keys per thread (key of index t + NT e in v[e]) of the first m / E threads descending:
// a bitonic network whose exchanges over a distance below 32 are shuffles and whose exchanges over NT
// and more stay inside a thread, so only the distances between go through shared memory and a barrier of
// the m / E threads (for 512 keys 10 of the 45 steps).
template <int NT, int E>
__device__ __forceinline__ void bitonic_regs(unsigned long long* buf, uint32_t m) {
    const uint32_t t = threadIdx.x, threads = E == 1 ? m : static_cast<uint32_t>(NT);
    auto bar = [&] { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); };
    unsigned long long v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = buf[t + static_cast<uint32_t>(NT) * e];
    for (uint32_t k = 2; k <= m; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            if (E > 1 && j >= static_cast<uint32_t>(NT)) {
#pragma unroll
                for (int de = E / 2; de > 0; de >>= 1) {  // compile-time register indices
                    if (j != static_cast<uint32_t>(NT) * de) continue;
#pragma unroll
                    for (int e = 0; e < E; ++e) {
                        if (e & de) continue;
                        const bool desc = ((t + static_cast<uint32_t>(NT) * e) & k) == 0;
                        const unsigned long long a = v[e], b = v[e + de];
                        if (desc ? (a < b) : (a > b)) {
                            v[e] = b;
                            v[e + de] = a;
                        }
                    }
                }
                continue;
            }
            if (j >= 32) {
                bar();  // the previous step's reads are done
#pragma unroll
                for (int e = 0; e < E; ++e) buf[t + static_cast<uint32_t>(NT) * e] = v[e];
                bar();
            }
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const unsigned long long o = j >= 32 ? buf[(t ^ j) + static_cast<uint32_t>(NT) * e]
                                                     : __shfl_xor_sync(0xffffffffu, v[e], j);
                // the lower index of a descending pair keeps the larger key
                const uint32_t i = t + static_cast<uint32_t>(NT) * e;
                const bool larger = ((i & k) == 0) == ((i & j) == 0);
                if (larger ? (o > v[e]) : (o < v[e])) v[e] = o;
            }
        }
    }
    bar();
#pragma unroll
    for (int e = 0; e < E; ++e) buf[t + static_cast<uint32_t>(NT) * e] = v[e];
}

// Sorts S.sortbuf[0..m) descending; m is a power of two, 32 <= m <= kMaxTopK (sort_size).
template <int NT>
__device__ __forceinline__ void bitonic_desc(SelectSmem& S, uint32_t m) {
    if (m <= static_cast<uint32_t>(NT)) {
        if (threadIdx.x < m) bitonic_regs<NT, 1>(S.sortbuf, m);
    } else if (m == 2u * NT) {
        bitonic_regs<NT, 2>(S.sortbuf, m);
    } else if (m == 4u * NT) {
        bitonic_regs<NT, 4>(S.sortbuf, m);
    } else if constexpr (kMaxTopK > 4 * NT) {
        bitonic_regs<NT, 8>(S.sortbuf, m);
    }
    __syncthreads();
}

// Keys a sort of n takes: the power of two at least n, at least a warp's 32.
__device__ inline uint32_t sort_size(uint32_t n) {
    uint32_t m = 32;
    while (m < n) m <<= 1;
    return m;
}

// Sorts n (<= kRankSort) distinct keys of S.sortbuf into `out` by counting, for each, the keys that precede
// it, NT / 256 threads to a key: no barrier between steps (256 keys: 1 us against 2 us by the network).
constexpr uint32_t kRankSort = 256;
template <int NT>
__device__ __forceinline__ void rank_sort(const SelectSmem& S, uint32_t n, unsigned long long* out) {
    constexpr uint32_t W = NT / kRankSort;  // 2 or 4 neighbouring lanes
    const uint32_t i = threadIdx.x / W, w = threadIdx.x % W;
    const unsigned long long key = i < n ? S.sortbuf[i] : 0ull;
    uint32_t before = 0;
    if (i < n) {
#pragma unroll 4
        for (uint32_t j = w; j < n; j += W) {
            const unsigned long long o = S.sortbuf[j];
            before += o > key || (o == key && j < i) ? 1u : 0u;
        }
    }
#pragma unroll
    for (uint32_t o = 1; o < W; o <<= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (i < n && w == 0) out[before] = key;
    __syncthreads();
}

// Zeros after the first `got` (<= kMaxTopK) keys of S.sortbuf up to the sort's size, which it returns.
template <int NT>
__device__ __forceinline__ uint32_t pad_sort(SelectSmem& S, uint32_t got) {
    const uint32_t m = sort_size(got);
    for (uint32_t i = got + threadIdx.x; i < m; i += NT) S.sortbuf[i] = 0ull;
    __syncthreads();
    return m;
}

// Brings the top `kq` (<= kMaxTopK) of n u64 keys key(i) (and possibly more) into S.sortbuf, unsorted,
// filled up with zeros to sort_size() entries, which it returns. Lists past 512 keys of which less than half is
// wanted are cut at a lower bound of the kq-th key first, so that the sort takes about kq keys.
constexpr uint32_t kCutKeys = 512;

template <int NT, class KeyFn>
__device__ __forceinline__ uint32_t gather_top_keys(KeyFn key, uint32_t n, uint32_t kq, SelectSmem& S) {
    uint32_t got;
    if (n <= kCutKeys || (n <= static_cast<uint32_t>(kMaxTopK) && n <= 2 * kq)) {
        for (uint32_t i = threadIdx.x; i < n; i += NT) S.sortbuf[i] = key(i);
        got = n;
    } else {
        const uint64_t lb =
            n <= static_cast<uint32_t>(kMaxTopK)
                ? static_cast<uint64_t>(kth_lower_bound<NT>(
                      [&](auto fn) {
                          for (uint32_t i = threadIdx.x; i < n; i += NT) fn(static_cast<uint32_t>(key(i) >> 32));
                      },
                      kq, 0u, 0xffffffffu, S))
                      << 32
                : kth_bound_u64<NT>(key, n, kq, S);
        if (threadIdx.x == 0) S.counter = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += NT) {
            const uint64_t v = key(i);
            if (v >= lb) {
                const uint32_t pos = next_place(&S.counter);
                if (pos < static_cast<uint32_t>(kMaxTopK)) S.sortbuf[pos] = v;
            }
        }
        __syncthreads();
        got = min(S.counter, static_cast<uint32_t>(kMaxTopK));
    }
    return pad_sort<NT>(S, got);
}

// ---------------------------------------------------------------------------------------------
// The threshold of a sample or of a first candidate pass. One CTA per query; bound by a chain of
// dependent steps (counts, entries, two digits), so the list is read once, into shared memory where it
// fits (`held` entries). 1,024 threads and long segments walked as they lie: with a threshold model,
// whose sample is kept as lists, 256 queries on 10M docs 1214 us a batch (K 1000: 1866) with 512 threads and
// a lookup per entry, 1190 (1785) now; 8-bit form, whose raises read long lists, 1M docs, 256 queries, K 100
// 877 -> 819; other raises even.
__global__ void __launch_bounds__(kST) sample_threshold_kernel(SampleThresholdLaunch L, uint32_t held) {
    constexpr int NT = kST;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HistSmem& S = *reinterpret_cast<HistSmem*>(smem_raw);
    float* cs = reinterpret_cast<float*>(smem_raw + sizeof(HistSmem));
    launch_dependents();
    wait_for_previous();
    const uint32_t qi = L.qlist ? L.qlist[blockIdx.x] : blockIdx.x;
    const uint32_t k = L.topk[qi];
    const uint32_t* counts = L.count + static_cast<uint64_t>(qi) * kMaxCandSegs;
    const float* sc = L.score + static_cast<uint64_t>(qi) * L.cap;
    bool lost = false;  // a sample segment that overflowed only lowers the sample's K-th best
    uint32_t key_lo, key_hi;
    const uint32_t n = load_list<NT, true>(S, counts, L.segs, L.seg_cap, sc, nullptr, cs, held, nullptr, &lost, &key_lo,
                                           &key_hi);
    auto visit = [&](auto fn) {
        if (n <= held) {
            for (uint32_t i = threadIdx.x; i < n; i += NT) fn(float_key(cs[i]));
        } else {
            walk_segments<NT, true>(counts, L.segs, L.seg_cap, sc, [](uint32_t) {}, [&](uint32_t, bool ok, float v) {
                if (ok) fn(float_key(v));
            });
        }
    };
    // with statistics, absolute digits: the features keep the 24-bit prefixes of the keys they stand for
    if (L.stats) {
        key_lo = 0;
        key_hi = 0xffffffffu;
    }
    float theta = L.raise_only ? L.theta[qi] : -INFINITY;
    if (k > 0 && n >= k) {
        // a lower bound of the K-th best serves the proof below as well as the K-th best itself
        const uint32_t kk = kth_lower_bound<NT>(visit, k, key_lo, key_hi, S);
        // k sample docs score >= t approximately, so the true K-th best exact score is >= t - eps_s;
        // a true top-K doc therefore scores >= t - eps_s - eps_m under the main pass's arithmetic.
        const float t = __fsub_rd(__fsub_rd(key_float(kk), L.eps_sample[qi]), L.eps_main[qi]);
        theta = L.raise_only ? fmaxf(theta, t) : t;
        if (L.stats && threadIdx.x == 0)
            L.stats[static_cast<uint64_t>(qi) * kSampleStats + kSampleRanks] = key_float(kk);
        if (L.theta_also && L.raise_only && threadIdx.x == 0) L.theta_also[qi] = fmaxf(L.theta_also[qi], t);
    } else if (L.stats && threadIdx.x == 0) {
        L.stats[static_cast<uint64_t>(qi) * kSampleStats + kSampleRanks] = -2.0f;  // no K-th best
    }
    __syncthreads();  // every thread has read the old theta
    if (threadIdx.x == 0) {
        L.theta[qi] = theta;
        if (L.theta_also && !L.raise_only) L.theta_also[qi] = theta;
    }
    if (L.stats) {
        // the sample's best scores at ranks 1, 2, 4, ..., 64: a lower bound of the key at rank
        // r = min(64, n) (its 24-bit prefix), then the (fewer than r) keys above that prefix's bucket,
        // each placed by counting the keys that precede it; a rank inside the bucket gets the bound (at
        // most 2^-15 relative below the score)
        float* st = L.stats + static_cast<uint64_t>(qi) * kSampleStats;
        const uint32_t r = min(n, 64u);
        uint32_t key_r = 0;
        if (r > 0) key_r = kth_lower_bound<NT>(visit, r, key_lo, key_hi, S);
        const uint32_t bucket_top = key_r | 0xFFu;
        __shared__ uint32_t above[64], ranked[64];
        if (threadIdx.x == 0) S.counter = 0;
        __syncthreads();
        if (r > 0)
            visit([&](uint32_t key) {
                if (key > bucket_top) {
                    const uint32_t slot = atomicAdd(&S.counter, 1u);
                    if (slot < 64u) above[slot] = key;
                }
            });
        __syncthreads();
        const uint32_t c = min(S.counter, 64u);  // < r unless keys were lost
        if (threadIdx.x < c) {
            const uint32_t key = above[threadIdx.x];
            uint32_t rank = 0;
            for (uint32_t j = 0; j < c; ++j) {
                const uint32_t o = above[j];
                rank += (o > key || (o == key && j < threadIdx.x)) ? 1u : 0u;
            }
            ranked[rank] = key;
        }
        __syncthreads();
        if (threadIdx.x < kSampleRanks) {
            const uint32_t rho = 1u << threadIdx.x;
            float v = -2.0f;
            if (rho <= r) v = key_float(rho <= c ? ranked[rho - 1] : key_r);
            st[threadIdx.x] = v;
        } else if (threadIdx.x == kSampleRanks) {
            st[kSampleRanks + 1] = static_cast<float>(n);
            for (uint32_t j = kSampleRanks + 2; j < kSampleStats; ++j) st[j] = 0.0f;
        }
    }
}

// The threshold of a doc sample whose pass wrote, for every query, the best score of each small group of
// sample docs (-inf for a group without a filtered doc). The group maxima are scores of distinct docs, so
// their K-th best bounds the docs' K-th best from below as a sample's K-th best does; where K is at most
// half the groups it lies at a rank not far past K (K = 100 of 4,096 groups: about 101). A dense array of
// an eighth of the docs replaces lists of all filtered docs with their counts and locations.
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) maxima_threshold_kernel(MaximaThresholdLaunch L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HistSmem& S = *reinterpret_cast<HistSmem*>(smem_raw);
    float4* cs = reinterpret_cast<float4*>(smem_raw + sizeof(HistSmem));
    launch_dependents();
    wait_for_previous();
    const uint32_t qi = L.qlist ? L.qlist[blockIdx.x] : blockIdx.x;
    const uint32_t k = L.topk[qi];
    const float eps_s = L.eps_sample[qi], eps_m = L.eps_main[qi];
    const float4* src = reinterpret_cast<const float4*>(L.best + static_cast<uint64_t>(qi) * L.cap);
    const uint32_t quads = L.groups / 4, cached = min(quads, kFastSample / 4);
    float lo = INFINITY, hi = -INFINITY;
    uint32_t n = 0;
    auto each = [](const float4& v, auto fn) {
        if (v.x > -INFINITY) fn(v.x);
        if (v.y > -INFINITY) fn(v.y);
        if (v.z > -INFINITY) fn(v.z);
        if (v.w > -INFINITY) fn(v.w);
    };
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < quads; i += NT) {
        const float4 v = src[i];
        if (i < cached) cs[i] = v;
        each(v, [&](float x) {
            lo = fminf(lo, x);
            hi = fmaxf(hi, x);
            ++n;
        });
    }
    if (threadIdx.x == 0) S.counter = 0;
    __syncthreads();
    n = warp_sum(n);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&S.counter, n);
    uint32_t a = float_key(lo), b = float_key(hi);  // no score: +inf, -inf
    block_minmax<NT>(a, b, S);
    float theta = -INFINITY;
    if (k > 0 && S.counter >= k) {
        const float t = kth_score_bound<NT>(
            [&](auto fn) {
                for (uint32_t i = threadIdx.x; i < cached; i += NT) each(cs[i], fn);
                for (uint32_t i = cached + threadIdx.x; i < quads; i += NT) each(src[i], fn);
            },
            k, key_float(a), key_float(b), S);
        theta = __fsub_rd(__fsub_rd(t, eps_s), eps_m);  // as in sample_threshold_kernel
    }
    if (threadIdx.x == 0) {
        L.theta[qi] = theta;
        if (L.theta_also) L.theta_also[qi] = theta;
    }
}

// Byte offsets of the query and of the cached scores in select_topk_kernel's shared memory.
__host__ __device__ inline size_t select_cand_offset(uint32_t dim) {
    return (sizeof(SelectSmem) + static_cast<size_t>(dim) * sizeof(float) + 15) & ~static_cast<size_t>(15);
}

// Exact scores of list(i), i < m, by groups of four lanes: lane j of a group holds dims 8 j .. 8 j + 7 of
// every 32 of its row (a 32-byte sector; eight 16-byte loads in flight cover 128 dims of the row), and the
// running sum goes round the four lanes, so that it still adds the products one by one in ascending order,
// as the ground truth does. 768 dims, batch 256, the select step: 132 us with pieces of 4 dims (twice the
// hand-overs), 122 with 8, 211 with 32 (a lane's loads then share no sector at a time, and L1 is too small
// to keep the other halves). A quad past the row is zero: adding +0 leaves a sum as it is (it is never
// -0). put(i, location, score) is called by one lane per row.
template <int NT, class List, class Put>
__device__ __forceinline__ void rescore_rows(const float* sq, const float* vec, uint32_t dim, uint32_t m, List list,
                                             Put put) {
    const uint32_t lane = threadIdx.x & 31, j = lane & 3;
    const uint32_t quads = dim / 4;
    for (uint32_t r0 = NT == 32 ? 0 : (threadIdx.x >> 5) * 8; r0 < m; r0 += NT / 4) {  // NT = 32: one warp's rows
        const uint32_t r = r0 + (lane >> 2);
        const bool ok = r < m;
        const uint32_t loc = list(ok ? r : r0);
        const float4* row = reinterpret_cast<const float4*>(vec + static_cast<uint64_t>(loc) * dim);
        float s = 0.0f;
        for (uint32_t f0 = 0; f0 < quads; f0 += 32) {
            float4 v[8];
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t f = f0 + 8 * (i / 2) + 2 * j + i % 2;
                v[i] = f < quads ? __ldg(row + f) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (uint32_t p = 0; p < 4; ++p) {
                if (f0 + 8 * p >= quads) break;  // uniform
#pragma unroll
                for (uint32_t i = 2 * p; i < 2 * p + 2; ++i) {
                    const uint32_t f = f0 + 8 * p + 2 * j + i % 2;
                    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (f < quads) q = *reinterpret_cast<const float4*>(sq + 4 * f);
                    v[i].x = __fmul_rn(q.x, v[i].x);
                    v[i].y = __fmul_rn(q.y, v[i].y);
                    v[i].z = __fmul_rn(q.z, v[i].z);
                    v[i].w = __fmul_rn(q.w, v[i].w);
                }
#pragma unroll
                for (uint32_t turn = 0; turn < 4; ++turn) {
                    // in turn u lane u of the group holds the sum so far and adds its 8 products
                    float n = s;
#pragma unroll
                    for (uint32_t i = 2 * p; i < 2 * p + 2; ++i) {
                        n = __fadd_rn(n, v[i].x);
                        n = __fadd_rn(n, v[i].y);
                        n = __fadd_rn(n, v[i].z);
                        n = __fadd_rn(n, v[i].w);
                    }
                    s = __shfl_sync(0xffffffffu, n, turn, 4);
                }
            }
        }
        if (ok && j == 0) put(r, loc, s);
    }
}

// A threshold above the proven one (a prediction) has to be checked: the list holds every doc
// with s~ >= theta, so a doc left out scores s < theta + eps, and the K best candidates are the
// K best docs when their K-th exact score s_K >= theta + eps. A query that fails goes back to a
// proven threshold: the larger of its proven one and s_K - eps (every true top-K doc scores at
// least s_K, the candidates' K-th best, hence s~ >= s_K - eps).
__device__ __forceinline__ void threshold_miss(const SelectLaunch& L, uint32_t qi, float raised) {
    if (threadIdx.x == 0) {
        const float t = fmaxf(L.theta_proven[qi], raised);
        L.theta[qi] = t;
        L.theta_proven[qi] = t;
        L.out_count[qi] = 0;
        atomicOr(L.status + qi, kStatusOverflow | kStatusThresholdMiss);
    }
}

// The end of the select step: the nf keys of a query (in S.sortbuf, or in ws) sorted, a predicted threshold
// checked, the first kq results written.
template <int NT>
__device__ __forceinline__ void finish_select(SelectSmem& S, const SelectLaunch& L, uint32_t qi, uint32_t k,
                                              uint32_t kq, uint32_t nf, bool in_smem, const unsigned long long* ws) {
    const uint32_t tid = threadIdx.x;
    __syncthreads();
    uint32_t m;
    const unsigned long long* sorted = S.sortbuf;
    if (in_smem && nf <= kRankSort) {
        unsigned long long* out = reinterpret_cast<unsigned long long*>(S.hist);  // free: the last list is read
        rank_sort<NT>(S, nf, out);
        sorted = out;
        m = 0;
    } else if (in_smem && (nf <= static_cast<uint32_t>(kSelT) || nf <= 2 * kq)) {
        m = pad_sort<NT>(S, nf);
    } else if (in_smem) {
        // more keys than a short sort takes: cut in place (each thread's keys go to registers first)
        constexpr int kOwn = kMaxTopK / NT;
        unsigned long long own[kOwn];
#pragma unroll
        for (int i = 0; i < kOwn; ++i) own[i] = tid + NT * i < nf ? S.sortbuf[tid + NT * i] : 0ull;
        uint32_t lo = 0xffffffffu, hi = 0;
#pragma unroll
        for (int i = 0; i < kOwn; ++i)
            if (tid + NT * i < nf) {
                lo = min(lo, static_cast<uint32_t>(own[i] >> 32));
                hi = max(hi, static_cast<uint32_t>(own[i] >> 32));
            }
        block_minmax<NT>(lo, hi, S);
        const uint32_t lb = kth_lower_bound<NT>(
            [&](auto fn) {
#pragma unroll
                for (int i = 0; i < kOwn; ++i)
                    if (tid + NT * i < nf) fn(static_cast<uint32_t>(own[i] >> 32));
            },
            kq, lo, hi, S);
        if (tid == 0) S.counter = 0;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kOwn; ++i)
            if (tid + NT * i < nf && static_cast<uint32_t>(own[i] >> 32) >= lb)
                S.sortbuf[next_place(&S.counter)] = own[i];
        __syncthreads();
        m = pad_sort<NT>(S, S.counter);
    } else {
        m = gather_top_keys<NT>([&](uint32_t i) { return static_cast<uint64_t>(ws[i]); }, nf, kq, S);
    }
    if (m) bitonic_desc<NT>(S, m);
    const float theta_q = L.theta[qi];
    if (L.theta_proven != nullptr && theta_q > L.theta_proven[qi]) {
        const float lo = kq == k && nf >= kq ? __fsub_rd(result_key_score(sorted[kq - 1]), L.eps_main[qi]) : -INFINITY;
        if (!(lo >= theta_q)) {  // uniform
            __syncthreads();  // every thread has read the thresholds
            threshold_miss(L, qi, lo);
            return;
        }
    }
    const uint32_t kout = min(kq, nf);  // kq, unless the bound is not a number
    const uint64_t orow = static_cast<uint64_t>(qi) * L.out_stride;
    for (uint32_t i = tid; i < kout; i += NT) {
        const uint64_t key = sorted[i];
        const uint32_t loc = result_key_loc(key);
        L.out_score[orow + i] = result_key_score(key);
        L.out_id[orow + i] = L.gdocid ? L.gdocid[loc] : static_cast<int64_t>(loc);
    }
    if (tid == 0) L.out_count[qi] = kout;
}

// ---------------------------------------------------------------------------------------------
// The select step, one CTA per query: a chain of dependent steps and the rescoring's row reads bound it.
//   * The list's scores are read once into shared memory (`fast` entries), the first locations with them.
//   * A list of at most kWholeFloats floats is rescored whole; a longer one is cut: t~ bounds the K-th
//     best approximate score from below, so only entries of at least t~ - 2 eps can be in the top K. Where
//     those are many, the entries of at least t~ (K of them at least) are rescored first: the least of
//     their exact scores, s, bounds the K-th exact score, and the rest needs only s - eps, about half the
//     band. (Lists of up to 512 entries whole, and two waves only past 512: 768 dims, 256 queries, K 10
//     473 us a batch, now 412; 1M docs x 128 dims, 256 queries, K 10 189, now 175; 131k docs, 32 queries,
//     K 100 82, now 72. Two waves from 2 K entries at any K: 768 dims, 256 queries, K 1000 832 -> 849.)
//   * Survivors are packed before they are rescored, so that every lane group has a row.
// SPLIT: the kernel ends with the survivors' list in L.work (and, of a list cut in two waves, the first
// wave's keys): rescore_kernel scores the rest with all SMs, select_final_kernel sorts. A query's rows
// are otherwise read by its own CTA, and the query with the most holds up the batch.
constexpr uint32_t kWholeFloats = 16384;

template <int NT, uint32_t FAST, bool SPLIT>
__global__ void __launch_bounds__(NT, NT == kSelT ? 2 : 1) select_topk_kernel(SelectLaunch L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SelectSmem& S = *reinterpret_cast<SelectSmem*>(smem_raw);
    float* sq = reinterpret_cast<float*>(smem_raw + sizeof(SelectSmem));
    float* cs = reinterpret_cast<float*>(smem_raw + select_cand_offset(L.dim));
    uint32_t* surv = S.hist;  // survivors' locations: after the last digit
    launch_dependents();
    wait_for_previous();
    const uint32_t qi = L.qlist ? L.qlist[blockIdx.x] : blockIdx.x;
    const uint32_t tid = threadIdx.x;
    const uint32_t k = L.topk[qi];
    const uint64_t row = static_cast<uint64_t>(qi) * L.cap;
    if (SPLIT && tid == 0) L.pending[qi] = make_uint2(1, 0);  // answered here, unless rows follow
    if (k > static_cast<uint32_t>(kMaxTopK)) {
        if (tid == 0) {
            L.out_count[qi] = 0;
            atomicOr(L.status + qi, kStatusTopKTooLarge);
        }
        return;
    }
    const uint32_t* counts = L.cand_count + static_cast<uint64_t>(qi) * kMaxCandSegs;
    const float* sc = L.cand_score + row;
    const uint32_t* lc = L.cand_loc + row;
    const float eps = L.eps_main[qi];
    const float theta_q = L.theta[qi];
    for (uint32_t i = tid; i < L.dim; i += NT) sq[i] = L.qry[static_cast<uint64_t>(qi) * L.dim + i];
    bool overflow = false;
    uint32_t key_lo, key_hi;
    const uint32_t n = load_list<NT, SPLIT>(S, counts, L.segs, L.seg_cap, sc, lc, cs, FAST, S.locs, &overflow, &key_lo,
                                            &key_hi);
    auto visit_keys = [&](auto fn) {
        if (n <= FAST) {
            for (uint32_t i = tid; i < n; i += NT) fn(float_key(cs[i]));
        } else {
            walk_segments<NT, SPLIT>(counts, L.segs, L.seg_cap, sc, [](uint32_t) {}, [&](uint32_t, bool ok, float v) {
                if (ok) fn(float_key(v));
            });
        }
    };
    const bool unproven = L.theta_proven != nullptr && theta_q > L.theta_proven[qi];
    if (overflow) {
        // The stored candidates are a subset of the qualifying docs, so their K-th best still bounds
        // the true K-th best from below: raise the threshold and let the host re-run this query.
        float theta = unproven ? L.theta_proven[qi] : theta_q;
        if (n >= k && k > 0) {
            const uint32_t kk = kth_lower_bound<NT>(visit_keys, k, key_lo, key_hi, S);
            theta = fmaxf(theta, __fsub_rd(key_float(kk), 2.0f * eps));
        }
        __syncthreads();  // every thread has read the old thresholds
        if (tid == 0) {
            L.theta[qi] = theta;
            if (L.theta_proven) L.theta_proven[qi] = theta;
            L.out_count[qi] = 0;
            atomicOr(L.status + qi, kStatusOverflow);
        }
        return;
    }
    if (n == 0 || k == 0) {
        __syncthreads();  // every thread has read the thresholds
        if (unproven && k > 0) {
            threshold_miss(L, qi, -INFINITY);
            return;
        }
        if (tid == 0) L.out_count[qi] = 0;
        return;
    }
    const uint32_t kq = min(k, n);
    unsigned long long* ws = L.work + row;
    uint32_t nf;
    bool in_smem;  // the keys: S.sortbuf or ws
    const bool whole = n <= static_cast<uint32_t>(kSelT) && (n <= kq || n * L.dim <= kWholeFloats);
    if (SPLIT && whole) {
        for (uint32_t i = tid; i < n; i += NT) ws[i] = S.locs[i];
        __syncthreads();
        if (tid == 0) L.pending[qi] = make_uint2(0, n);
        return;
    }
    if (whole) {
        rescore_rows<NT>(sq, L.vec, L.dim, n, [&](uint32_t i) { return S.locs[i]; },
                         [&](uint32_t i, uint32_t loc, float e) { S.sortbuf[i] = result_key(e, loc); });
        nf = n;
        in_smem = true;
    } else {
        const float t = n > kq ? key_float(kth_lower_bound<NT>(visit_keys, kq, key_lo, key_hi, S)) : -INFINITY;
        const float cut2 = __fsub_rd(t, 2.0f * eps);
        // fn(score, location) of every entry
        auto visit_entries = [&](auto fn) {
            if (n <= min(FAST, static_cast<uint32_t>(kMaxTopK))) {
                for (uint32_t i = tid; i < n; i += NT) fn(cs[i], [&] { return S.locs[i]; });
            } else {
                walk_segments<NT, SPLIT>(counts, L.segs, L.seg_cap, sc, [](uint32_t) {},
                                         [&](uint32_t at, bool ok, float v) {
                                             if (ok) fn(v, [&] { return lc[at]; });
                                         });
            }
        };
        // how many clear the cut at all
        if (tid == 0) S.counter = 0;
        __syncthreads();
        uint32_t mine = 0;
        visit_keys([&](uint32_t key) { mine += key_float(key) >= cut2 ? 1u : 0u; });
        mine = warp_sum(mine);
        if ((tid & 31) == 0 && mine) atomicAdd(&S.counter, mine);
        __syncthreads();
        const uint32_t all = S.counter;
        // a first wave pays where it spares reading about as many rows again, or kSelT; in the split form,
        // where this CTA alone reads it and all SMs the rest, later
        const uint32_t limit = SPLIT ? 2 * kq + 256 : min(static_cast<uint32_t>(kSelT), max(2 * kq, 128u));
        const bool two = all > limit && all > kq && t > -INFINITY;
        float lo = two ? t : cut2, hi = INFINITY, low_exact = INFINITY;
        nf = 0;
        in_smem = all <= static_cast<uint32_t>(kMaxTopK);
        for (int wave = 0; wave < (two ? 2 : 1); ++wave) {
            __syncthreads();  // the survivors' list is free
            if (tid == 0) S.total = 0;
            __syncthreads();
            const bool last = !two || wave == 1;
            visit_entries([&](float v, auto loc) {
                if (v >= lo && (wave == 0 || v < hi)) {
                    const uint32_t at = next_place(&S.total);
                    if (in_smem)
                        surv[at] = loc();
                    else
                        ws[nf + at] = loc();
                }
            });
            __syncthreads();
            const uint32_t m = S.total;
            if (SPLIT && last) {
                if (in_smem)
                    for (uint32_t i = tid; i < m; i += NT) ws[nf + i] = surv[i];
                if (tid == 0) L.pending[qi] = make_uint2(nf, nf + m);
                return;
            }
            float least = INFINITY;
            rescore_rows<NT>(
                sq, L.vec, L.dim, m,
                [&](uint32_t i) { return in_smem ? surv[i] : static_cast<uint32_t>(ws[nf + i]); },
                [&](uint32_t i, uint32_t loc, float e) {
                    const unsigned long long key = result_key(e, loc);
                    if (in_smem && !SPLIT)
                        S.sortbuf[nf + i] = key;
                    else
                        ws[nf + i] = key;
                    least = fminf(least, e);
                });
            nf += m;
            if (last) break;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) least = fminf(least, __shfl_xor_sync(0xffffffffu, least, o));
            if ((tid & 31) == 0) S.wsum[tid >> 5] = float_bits(least);
            __syncthreads();
            for (int w = 0; w < NT / 32; ++w) low_exact = fminf(low_exact, bits_float(S.wsum[w]));
            hi = t;
            lo = fmaxf(cut2, __fsub_rd(low_exact, eps));
        }
    }
    finish_select<NT>(S, L, qi, k, kq, nf, in_smem, ws);
}

// Exact scores of every query's pending rows (L.work from L.pending.x to .y), eight rows to a warp, the
// groups of eight dealt out evenly over all warps of the grid: bound by the rows' reads, where the query
// with the most rows bound the one-kernel step (8-bit form, 768 dims, 300k docs, 128 queries, K 10: select
// step 975 -> 239 us; K 100: 10.0 -> 1.37 ms).
constexpr int kRescoreT = 256;

__global__ void __launch_bounds__(kRescoreT, 4) rescore_kernel(SelectLaunch L) {
    extern __shared__ uint32_t group_end[];  // [nq_list] groups of the queries up to and with this one
    __shared__ uint32_t wsum[kRescoreT / 32];
    launch_dependents();
    wait_for_previous();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t carry = 0;
    for (uint32_t i0 = 0; i0 < L.nq_list; i0 += kRescoreT) {
        const uint32_t i = i0 + tid;
        uint32_t x = 0;
        if (i < L.nq_list) {
            const uint2 p = L.pending[L.qlist ? L.qlist[i] : i];
            x = p.y > p.x ? (p.y - p.x + 7) / 8 : 0u;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= static_cast<uint32_t>(o)) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        uint32_t before = 0, all = 0;
        for (uint32_t w = 0; w < kRescoreT / 32; ++w) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        if (i < L.nq_list) group_end[i] = carry + before + x;
        carry += all;
        __syncthreads();
    }
    const uint32_t step = gridDim.x * (kRescoreT / 32);
    for (uint32_t g = blockIdx.x * (kRescoreT / 32) + warp; g < carry; g += step) {
        uint32_t lo = 0, hi = L.nq_list - 1;  // the first query whose end is past g
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (group_end[mid] > g)
                hi = mid;
            else
                lo = mid + 1;
        }
        const uint32_t qi = L.qlist ? L.qlist[lo] : lo;
        const uint2 p = L.pending[qi];
        const uint32_t first = p.x + 8 * (g - (lo ? group_end[lo - 1] : 0u));
        unsigned long long* ws = L.work + static_cast<uint64_t>(qi) * L.cap + first;
        rescore_rows<32>(L.qry + static_cast<uint64_t>(qi) * L.dim, L.vec, L.dim, min(8u, p.y - first),
                         [&](uint32_t i) { return static_cast<uint32_t>(ws[i]); },
                         [&](uint32_t i, uint32_t loc, float e) { ws[i] = result_key(e, loc); });
    }
}

// The keys of L.work sorted and written out, one CTA per query.
__global__ void __launch_bounds__(kSelT, 2) select_final_kernel(SelectLaunch L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SelectSmem& S = *reinterpret_cast<SelectSmem*>(smem_raw);
    launch_dependents();
    wait_for_previous();
    const uint32_t qi = L.qlist ? L.qlist[blockIdx.x] : blockIdx.x;
    const uint2 p = L.pending[qi];
    if (p.x > p.y) return;  // the first kernel has written this query's outcome
    const uint32_t nf = p.y, k = L.topk[qi];
    const unsigned long long* ws = L.work + static_cast<uint64_t>(qi) * L.cap;
    const bool in_smem = nf <= static_cast<uint32_t>(kMaxTopK);
    if (in_smem)
        for (uint32_t i = threadIdx.x; i < nf; i += kSelT) S.sortbuf[i] = ws[i];
    finish_select<kSelT>(S, L, qi, k, min(k, nf), nf, in_smem, ws);
}

// ---------------------------------------------------------------------------------------------
// Aggregator: stable compaction. A CTA scatters 4,096 docs (64 bitmap words); where they go needs the
// kept docs before them, which it finds by
//   own     counting the bitmap's earlier words itself (one launch),
//   sums    adding up the earlier blocks' counts, which aggregate_count_kernel left (two launches), or
//   scanned reading its offset after aggregate_scan_kernel (three launches, very long lists).
// All three are bound by launches and one dependent chain of loads, not by bandwidth, at the sizes of a
// query's docs: 1.3M docs, a tenth kept, 15 us in three launches with 1,024 docs a CTA, now 8 us; 10M
// docs 24 us. (8,192 docs a CTA of 1,024 threads: one CTA per SM at 56 registers, 28 us at 10M; held to
// 32 registers it spills, 27 us.) The rule is at launch_aggregate.
constexpr int kAggT = 512;                  // threads of a scatter CTA
constexpr uint32_t kAggWords = 64;          // bitmap words a scatter CTA covers
constexpr uint32_t kAggDocs = kAggWords * 64;
enum AggPrefix : int { kAggOwn = 0, kAggSums = 1, kAggScanned = 2 };

// Bitmap word w of n docs, docs past n cleared.
__device__ __forceinline__ uint64_t agg_word(const uint64_t* bits, uint64_t w, uint32_t n) {
    const uint64_t d0 = w * 64;
    if (d0 >= n) return 0;
    const uint64_t left = n - d0;
    const uint64_t v = bits[w];
    return left >= 64 ? v : v & ((1ull << left) - 1);
}

// Kept docs of each block of kAggDocs docs, one warp per block.
__global__ void __launch_bounds__(256) aggregate_count_kernel(const uint64_t* __restrict__ bits, uint32_t n,
                                                              uint32_t nb, uint32_t* __restrict__ block_count) {
    launch_dependents();
    const uint32_t b = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b >= nb) return;
    uint32_t c = 0;
#pragma unroll
    for (uint32_t i = 0; i < kAggWords / 32; ++i)
        c += __popcll(agg_word(bits, static_cast<uint64_t>(b) * kAggWords + lane + 32u * i, n));
    c = warp_sum(c);
    if (lane == 0) block_count[b] = c;
}

// Exclusive scan of nb block counts in place (one CTA).
__global__ void __launch_bounds__(1024) aggregate_scan_kernel(uint32_t* block_count, uint32_t nb) {
    __shared__ uint32_t warp_tot[32];
    __shared__ uint32_t carry;
    launch_dependents();
    wait_for_previous();
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t b0 = 0; b0 < nb; b0 += blockDim.x) {
        const uint32_t i = b0 + threadIdx.x;
        const uint32_t v = i < nb ? block_count[i] : 0;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= static_cast<uint32_t>(o)) x += y;
        }
        if (lane == 31) warp_tot[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t t = warp_tot[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= static_cast<uint32_t>(o)) t += y;
            }
            warp_tot[lane] = t;  // inclusive over warps
        }
        __syncthreads();
        const uint32_t warp_excl = warp ? warp_tot[warp - 1] : 0;
        const uint32_t excl = carry + warp_excl + x - v;
        if (i < nb) block_count[i] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + v;
        __syncthreads();
    }
}

template <int MODE>
__global__ void __launch_bounds__(kAggT) aggregate_scatter_kernel(const uint64_t* bits,
                                                                  const float* scores,
                                                                  const uint32_t* loc_in, uint32_t n,
                                                                  const uint32_t* blocks,
                                                                  float* out_scores,
                                                                  uint32_t* out_loc,
                                                                  uint32_t* total) {
    __shared__ uint32_t wsum[kAggT / 32];
    __shared__ uint32_t woff[kAggWords];
    __shared__ uint64_t wbits[kAggWords];
    launch_dependents();
    wait_for_previous();
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5, b = blockIdx.x;
    // kept docs before this block: this thread's share of them
    uint32_t before = 0;
    if (MODE == kAggOwn) {
        // whole words below the block; the bitmap is only 8-byte aligned
        const uint32_t words = b * kAggWords;
#pragma unroll 8
        for (uint32_t w = t; w < words; w += kAggT) before += __popcll(bits[w]);
    } else if (MODE == kAggSums) {
        for (uint32_t i = t; i < b; i += kAggT) before += blocks[i];
    } else if (t == 0) {
        before = blocks[b];
    }
    uint32_t c = 0;
    if (t < kAggWords) {
        const uint64_t v = agg_word(bits, static_cast<uint64_t>(b) * kAggWords + t, n);
        wbits[t] = v;
        c = static_cast<uint32_t>(__popcll(v));
    }
    // exclusive offsets of the block's words (the first two warps), and the sum of every thread's share
    uint32_t x = c;
    if (t < kAggWords) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= static_cast<uint32_t>(o)) x += y;
        }
        woff[t] = x - c;
    }
    before = warp_sum(before);
    __shared__ uint32_t qsum[kAggWords / 32];
    if (lane == 31 && warp < kAggWords / 32) qsum[warp] = x;
    if (lane == 0) wsum[warp] = before;
    __syncthreads();
    const uint32_t base = warp_sum(lane < kAggT / 32 ? wsum[lane] : 0u);
    // a warp takes four words (256 docs): 8 coalesced loads per thread in flight, only for kept docs
    const uint32_t w0 = warp * 4u;
    uint32_t off = base;
#pragma unroll
    for (uint32_t i = 0; i < kAggWords / 32; ++i)
        if (i < w0 / 32u) off += qsum[i];
    float s[8];
    uint32_t l[8], at[8];
    uint32_t hits = 0;
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
        const uint64_t wv = wbits[w0 + j / 2];
        const uint32_t low = static_cast<uint32_t>(wv);
        const uint32_t half = j & 1u ? static_cast<uint32_t>(wv >> 32) : low;
        const uint64_t doc = static_cast<uint64_t>(b) * kAggDocs + (w0 + j / 2) * 64u + (j & 1u) * 32u + lane;
        at[j] = off + woff[w0 + j / 2] + (j & 1u ? __popc(low) : 0) + __popc(half & ((1u << lane) - 1u));
        if ((half >> lane) & 1u) {
            hits |= 1u << j;
            s[j] = scores[doc];
            l[j] = loc_in ? loc_in[doc] : static_cast<uint32_t>(doc);
        }
    }
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j)
        if ((hits >> j) & 1u) {
            out_scores[at[j]] = s[j];
            out_loc[at[j]] = l[j];
        }
    if (b == gridDim.x - 1 && t == 0) {
        uint32_t sum = base;
#pragma unroll
        for (uint32_t i = 0; i < kAggWords / 32; ++i) sum += qsum[i];
        *total = sum;
    }
}

// ---------------------------------------------------------------------------------------------
// TOPK operator: exact top K of one compacted list, one thread-block cluster. The list's length is only
// known on the device and the caller gives no scratch, so the CTAs of one cluster work together through
// distributed shared memory: a 12-bit digit histogram of the keys per CTA, summed over the cluster,
// picks the digit of the K-th key; as soon as the keys at or above its bucket fit the sort buffer they
// go to the first CTA, which sorts them. For real scores that is one digit: the scores are read twice.
// A list longer than kTopkSample is first bounded from below by an evenly spaced sample, so that the
// histogram only counts keys that can still be among the top K (shared-memory atomics on a few crowded
// bins would bound the pass otherwise). One CTA over eight digits took 357 us for the top 100 of
// 131,072 scores; 16 CTAs take 11 us.
constexpr uint32_t kTopkSample = 65536;

__global__ void __launch_bounds__(kST) topk_op_kernel(const float* scores,
                                                      const uint32_t* locs,
                                                      const uint32_t* count, uint32_t k,
                                                      float* out_scores, uint32_t* out_locs,
                                                      uint32_t* out_count) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SelectSmem& S = *reinterpret_cast<SelectSmem*>(smem_raw);
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t C = cluster.num_blocks(), rank = cluster.block_rank(), t = threadIdx.x;
    wait_for_previous();
    const uint32_t n = *count;
    const uint32_t kq = min(k, n);
    uint32_t m;  // keys to sort
    if (kq == 0 || n <= static_cast<uint32_t>(kMaxTopK)) {  // uniform over the cluster: no remote access follows
        if (rank != 0) return;
        if (kq == 0) {
            if (t == 0) *out_count = 0;
            return;
        }
        m = gather_top_keys<kST>([&](uint32_t i) { return result_key(scores[i], locs[i]); }, n, kq, S);
    } else {
        uint32_t* hist = S.hist;
        const uint32_t gt = rank * kST + t, gthreads = C * kST;
        // fn(index, score) for the entries mul * i, i < cnt, 4 loads in flight
        auto visit = [&](uint32_t cnt, uint32_t mul, auto fn) {
            for (uint64_t i = gt; i < cnt; i += 4ull * gthreads) {
                float v[4];
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const uint64_t at = i + static_cast<uint64_t>(u) * gthreads;
                    v[u] = at < cnt ? scores[at * mul] : 0.0f;
                }
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const uint64_t at = i + static_cast<uint64_t>(u) * gthreads;
                    if (at < cnt) fn(static_cast<uint32_t>(at * mul), v[u]);
                }
            }
        };
        // the histograms of all CTAs summed into every CTA's own: each sums a slice of the bins, then
        // gathers the others' slices (a CTA's histogram and slice are not written again before every
        // CTA has read them: the next pass writes its histogram after the second barrier, its slice
        // after the next pass's first)
        auto sum_cluster = [&] {
            cluster.sync();
            const uint32_t slice = 4096u / C;
            if (t < slice) {
                uint32_t s = 0;
                for (uint32_t r = 0; r < C; ++r) s += cluster.map_shared_rank(hist, r)[rank * slice + t];
                S.locs[t] = s;
            }
            cluster.sync();
            for (uint32_t i = t; i < 4096u; i += kST) hist[i] = cluster.map_shared_rank(S.locs, i / slice)[i % slice];
            __syncthreads();
        };
        auto clear = [&] {
            for (uint32_t i = t; i < 4096u; i += kST) hist[i] = 0;
            __syncthreads();
        };
        uint32_t floor_key = 0;  // keys below it are not among the top K
        if (n > 2u * kTopkSample) {
            clear();
            visit(kTopkSample, n / kTopkSample, [&](uint32_t, float v) { atomicAdd(&hist[float_key(v) >> 20], 1u); });
            sum_cluster();
            uint32_t kr = kq;  // kq <= kMaxTopK < kTopkSample
            floor_key = pick_digit4096<kST>(hist, &kr, S) << 20;
        }
        uint64_t prefix = 0, mask = 0;
        uint32_t krem = kq, in_bin = 0;
        const int shifts[6] = {52, 40, 32, 20, 8, 0};
        bool fits = false;
        for (int p = 0; p < 6 && !fits; ++p) {
            const int shift = shifts[p];
            const uint64_t digit = p == 2 || p == 5 ? 255ull : 4095ull;
            clear();
            visit(n, 1u, [&](uint32_t i, float v) {
                const uint32_t hi = float_key(v);
                if (hi < floor_key || ((static_cast<uint64_t>(hi) << 32) & mask) >> 32 != prefix >> 32) return;
                uint64_t key = static_cast<uint64_t>(hi) << 32;
                if (p >= 3) {
                    key = result_key(v, locs[i]);
                    if ((key & mask) != prefix) return;
                }
                atomicAdd(&hist[(key >> shift) & digit], 1u);
            });
            sum_cluster();
            const uint64_t d = pick_digit4096<kST>(hist, &krem, S, &in_bin);
            prefix |= d << shift;
            mask |= digit << shift;
            fits = (kq - krem) + in_bin <= static_cast<uint32_t>(kMaxTopK);
        }
        // the keys above the bucket (kq - krem of them), then the bucket's own, into the first CTA's
        // buffer: all of them when they fit; otherwise every bit is fixed, the bucket holds copies of
        // one key (an entry listed more than once) and the first krem of them are as good as any
        if (t == 0) {
            S.counter = 0;
            S.total = 0;
        }
        cluster.sync();
        SelectSmem* S0 = cluster.map_shared_rank(&S, 0);
        const uint32_t above = kq - krem;
        visit(n, 1u, [&](uint32_t i, float v) {
            const uint32_t hi = float_key(v);
            if (hi < static_cast<uint32_t>(prefix >> 32)) return;
            const uint64_t key = result_key(v, locs[i]);
            if ((key & mask) < prefix) return;
            if ((key & mask) > prefix) {
                S0->sortbuf[atomicAdd(&S0->counter, 1u)] = key;
            } else {
                const uint32_t at = above + atomicAdd(&S0->total, 1u);
                if (at < static_cast<uint32_t>(kMaxTopK)) S0->sortbuf[at] = key;
            }
        });
        cluster.sync();
        if (rank != 0) return;
        const uint32_t got = min(above + S.total, static_cast<uint32_t>(kMaxTopK));
        m = pad_sort<kST>(S, got);
    }
    bitonic_desc<kST>(S, m);
    for (uint32_t i = t; i < kq; i += kST) {
        const uint64_t key = S.sortbuf[i];
        out_scores[i] = result_key_score(key);
        out_locs[i] = result_key_loc(key);
    }
    if (t == 0) *out_count = kq;
}

// Per-query error bounds: eps = c * ||q||_2 * max_doc ||v||_2 (Cauchy-Schwarz on sum |q_i v_i|),
// computed in double and rounded up to float.
// Bounds of queries qlist[0..nq) (or 0..nq-1 when qlist is null), written at the query's own index.
__global__ void query_eps_kernel(const float* qry, const uint32_t* qlist, uint32_t nq,
                                 uint32_t dim, float max_norm, double c_main, double c_sample,
                                 float* eps_main, float* eps_sample) {
    // beside the batch's filter, as stage_queries_kernel
    launch_dependents();
    const uint32_t r = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const uint32_t lane = threadIdx.x & 31;
    if (r >= nq) {
        wait_for_previous();
        return;
    }
    const uint32_t q = qlist ? qlist[r] : r;
    double s = 0.0;
    for (uint32_t d = lane; d < dim; d += 32) {
        const double x = qry[static_cast<uint64_t>(q) * dim + d];
        s += x * x;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
        const double base = sqrt(s) * (1.0 + 1e-12) * static_cast<double>(max_norm);
        eps_main[q] = __double2float_ru(c_main * base + 1e-30);
        eps_sample[q] = __double2float_ru(c_sample * base + 1e-30);
    }
    wait_for_previous();
}

// Opts a kernel into more than 48 KB of dynamic shared memory, always to the same ceiling: searchers
// on other threads launch the same kernel concurrently with their own sizes, and a per-call value
// could drop below another caller's launch.
template <class K>
cudaError_t set_smem(K kernel, size_t bytes) {
    constexpr size_t kCeiling = 216 * 1024;
    if (bytes <= 48 * 1024) return cudaSuccess;
    if (bytes > kCeiling) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kCeiling));
}

}  // namespace

namespace {
bool bad_segments(uint32_t segs, uint32_t seg_cap, uint32_t cap) {
    return segs == 0 || segs > kMaxCandSegs || seg_cap == 0 || static_cast<uint64_t>(segs) * seg_cap > cap;
}
}  // namespace

// Two CTAs an SM, but one with room for a whole sample of the default size where the statistics of few queries walk
// it five more times (64 queries, 32,768 docs: 57 -> 36 us).
cudaError_t launch_sample_threshold(const SampleThresholdLaunch& L, cudaStream_t stream) {
    if (L.nq_list == 0) return cudaSuccess;
    if (bad_segments(L.segs, L.seg_cap, L.cap)) return cudaErrorInvalidValue;
    const uint32_t held = L.stats && L.nq_list <= device_sms() ? kFastLarge : kFastSample;
    const size_t smem = sizeof(HistSmem) + held * sizeof(float);
    cudaError_t e = set_smem(sample_threshold_kernel, smem);
    if (e != cudaSuccess) return e;
    return launch_dependent(sample_threshold_kernel, dim3(L.nq_list), kST, smem, stream, 1, L, held);
}

// Up to as many queries as SMs every CTA has one to itself: this kernel and the select step then take 1,024
// threads (more, and two CTAs of 512 threads per SM hide each other's steps better).
cudaError_t launch_maxima_threshold(const MaximaThresholdLaunch& L, cudaStream_t stream) {
    if (L.nq_list == 0) return cudaSuccess;
    if (L.groups == 0 || L.groups % 4 || L.cap % 4 || L.groups > L.cap || (reinterpret_cast<uintptr_t>(L.best) & 15u))
        return cudaErrorInvalidValue;
    const size_t smem = sizeof(HistSmem) + (L.groups < kFastSample ? L.groups : kFastSample) * sizeof(float);
    const bool wide = L.nq_list <= device_sms();
    auto kernel = wide ? maxima_threshold_kernel<kST> : maxima_threshold_kernel<kSelT>;
    cudaError_t e = set_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    return launch_dependent(kernel, dim3(L.nq_list), wide ? kST : kSelT, smem, stream, 1, L);
}

cudaError_t launch_select_topk(const SelectLaunch& L, cudaStream_t stream) {
    if (L.nq_list == 0) return cudaSuccess;
    if (bad_segments(L.segs, L.seg_cap, L.cap) || L.segs > static_cast<uint32_t>(kST)) return cudaErrorInvalidValue;
    const bool wide = L.fast_large || L.nq_list <= device_sms();
    const size_t smem = select_cand_offset(L.dim) + (wide ? kFastLarge : kFast) * sizeof(float);
    const bool split = L.pending != nullptr;
    auto kernel = wide ? (split ? select_topk_kernel<kST, kFastLarge, true> : select_topk_kernel<kST, kFastLarge, false>)
                       : (split ? select_topk_kernel<kSelT, kFast, true> : select_topk_kernel<kSelT, kFast, false>);
    cudaError_t e = set_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    e = launch_dependent(kernel, dim3(L.nq_list), wide ? kST : kSelT, smem, stream, 1, L);
    if (e != cudaSuccess || !split) return e;
    e = launch_dependent(rescore_kernel, dim3(4 * device_sms()), kRescoreT, L.nq_list * sizeof(uint32_t), stream, 1, L);
    if (e != cudaSuccess) return e;
    e = set_smem(select_final_kernel, sizeof(SelectSmem));
    if (e != cudaSuccess) return e;
    return launch_dependent(select_final_kernel, dim3(L.nq_list), kSelT, sizeof(SelectSmem), stream, 1, L);
}

cudaError_t launch_query_eps(const float* qry, const uint32_t* qlist, uint32_t nq, uint32_t dim, float max_norm,
                             double c_main, double c_sample, float* eps_main, float* eps_sample, cudaStream_t stream) {
    if (nq == 0) return cudaSuccess;
    return launch_dependent(query_eps_kernel, dim3((nq + 7) / 8), 256, 0, stream, 1, qry, qlist, nq, dim, max_norm,
                            c_main, c_sample, eps_main, eps_sample);
}

size_t aggregate_workspace_bytes(uint32_t n) {
    const size_t nb = (static_cast<size_t>(n) + 1023) / 1024;
    return (nb > 0 ? nb : 1) * sizeof(uint32_t);
}

// One launch while a CTA counts the bitmap below it about as fast as a second launch starts (the last
// CTA's chain is the longest, 4 KB of words a step, 128 KB at 2^20 docs: 8.0 us there against 9.3 us for
// two launches at 1.5M, 6.7 us below 500,000); block counts added up by every CTA while they are few; a
// scan of them beyond.
cudaError_t launch_aggregate(const uint64_t* bits, const float* scores, const uint32_t* loc_in, uint32_t n,
                             float* out_scores, uint32_t* out_loc, uint32_t* total, uint32_t* workspace,
                             cudaStream_t stream) {
    constexpr uint32_t kOwnDocs = 1u << 20;
    constexpr uint32_t kSumBlocks = 16384;
    const uint32_t nb = static_cast<uint32_t>((static_cast<uint64_t>(n) + kAggDocs - 1) / kAggDocs);
    if (nb == 0) return cudaMemsetAsync(total, 0, sizeof(uint32_t), stream);
    if (n <= kOwnDocs) {
        return launch_dependent(aggregate_scatter_kernel<kAggOwn>, dim3(nb), kAggT, 0, stream, 1, bits, scores, loc_in,
                                n, workspace, out_scores, out_loc, total);
    }
    aggregate_count_kernel<<<(nb + 7) / 8, 256, 0, stream>>>(bits, n, nb, workspace);
    if (nb <= kSumBlocks) {
        return launch_dependent(aggregate_scatter_kernel<kAggSums>, dim3(nb), kAggT, 0, stream, 1, bits, scores, loc_in,
                                n, workspace, out_scores, out_loc, total);
    }
    cudaError_t e = launch_dependent(aggregate_scan_kernel, dim3(1), 1024, 0, stream, 1, workspace, nb);
    if (e != cudaSuccess) return e;
    return launch_dependent(aggregate_scatter_kernel<kAggScanned>, dim3(nb), kAggT, 0, stream, 1, bits, scores, loc_in,
                            n, workspace, out_scores, out_loc, total);
}

// Scratch of the allocation-free aggregator: one word per 1,024 docs, kAggStaticBlocks of them (64 KB,
// docNumber <= 16,777,216; the count kernel writes one per kAggDocs docs). Module-scope, so it exists once per
// device for the life of the process and every call on that device shares it. The count kernel writes every
// entry a call reads before the scan reads it, so a call never sees an earlier call's contents and nothing has
// to be cleared; two calls that overlap on the GPU (different streams, no ordering) do race on it.
static __device__ __align__(256) uint32_t g_aggregate_scratch[kAggStaticBlocks];
static_assert(kAggStaticMaxDocs == kAggStaticBlocks * 1024u && kAggDocs >= 1024u,
              "a block count per 1,024 docs at most");

cudaError_t aggregate_static_scratch(uint32_t** scratch) {
    return cudaGetSymbolAddress(reinterpret_cast<void**>(scratch), g_aggregate_scratch);
}

// CTAs of the TOPK operator's cluster on the current device: 16 where a GPC holds them, else the portable
// 8. A property of the device, asked once (the query costs more host time than the launch).
static unsigned topk_cluster(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr) {
    constexpr int kDevices = 64;
    static std::atomic<unsigned> known[kDevices];
    int dev = 0;
    const bool keep = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kDevices;
    unsigned size = keep ? known[dev].load(std::memory_order_relaxed) : 0u;
    if (size) return size;
    size = 16;
    attr.val.clusterDim.x = size;
    cfg.gridDim = dim3(size, 1, 1);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, topk_op_kernel, &cfg) != cudaSuccess || clusters < 1) {
        cudaGetLastError();
        size = 8;
    }
    if (keep) known[dev].store(size, std::memory_order_relaxed);
    return size;
}

cudaError_t launch_topk_op(const float* scores, const uint32_t* locs, const uint32_t* count, uint32_t k,
                           float* out_scores, uint32_t* out_locs, uint32_t* out_count, cudaStream_t stream) {
    if (k > static_cast<uint32_t>(kMaxTopK)) return cudaErrorInvalidValue;
    const size_t smem = sizeof(SelectSmem);
    cudaError_t e = set_smem(topk_op_kernel, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(topk_op_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kST, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const unsigned size = topk_cluster(cfg, attr[0]);
    return launch_dependent(topk_op_kernel, dim3(size), kST, smem, stream, size, scores, locs, count, k, out_scores,
                            out_locs, out_count);
}


// ---------------------------------------------------------------------------------------------
// Cross-shard merge (the reference's k-way merge of per-shard results, run_context.cpp:86-118 and
// 237-270): the shards' sorted lists are merged by score descending, equal scores taking the lower
// shard first (within a shard, list order). Every entry finds its output position directly: its
// index in its own list plus, for every other shard, how many of that shard's entries precede it
// (a binary search on the score), so one thread places one entry and no thread waits on another.
// Only entries that can be among the top K take part: where m shards hold at least j = ceil(K / m)
// entries, K entries score at least tau, the least of those shards' j-th scores, and a list's entries
// from tau up are a prefix of it. The prefixes (a little over K entries in all when the shards are
// alike) are ranked in shared memory, where the searches' instructions bound the kernel: eight lists of
// 1,000 for 256 queries took 98 us when every entry searched every list in global memory, 29 us with the
// prefixes in shared memory and general binary searches, and take 17 us with padded lists of keys.
namespace {
// Entries of a list sorted by score descending that come before score x: those with score > x, or
// with score >= x when `ties_first` (a lower shard).
__device__ inline uint32_t preceding(const float* sc, uint32_t n, float x, bool ties_first) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        const float v = sc[mid];
        if (ties_first ? (v >= x) : (v > x))
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

constexpr int kMergeT = 1024;
// Up to as many keys a CTA has a thread for each and cuts nothing: the cut's steps, and 1,024 threads, would be most
// of the time (2 lists of 10, 256 queries 3.9 -> 3.0 us, 4 of 100 4.3 -> 3.7). Of more than eight lists half as many,
// since a thread searches every list (16 lists of 16: 6.4 us cut, 7.5 not).
constexpr int kMergeFew = 512;
constexpr uint32_t kMergeCap = 12000;  // keys held in shared memory (with the rest within 48 KB)

// One shard's lists as they are (256 queries x 2,000: 10.5 us through the searches below, 6.0 here).
constexpr int kCopyT = 512;
__global__ void __launch_bounds__(kCopyT) copy_shard_kernel(const __grid_constant__ ShardMergeLaunch L) {
    const uint32_t q = blockIdx.x, n = min(L.counts[0][q], min(L.in_stride, L.topk));
    const uint64_t in = static_cast<uint64_t>(q) * L.in_stride, out = static_cast<uint64_t>(q) * L.out_stride;
    if (threadIdx.x == 0) L.out_count[q] = n;
    const float* sc = L.scores[0] + in;
    const int64_t* id = L.ids[0] + in;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < n; i += kCopyT) {
        const float s = __ldg(sc + i);
        const long long x = __ldg(reinterpret_cast<const long long*>(id + i));
        L.out_score[out + i] = s;
        L.out_id[out + i] = x;
    }
}

template <int NT>
__global__ void __launch_bounds__(NT) merge_shards_kernel(const __grid_constant__ ShardMergeLaunch L) {
    extern __shared__ __align__(16) uint32_t merge_key[];  // [shards][P]
    __shared__ uint32_t s_n[kMaxShards];
    __shared__ float s_tau;
    __shared__ int s_all;
    const uint32_t q = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t row = static_cast<uint64_t>(q) * L.in_stride;
    if (warp == 0) {
        // lane l holds the counts of shards l and l + 32
        const uint32_t most = min(L.in_stride, L.topk);
        const uint32_t c0 = lane < L.shards ? min(L.counts[lane][q], most) : 0u;
        const uint32_t c1 = lane + 32 < L.shards ? min(L.counts[lane + 32][q], most) : 0u;
        const uint32_t total = warp_sum(c0 + c1);
        // the most shards m that hold ceil(topk / m) entries each
        uint32_t j = 0;
        if (NT != kMergeFew && total > L.topk)
            for (uint32_t m = L.shards; m > 0 && j == 0; --m) {
                const uint32_t want = (L.topk + m - 1) / m;
                const uint32_t have = __popc(__ballot_sync(0xffffffffu, c0 >= want)) +
                                      __popc(__ballot_sync(0xffffffffu, c1 >= want));
                if (want > 0 && have >= m) j = want;
            }
        float tau = INFINITY;
        if (j > 0) {
            const float a = c0 >= j ? L.scores[lane][row + j - 1] : INFINITY;
            const float b = c1 >= j ? L.scores[lane + 32][row + j - 1] : INFINITY;
            tau = fminf(a, b);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tau = fminf(tau, __shfl_xor_sync(0xffffffffu, tau, o));
        s_n[lane] = c0;
        s_n[lane + 32] = c1;
        if (lane == 0) {
            s_tau = tau;
            s_all = j == 0;
            L.out_count[q] = min(total, L.topk);
        }
    }
    __syncthreads();
    if (!s_all) {
        // each list's entries that are not below tau: a 32-way search per warp (a NaN is not below it)
        const float tau = s_tau;
        for (uint32_t s = warp; s < L.shards; s += NT / 32) {
            const float* sc = L.scores[s] + row;
            uint32_t lo = 0, hi = s_n[s];  // entries before lo are in, those from hi on are out
            while (lo < hi) {
                const uint32_t step = (hi - lo + 31) / 32;
                const uint32_t at = lo + lane * step;
                const bool in = at < hi && !(sc[at] < tau);
                const uint32_t ins = __popc(__ballot_sync(0xffffffffu, in));  // a prefix of the lanes
                if (ins == 0) {
                    hi = lo;
                } else {
                    hi = min(hi, lo + ins * step);
                    lo = lo + (ins - 1) * step + 1;
                }
            }
            __syncwarp();
            if (lane == 0) s_n[s] = lo;
        }
        __syncthreads();
    }
    // The prefixes' scores as order-preserving keys, each list padded with zeros to the same power of two:
    // a search for how many keys of list t exceed a key is then log2(P) identical steps. An equal key of a
    // lower shard precedes: it exceeds the key minus one.
    uint32_t longest = max(s_n[lane], s_n[lane + 32]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
    if (longest == 0) return;
    const uint32_t log_p = 32u - __clz(longest), P = 1u << log_p;  // P > longest: the search can pass every entry
    if (L.shards * static_cast<uint64_t>(P) <= kMergeCap) {
        for (uint32_t e = threadIdx.x; e < L.shards * P; e += NT) {
            const uint32_t s = e >> log_p, i = e & (P - 1u);
            merge_key[e] = i < s_n[s] ? float_key(L.scores[s][row + i]) : 0u;
        }
        __syncthreads();
        for (uint32_t e = threadIdx.x; e < L.shards * P; e += NT) {
            const uint32_t s = e >> log_p, i = e & (P - 1u);
            if (i >= s_n[s]) continue;
            const uint32_t key = merge_key[e];
            const int64_t id = L.ids[s][row + i];
            uint32_t pos = i;
            for (uint32_t t = 0; t < L.shards; t += 2) {  // two searches at a time
                const bool b = t + 1 < L.shards;
                const uint32_t ka = key - (t < s ? 1u : 0u), kb = key - (t + 1 < s ? 1u : 0u);
                const uint32_t *pa = merge_key + t * P - 1, *pb = b ? pa + P : pa;
                uint32_t na = 0, nb = 0;
                for (uint32_t step = P >> 1; step > 0; step >>= 1) {
                    na += pa[na + step] > ka ? step : 0u;
                    nb += pb[nb + step] > kb ? step : 0u;
                }
                pos += (t != s ? na : 0u) + (b && t + 1 != s ? nb : 0u);
            }
            if (pos < L.topk) {
                const uint64_t o = static_cast<uint64_t>(q) * L.out_stride + pos;
                L.out_score[o] = L.scores[s][row + i];
                L.out_id[o] = id;
            }
        }
        return;
    }
    // prefixes past the buffer: searched in global memory
    for (uint32_t s = 0; s < L.shards; ++s)
        for (uint32_t i = threadIdx.x; i < s_n[s]; i += NT) {
            const float x = L.scores[s][row + i];
            uint32_t pos = i;
            for (uint32_t t = 0; t < L.shards && pos < L.topk; ++t)
                if (t != s) pos += preceding(L.scores[t] + row, s_n[t], x, t < s);
            if (pos < L.topk) {
                const uint64_t o = static_cast<uint64_t>(q) * L.out_stride + pos;
                L.out_score[o] = x;
                L.out_id[o] = L.ids[s][row + i];
            }
        }
}
}  // namespace

cudaError_t launch_merge_shards(const ShardMergeLaunch& L, cudaStream_t stream) {
    if (L.nq == 0) return cudaSuccess;
    if (L.shards == 0 || L.shards > kMaxShards || L.topk > static_cast<uint32_t>(kMaxTopK) || L.topk > L.out_stride ||
        !L.out_score || !L.out_id || !L.out_count)
        return cudaErrorInvalidValue;
    for (uint32_t s = 0; s < L.shards; ++s)
        if (!L.scores[s] || !L.ids[s] || !L.counts[s]) return cudaErrorInvalidValue;
    uint64_t keys = 1;  // the lists padded, uncut
    while (keys <= (L.in_stride < L.topk ? L.in_stride : L.topk)) keys *= 2;
    keys *= L.shards;
    if (L.shards == 1) {
        copy_shard_kernel<<<L.nq, kCopyT, 0, stream>>>(L);
    } else if (keys <= (L.shards <= 8 ? kMergeFew : kMergeFew / 2)) {
        merge_shards_kernel<kMergeFew><<<L.nq, kMergeFew, keys * sizeof(uint32_t), stream>>>(L);
    } else {
        const size_t held = keys < kMergeCap ? keys : kMergeCap;
        merge_shards_kernel<kMergeT><<<L.nq, kMergeT, held * sizeof(uint32_t), stream>>>(L);
    }
    return cudaGetLastError();
}

}  // namespace hss
