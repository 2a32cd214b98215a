// score.cu -- scoring kernels.
//
//  * exact_score_kernel: the materialised score matrix C[m x n] = Q . D^T of the reference's
//    kernel_vector_mmad (kernel_vector_mmad_op.cpp:3-11), computed in the ground truth's own
//    arithmetic (FP32, sequential over d, separate multiply and add), so every entry is bit-identical
//    to the CPU oracle's score. Used by the operator-level API and the parity tests.
//  * cand_simt_kernel: the bulk candidate pass on FP32 SIMT cores. Scores a 128-doc x 64-query tile
//    with FFMA (any summation order, error <= gamma_d * sum|q_i v_i|), tests the filter bit and the
//    per-query threshold in the epilogue and appends survivors to per-query candidate lists. The
//    B x N score matrix is never written.
#include "hss_device.cuh"
#include "hss_kernels.h"

namespace hss {
namespace {

// ---------------------------------------------------------------------------------------------
// Exact materialised scorer. Every output is one sequential chain of dim separate multiplies and adds,
// so the kernel is bound by FP32 issue: 2 m n dim lane operations at 128 per clock per SM (29 us for
// 32 x 131,072 x 128 at 1965 MHz), with the doc rows' 67 MB behind that (10 us). A thread keeps TQ x TD
// chains in registers, so a query value from shared memory serves TD docs and a doc value TQ queries:
// at 8 x 4, 12 16-byte shared loads feed 256 operations (one thread per doc, which re-read its row from
// L1 for every query and had one chain in flight, took 535 us there; this takes 45 us). Stages of 16
// dims, or one stage of 32, let 7 CTAs share an SM instead of 5 but took 51 and 53 us (more barriers;
// spills at 72 registers). Doc rows are copied as they lie (cp.async, two stages of 32 dims) with a
// row pitch of 36 floats, which keeps the 16-byte reads of 8 neighbouring rows on distinct banks.
// Packed f32x2 multiplies and adds are not used: they came out contracted into a fused multiply-add,
// which rounds once where the ground truth rounds twice.
// ---------------------------------------------------------------------------------------------
constexpr int kExactT = 128;        // threads: 4 warps, WQ of them side by side over the queries
constexpr int kExactK = 32;         // dims per stage
constexpr int kExactPitch = kExactK + 4;

// 16 bytes, or four 4-byte copies where a matrix is only 4-byte aligned (VEC false).
template <bool VEC>
__device__ __forceinline__ void copy4_async(float* smem, const float* gmem) {
    const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    if (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s + 4u * i), "l"(gmem + i) : "memory");
    }
}

template <int TQ, int TD, int WQ>
struct ExactTile {
    static constexpr int QT = TQ * WQ;             // queries per CTA
    static constexpr int DT = 32 * TD * (4 / WQ);  // docs per CTA
    static constexpr int stage_floats = DT * kExactPitch + QT * kExactK;
    static constexpr size_t smem = 2 * static_cast<size_t>(stage_floats) * sizeof(float);
};

template <int TQ, int TD, int WQ, bool VEC>
__global__ void __launch_bounds__(kExactT) exact_score_kernel(const float* __restrict__ qry,
                                                              const float* __restrict__ docs, float* __restrict__ out,
                                                              uint32_t m, uint32_t n, uint32_t dim, uint64_t ldc) {
    using T = ExactTile<TQ, TD, WQ>;
    extern __shared__ __align__(16) float exact_smem[];
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t wq = warp % WQ, wd = warp / WQ;
    const uint64_t doc0 = static_cast<uint64_t>(blockIdx.x) * T::DT;
    const uint32_t q0 = blockIdx.y * T::QT;
    const uint32_t chunks = (dim + kExactK - 1) / kExactK;

    // Rows past the matrices are not written and their outputs not stored: docs copy the last row (in bounds),
    // absent queries nothing (copies of the last query by every CTA met in one place: 100,000 docs x 100, 6
    // queries 47 us, 19 now)
    auto stage = [&](uint32_t c) {
        float* sd = exact_smem + (c & 1u) * T::stage_floats;
        float* sq = sd + T::DT * kExactPitch;
        const uint32_t k0 = c * kExactK, k4 = min(static_cast<uint32_t>(kExactK), dim - k0) / 4;
        for (uint32_t f = t; f < T::DT * (kExactK / 4); f += kExactT) {
            const uint32_t r = f / (kExactK / 4), part = f % (kExactK / 4);
            if (part < k4) {
                const uint64_t doc = min(doc0 + r, static_cast<uint64_t>(n) - 1);
                copy4_async<VEC>(sd + r * kExactPitch + part * 4, docs + doc * dim + k0 + part * 4);
            }
        }
        for (uint32_t f = t; f < T::QT * (kExactK / 4); f += kExactT) {
            const uint32_t r = f / (kExactK / 4), part = f % (kExactK / 4);
            if (part < k4 && q0 + r < m)
                copy4_async<VEC>(sq + r * kExactK + part * 4,
                                 qry + static_cast<uint64_t>(q0 + r) * dim + k0 + part * 4);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[TQ][TD];
#pragma unroll
    for (int i = 0; i < TQ; ++i)
#pragma unroll
        for (int j = 0; j < TD; ++j) acc[i][j] = 0.0f;

    stage(0);
    for (uint32_t c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) {
            stage(c + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const float* sd = exact_smem + (c & 1u) * T::stage_floats + (wd * 32u * TD + lane) * kExactPitch;
        const float* sq = exact_smem + (c & 1u) * T::stage_floats + T::DT * kExactPitch + wq * TQ * kExactK;
        const uint32_t kc = min(static_cast<uint32_t>(kExactK), dim - c * kExactK);
#pragma unroll 4
        for (uint32_t k = 0; k < kc; k += 4) {
            float4 d[TD];
#pragma unroll
            for (int j = 0; j < TD; ++j) d[j] = *reinterpret_cast<const float4*>(sd + j * 32 * kExactPitch + k);
#pragma unroll
            for (int i = 0; i < TQ; ++i) {
                const float4 q = *reinterpret_cast<const float4*>(sq + i * kExactK + k);
#pragma unroll
                for (int j = 0; j < TD; ++j) {
                    float s = acc[i][j];
                    s = __fadd_rn(s, __fmul_rn(q.x, d[j].x));
                    s = __fadd_rn(s, __fmul_rn(q.y, d[j].y));
                    s = __fadd_rn(s, __fmul_rn(q.z, d[j].z));
                    s = __fadd_rn(s, __fmul_rn(q.w, d[j].w));
                    acc[i][j] = s;
                }
            }
        }
        __syncthreads();  // the stage is read before the next-but-one chunk is copied into it
    }
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
        const uint32_t q = q0 + wq * TQ + i;
        if (q >= m) break;
#pragma unroll
        for (int j = 0; j < TD; ++j) {
            const uint64_t doc = doc0 + wd * 32u * TD + lane + 32u * j;
            if (doc < n) out[q * ldc + doc] = acc[i][j];
        }
    }
}

template <int TQ, int TD, int WQ>
cudaError_t launch_exact_tile(const float* qry, const float* docs, float* out, uint32_t m, uint32_t n, uint32_t dim,
                              uint64_t ldc, cudaStream_t stream) {
    using T = ExactTile<TQ, TD, WQ>;
    const bool vec = ((reinterpret_cast<uintptr_t>(qry) | reinterpret_cast<uintptr_t>(docs)) & 15u) == 0;
    auto kernel = vec ? exact_score_kernel<TQ, TD, WQ, true> : exact_score_kernel<TQ, TD, WQ, false>;
    if (T::smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(T::smem));
        if (e != cudaSuccess) return e;
    }
    const dim3 grid(static_cast<uint32_t>((static_cast<uint64_t>(n) + T::DT - 1) / T::DT), (m + T::QT - 1) / T::QT);
    kernel<<<grid, kExactT, T::smem, stream>>>(qry, docs, out, m, n, dim, ldc);
    return cudaGetLastError();
}

// Rows of at most kShortDim floats: bound by the doc rows' and the outputs' bytes, at launch latency in the sizes in
// use, and a staged tile would wait for a copy of a few sectors a row through shared memory. A thread reads its doc's
// row into registers and forms every query's chain from it, up to 32 queries to a CTA (broadcast from shared memory).
// 300,000 docs, us staged -> so: 4 dims 1 query 7.0 -> 3.6, 8 queries 21.9 -> 3.9, 32 queries 16.8 -> 7.8; 16 dims 1
// query 7.0 -> 5.2, 32 queries 19.6 -> 18.4; 28 dims 1 query 8.0 -> 6.3, 8 queries 40.5 -> 11.5, 32 queries even. Past
// 16 dims a second CTA's worth of queries is better staged (100,000 docs x 28, 100 queries: 40 us).
constexpr uint32_t kShortDim = 28, kShortDimMany = 16, kShortQueries = 32;
constexpr int kShortT = 128;

template <int QUADS, bool VEC>
__global__ void __launch_bounds__(kShortT) exact_short_kernel(const float* __restrict__ qry,
                                                              const float* __restrict__ docs, float* __restrict__ out,
                                                              uint32_t m, uint32_t n, uint64_t ldc, uint32_t per) {
    __shared__ __align__(16) float sq[kShortQueries * QUADS * 4];
    const uint32_t q0 = blockIdx.y * per, queries = min(per, m - q0);
    for (uint32_t i = threadIdx.x; i < queries * QUADS * 4; i += kShortT)
        sq[i] = qry[static_cast<uint64_t>(q0) * QUADS * 4 + i];
    const uint64_t doc = static_cast<uint64_t>(blockIdx.x) * kShortT + threadIdx.x;
    float4 v[QUADS];
    if (doc < n) {
        const float* row = docs + doc * (QUADS * 4);
#pragma unroll
        for (int i = 0; i < QUADS; ++i)
            v[i] = VEC ? *reinterpret_cast<const float4*>(row + 4 * i)
                       : make_float4(row[4 * i], row[4 * i + 1], row[4 * i + 2], row[4 * i + 3]);
    }
    __syncthreads();
    if (doc >= n) return;
    for (uint32_t q = 0; q < queries; ++q) {
        float s = 0.0f;
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(sq + (q * QUADS + i) * 4);
            s = __fadd_rn(s, __fmul_rn(x.x, v[i].x));
            s = __fadd_rn(s, __fmul_rn(x.y, v[i].y));
            s = __fadd_rn(s, __fmul_rn(x.z, v[i].z));
            s = __fadd_rn(s, __fmul_rn(x.w, v[i].w));
        }
        out[(static_cast<uint64_t>(q0) + q) * ldc + doc] = s;
    }
}

template <int QUADS>
cudaError_t launch_exact_short(const float* qry, const float* docs, float* out, uint32_t m, uint32_t n, uint64_t ldc,
                               cudaStream_t stream) {
    const bool vec = (reinterpret_cast<uintptr_t>(docs) & 15u) == 0;
    auto kernel = vec ? exact_short_kernel<QUADS, true> : exact_short_kernel<QUADS, false>;
    // fewer queries to a CTA where the docs alone would leave SMs with less than four CTAs
    const uint64_t tiles = (n - 1) / kShortT + 1;
    uint32_t per = kShortQueries;
    const uint64_t ctas = 4ull * device_sms();
    while (per > 2 && tiles * ((m - 1) / per + 1) < ctas) per /= 2;
    const dim3 grid(static_cast<uint32_t>(tiles), (m - 1) / per + 1);
    kernel<<<grid, kShortT, 0, stream>>>(qry, docs, out, m, n, ldc, per);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// SIMT candidate pass, bound by the FP32 pipe: 2 nq n dim flop at 74 TFLOP/s (64 queries x 1M docs x 128:
// 220 us). A CTA of 8 warps scores 128 docs for 8 TQ queries at a time: a warp is one group of TQ queries
// (so the epilogue's per-query ballots are warp-uniform), a lane has docs lane + 32 r, r < 4. Rows are
// staged as they lie (cp.async, three stages of 32 dims, a pitch of 36 floats: the 16-byte reads of 8
// neighbouring rows fall on distinct banks) and products are taken two dims at a time by packed
// multiply-adds: an accumulator holds the even and the odd dims' sums, added at the end (the pass's error
// bound holds for any order of summation). A packed instruction takes the pipe as long as two plain ones
// but one issue slot (in registers alone 4 x 8 outputs run at 63 TFLOP/s this way, 44 with plain
// multiply-adds). 64 queries x 1M docs x 128: 670 us with 4-byte transposed stores, one stage and plain
// multiply-adds, 455 us now (two stages with two barriers each: 468; 16 queries a thread in CTAs of 4 warps:
// 485, too few warps to hide the reads).
// ---------------------------------------------------------------------------------------------
constexpr int kCT = 256;           // threads: 8 warps
constexpr uint32_t kCWarps = kCT / 32;
constexpr int kCK = 32;            // dims per stage
constexpr int kCPitch = kCK + 4;
static_assert(kSimtGroup == 4, "a thread's docs of a tile are one group");
static_assert(kSampleRun * kSampleRuns == kDocTile && kCT / 8 == 2 * kSampleRun && kSampleRun == 16,
              "a sample tile's rows");

__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

template <int TQ>
struct SimtTile {
    static constexpr uint32_t QT = kCWarps * TQ;  // queries per chunk
    static constexpr uint32_t stage_floats = (kDocTile + QT) * kCPitch;
    // three stages, four chunks' filter words; then the queries' counts and thresholds
    static constexpr size_t fixed = 3 * stage_floats * sizeof(float) + 4 * QT * 16;
};

// MAXIMA: the pass writes group maxima (CandLaunch::best) of sample tiles instead of candidates.
template <int TQ, bool MAXIMA>
__global__ void __launch_bounds__(kCT, 2) cand_simt_kernel(CandLaunch L) {
    using T = SimtTile<TQ>;
    extern __shared__ __align__(16) unsigned char simt_smem[];
    float* ring = reinterpret_cast<float*>(simt_smem);
    uint4* sBits = reinterpret_cast<uint4*>(ring + 3 * T::stage_floats);  // [4][QT]: 128 docs' filter bits
    uint32_t* sCount = reinterpret_cast<uint32_t*>(sBits + 4 * T::QT);  // [nq_list] candidates found per query
    float* sTheta = reinterpret_cast<float*>(sCount + L.nq_list);

    const uint32_t tid = threadIdx.x, lane = tid & 31, qg = tid >> 5;
    const uint32_t nchunks = (L.nq_list + T::QT - 1) / T::QT;
    const uint32_t kchunks = (L.dim + kCK - 1) / kCK;
    launch_dependents();
    wait_for_previous();
    for (uint32_t i = tid; i < L.nq_list; i += kCT) {
        sCount[i] = 0;
        sTheta[i] = L.theta[L.qlist ? L.qlist[i] : i];
    }

    auto copy16 = [](void* smem, const void* gmem) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(smem))),
                     "l"(gmem)
                     : "memory");
    };
    // dims [32 kc, +32) of a tile's docs and a chunk's queries; with kc = 0 the chunk's filter words too
    auto copy_stage = [&](uint32_t tile, uint32_t chunk, uint32_t kc, uint32_t stage, uint32_t bits) {
        const uint32_t k0 = kc * kCK, part = tid & 7;
        float* sd = ring + stage * T::stage_floats + (tid >> 3) * kCPitch + part * 4;
        if (part * 4 < L.dim - k0) {
            // row tid / 8, then every 32nd: of the tile, or (MAXIMA) of the sample tile, whose rows 32 apart
            // are two runs apart
            const uint64_t row = tid >> 3;
            const uint64_t doc = MAXIMA ? (row / kSampleRun * L.sample_tiles + tile) * kSampleRun + row % kSampleRun
                                        : static_cast<uint64_t>(tile) * kDocTile + row;
            const uint64_t step = MAXIMA ? static_cast<uint64_t>(L.sample_tiles) * (kCT / 8) : kCT / 8;
            const float* v = L.vec + doc * L.dim + k0 + part * 4;
#pragma unroll
            for (uint32_t i = 0; i < kDocTile * 8 / kCT; ++i)
                copy16(sd + i * (kCT / 8) * kCPitch, v + i * step * L.dim);
#pragma unroll
            for (uint32_t i = 0; i < (T::QT * 8 + kCT - 1) / kCT; ++i) {
                const uint32_t r = (tid >> 3) + i * (kCT / 8);
                const uint32_t li = min(chunk * T::QT + r, L.nq_list - 1);  // past the list: not emitted
                const uint32_t qi = L.qlist ? L.qlist[li] : li;
                if (r < T::QT)
                    copy16(sd + (kDocTile + i * (kCT / 8)) * kCPitch,
                           L.qry + static_cast<uint64_t>(qi) * L.dim + k0 + part * 4);
            }
        }
        if (kc == 0 && tid < T::QT) {
            const uint32_t li = min(chunk * T::QT + tid, L.nq_list - 1);
            const uint32_t qi = L.qlist ? L.qlist[li] : li;
            const uint64_t* brow = L.bits + static_cast<uint64_t>(qi) * L.bits_stride;
            if (MAXIMA) {  // 16 bits of every run
                const uint16_t* p = reinterpret_cast<const uint16_t*>(brow) + tile;
                uint32_t b[kSampleRuns];
#pragma unroll
                for (uint32_t r = 0; r < kSampleRuns; ++r) b[r] = p[static_cast<uint64_t>(r) * L.sample_tiles];
                sBits[bits * T::QT + tid] =
                    make_uint4(b[0] | b[1] << 16, b[2] | b[3] << 16, b[4] | b[5] << 16, b[6] | b[7] << 16);
            } else {
                // bitmap rows and tiles are multiples of 16 bytes (segments of 128 docs)
                copy16(sBits + bits * T::QT + tid, brow + tile * 2ull);
            }
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };

    // The it-th tile of the pass (32-bit: the launcher checks tile_walk_fits).
    auto tile_at = [&](uint32_t it) {
        if (MAXIMA) return sample_tile_of(it, L.block_step);
        return L.tile_skip >= 2 ? it + it / (L.tile_skip - 1) + 1
                                : static_cast<uint32_t>(L.tile_begin) + it * static_cast<uint32_t>(L.tile_step);
    };
    // Stages in order, tile by tile, chunk by chunk, k by k, are copied two ahead into a ring of three. The
    // next one to copy:
    const uint32_t count = static_cast<uint32_t>(L.tile_count);
    uint32_t c_it = blockIdx.x, c_chunk = 0, c_k = 0, c_stage = 0, c_bits = 0;
    auto copy_next = [&] {
        if (c_it < count) {
            copy_stage(tile_at(c_it), c_chunk, c_k, c_stage, c_bits);
            c_stage = c_stage == 2 ? 0 : c_stage + 1;
            if (++c_k == kchunks) {
                c_k = 0;
                c_bits = (c_bits + 1) & 3;
                if (++c_chunk == nchunks) {
                    c_chunk = 0;
                    c_it += gridDim.x;
                }
            }
        }
        commit();
    };
    copy_next();
    copy_next();
    uint32_t stage = 0, bits = 0;
    for (uint32_t it = blockIdx.x; it < count; it += gridDim.x) {
        const uint32_t doc0 = tile_at(it) * kDocTile;
        for (uint32_t chunk = 0; chunk < nchunks; ++chunk, bits = (bits + 1) & 3) {
            unsigned long long acc[4][TQ];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int j = 0; j < TQ; ++j) acc[r][j] = 0;
            for (uint32_t kc = 0; kc < kchunks; ++kc, stage = stage == 2 ? 0 : stage + 1) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncthreads();  // the stage has landed; the one copied into next was read by every warp
                copy_next();
                const float* sd = ring + stage * T::stage_floats + lane * kCPitch;
                const float* sq = ring + stage * T::stage_floats + (kDocTile + qg * TQ) * kCPitch;
                const uint32_t kn = min(static_cast<uint32_t>(kCK), L.dim - kc * kCK);
#pragma unroll 2
                for (uint32_t k = 0; k < kn; k += 4) {
                    ulonglong2 d[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        d[r] = *reinterpret_cast<const ulonglong2*>(sd + r * 32 * kCPitch + k);
#pragma unroll
                    for (int j = 0; j < TQ; ++j) {
                        const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(sq + j * kCPitch + k);
#pragma unroll
                        for (int r = 0; r < 4; ++r) fma2(acc[r][j], d[r].x, q.x);
#pragma unroll
                        for (int r = 0; r < 4; ++r) fma2(acc[r][j], d[r].y, q.y);
                    }
                }
            }

            // Epilogue: filter bit && score >= theta -> append (score, location) to this CTA's segment
            // of the query's list (a shared-memory count per query; no global atomics).
#pragma unroll
            for (int j = 0; j < TQ; ++j) {
                const uint32_t li = chunk * T::QT + qg * TQ + j;
                if (li >= L.nq_list) break;  // warp-uniform
                const uint4 w = sBits[bits * T::QT + qg * TQ + j];
                const uint32_t word[4] = {w.x, w.y, w.z, w.w};
                float s[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float2 x = *reinterpret_cast<const float2*>(&acc[r][j]);
                    s[r] = (word[r] >> lane) & 1u ? x.x + x.y : -INFINITY;
                }
                if constexpr (MAXIMA) {
                    const uint32_t qi = L.qlist ? L.qlist[li] : li;
                    L.best[static_cast<uint64_t>(qi) * L.cap + it * (kDocTile / kSimtGroup) + lane] =
                        fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
                    continue;
                }
                const float th = sTheta[li];
                if (!__any_sync(0xffffffffu, fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3])) >= th)) continue;
                const uint32_t qi = L.qlist ? L.qlist[li] : li;
                const uint64_t seg =
                    static_cast<uint64_t>(qi) * L.cap + static_cast<uint64_t>(L.seg_base + blockIdx.x) * L.seg_cap;
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const bool pred = ((word[r] >> lane) & 1u) && s[r] >= th;
                    const uint32_t mask = __ballot_sync(0xffffffffu, pred);
                    if (mask == 0) continue;
                    // the query is this warp's alone: no atomic
                    const uint32_t base = sCount[li];
                    __syncwarp();
                    if (lane == 0) sCount[li] = base + __popc(mask);
                    __syncwarp();
                    if (pred) {
                        const uint32_t idx = base + __popc(mask & ((1u << lane) - 1u));
                        if (idx < L.seg_cap) {
                            L.cand_score[seg + idx] = s[r];
                            L.cand_loc[seg + idx] = doc0 + 32u * r + lane;
                        }
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (MAXIMA) return;
    __syncthreads();
    for (uint32_t i = tid; i < L.nq_list; i += kCT) {
        const uint32_t qi = L.qlist ? L.qlist[i] : i;
        L.cand_count[static_cast<uint64_t>(qi) * kMaxCandSegs + L.seg_base + blockIdx.x] = sCount[i];
    }
}

template <int TQ>
cudaError_t launch_cand_simt_tile(const CandLaunch& L, cudaStream_t stream) {
    const size_t smem = SimtTile<TQ>::fixed + static_cast<size_t>(L.nq_list) * 8;
    // the most any caller's batch needs: searchers on other threads launch the same kernel
    constexpr size_t kCeiling = SimtTile<TQ>::fixed + static_cast<size_t>(kMaxSimtBatch) * 8;
    auto kernel = L.best ? cand_simt_kernel<TQ, true> : cand_simt_kernel<TQ, false>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kCeiling));
    if (e != cudaSuccess) return e;
    return launch_dependent(kernel, dim3(L.segs), kCT, smem, stream, 1, L);
}

}  // namespace

// Short rows go straight to registers (exact_short_kernel). The tile of longer ones: few queries take narrow ones
// (the pass is then bound by the doc rows, so no thread should carry chains of absent queries); from 5 queries on,
// 32 x 128 where that pads the batch to at most a tenth more queries than 16 x 64 does and still gives every SM a
// CTA, else 16 x 64.
cudaError_t launch_exact_score(const float* qry, const float* docs, float* out, uint32_t m, uint32_t n, uint32_t dim,
                               uint64_t ldc, cudaStream_t stream) {
    if (m == 0 || n == 0) return cudaSuccess;
    if ((static_cast<uint64_t>(m) + 7) / 8 > 65535u) return cudaErrorInvalidValue;
    const uint64_t sms = device_sms();
    if (dim <= (m <= kShortQueries ? kShortDim : kShortDimMany)) {
        switch (dim / 4) {
            case 1: return launch_exact_short<1>(qry, docs, out, m, n, ldc, stream);
            case 2: return launch_exact_short<2>(qry, docs, out, m, n, ldc, stream);
            case 3: return launch_exact_short<3>(qry, docs, out, m, n, ldc, stream);
            case 4: return launch_exact_short<4>(qry, docs, out, m, n, ldc, stream);
            case 5: return launch_exact_short<5>(qry, docs, out, m, n, ldc, stream);
            case 6: return launch_exact_short<6>(qry, docs, out, m, n, ldc, stream);
            case 7: return launch_exact_short<7>(qry, docs, out, m, n, ldc, stream);
        }
    }
    if (m <= 2) return launch_exact_tile<2, 1, 1>(qry, docs, out, m, n, dim, ldc, stream);
    if (m <= 4)
        return n >= sms * 256 ? launch_exact_tile<4, 2, 1>(qry, docs, out, m, n, dim, ldc, stream)
                               : launch_exact_tile<4, 1, 1>(qry, docs, out, m, n, dim, ldc, stream);
    const uint32_t pad32 = (m + 31) / 32 * 32, pad16 = (m + 15) / 16 * 16;
    const uint64_t ctas = static_cast<uint64_t>(pad32 / 32) * ((static_cast<uint64_t>(n) + 127) / 128);
    if (10ull * pad32 <= 11ull * pad16 && ctas >= sms)
        return launch_exact_tile<8, 4, 4>(qry, docs, out, m, n, dim, ldc, stream);
    return launch_exact_tile<4, 2, 4>(qry, docs, out, m, n, dim, ldc, stream);
}

uint32_t cand_simt_segments(uint64_t tile_count, int num_sms, uint32_t cap) {
    uint64_t g = static_cast<uint64_t>(num_sms) * 2;  // the CTAs resident at a time
    g = tile_count < g ? tile_count : g;
    g = g < kMaxCandSegs / 2 ? g : kMaxCandSegs / 2;  // one segment per CTA, room for two passes
    const uint64_t by_cap = cap / (2 * kMinSegCap) > 0 ? cap / (2 * kMinSegCap) : 1;
    return static_cast<uint32_t>(g < by_cap ? g : by_cap);
}

cudaError_t launch_cand_simt(const CandLaunch& L, int num_sms, cudaStream_t stream) {
    if (L.tile_count == 0 || L.nq_list == 0) return cudaSuccess;
    const uint64_t seg_end = static_cast<uint64_t>(L.seg_base) + L.segs;
    if (L.segs != cand_simt_segments(L.tile_count, num_sms, L.cap) || L.seg_cap == 0 || seg_end > kMaxCandSegs ||
        seg_end * L.seg_cap > L.cap || L.nq_list > kMaxSimtBatch ||
        !tile_walk_fits(L.tile_begin, L.tile_step, L.tile_skip, L.tile_count, L.segs))
        return cudaErrorInvalidValue;
    if (L.best && (L.tile_count * (kDocTile / kSimtGroup) > L.cap || L.bits_stride < 2ull * L.sample_tiles ||
                   !sample_fits(L.tile_count, L.block_step, L.sample_tiles)))
        return cudaErrorInvalidValue;
    // the filter words and rows are copied 16 bytes at a time
    if ((L.bits_stride & 1u) || (reinterpret_cast<uintptr_t>(L.bits) & 15u) || (reinterpret_cast<uintptr_t>(L.vec) & 15u) ||
        (reinterpret_cast<uintptr_t>(L.qry) & 15u))
        return cudaErrorInvalidValue;
    // chunks as narrow as the batch: a chunk's pipe time is that of all its queries
    if (L.nq_list <= 8) return launch_cand_simt_tile<1>(L, stream);
    if (L.nq_list <= 16) return launch_cand_simt_tile<2>(L, stream);
    if (L.nq_list <= 32) return launch_cand_simt_tile<4>(L, stream);
    return launch_cand_simt_tile<8>(L, stream);
}

}  // namespace hss
