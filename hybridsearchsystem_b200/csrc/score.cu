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

    // rows past the matrices copy the last row instead (in bounds; their outputs are not stored)
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
            if (part < k4)
                copy4_async<VEC>(sq + r * kExactK + part * 4,
                                 qry + static_cast<uint64_t>(min(q0 + r, m - 1)) * dim + k0 + part * 4);
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

// ---------------------------------------------------------------------------------------------
// SIMT candidate pass.
// 256 threads = 32 doc groups (4 docs each) x 8 query groups (8 queries each); a warp is one query
// group, so the epilogue's per-query ballots are warp-uniform.
// ---------------------------------------------------------------------------------------------
constexpr int kCT = 256;
constexpr int kCQ = 64;   // queries per chunk
constexpr int kCK = 32;   // dims per smem stage
static_assert(kSimtGroup == 4, "a thread's docs of a tile are one group");
constexpr int kDPad = kDocTile + 4;
constexpr int kQPad = kCQ + 4;

// MAXIMA: the pass writes group maxima (CandLaunch::best) instead of candidates.
template <bool MAXIMA>
__global__ void __launch_bounds__(kCT) cand_simt_kernel(CandLaunch L) {
    extern __shared__ uint32_t sCount[];  // [nq_list] candidates this CTA found per query
    __shared__ __align__(16) float sD[kCK][kDPad];
    __shared__ __align__(16) float sQ[kCK][kQPad];
    __shared__ uint64_t sBits[kCQ][2];
    __shared__ float sTheta[kCQ];
    __shared__ uint32_t sQi[kCQ];

    const uint32_t tid = threadIdx.x;
    const uint32_t dg = tid & 31;  // lane
    const uint32_t qg = tid >> 5;  // warp
    const uint32_t nchunks = (L.nq_list + kCQ - 1) / kCQ;
    const uint32_t kchunks = (L.dim + kCK - 1) / kCK;
    launch_dependents();
    wait_for_previous();
    for (uint32_t i = tid; i < L.nq_list; i += kCT) sCount[i] = 0;

    TileWalk walk(L.tile_begin, L.tile_step, L.tile_skip, blockIdx.x, gridDim.x);
    for (uint64_t it = blockIdx.x; it < L.tile_count; it += gridDim.x, walk.advance()) {
        const uint64_t tile = walk.tile();
        const uint64_t doc0 = tile * kDocTile;
        for (uint32_t chunk = 0; chunk < nchunks; ++chunk) {
            float acc[4][8];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[r][j] = 0.0f;

            for (uint32_t kc = 0; kc < kchunks; ++kc) {
                __syncthreads();
                const uint32_t k0 = kc * kCK;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t f = tid + kCT * i;
                    const uint32_t doc = f >> 3, part = f & 7;
                    const uint32_t k = k0 + part * 4;
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (k < L.dim) v = *reinterpret_cast<const float4*>(L.vec + (doc0 + doc) * L.dim + k);
                    sD[part * 4 + 0][doc] = v.x;
                    sD[part * 4 + 1][doc] = v.y;
                    sD[part * 4 + 2][doc] = v.z;
                    sD[part * 4 + 3][doc] = v.w;
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t f = tid + kCT * i;
                    const uint32_t qq = f >> 3, part = f & 7;
                    const uint32_t k = k0 + part * 4;
                    const uint32_t li = chunk * kCQ + qq;
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (li < L.nq_list && k < L.dim) {
                        const uint32_t qi = L.qlist ? L.qlist[li] : li;
                        v = *reinterpret_cast<const float4*>(L.qry + static_cast<uint64_t>(qi) * L.dim + k);
                    }
                    sQ[part * 4 + 0][qq] = v.x;
                    sQ[part * 4 + 1][qq] = v.y;
                    sQ[part * 4 + 2][qq] = v.z;
                    sQ[part * 4 + 3][qq] = v.w;
                }
                if (kc == 0 && tid < kCQ) {
                    const uint32_t li = chunk * kCQ + tid;
                    uint64_t b0 = 0, b1 = 0;
                    float th = INFINITY;
                    uint32_t qi = 0xffffffffu;
                    if (li < L.nq_list) {
                        qi = L.qlist ? L.qlist[li] : li;
                        const uint64_t* brow = L.bits + static_cast<uint64_t>(qi) * L.bits_stride + tile * 2;
                        b0 = brow[0];
                        b1 = brow[1];
                        th = L.theta[qi];
                    }
                    sBits[tid][0] = b0;
                    sBits[tid][1] = b1;
                    sTheta[tid] = th;
                    sQi[tid] = qi;
                }
                __syncthreads();
#pragma unroll 8
                for (int k = 0; k < kCK; ++k) {
                    const float4 d4 = *reinterpret_cast<const float4*>(&sD[k][dg * 4]);
                    const float4 qa = *reinterpret_cast<const float4*>(&sQ[k][qg * 8]);
                    const float4 qb = *reinterpret_cast<const float4*>(&sQ[k][qg * 8 + 4]);
                    const float dv[4] = {d4.x, d4.y, d4.z, d4.w};
                    const float qv[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
                    for (int r = 0; r < 4; ++r)
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[r][j] = fmaf(dv[r], qv[j], acc[r][j]);
                }
            }

            // Epilogue: filter bit && score >= theta -> append (score, location) to this CTA's segment
            // of the query's list (a shared-memory count per query; no global atomics).
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t qq = qg * 8 + j;
                const uint32_t qi = sQi[qq];
                if (qi == 0xffffffffu) continue;  // warp-uniform
                const float th = sTheta[qq];
                const uint64_t w0 = sBits[qq][0], w1 = sBits[qq][1];
                if constexpr (MAXIMA) {
                    float b = -INFINITY;
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const uint32_t dl = dg * 4 + r;
                        if (((dl < 64 ? w0 : w1) >> (dl & 63)) & 1ull) b = fmaxf(b, acc[r][j]);
                    }
                    L.best[static_cast<uint64_t>(qi) * L.cap + it * (kDocTile / kSimtGroup) + dg] = b;
                    continue;
                }
                const uint64_t seg =
                    static_cast<uint64_t>(qi) * L.cap + static_cast<uint64_t>(L.seg_base + blockIdx.x) * L.seg_cap;
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const uint32_t dl = dg * 4 + r;
                    const uint64_t w = dl < 64 ? w0 : w1;
                    const bool pred = ((w >> (dl & 63)) & 1ull) && acc[r][j] >= th;
                    const uint32_t mask = __ballot_sync(0xffffffffu, pred);
                    if (mask == 0) continue;
                    uint32_t base = 0;
                    const uint32_t leader = __ffs(mask) - 1;
                    if (dg == leader) base = atomicAdd(&sCount[chunk * kCQ + qq], __popc(mask));
                    base = __shfl_sync(0xffffffffu, base, leader);
                    if (pred) {
                        const uint32_t idx = base + __popc(mask & ((1u << dg) - 1u));
                        if (idx < L.seg_cap) {
                            L.cand_score[seg + idx] = acc[r][j];
                            L.cand_loc[seg + idx] = static_cast<uint32_t>(doc0 + dl);
                        }
                    }
                }
            }
        }
    }
    if (MAXIMA) return;
    __syncthreads();
    for (uint32_t i = tid; i < L.nq_list; i += kCT) {
        const uint32_t qi = L.qlist ? L.qlist[i] : i;
        L.cand_count[static_cast<uint64_t>(qi) * kMaxCandSegs + L.seg_base + blockIdx.x] = sCount[i];
    }
}

}  // namespace

// The tile: few queries take narrow ones (the pass is then bound by the doc rows, so no thread should
// carry chains of absent queries); from 5 queries on, 32 x 128 where that pads the batch to at most a
// tenth more queries than 16 x 64 does and still gives every SM a CTA, else 16 x 64.
cudaError_t launch_exact_score(const float* qry, const float* docs, float* out, uint32_t m, uint32_t n, uint32_t dim,
                               uint64_t ldc, cudaStream_t stream) {
    if (m == 0 || n == 0) return cudaSuccess;
    if ((static_cast<uint64_t>(m) + 7) / 8 > 65535u) return cudaErrorInvalidValue;
    constexpr uint64_t kSms = 148;
    if (m <= 2) return launch_exact_tile<2, 1, 1>(qry, docs, out, m, n, dim, ldc, stream);
    if (m <= 4)
        return n >= kSms * 256 ? launch_exact_tile<4, 2, 1>(qry, docs, out, m, n, dim, ldc, stream)
                               : launch_exact_tile<4, 1, 1>(qry, docs, out, m, n, dim, ldc, stream);
    const uint32_t pad32 = (m + 31) / 32 * 32, pad16 = (m + 15) / 16 * 16;
    const uint64_t ctas = static_cast<uint64_t>(pad32 / 32) * ((static_cast<uint64_t>(n) + 127) / 128);
    if (10ull * pad32 <= 11ull * pad16 && ctas >= kSms)
        return launch_exact_tile<8, 4, 4>(qry, docs, out, m, n, dim, ldc, stream);
    return launch_exact_tile<4, 2, 4>(qry, docs, out, m, n, dim, ldc, stream);
}

uint32_t cand_simt_segments(uint64_t tile_count, int num_sms, uint32_t cap) {
    uint64_t g = static_cast<uint64_t>(num_sms) * 3;
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
    const size_t smem = static_cast<size_t>(L.nq_list) * sizeof(uint32_t);
    if (L.best && L.tile_count * (kDocTile / kSimtGroup) > L.cap) return cudaErrorInvalidValue;
    return launch_dependent(L.best ? cand_simt_kernel<true> : cand_simt_kernel<false>, dim3(L.segs), kCT, smem, stream,
                            1, L);
}

}  // namespace hss
