// The kernels around the attention for sm_100a: the merge of split items, the arrival flags and the push of the fused all-gather, the
// cache write, and small helpers.
#include <cuda_bf16.h>
#include <cfloat>
#include "defs.h"
#include "ptx.cuh"
#include "rows.cuh"

namespace dsa {

__global__ void debug_rows_kernel(AttnParams p, int total_q, int32_t* rows_out) {
    const long long n = (long long)total_q * p.topk;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int q = (int)(i / p.topk);
        rows_out[i] = translate_row(__ldg(p.indices + i), q / p.s_q, p);
    }
}

// ------------------------------------------------------------------ split merge
// Same arithmetic as the reference's two-pass merge (opus_attn/dsa_v32/common/mla_reduce.hpp:92-156): m = max lse_i,
// w_i = exp2((lse_i - m) log2e) (0 for an empty split), out = sum w_i O_i / sum w_i, lse = m + ln(sum w_i); all
// empty -> 0, +inf.
// The partials were written by the kernel before and come from L2 (16 splits x 128 heads: 4 MB), so the time is a
// chain of load latencies, not bytes: the plan's tables are read before the wait for the attention kernel, lane i then
// fetches the lse of split i while the first partial rows (eight or sixteen float4 per lane) are already on their way.
// kV = float4 per lane and split: a warp covers 128 kV columns of one tile row, a block four warps.  kV = 1 (a block per
// row) while all blocks are resident at once, else kV = 4 (a warp per row), which needs a quarter of the blocks.
// Measured: decode of one sequence (16 splits) 25.3 -> 19.8 us, batch 16 37.1 -> 35.4 us, two sequences of 16 heads on a bf16
// cache 21.5 -> 15.9 us, against one warp per row that walked the splits one by one (slot, then lse, then four float4).
// With kV = 1 throughout, a prefill chunk of 64 split rows x 64 heads took 8.9 us for its merge instead of 5.2.
// kFlight = float4 in flight per lane: 16, so that the 16 splits of a row come in one round, where four blocks an SM are enough (one sequence 16.55 -> 16.15 us,
// two sequences of 16 heads on a bf16 cache 12.42 -> 12.00; with 16 throughout, 16 sequences 30.35 -> 30.45, 100 92.2 -> 94.5), else 8.
constexpr int kMergeBlocks = 8;                       // blocks per SM of the form with kV = 1, kFlight = 8 (64 registers per thread)
constexpr int kMergeBlocksDeep = 4;                   // and with kFlight = 16
template <int kV, int kFlight>
__global__ void __launch_bounds__(128, kFlight == 16 ? kMergeBlocksDeep : kV == 1 ? kMergeBlocks : kMergeBlocks - 1) combine_kernel(const float* __restrict__ o_accum, const float* __restrict__ lse_accum,
                                                      const int32_t* __restrict__ reduce_indptr,
                                                      const int32_t* __restrict__ reduce_slots,
                                                      const ReduceDst* __restrict__ reduce_dst, const OutTargets tgt,
                                                      int64_t stride_o_row, int64_t stride_o_head, int H) {
    constexpr int kF = kFlight / kV;    // splits in flight
    const int rr = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hrow = kV == 1 ? blockIdx.y : blockIdx.y * 4 + warp;   // row of the 128-row tile
    const int col = (kV == 1 ? warp * 128 : 0) + lane * 4;
    // the tables belong to the plan: no kernel writes them
    const ReduceDst dst = reduce_dst[rr];
    const int s0 = reduce_indptr[rr], ns = reduce_indptr[rr + 1] - s0;
    int slot = lane < ns ? __ldg(reduce_slots + s0 + lane) : 0;
    grid_dependency_wait();   // launched ahead of the attention kernel's end (programmatic stream serialization)
    int head = dst.head_block * kHeadsPerBlock + hrow, q_row = dst.q_row;
    if (dst.head_block < 0) {   // stacked unit: -head_block query rows of H heads each
        const int sub = hrow / H;
        if (sub >= -dst.head_block) return;
        head = hrow - sub * H;
        q_row += sub;
    }
    if (head >= H || hrow >= kHeadsPerBlock) return;
    float lse_i = lane < ns ? lse_accum[(size_t)slot * kHeadsPerBlock + hrow] : -FLT_MAX;
    const float* src = o_accum + (size_t)hrow * kDV + col;
    float4 x[kF][kV];
    auto load = [&](int j, int n) {   // splits [j, j + kF) of the chunk's n; j + k <= 31, so the source lane is always in range
#pragma unroll
        for (int k = 0; k < kF; ++k) {
            const int sl = __shfl_sync(0xffffffffu, slot, j + k);
#pragma unroll
            for (int v = 0; v < kV; ++v) {
                x[k][v] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (j + k < n) x[k][v] = *reinterpret_cast<const float4*>(src + (size_t)sl * kHeadsPerBlock * kDV + v * 128);
            }
        }
    };
    load(0, min(32, ns));
    float m = lse_i;
    for (int i = lane + 32; i < ns; i += 32) m = fmaxf(m, lse_accum[(size_t)reduce_slots[s0 + i] * kHeadsPerBlock + hrow]);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    float4 acc[kV];
#pragma unroll
    for (int v = 0; v < kV; ++v) acc[v] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float denom = 0.0f;
    for (int c0 = 0; c0 < ns; c0 += 32) {
        if (c0) {
            slot = c0 + lane < ns ? __ldg(reduce_slots + s0 + c0 + lane) : 0;
            lse_i = c0 + lane < ns ? lse_accum[(size_t)slot * kHeadsPerBlock + hrow] : -FLT_MAX;
        }
        // an empty piece has no weight, one of infinite lse (an infinite sink) all of it; a NaN stays one
        const float wgt = lse_i == -FLT_MAX ? 0.0f : lse_i == m ? 1.0f : exp2f((lse_i - m) * 1.4426950408889634f);
        const int n = min(32, ns - c0);
        for (int j = 0; j < n; j += kF) {
            if (c0 + j) load(j, n);
#pragma unroll
            for (int k = 0; k < kF; ++k) {   // in split order, whatever the number in flight; past the end the weight is 0
                const float wk = __shfl_sync(0xffffffffu, wgt, j + k);
                denom += wk;
#pragma unroll
                for (int v = 0; v < kV; ++v) {
                    acc[v].x += wk * x[k][v].x;
                    acc[v].y += wk * x[k][v].y;
                    acc[v].z += wk * x[k][v].z;
                    acc[v].w += wk * x[k][v].w;
                }
            }
        }
    }
    const float inv = denom == 0.0f ? 0.0f : 1.0f / denom;
    const float lse_val = denom == 0.0f ? INFINITY : m + log2f(denom) * 0.69314718055994531f;
    for (int d = 0; d < tgt.n_peers; ++d) {   // one destination, or every peer's gathered buffer
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(tgt.out[d]) + (size_t)q_row * stride_o_row + (size_t)head * stride_o_head + col;
#pragma unroll
        for (int v = 0; v < kV; ++v) {
            uint2 u;
            u.x = pack_bf16x2(acc[v].x * inv, acc[v].y * inv);
            u.y = pack_bf16x2(acc[v].z * inv, acc[v].w * inv);
            *reinterpret_cast<uint2*>(o + v * 128) = u;
        }
        if (col == 0 && tgt.lse[d] != nullptr) tgt.lse[d][(size_t)q_row * tgt.lse_stride_row + head] = lse_val;
    }
}

// ------------------------------------------------------------------ arrival flags of the fused all-gather
// After the kernels that stored this rank's rows into the peers' buffers: publish the step in every peer's
// flag array (system-scope release after a system-scope fence, so the rows are visible before the flag),
// then wait until every peer has published the same step here.  The wait is bounded (one second); on expiry
// the status word gets DSA_V32_ERR_DEVICE_WAIT and the kernel returns.
__global__ void __launch_bounds__(32) peer_signal_wait_kernel(const PeerSync s) {
    const int lane = threadIdx.x;
    __threadfence_system();
    if (lane < s.n_peers) {
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(s.flags[lane] + s.my_rank), "r"(s.step) : "memory");
        const uint32_t* mine = s.flags[s.my_rank] + lane;
        const uint64_t t0 = global_ns();
        bool ok = false;
        for (uint32_t it = 0; it < DSA_WAIT_LIMIT; ++it) {
            uint32_t v;
            asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(mine) : "memory");
            if (static_cast<int32_t>(v - s.step) >= 0) {
                ok = true;
                break;
            }
            if (global_ns() - t0 > 1000000000ull) break;
            __nanosleep(200);
        }
        if (!ok) atomicExch(s.status, DSA_V32_ERR_DEVICE_WAIT);
    }
}

// ------------------------------------------------------------------ cache write path
// One warp per row: per 128 values amax -> scale = amax / 448, e4m3(x / scale) with RNE and
// saturation (cvt.rn.satfinite), scales and rope appended.
// Eight lanes hold a group of 128 values (lane i of the eight: values 4 i + 32 j ..), so three shuffles give all four
// maxima at once, every load instruction takes four whole lines, and all loads of a row are in flight together.
// What bounds a few thousand rows is instruction issue, most of it the divisions.  The sixteen quotients of a lane share
// their divisor: with r = the rounded 1 / scale, q = x r and q + r (x - q scale) in fused steps is the rounded quotient
// (Markstein, IBM J. Res. Dev. 34, 1990); scales so small or large that a step could underflow or overflow divide.
// 8192 rows: 8.5 -> 6.1 us a call (host and kernel; a warp per row with 20 shuffles and 20 divisions per lane before).
__global__ void __launch_bounds__(256) pack_fp8_rows_kernel(const float* __restrict__ latent,
                                                            const __nv_bfloat16* __restrict__ rope,
                                                            const int64_t* __restrict__ dst_rows, uint8_t* __restrict__ out,
                                                            int64_t num_rows) {
    const int lane = threadIdx.x & 31, g = lane >> 3, i = lane & 7;
    const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= num_rows) return;
    const float4* x = reinterpret_cast<const float4*>(latent + r * kDV + g * 128) + i;
    float4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __ldg(x + 8 * j);
    const uint32_t rp = __ldg(reinterpret_cast<const uint32_t*>(rope + r * kDRope) + lane);
    const int64_t dr = dst_rows ? __ldg(reinterpret_cast<const long long*>(dst_rows) + r) : r;
    uint8_t* row = out + dr * kFp8RowBytes;
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    const float scale = amax > 0.0f ? __fdiv_rn(amax, 448.0f) : 1.0f;
    const float recip = __frcp_rn(scale);
    const bool plain = scale >= 0x1p-80f && scale <= 0x1p80f;   // (a NaN or infinite row divides)
    auto quotient = [&](float a) -> float {
        if (!plain) return __fdiv_rn(a, scale);
        const float q = __fmul_rn(a, recip);
        const float f = __fmaf_rn(__fmaf_rn(-q, scale, a), recip, q);
        return copysignf(f, a);   // -0 / scale
    };
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint16_t lo, hi;
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(quotient(v[j].y)), "f"(quotient(v[j].x)));
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(quotient(v[j].w)), "f"(quotient(v[j].z)));
        w[j] = (uint32_t)lo | ((uint32_t)hi << 16);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) reinterpret_cast<uint32_t*>(row + g * 128)[i + 8 * j] = w[j];
    if (i == 0) reinterpret_cast<float*>(row + kDV)[g] = scale;
    reinterpret_cast<uint32_t*>(row + kDV + 16)[lane] = rp;
}

// ------------------------------------------------------------------ self-test of the bounded waits
// Four warps wait on an initialised barrier that nothing ever arrives at: one by time, with a short budget, three in the short forms (with a
// complete phase beside the one that is not).  The first must give up and raise the CTA's abort flag, which must end the others; the kernel records
// DSA_V32_ERR_DEVICE_WAIT in the status word - the path every wait of the attention kernels takes when its peer never answers - and must exit
// normally.  result[0] = 1 when all waits returned false, result[1] = the abort flag they left.
__global__ void __launch_bounds__(128) wait_expiry_selftest_kernel(int32_t* status, int32_t* result, unsigned long long budget_ns) {
    __shared__ uint64_t bar;
    __shared__ int abort_flag, gave_up;
    const uint32_t b = smem_u32(&bar);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    if (threadIdx.x == 0) {
        mbar_init(b, 1);
        abort_flag = gave_up = 0;
        fence_mbar_init();
    }
    __syncthreads();
    // phase 0 is not complete, the one before it (parity 1) is
    const bool ok = warp == 0   ? __all_sync(0xffffffffu, mbar_wait_budget(b, 0, &abort_flag, budget_ns))
                    : warp == 1 ? warp_wait_short(b, 0, &abort_flag)
                    : warp == 2 ? warp_wait_short2(b, 1, b, 0, &abort_flag)
                                : warp_wait_short3(b, 1, b, 0, b, 1, &abort_flag);
    if (!ok && (threadIdx.x & 31) == 0) atomicAdd(&gave_up, 1);
    __syncthreads();
    if (abort_flag) settle_in_flight();
    if (threadIdx.x == 0) {
        if (abort_flag) atomicExch(status, DSA_V32_ERR_DEVICE_WAIT);
        result[0] = gave_up == 4 ? 1 : 0;
        result[1] = abort_flag;
    }
}

// ------------------------------------------------------------------ launch helpers (called from capi.cu)
cudaError_t launch_combine(const float* o_accum, const float* lse_accum, const int32_t* reduce_indptr,
                           const int32_t* reduce_slots, const ReduceDst* reduce_dst, int num_reduce_rows, const OutTargets& tgt,
                           int64_t stride_o_row, int64_t stride_o_head, int H, int tile_rows, cudaStream_t stream) {
    if (num_reduce_rows <= 0) return cudaSuccess;
    int sms = 0;
    cudaError_t e = sm_count(&sms);
    if (e != cudaSuccess) return e;
    const int64_t rows = (int64_t)num_reduce_rows * tile_rows;
    const bool wide = rows > int64_t(sms) * kMergeBlocks, deep = rows <= int64_t(sms) * kMergeBlocksDeep;
    dim3 grid(num_reduce_rows, wide ? (tile_rows + 3) / 4 : tile_rows);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = grid;
    cfg.blockDim = dim3(128, 1, 1);
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, wide ? combine_kernel<4, 8> : deep ? combine_kernel<1, 16> : combine_kernel<1, 8>, o_accum, lse_accum, reduce_indptr, reduce_slots, reduce_dst, tgt, stride_o_row,
                              stride_o_head, H);
}

// Pushes a contiguous block of this GPU's gathered buffer to the same place in every peer's (plain 16-byte
// stores through the peer mappings, all SMs): the sequence-sharded form of the fused all-gather.
struct PeerPush {
    int32_t n_peers, my_rank;
    const uint4* src;
    uint4* dst[DSA_V32_MAX_PEERS];
    int64_t n16;   // 16-byte words
};
__global__ void __launch_bounds__(512) peer_push_kernel(const PeerPush s) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < s.n16; i += (int64_t)gridDim.x * blockDim.x) {
        const uint4 v = s.src[i];
        for (int r = 0; r < s.n_peers; ++r)
            if (r != s.my_rank) s.dst[r][i] = v;
    }
}
cudaError_t launch_peer_push(int n_peers, int my_rank, const void* src, void* const* dst, int64_t bytes, cudaStream_t stream) {
    if (bytes <= 0 || n_peers <= 1) return cudaSuccess;
    PeerPush s;
    s.n_peers = n_peers;
    s.my_rank = my_rank;
    s.src = reinterpret_cast<const uint4*>(src);
    for (int r = 0; r < DSA_V32_MAX_PEERS; ++r) s.dst[r] = r < n_peers ? reinterpret_cast<uint4*>(dst[r]) : nullptr;
    s.n16 = bytes / 16;
    peer_push_kernel<<<148 * 2, 512, 0, stream>>>(s);
    return cudaGetLastError();
}

cudaError_t launch_peer_sync(const PeerSync& s, cudaStream_t stream) {
    peer_signal_wait_kernel<<<1, 32, 0, stream>>>(s);
    return cudaGetLastError();
}

cudaError_t launch_wait_selftest(int32_t* status, int32_t* result, unsigned long long budget_ns, cudaStream_t stream) {
    wait_expiry_selftest_kernel<<<1, 128, 0, stream>>>(status, result, budget_ns);
    return cudaGetLastError();
}

cudaError_t launch_debug_rows(const AttnParams& p, int total_q, int32_t* rows_out, cudaStream_t stream) {
    debug_rows_kernel<<<256, 256, 0, stream>>>(p, total_q, rows_out);
    return cudaGetLastError();
}

cudaError_t launch_pack_fp8(const float* latent, const void* rope, const int64_t* dst_rows, void* out, int64_t num_rows,
                            cudaStream_t stream) {
    if (num_rows <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((num_rows + 7) / 8);
    pack_fp8_rows_kernel<<<blocks, 256, 0, stream>>>(latent, reinterpret_cast<const __nv_bfloat16*>(rope), dst_rows,
                                                     reinterpret_cast<uint8_t*>(out), num_rows);
    return cudaGetLastError();
}

}  // namespace dsa
