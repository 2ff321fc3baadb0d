// Top-k selection of the sparse-attention index lists: for every query row, the positions of the k largest
// indexer scores among the row's valid positions, as the int32 list the attention kernels consume (-1 padding).
// This is the output stage of the DSA indexer that produces `indices` upstream of the attention; the
// reference lab has no counterpart (its harness draws the lists at random, common/host.cc:239-261).
//
// One cluster of C CTAs per query row (C = 1 when there are rows enough to fill the chip), every CTA a contiguous
// slice of the row's positions.  Exact radix select on order-preserving 32-bit keys, 12 + 10 + 10 bits from the top:
// a CTA reads its slice once and keeps the keys in registers; the first pass counts all of them in a shared-memory
// histogram, the keys of the bin that holds the k-th largest one are compacted into a short list, and the two other
// passes look at that list only.  One warp finds a bin from the histograms of all CTAs of the cluster (64 coarse sums,
// then the bins of the coarse one; remote ones through distributed shared memory).  Then the positions above the
// threshold and the lowest ones equal to it are written in ascending order by one prefix sum over (round, warp)
// counts - the list is deterministic.
//
// What bounds it: instruction issue while there are many rows (every key is touched four times: made, counted, tested
// for the list, written), and the chain of block- and cluster-wide steps when there are few.  Measured against one CTA of
// 512 threads per row that reads the row in each of five passes and scans every 512 positions: 64 rows of 32768 84.0 ->
// 14.4 us, 2048 rows of up to 8192 247.6 -> 51.6 us (0.6 and 1.5 TB/s of scores and lists).
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>
#include "defs.h"

namespace dsa {

constexpr int kSelBits0 = 12;                       // first pass; the two others take ten bits each
constexpr int kSelBins = 1 << kSelBits0;

constexpr int kSelList = 2048;                      // keys kept for the two later passes; more are read again instead

// float -> key with the same order as the values, at least 1: NaN (canonical after the addition) sorts lowest of all, so it
// is never preferred, -0.0 ties with +0.0, and 0 is left for "no position"
__device__ __forceinline__ uint32_t order_key(float x) {
    const uint32_t b = __float_as_uint(x + 0.0f);
    const uint32_t k = b ^ (static_cast<uint32_t>(static_cast<int32_t>(b) >> 31) | 0x80000000u);
    return x != x ? 1u : k;
}

struct alignas(16) SelShared {
    int hist[kSelBins];     // first pass
    int hist2[2][1024];     // the two others
    int coarse[3][64];
    uint32_t list[kSelList];
    int counts[1024];       // (round, warp): positions taken for sure | positions equal to the threshold, prefix sums later
    int list_n;
    int total[2];           // this CTA's sums of the two
    int found[3];           // bin, how many more to take in it, how many it holds
};
static_assert(alignof(SelShared) == 16 && offsetof(SelShared, hist) % 16 == 0 && offsetof(SelShared, hist2) % 16 == 0, "cleared 16 bytes at a time");

__device__ __forceinline__ void count_in(int* bin) {
    asm volatile("red.shared::cta.add.u32 [%0], 1;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(bin))) : "memory");
}
__device__ __forceinline__ const SelShared* sel_peer(const SelShared* s, uint32_t rank) {
    uint64_t out;
    asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<uint64_t>(s)), "r"(rank));
    return reinterpret_cast<const SelShared*>(out);
}
template <bool kShared> __device__ __forceinline__ void sel_sync() {
    if (kShared) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// One warp: v0, v1 = the counts of bins 2 lane and 2 lane + 1.  The highest bin with (sum of the bins above it) < need
// <= (that sum + the bin itself), what is left of `need` inside it, and how many keys it holds.
__device__ __forceinline__ void sel_find_bin(int v0, int v1, int need, int& bin, int& left, int& holds) {
    const int lane = threadIdx.x & 31;
    int incl = v0 + v1;                              // suffix sum over lanes
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_down_sync(0xffffffffu, incl, off);
        if (lane + off < 32) incl += o;
    }
    const int above = incl - v0 - v1;                // keys in the bins of higher lanes
    const uint32_t who = __ballot_sync(0xffffffffu, above < need && incl >= need);
    const int src = who ? __ffs(who) - 1 : 0;        // always one lane: 1 <= need <= all keys
    const bool hi = above + v1 >= need;
    bin = __shfl_sync(0xffffffffu, 2 * lane + (hi ? 1 : 0), src);
    left = __shfl_sync(0xffffffffu, need - above - (hi ? 0 : v1), src);
    holds = __shfl_sync(0xffffffffu, hi ? v1 : v0, src);
}

// The k largest of the first n positions of a row (0 < k < n), by one CTA or (kShared) by all n_cta of a cluster, a slice each.
// kThreads x kPer positions per CTA are kept in registers; kReload: slices of any length, read again in every pass.
template <int kThreads, int kPer, bool kShared, bool kReload>
__device__ __forceinline__ void select_row(SelShared& sh, const float* __restrict__ row, int32_t* __restrict__ out, int n, int k, int rank, int n_cta, int vec_ok) {
    static_assert(kShared || !kReload, "a row longer than the registers of one CTA is cut over a cluster first");
    static_assert(kPer % 4 == 0 && kThreads * kPer / 128 <= 1024, "counts table");
    constexpr int kChunk = kThreads * kPer;          // positions per round of the register file
    constexpr int kWarps = kThreads / 32;
    constexpr int kRounds = kPer / 4;                // four consecutive positions per thread and round
    constexpr int kRound = 4 * kThreads;             // positions of a round
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per_cta = ((n + n_cta - 1) / n_cta + 3) & ~3;
    const int begin = min(rank * per_cta, n), end = min(begin + per_cta, n);
    const int n_chunks = kReload ? (per_cta + kChunk - 1) / kChunk : 1;
    // Rounds that hold a position: the work follows the row's own length, not the width that the form is made for.
    constexpr bool kGuard = !kReload;
    const int live = kGuard ? min(kRounds, (max(0, end - begin) + kRound - 1) / kRound) : kRounds;

    uint32_t key[kPer];
    auto load_chunk = [&](int c) {
        const int base = begin + c * kChunk + 4 * tid;
        if (vec_ok && base + (kRounds - 1) * kRound + 4 <= end) {   // all of the thread's positions are there
#pragma unroll
            for (int r = 0; r < kRounds; ++r) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(row + base + r * kRound));
                key[4 * r + 0] = order_key(v.x);
                key[4 * r + 1] = order_key(v.y);
                key[4 * r + 2] = order_key(v.z);
                key[4 * r + 3] = order_key(v.w);
            }
        } else {
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int p = base + (j >> 2) * kRound + (j & 3);
                key[j] = p < end ? order_key(__ldg(row + p)) : 0u;
            }
        }
    };
    if (!kReload) load_chunk(0);
    for (int i = 4 * tid; i < kSelBins; i += kRound) *reinterpret_cast<int4*>(sh.hist + i) = make_int4(0, 0, 0, 0);
    for (int i = 4 * tid; i < 2048; i += kRound) *reinterpret_cast<int4*>(&sh.hist2[0][0] + i) = make_int4(0, 0, 0, 0);
    if (tid == 0) sh.list_n = 0;
    __syncthreads();

    // ---- the k-th largest key: bits [20, 32), [10, 20), [0, 10)
    uint32_t prefix = 0;
    int need = k;           // how many more to take among the keys that match the prefix
    bool tie = false;       // more keys equal the threshold than are needed
#pragma unroll
    for (int pass = 0; pass < 3; ++pass) {
        constexpr int kShift[3] = {20, 10, 0};
        const int shift = kShift[pass];
        const int per_coarse = pass == 0 ? 64 : 16;            // 64 coarse bins in every pass
        int* hist = pass == 0 ? sh.hist : sh.hist2[pass - 1];
        const uint32_t want = pass == 0 ? 0u : prefix >> (shift + 10);
        if (pass == 0) {
            for (int c = 0; c < n_chunks; ++c) {
                if (kReload) load_chunk(c);
#pragma unroll
                for (int r = 0; r < kRounds; ++r)
                    if (r < live)
#pragma unroll
                        for (int j = 4 * r; j < 4 * r + 4; ++j) count_in(&hist[key[j] >> 20]);
            }
        } else if (sh.list_n <= kSelList) {
            for (int i = tid; i < sh.list_n; i += kThreads) {
                const uint32_t x = sh.list[i];
                if ((x >> (shift + 10)) == want) count_in(&hist[(x >> shift) & 1023u]);
            }
        } else {            // too many keys share the first twelve bits: all of the slice again
#pragma unroll 1
            for (int c = 0; c < n_chunks; ++c) {
                if (kReload) load_chunk(c);
#pragma unroll
                for (int j = 0; j < kPer; ++j)
                    if (key[j] != 0u && (key[j] >> (shift + 10)) == want) count_in(&hist[(key[j] >> shift) & 1023u]);
            }
        }
        __syncthreads();
        if (pass == 0 && tid == 0) hist[0] -= (kGuard ? live * kRound : n_chunks * kChunk) - (end - begin);   // "no position" keys do not count
        if (pass == 0) __syncthreads();
        for (int b = warp; b < 64; b += kWarps) {
            int s = 0;
            for (int i = lane; i < per_coarse; i += 32) s += hist[b * per_coarse + i];
            s = __reduce_add_sync(0xffffffffu, s);
            if (lane == 0) sh.coarse[pass][b] = s;
        }
        sel_sync<kShared>();
        if (warp == 0) {
            int v0 = 0, v1 = 0, cb, fb, left, holds;
            for (int r = 0; r < n_cta; ++r) {
                const SelShared* p = kShared ? sel_peer(&sh, r) : &sh;
                v0 += p->coarse[pass][2 * lane];
                v1 += p->coarse[pass][2 * lane + 1];
            }
            sel_find_bin(v0, v1, need, cb, left, holds);
            v0 = v1 = 0;
            if (2 * lane < per_coarse)
                for (int r = 0; r < n_cta; ++r) {
                    const SelShared* p = kShared ? sel_peer(&sh, r) : &sh;
                    const int* h = (pass == 0 ? p->hist : p->hist2[pass == 0 ? 0 : pass - 1]) + cb * per_coarse;
                    v0 += h[2 * lane];
                    v1 += h[2 * lane + 1];
                }
            sel_find_bin(v0, v1, left, fb, left, holds);
            if (lane == 0) {
                sh.found[0] = cb * per_coarse + fb;
                sh.found[1] = left;
                sh.found[2] = holds;
            }
        }
        __syncthreads();
        prefix |= (uint32_t)sh.found[0] << shift;
        need = sh.found[1];
        tie = sh.found[2] > need;
        if (pass == 0) {    // the keys of the bin, for the two later passes
#pragma unroll 1
            for (int c = 0; c < n_chunks; ++c) {
                if (kReload) load_chunk(c);
#pragma unroll
                for (int r = 0; r < kRounds; ++r)
                    if (r < live)
#pragma unroll
                        for (int j = 4 * r; j < 4 * r + 4; ++j)
                            if ((key[j] ^ prefix) < (1u << 20) && key[j] != 0u) {
                                const int at = atomicAdd(&sh.list_n, 1);
                                if (at < kSelList) sh.list[at] = key[j];
                            }
            }
            __syncthreads();
        }
    }

    // ---- counts per (round, warp), in position order, and their prefix sums.  Without ties every key at or above the
    // threshold is taken; with them the keys equal to it are counted apart and the first `need` of the row are taken.
    const uint32_t floor_key = tie ? prefix + 1u : prefix;
    int gt_base = 0, eq_base = 0;       // positions of the row before this CTA's slice (and before the chunk)
    auto add_slices_before = [&]() {    // a CTA's first output slot depends on the CTAs before it
        sel_sync<kShared>();
        for (int r = 0; r < rank; ++r) {
            const SelShared* p = sel_peer(&sh, r);
            gt_base += p->total[0];
            eq_base += p->total[1];
        }
    };
    if (kReload) {                      // the slices' sums take a reading of their own
        int g = 0, e = 0;
        for (int c = 0; c < n_chunks; ++c) {
            load_chunk(c);
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                g += key[j] >= floor_key;
                e += tie && key[j] == prefix;
            }
        }
        if (tid < 2) sh.total[tid] = 0;
        __syncthreads();
        g = __reduce_add_sync(0xffffffffu, g);
        e = __reduce_add_sync(0xffffffffu, e);
        if (lane == 0) {
            atomicAdd(&sh.total[0], g);
            atomicAdd(&sh.total[1], e);
        }
        add_slices_before();
    }
    for (int c = 0; c < n_chunks; ++c) {
        if (kReload) load_chunk(c);
        // four rounds to a word of four byte-wide fields (a warp has at most 128 of a round's positions)
        uint32_t before_g[(kRounds + 3) / 4], before_e[(kRounds + 3) / 4];   // of the lanes before this one
#pragma unroll
        for (int w = 0; w < (kRounds + 3) / 4; ++w) {
            if (4 * w >= live) break;
            uint32_t g = 0, e = 0;
#pragma unroll
            for (int j = 0; j < 16 && 16 * w + j < kPer; ++j) {
                g += key[16 * w + j] >= floor_key ? 1u << (8 * (j >> 2)) : 0u;
                if (tie) e += key[16 * w + j] == prefix ? 1u << (8 * (j >> 2)) : 0u;
            }
            uint32_t gi = g, ei = e;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, gi, off);
                if (lane >= off) gi += o;
            }
            if (tie)
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const uint32_t o = __shfl_up_sync(0xffffffffu, ei, off);
                    if (lane >= off) ei += o;
                }
            before_g[w] = gi - g;
            before_e[w] = ei - e;
            if (lane == 31)
#pragma unroll
                for (int r = 0; r < 4 && 4 * w + r < kRounds; ++r)
                    sh.counts[(4 * w + r) * kWarps + warp] = ((gi >> (8 * r)) & 255u) | (((ei >> (8 * r)) & 255u) << 16);
        }
        __syncthreads();
        if (warp == 0) {                // exclusive prefix sums over the (round, warp) counts
            constexpr int kN = kRounds * kWarps, kEach = (kN + 31) / 32;
            int v[kEach], g = 0, e = 0;
#pragma unroll
            for (int i = 0; i < kEach; ++i) {
                v[i] = lane * kEach + i < live * kWarps ? sh.counts[lane * kEach + i] : 0;
                g += v[i] & 0xFFFF;
                e += v[i] >> 16;
            }
            int gi = g, ei = e;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int a = __shfl_up_sync(0xffffffffu, gi, off), b = __shfl_up_sync(0xffffffffu, ei, off);
                if (lane >= off) {
                    gi += a;
                    ei += b;
                }
            }
            // the two sums of a chunk fit 16 bits each: at most kChunk <= 32768 positions
            int run = (gi - g) | ((ei - e) << 16);
#pragma unroll
            for (int i = 0; i < kEach; ++i) {
                if (lane * kEach + i < kN) sh.counts[lane * kEach + i] = run;
                run += v[i];
            }
            if (lane == 31) {
                int* sums = kReload ? sh.found : sh.total;
                sums[0] = gi;
                sums[1] = ei;
            }
        }
        if (kShared && !kReload) add_slices_before();
        else __syncthreads();
        const int base = begin + c * kChunk + 4 * tid;
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            if (r >= live) break;
            const uint32_t before = (uint32_t)sh.counts[r * kWarps + warp];
            int g = gt_base + (int)(before & 0xFFFFu) + (int)((before_g[r >> 2] >> (8 * (r & 3))) & 255u);
            if (!tie) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (key[4 * r + j] >= floor_key) out[g++] = base + r * kRound + j;
            } else {
                int e = eq_base + (int)(before >> 16) + (int)((before_e[r >> 2] >> (8 * (r & 3))) & 255u);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool eq = key[4 * r + j] == prefix, gt = key[4 * r + j] > prefix;
                    if (gt || (eq && e < need)) out[g + min(e, need)] = base + r * kRound + j;
                    g += gt;
                    e += eq;
                }
            }
        }
        if (kReload) {
            gt_base += sh.found[0];
            eq_base += sh.found[1];
            __syncthreads();
        }
    }
    if (kShared) sel_sync<kShared>();   // no CTA leaves while another may still read its tables
}

// Not inlined: the registers of the cluster's own path are not shared with it.
template <int kThreads, int kPer>
__device__ __noinline__ void select_row_alone(SelShared* sh, const float* row, int32_t* out, int n, int k, int vec_ok) {
    select_row<kThreads, kPer, false, false>(*sh, row, out, n, k, 0, 1, vec_ok);
}

// One CTA or one cluster per row.  The lengths are on the device and the form is chosen by the buffer's width, so a row that fits the
// registers of one CTA is left to the first of its cluster, and one whose valid positions are all selected needs no selection.
// Rows of 2100-3000 in a buffer of 131072: 160 rows 23 us (74 when the whole cluster worked on the width; one CTA of 512 threads that
// scanned the row five times 31), 300 rows 40 (146; 33).  Small CTAs for the short rows in a launch before, and then clusters that
// stay and deal the long ones out among themselves, took 12.5 us for the 300, but 5 to 12 % more for full rows and up to 65 % for mixed
// ones, whose order they fix beforehand.
template <int kThreads, int kPer, bool kCluster, bool kReload>
__global__ void __launch_bounds__(kThreads, kThreads == 512 ? (kCluster ? 2 : 3) : 1) topk_select_kernel(const float* __restrict__ scores, int64_t stride_row,
                                                                const int32_t* __restrict__ valid_len, int kv_len, int topk,
                                                                int n_cta, int vec_ok, int32_t* __restrict__ indices_out) {
    __shared__ SelShared sh;
    const int rank = kCluster ? (int)(blockIdx.x % n_cta) : 0;
    const int q = kCluster ? (int)(blockIdx.x / n_cta) : (int)blockIdx.x;
    const float* row = scores + (size_t)q * stride_row;
    int32_t* out = indices_out + (size_t)q * topk;
    int n = valid_len ? valid_len[q] : kv_len;
    n = n < 0 ? 0 : (n > kv_len ? kv_len : n);
    if (n <= topk) {   // everything valid is selected
        for (int i = rank * kThreads + threadIdx.x; i < topk; i += n_cta * kThreads) out[i] = i < n ? i : -1;
        return;
    }
    if (!kCluster || n <= kThreads * kPer) {
        if (rank == 0) {
            if constexpr (kCluster) select_row_alone<kThreads, kPer>(&sh, row, out, n, topk, vec_ok);
            else select_row<kThreads, kPer, false, false>(sh, row, out, n, topk, 0, 1, vec_ok);
        }
        return;
    }
    if constexpr (kCluster) select_row<kThreads, kPer, true, kReload>(sh, row, out, n, topk, rank, n_cta, vec_ok);
}

template <int kThreads, int kPer, bool kCluster, bool kReload>
static cudaError_t launch_sel(const float* scores, int64_t stride_row, const int32_t* valid_len, int total_q, int kv_len, int topk,
                              int n_cta, int vec_ok, int32_t* indices_out, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3((unsigned)total_q * n_cta, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.stream = stream;
    if (kCluster) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = n_cta;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, topk_select_kernel<kThreads, kPer, kCluster, kReload>, scores, stride_row, valid_len, kv_len, topk, n_cta, vec_ok, indices_out);
}

cudaError_t launch_topk_select(const float* scores, int64_t stride_row, const int32_t* valid_len, int total_q, int kv_len, int topk,
                               int32_t* indices_out, cudaStream_t stream) {
    if (total_q <= 0) return cudaSuccess;
    const int vec_ok = (stride_row % 4 == 0 && (reinterpret_cast<uintptr_t>(scores) & 15u) == 0) ? 1 : 0;
    int sms = 0;
    cudaError_t e = sm_count(&sms);
    if (e != cudaSuccess) return e;
    // CTAs per row: up to two waves' worth of an SM each (64 rows of 32768 positions: four CTAs of 512 threads 14.8 us, one of
    // 1024 threads 15.0, eight 27, the exchange of a cluster growing with its size), and enough that a slice fits the
    // registers.
    int n_cta = 1;
    while (n_cta < 8 && (((int64_t)total_q * n_cta * 2 <= 2 * sms && kv_len / (2 * n_cta) >= 4096) || kv_len > n_cta * 32768)) n_cta *= 2;
    const int per_cta = ((kv_len + n_cta - 1) / n_cta + 3) & ~3;
    // Slices of up to 8192 positions: 16 keys per thread, three CTAs on an SM (2048 rows of 8192: 49.6 us; 32 keys in 256
    // threads 51.6, 8 in 1024 threads 61.7).
    auto launch = [&](auto form) { return form(scores, stride_row, valid_len, total_q, kv_len, topk, n_cta, vec_ok, indices_out, stream); };
    if (per_cta <= 8192) return launch(n_cta > 1 ? launch_sel<512, 16, true, false> : launch_sel<512, 16, false, false>);
    if (per_cta <= 32768) return launch(n_cta > 1 ? launch_sel<1024, 32, true, false> : launch_sel<1024, 32, false, false>);
    return launch(launch_sel<1024, 32, true, true>);   // only a cluster of eight gets here
}

}  // namespace dsa
