// Sparse MLA attention for few heads: work items of at most 32 tile rows (fp8 cache: 16; 16 or 32 heads of a head-sharded
// deployment, or the stacked rows of an MTP pair) that hold enough slots on average (few_heads_form in plan.h).
//
// The 128-row kernels put the heads on the 128 rows of the tensor-core tile, so an item of 16 heads pays
// for 128: a tile of 32 slots takes the same 1 800-2 600 cycles whatever H is, while the rows it gathers would take
// 900 cycles of the SM pair's share of HBM.  Here the product is turned round:
//       S^T [slots x heads]          = K [slots x 576] Q^T         (A = the gathered tile, B = Q in shared memory)
//       O^T [512 columns x heads]   += V^T [512 x slots] P^T       (A = the same tile seen MN-major, B = P in shared memory)
// The wide dimension of both products is now the gathered data, the output takes 4 x 16 (32) TMEM columns instead of
// 512, and one CTA holds all 576 columns of an item: no partial scores cross the SM-to-SM link.
//
// The two CTAs of a pair share a work list and split every item by slots: each attends to half of the piece's
// slots; at the end each sends the other the fp32 sums of 256 output columns, the row maxima and the row sums through
// distributed shared memory, and merges and writes its own 256 columns.
//
// Warp roles (20 warps):
//   warps 0-3   softmax: thread = slot (the M = 64 accumulator puts its rows on lanes 0-15 of every TMEM lane
//              quadrant), holding the scores of its slot, 16 heads at a time.  A head's reference maximum is only moved
//              when a score exceeds it by more than the lazy margin of 8 - one vote of the four warps per tile (taking the
//              exponentials while it is under way gained nothing); the row sums stay per slot in fp32 registers and cross
//              the lanes once per item.  P goes to shared memory (fp8 cache: one copy per 128-column scale group, pre-multiplied by that
//              group's row scale).  Epilogue: merge, normalise, store.
//   warp 4      score issuer; it also fetches the item's Q (TMA).     warp 5  P V issuer.     warps 6, 7 idle.
//   warps 8-19  row loaders, four rows of every tile each.  bf16 cache: 16-byte cp.async copies straight into the
//              swizzled tile; fp8 cache: a row's bytes are loaded into registers one tile ahead (asked into L2 three tiles
//              ahead), converted e4m3 -> bf16 exactly and stored.  No staging of raw rows: the room it would take is the
//              third tile stage.
//
// What bounds it (cycle stamps of an instrumented copy, fp8, 16 heads): a tile holds its stage for 8 500 cycles (load and convert 900, the other warps'
// rows 700, scores 2 000, softmax 2 100, P V 750 and the hand-offs between them), three stages: 2 850-3 300 cycles per
// 48 slots; its MMAs take 2 000 of them to issue (36 for the scores of M = 64, N = 16 at 33 cycles, 12 for P V at 62), though
// the counter has the tensor pipe active for 8 %.
// Measured against paired_fp8.cu: 74 rows of 16 heads x 2048 slots 57.8 -> 50.9 us, 200 x 1024 90.3 -> 73.1 (52 and 75 since its loaders look for NaN codes).  (For 17 to 32 rows of an fp8 cache it
// had a form, too: 71 us for 74 x 2048 where paired_fp8.cu takes 60.)  Against paired_heads.cu: bf16, 296 rows of 16 heads x 1024 slots 86.6 -> 78.9,
// eight sequences of 16 heads x 2048 in pieces 15.1 -> 14.2 with the merge; more shapes beside the rule (few_heads_form in plan.h).
// out against 64 bits: 2.08e-3 (1.68e-3 in paired_fp8.cu), lse at most 1.4e-6 (1.7e-6).
//
// Every mbarrier wait is bounded, as in the 128-row kernels, and the warps of the softmax group meet on mbarriers only, so a
// warp that gave up never leaves the others in a hardware barrier.
#include <cuda_bf16.h>
#include <cfloat>
#include <cstddef>
#include <mutex>
#include "defs.h"
#include "ptx.cuh"
#include "rows.cuh"

namespace dsa {
namespace small {

constexpr int kSlots = 48;                         // slots per tile: rows 0-47 of the M = 64 score MMA (its last 16 rows read the bytes
                                                   // after a block, and nothing reads their scores)
constexpr int kStages = 3;
constexpr int kBlocks = kDQK / 64;                 // nine 64-column blocks of a row
constexpr int kKvBlock = kSlots * 128;             // 6144 bytes: one 64-column block of a tile
constexpr int kTileBytes = kBlocks * kKvBlock;     // 55 296
constexpr int kXBytes = 2 * 128 * 16 * 4;          // 16 384: the peer's sums of this CTA's 256 columns, 16 heads at a time (overlays the P copies)
constexpr int kLoadWarp0 = 8;
constexpr int kLoadWarps = kSlots / 4;             // 12: four rows of every tile each, eight lanes per row
constexpr int kWarps = kLoadWarp0 + kLoadWarps;    // 20: five warpgroups
// Registers per thread after the role split (setmaxnreg): softmax warpgroup + issuers' + three of loaders <= 480, five times the
// launch's 96.  fp8: the loaders hold the next row and the one being converted (64 sequences 53 -> 51 us against loading
// it after the conversion); bf16: the rows never pass through registers.
template <bool kFp8> constexpr int kRegsLoaders = kFp8 ? 104 : 72;
template <bool kFp8> constexpr int kRegsSoftmax = kFp8 ? 112 : 152;
constexpr int kRegsIssuers = 56;
constexpr int kCtlBytes = 5120;

// kN: tile rows (heads) an item may have = N of both MMAs, 16 or 32
template <int kN>
struct Cfg {
    static constexpr int kHalves = kN / 16;            // a softmax thread works on 16 heads at a time
    static constexpr int kQBlock = kN * 128;
    static constexpr int kQBytes = kBlocks * kQBlock;
    static constexpr int kPCopy = kSlots * kN * 2;     // one copy of P: a row of kN bf16 per slot
    static constexpr int kOffQ = kStages * kTileBytes;
    static constexpr int kOffP = kOffQ + kQBytes;
    static constexpr int kOffCtl = kOffP + kXBytes;
    static constexpr int kSmemBytes = kOffCtl + kCtlBytes + 1024;   // + slack for 1024-byte alignment
    // TMEM columns: O^T four 128-column groups x kN heads | S^T two buffers of 5 (fp8: four scale groups and the rope) x kN
    static constexpr uint32_t kColS = 4 * kN, kSBuf = 5 * kN, kTmemCols = kN == 16 ? 256 : 512;
    static_assert(kN == 16 || kN == 32, "rows of 32 or 64 bytes");
    static_assert(4 * kPCopy <= kXBytes, "the P copies fit under the exchange buffer");
    static_assert(kSmemBytes <= 232448, "227 KB per CTA");
    static_assert(kColS + 2 * kSBuf <= kTmemCols, "TMEM");
};

struct Ctl {
    float4 row_scale[kStages][kSlots];   // fp8 cache: a slot's four scales
    float wmax[4][32];                   // per softmax warp: column maxima of a tile whose references move
    float ref[2][32];                    // reference maxima: the current ones and the ones before the last move
    float lsum[2][4][32];                // per softmax warp: row sums of an item, by item parity
    float peer_m[16], peer_l[16];        // the peer CTA's reference maxima and row sums of the heads being merged
    uint32_t vote[2][4];                 // read as one 16-byte word
    uint64_t kv_full[kStages], kv_empty[kStages];
    uint64_t s_full[2], s_empty[2];
    uint64_t p_full, pv_done, q_full, q_empty, o_full, o_free, team, x_ready, x_full;
    uint8_t ok[kStages][64];             // the slot holds a row (not padding)
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(Ctl) <= kCtlBytes && offsetof(Ctl, vote) % 16 == 0 && offsetof(Ctl, wmax) % 16 == 0 && offsetof(Ctl, ref) % 16 == 0, "control block");

// What this CTA does of a work item: its half of the slots, all tile rows.
struct Part {
    int k_begin, k_end, n_tiles, n_rows;
};
__device__ __forceinline__ Part part_of(const dsa_v32_work_info& w, int half, int H) {
    Part a;
    const int mid = w.k_begin + (w.k_end - w.k_begin + 1) / 2;
    a.k_begin = half ? mid : w.k_begin;
    a.k_end = half ? w.k_end : mid;
    a.n_rows = w.stacked_rows > 1 ? w.stacked_rows * H : H;
    // a CTA without slots still runs one tile, all masked: its sums are then zeros and not stale accumulators
    a.n_tiles = max(1, (a.k_end - a.k_begin + kSlots - 1) / kSlots);
    return a;
}

__device__ __forceinline__ bool wait_on(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    const uint32_t b = smem_u32(bar);
    if (__all_sync(0xffffffffu, mbar_test_wait(b, parity))) return true;
    return warp_wait(b, parity, abort_flag);
}
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(bar));
}

// Position in a ring of kStages tiles: stage and the parity of its current use.
struct Ring {
    uint32_t s = 0, ph = 0;
    __device__ __forceinline__ void next() {
        if (++s == kStages) {
            s = 0;
            ph ^= 1u;
        }
    }
};

// 16 values per lane -> lane i (and i + 16) holds the reduction of value i over its half warp of 16 lanes
template <bool kMax>
__device__ __forceinline__ float reduce16(float (&v)[16], int lane) {
#pragma unroll
    for (int off = 8; off >= 1; off >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int j = 0; j < off; ++j) {
            const float keep = up ? v[j + off] : v[j], send = up ? v[j] : v[j + off];
            const float got = __shfl_xor_sync(0xffffffffu, send, off);
            v[j] = kMax ? fmaxf(keep, got) : keep + got;
        }
    }
    return v[0];
}

template <bool kFp8, int kN>
__global__ void __launch_bounds__(32 * kWarps, 1)
small_heads_kernel(const __grid_constant__ CUtensorMap tm_q, const AttnParams p) {
    using C = Cfg<kN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // the same offset in both CTAs of a pair
    uint8_t* sKV = smem;
    uint8_t* sQ = smem + C::kOffQ;
    uint8_t* sP = smem + C::kOffP;
    Ctl* ctl = reinterpret_cast<Ctl*>(smem + C::kOffCtl);
    volatile int* abort_flag = &ctl->abort_flag;
    // fp8: the warp's number by a shuffle, so known to be the same in all lanes: fewer instructions (200 rows of 16 heads x 1024 slots 74.7 -> 72.0 us;
    // bf16, two rows x 2048: 12.26 -> 12.37)
    const int tid = threadIdx.x, warp = kFp8 ? __shfl_sync(0xffffffffu, tid >> 5, 0) : tid >> 5, lane = tid & 31;
    const int list = blockIdx.x >> 1;
    const int half = (int)cluster_ctarank(), peer = half ^ 1;
    const int w_begin = __ldg(p.list_indptr + list), w_end = __ldg(p.list_indptr + list + 1);
    constexpr int kCopies = kFp8 ? 4 : 1;

    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) {
            // fp8: the loading warps; bf16: each of their lanes (its copies) and one plain arrival per warp (the slots' flags)
            mbar_init(smem_u32(&ctl->kv_full[i]), kFp8 ? kLoadWarps : kLoadWarps * 33);
            mbar_init(smem_u32(&ctl->kv_empty[i]), 1);
        }
        mbar_init(smem_u32(&ctl->p_full), 4);
        mbar_init(smem_u32(&ctl->pv_done), 1);
        fence_mbar_init();
    } else if (tid == 32) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&ctl->s_full[i]), 1);
            mbar_init(smem_u32(&ctl->s_empty[i]), 4);
        }
        mbar_init(smem_u32(&ctl->q_full), 1);
        mbar_init(smem_u32(&ctl->q_empty), 1);
        fence_mbar_init();
    } else if (tid == 64) {
        mbar_init(smem_u32(&ctl->o_full), 1);
        mbar_init(smem_u32(&ctl->o_free), 4);
        mbar_init(smem_u32(&ctl->team), 4);
        mbar_init(smem_u32(&ctl->x_ready), 1);
        mbar_init(smem_u32(&ctl->x_full), 1);
        ctl->abort_flag = 0;
        fence_mbar_init();
    }
    for (int i = tid * 16; i < C::kQBytes; i += 32 * kWarps * 16) *reinterpret_cast<uint4*>(sQ + i) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async_smem();   // tile rows that no head fills are read by the MMAs (their results are not)
    if (warp == 4) {
        tmem_alloc(smem_u32(&ctl->tmem_base), C::kTmemCols);
        tmem_relinquish();
        if (lane == 0) prefetch_tensormap(&tm_q);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer's barriers exist before anything is sent to it
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    grid_dependency_wait();   // everything above may overlap the tail of the kernel before this one
    const uint32_t peer_abort = map_to_cta(smem_u32(&ctl->abort_flag), peer);

    if (warp < 4) {
        // ============================================================ softmax + epilogue
        setmaxnreg_inc<kRegsSoftmax<kFp8>>();
        static_assert(kRegsSoftmax<kFp8> + kRegsIssuers + 3 * kRegsLoaders<kFp8> <= 5 * 96, "more registers than the launch has");
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(warp * 32) << 16);
        const bool live_lane = lane < 16 && warp < kSlots / 16;   // this thread has a slot
        const int slot = 16 * warp + (lane & 15);
        uint32_t team_n = 0, xn = 0, it = 0, rb = 0;   // rb: which of ctl->ref holds the current references
        Ring ring;
        const uint64_t c2 = pack2(p.scale_log2, p.scale_log2);
        // the four softmax warps meet: what they wrote to shared memory before is visible after
        auto meet = [&]() -> bool {
            warp_arrive(&ctl->team, lane);
            const bool ok = wait_on(&ctl->team, team_n & 1u, abort_flag);
            ++team_n;
            return ok;
        };
        int item_n = 0;
        for (int w = w_begin; w < w_end; ++w, ++item_n) {
            const dsa_v32_work_info wi = p.works[w];
            const Part pt = part_of(wi, half, p.H);
            const int n_halves = (kN > 16 && pt.n_rows > 16) ? 2 : 1;
            float l[kN];   // row sums of this slot's P
#pragma unroll
            for (int j = 0; j < kN; ++j) l[j] = 0.0f;
            for (int t = 0; t < pt.n_tiles; ++t, ++it, ring.next()) {
                const uint32_t sb = it & 1u;
                if (!wait_on(&ctl->kv_full[ring.s], ring.ph, abort_flag)) goto done;   // flags and scales of the tile
                const bool ok_slot = live_lane && ctl->ok[ring.s][slot] != 0;
                float4 sc = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                if (kFp8 && live_lane) sc = ctl->row_scale[ring.s][slot];
                if (!wait_on(&ctl->s_full[sb], (it >> 1) & 1u, abort_flag)) goto done;
                tc_fence_after();
                // ---- scores of this slot: v = sum_g scale_g S_g + S_rope, 16 heads at a time
                uint64_t v2[kN / 2];
                bool over = false;   // does a score exceed its head's reference by more than the margin?
#pragma unroll
                for (int hh = 0; hh < C::kHalves; ++hh) {
                    if (hh && n_halves < 2) break;
                    const uint32_t s0 = lane_base + C::kColS + sb * C::kSBuf + 16 * hh;
                    if (kFp8) {
                        const uint64_t sx = pack2(sc.x, sc.x), sy = pack2(sc.y, sc.y), sz = pack2(sc.z, sc.z), sw = pack2(sc.w, sc.w);
                        uint32_t a[16], b[16], c[16], d[16], e[16];
                        tmem_ld_n<16>(s0, a);
                        tmem_ld_n<16>(s0 + 4 * kN, e);
                        tmem_ld_n<16>(s0 + kN, b);
                        tmem_ld_n<16>(s0 + 2 * kN, c);
                        tmem_ld_n<16>(s0 + 3 * kN, d);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            uint64_t r = fma2(sx, pack2u(a[2 * j], a[2 * j + 1]), pack2u(e[2 * j], e[2 * j + 1]));
                            r = fma2(sy, pack2u(b[2 * j], b[2 * j + 1]), r);
                            r = fma2(sz, pack2u(c[2 * j], c[2 * j + 1]), r);
                            v2[8 * hh + j] = fma2(sw, pack2u(d[2 * j], d[2 * j + 1]), r);
                        }
                    } else {
                        uint32_t a[16];
                        tmem_ld_n<16>(s0, a);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 8; ++j) v2[8 * hh + j] = pack2u(a[2 * j], a[2 * j + 1]);
                    }
                    if (hh + 1 == n_halves) {
                        tc_fence_before();
                        warp_arrive(&ctl->s_empty[sb], lane);
                    }
                    if (t > 0) {
                        const float4* rf = reinterpret_cast<const float4*>(&ctl->ref[rb][16 * hh]);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float4 r4 = rf[j];
                            float y0, y1, y2, y3;
                            unpack2(mul2(v2[8 * hh + 2 * j], c2), y0, y1);
                            unpack2(mul2(v2[8 * hh + 2 * j + 1], c2), y2, y3);
                            over |= (y0 > r4.x + 8.0f) | (y1 > r4.y + 8.0f) | (y2 > r4.z + 8.0f) | (y3 > r4.w + 8.0f);
                        }
                    }
                }
                bool move = t == 0;   // the first tile sets the references
                if (t > 0) {
                    over = __any_sync(0xffffffffu, over && ok_slot);
                    if (lane == 0) ctl->vote[sb][warp] = over;
                    if (!meet()) goto done;
                    const uint4 vt = *reinterpret_cast<const uint4*>(ctl->vote[sb]);
                    move = (vt.x | vt.y | vt.z | vt.w) != 0u;
                }
                if (move) {
                    // ---- rare after the first tile: column maxima over the tile, references moved where needed
#pragma unroll
                    for (int hh = 0; hh < C::kHalves; ++hh) {
                        if (hh && n_halves < 2) break;
                        float y[16];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            unpack2(mul2(v2[8 * hh + j], c2), y[2 * j], y[2 * j + 1]);
                            if (!ok_slot) y[2 * j] = y[2 * j + 1] = -INFINITY;
                        }
                        const float cm = reduce16<true>(y, lane);
                        if (lane < 16) ctl->wmax[warp][16 * hh + lane] = cm;
                    }
                    if (!meet()) goto done;
                    if (tid < kN) {   // thread = head; the other copy of the references was last read before an earlier meeting
                        const float mx = fmaxf(fmaxf(ctl->wmax[0][tid], ctl->wmax[1][tid]), fmaxf(ctl->wmax[2][tid], ctl->wmax[3][tid]));
                        const float old = t > 0 ? ctl->ref[rb][tid] : -INFINITY;
                        ctl->ref[rb ^ 1u][tid] = mx > old + 8.0f ? mx : old;
                    }
                    if (!meet()) goto done;
                    rb ^= 1u;
                    if (t > 0) {
                        // the row sums, and O so far (complete once the previous tile's product is), go to the new references
                        if (!wait_on(&ctl->pv_done, (it - 1) & 1u, abort_flag)) goto done;
                        tc_fence_after();
#pragma unroll
                        for (int hh = 0; hh < C::kHalves; ++hh) {
                            if (hh && n_halves < 2) break;
                            float f[16];
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const float old = ctl->ref[rb ^ 1u][16 * hh + j], now = ctl->ref[rb][16 * hh + j];
                                f[j] = old == now ? 1.0f : ex2_approx(old - now);   // old = -inf: 0
                                l[16 * hh + j] *= f[j];
                            }
#pragma unroll 1
                            for (int g = 0; g < 4; ++g) {
                                const uint32_t oc = lane_base + g * kN + 16 * hh;
                                uint32_t o[16];
                                tmem_ld_n<16>(oc, o);
                                tmem_wait_ld();
#pragma unroll
                                for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f[j]);
                                tmem_st_n<16>(oc, o);
                            }
                        }
                        tmem_wait_st();
                    }
                }
                // ---- P = 2^(score - reference), at most 2^8; a masked slot gives 0
#pragma unroll
                for (int hh = 0; hh < C::kHalves; ++hh) {
                    if (hh && n_halves < 2) break;
                    const float4* rf = reinterpret_cast<const float4*>(&ctl->ref[rb][16 * hh]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 r4 = rf[j];
                        const float rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const int i = 8 * hh + 2 * j + k;
                            const float r0 = rr[2 * k] == -INFINITY ? 0.0f : rr[2 * k], r1 = rr[2 * k + 1] == -INFINITY ? 0.0f : rr[2 * k + 1];
                            float y0, y1;
                            unpack2(fma2(v2[i], c2, pack2(-r0, -r1)), y0, y1);
                            const float p0 = ok_slot ? ex2_approx(y0) : 0.0f, p1 = ok_slot ? ex2_approx(y1) : 0.0f;
                            l[2 * i] += p0;
                            l[2 * i + 1] += p1;
                            v2[i] = pack2(p0, p1);
                        }
                    }
                }
                if (it > 0)   // the product that read the P buffer last is complete
                    if (!wait_on(&ctl->pv_done, (it - 1) & 1u, abort_flag)) goto done;
                if (live_lane) {
                    // MN-major operand: a row of kN bf16 per slot, 32- or 64-byte swizzle (the 16-byte chunks of a row are
                    // permuted by address bits 7 (and 8), which count groups of four (two) rows)
                    const float scv[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
                    for (int hh = 0; hh < C::kHalves; ++hh) {
                        if (hh && n_halves < 2) break;   // nothing reads the output columns of heads that are not there
                        const uint32_t lin = static_cast<uint32_t>(slot) * (2 * kN) + 32 * hh;
                        const uint32_t x = (lin >> 3) & (kN == 16 ? 16u : 48u);
#pragma unroll
                        for (int g = 0; g < kCopies; ++g) {
                            uint32_t u[8];
                            const uint64_t sg = pack2(scv[g], scv[g]);
#pragma unroll
                            for (int j = 0; j < 8; ++j) u[j] = pack_bf16x2_from2(kFp8 ? mul2(v2[8 * hh + j], sg) : v2[8 * hh + j]);
                            *reinterpret_cast<uint4*>(sP + g * C::kPCopy + (lin ^ x)) = make_uint4(u[0], u[1], u[2], u[3]);
                            *reinterpret_cast<uint4*>(sP + g * C::kPCopy + ((lin + 16u) ^ x)) = make_uint4(u[4], u[5], u[6], u[7]);
                        }
                    }
                }
                fence_proxy_async_smem();
                tc_fence_before();
                warp_arrive(&ctl->p_full, lane);
            }
            // ---- epilogue: row sums over the slots, exchange with the peer CTA, output
            {
                const int ip = item_n & 1;
#pragma unroll
                for (int hh = 0; hh < C::kHalves; ++hh) {
                    float lv[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) lv[j] = l[16 * hh + j];
                    const float lw = reduce16<false>(lv, lane);
                    if (lane < 16) ctl->lsum[ip][warp][16 * hh + lane] = lw;
                }
                if (!meet()) goto done;
                if (!wait_on(&ctl->o_full, item_n & 1, abort_flag)) goto done;
                tc_fence_after();
                const uint32_t pbar = map_to_cta(smem_u32(&ctl->x_full), peer);
                const uint32_t xout = map_to_cta(smem_u32(sP), peer) + static_cast<uint32_t>(tid) * 16u;
#pragma unroll 1
                for (int hh = 0; hh < n_halves; ++hh) {
                    const int h = lane & 15, r = 16 * hh + h;   // lane h (and h + 16) carries tile row r's numbers; the loops below broadcast them
                    int sub = 0, head = r;
                    if (wi.stacked_rows > 1) {
                        sub = r / p.H;
                        head = r - sub * p.H;
                    }
                    const bool live = r < pt.n_rows;
                    float m = ctl->ref[rb][r];
                    float ls = (ctl->lsum[ip][0][r] + ctl->lsum[ip][1][r]) + (ctl->lsum[ip][2][r] + ctl->lsum[ip][3][r]);
                    if (p.attn_sink != nullptr && wi.k_begin == 0 && half == 0) {
                        // attention sink: one more term exp(sink - m) in the denominator, in the piece that starts the list
                        const float sink2 = live ? __ldg(p.attn_sink + head) * 1.4426950408889634f : -INFINITY;
                        // (a NaN is no term, nor an infinite sink where there is no score)
                        if (sink2 > -INFINITY) {
                            if (m == -INFINITY) m = sink2;
                            const float d = sink2 - m;
                            if (d == d) ls += ex2_approx(d);
                        }
                    }
                    // this CTA's P buffer is free (every product of the item is complete; all four warps have met since they
                    // read the last exchange), so the peer may write its sums over it
                    if (hh > 0)
                        if (!meet()) goto done;
                    if (tid == 0) {
                        mbar_arrive_expect_tx(smem_u32(&ctl->x_full), kXBytes + 2 * 16 * 4);
                        mbar_arrive_cluster(map_to_cta(smem_u32(&ctl->x_ready), peer));
                    }
                    uint32_t u[2][16];
                    tmem_ld_n<16>(lane_base + (2 * half) * kN + 16 * hh, u[0]);
                    tmem_ld_n<16>(lane_base + (2 * half + 1) * kN + 16 * hh, u[1]);
                    {
                        uint32_t o[2][16];
                        tmem_ld_n<16>(lane_base + (2 * peer) * kN + 16 * hh, o[0]);
                        tmem_ld_n<16>(lane_base + (2 * peer + 1) * kN + 16 * hh, o[1]);
                        tmem_wait_ld();
                        if (hh + 1 == n_halves) {   // the next item's products may overwrite O
                            tc_fence_before();
                            warp_arrive(&ctl->o_free, lane);
                        }
                        if (!warp_wait_cluster(smem_u32(&ctl->x_ready), xn & 1u, abort_flag)) goto done;
                        if (tid < 16) {
                            st_async_u32(map_to_cta(smem_u32(&ctl->peer_m[tid]), peer), __float_as_uint(m), pbar);
                            st_async_u32(map_to_cta(smem_u32(&ctl->peer_l[tid]), peer), __float_as_uint(ls), pbar);
                        }
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            st_async_b32x4(xout + c * 2048, o[c >> 2][4 * (c & 3)], o[c >> 2][4 * (c & 3) + 1], o[c >> 2][4 * (c & 3) + 2],
                                           o[c >> 2][4 * (c & 3) + 3], pbar);
                    }
                    if (!warp_wait_cluster(smem_u32(&ctl->x_full), xn & 1u, abort_flag)) goto done;
                    ++xn;
                    const float pm = ctl->peer_m[h], pl = ctl->peer_l[h];
                    const float mm = fmaxf(m, pm);
                    // an infinite sink is the reference of a row without positions: its zeros stay zeros
                    const float f_own = m == -INFINITY ? 0.0f : (m == mm ? 1.0f : ex2_approx(m - mm));
                    const float f_peer = pm == -INFINITY ? 0.0f : (pm == mm ? 1.0f : ex2_approx(pm - mm));
                    ls = ls * f_own + pl * f_peer;
                    m = mm;
                    const float inv = ls == 0.0f ? 0.0f : 1.0f / ls;   // (a NaN stays one, in lse too)
                    const float lse_nat = ls == 0.0f ? INFINITY : (m + __log2f(ls)) * 0.69314718055994531f;
                    const float k_own = f_own * inv, k_peer = f_peer * inv;
                    if (warp == 0 && lane < 16 && live && half == 0) {
                        if (wi.partial_slot >= 0) {
                            p.lse_accum[(size_t)wi.partial_slot * kHeadsPerBlock + r] = ls == 0.0f ? -FLT_MAX : lse_nat;
                        } else {
                            const size_t off = (size_t)(wi.q_row + sub) * p.lse_stride_row + head;
                            if (p.n_peers > 0) {
                                for (int d = 0; d < p.n_peers; ++d)
                                    if (p.lse_peers[d] != nullptr) p.lse_peers[d][off] = lse_nat;
                            } else if (p.lse != nullptr) {
                                p.lse[off] = lse_nat;
                            }
                        }
                    }
                    const float4* xin = reinterpret_cast<const float4*>(sP + tid * 16);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 x0 = xin[c * 128], x1 = xin[(c + 4) * 128];
                        const float xv[2][4] = {{x0.x, x0.y, x0.z, x0.w}, {x1.x, x1.y, x1.z, x1.w}};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int j = 4 * c + k;
                            const float ko = __shfl_sync(0xffffffffu, k_own, j), kp = __shfl_sync(0xffffffffu, k_peer, j);
                            u[0][j] = __float_as_uint(__uint_as_float(u[0][j]) * ko + xv[0][k] * kp);
                            u[1][j] = __float_as_uint(__uint_as_float(u[1][j]) * ko + xv[1][k] * kp);
                        }
                    }
                    const int col = 2 * half * 128 + warp * 32 + lane;   // of group 0; group 1 is 128 columns on
                    if (wi.partial_slot >= 0) {
                        float* dst = p.o_accum + ((size_t)wi.partial_slot * kHeadsPerBlock + 16 * hh) * kDV + col;
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (16 * hh + j < pt.n_rows) {
                                dst[(size_t)j * kDV] = __uint_as_float(u[0][j]);
                                dst[(size_t)j * kDV + 128] = __uint_as_float(u[1][j]);
                            }
                    } else {
                        // two neighbouring lanes exchange half of their heads: each then stores two columns (4 bytes) of eight heads
                        const bool odd = lane & 1;
                        const int row0 = 16 * hh + (odd ? 8 : 0);
                        int rs = 0, rh = row0;
                        if (wi.stacked_rows > 1) {
                            rs = row0 / p.H;
                            rh = row0 - rs * p.H;
                        }
                        size_t off = (size_t)(wi.q_row + rs) * p.stride_o_row + (size_t)rh * p.stride_o_head + (col & ~1);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            uint32_t w2[2];
#pragma unroll
                            for (int g = 0; g < 2; ++g) {
                                const float a = __uint_as_float(u[g][j]), b = __uint_as_float(u[g][j + 8]);
                                const float got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
                                w2[g] = odd ? pack_bf16x2(got, b) : pack_bf16x2(a, got);
                            }
                            if (row0 + j < pt.n_rows) {
                                for (int d = 0; d < (p.n_peers > 0 ? p.n_peers : 1); ++d) {
                                    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.n_peers > 0 ? p.out_peers[d] : p.out) + off;
                                    *reinterpret_cast<uint32_t*>(o) = w2[0];
                                    *reinterpret_cast<uint32_t*>(o + 128) = w2[1];
                                }
                            }
                            off += p.stride_o_head;
                            if (++rh == p.H) {   // the next stacked query row
                                rh = 0;
                                off += p.stride_o_row - (int64_t)p.H * p.stride_o_head;
                            }
                        }
                    }
                }
            }
        }
    } else if (warp < kLoadWarp0) {
        setmaxnreg_dec<kRegsIssuers>();
        if (warp == 4) {
            // ======================================================== Q and score issuer
            const uint32_t el = elect_one() ? 1u : 0u;
            constexpr uint32_t idesc = make_idesc_bf16(64, kN, false);
            const uint64_t q_desc = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
            const uint64_t k_desc0 = make_smem_desc_sw128(smem_u32(sKV), 16, 1024);
            const uint32_t q_lo = static_cast<uint32_t>(q_desc), q_hi = static_cast<uint32_t>(q_desc >> 32);
            uint32_t it = 0;
            Ring ring;
            int item_n = 0;
            for (int w = w_begin; w < w_end; ++w, ++item_n) {
                const dsa_v32_work_info wi = p.works[w];
                const Part pt = part_of(wi, half, p.H);
                if (item_n > 0)   // the products of the item before have read their Q
                    if (!wait_on(&ctl->q_empty, (item_n - 1) & 1, abort_flag)) goto done;
                if (lane == 0) {   // one box = the H heads of one query row; a stacked item has one per query row, H heads apart
                    const int n_box = wi.stacked_rows > 1 ? wi.stacked_rows : 1;
                    const uint32_t bar = smem_u32(&ctl->q_full);
                    mbar_arrive_expect_tx(bar, static_cast<uint32_t>(n_box * p.H * 128 * kBlocks));
                    for (int b = 0; b < n_box; ++b)
                        for (int kb = 0; kb < kBlocks; ++kb)
                            tma_load_3d(smem_u32(sQ) + static_cast<uint32_t>(kb * C::kQBlock + b * p.H * 128), &tm_q, bar, kb * 64, 0, wi.q_row + b);
                }
                __syncwarp();
                if (!wait_on(&ctl->q_full, item_n & 1, abort_flag)) goto done;
                for (int t = 0; t < pt.n_tiles; ++t, ++it, ring.next()) {
                    const uint32_t sb = it & 1u;
                    if (!wait_on(&ctl->kv_full[ring.s], ring.ph, abort_flag)) goto done;
                    if (!kFp8) fence_proxy_async_smem();   // written by cp.async (generic proxy)
                    if (it >= 2)
                        if (!wait_on(&ctl->s_empty[sb], ((it >> 1) & 1u) ^ 1u, abort_flag)) goto done;
                    tc_fence_after();
                    const uint64_t k_desc = k_desc0 + static_cast<uint64_t>((ring.s * kTileBytes) >> 4);
                    const uint32_t k_lo = static_cast<uint32_t>(k_desc), k_hi = static_cast<uint32_t>(k_desc >> 32);
                    const uint32_t d0 = tmem + C::kColS + sb * C::kSBuf;
#pragma unroll
                    for (int kb = 0; kb < kBlocks; ++kb)   // fp8: one accumulator per scale group (two blocks), one for the rope
                        umma_ss_x4_el(kFp8 ? d0 + (kb >> 1) * kN : d0, k_lo + ((kb * kKvBlock) >> 4), k_hi, q_lo + ((kb * C::kQBlock) >> 4), q_hi, idesc,
                                      kFp8 ? (kb & 1) : (kb ? 1u : 0u), el);
                    tc_commit_el(smem_u32(&ctl->s_full[sb]), el);
                }
                tc_commit_el(smem_u32(&ctl->q_empty), el);
            }
        } else if (warp == 5) {
            // ======================================================== P V issuer
            const uint32_t el = elect_one() ? 1u : 0u;
            constexpr uint32_t idesc = make_idesc_bf16(128, kN, true) | kIdescATransposed;
            const uint64_t v_desc0 = make_smem_desc_sw128(smem_u32(sKV), kKvBlock, 1024);   // MN-major: 64-column blocks kKvBlock apart
            const uint64_t p_desc = make_smem_desc_mn_narrow<kN>(smem_u32(sP), C::kPCopy);
            uint32_t it = 0;
            Ring ring;
            int item_n = 0;
            for (int w = w_begin; w < w_end; ++w, ++item_n) {
                const Part pt = part_of(p.works[w], half, p.H);
                for (int t = 0; t < pt.n_tiles; ++t, ++it, ring.next()) {
                    if (!wait_on(&ctl->p_full, it & 1u, abort_flag)) goto done;
                    if (!kFp8) {   // the tile was written by cp.async: observe its barrier, then fence
                        if (!wait_on(&ctl->kv_full[ring.s], ring.ph, abort_flag)) goto done;
                        fence_proxy_async_smem();
                    }
                    if (t == 0 && item_n > 0)   // the previous item's O has been read out
                        if (!wait_on(&ctl->o_free, (item_n - 1) & 1, abort_flag)) goto done;
                    tc_fence_after();
                    const uint64_t v_desc = v_desc0 + static_cast<uint64_t>((ring.s * kTileBytes) >> 4);
#pragma unroll
                    for (int ks = 0; ks < kSlots / 16; ++ks)
#pragma unroll
                        for (int g = 0; g < 4; ++g)
                            umma_ss_el(tmem + g * kN, v_desc + static_cast<uint64_t>((2 * g * kKvBlock + ks * 2048) >> 4),
                                       p_desc + static_cast<uint64_t>(((kFp8 ? g * C::kPCopy : 0) + ks * 16 * 2 * kN) >> 4), idesc, (t > 0 || ks > 0) ? 1u : 0u, el);
                    tc_commit_el(smem_u32(&ctl->kv_empty[ring.s]), el);
                    tc_commit_el(smem_u32(&ctl->pv_done), el);
                    if (t + 1 == pt.n_tiles) tc_commit_el(smem_u32(&ctl->o_full), el);
                }
            }
        }
    } else {
        if constexpr (kFp8) setmaxnreg_inc<kRegsLoaders<kFp8>>();
        else setmaxnreg_dec<kRegsLoaders<kFp8>>();
        {
            // ======================================================== row loaders: four rows of every tile per warp, eight lanes per row
            const int r = 4 * (warp - kLoadWarp0) + (lane >> 3);   // tile row
            const int oc = lane & 7;                               // 16-byte chunks oc, oc + 8, ... of the row
            const uint8_t* kv_bytes = reinterpret_cast<const uint8_t*>(p.kv);
            constexpr uint32_t row_bytes = kFp8 ? kFp8RowBytes : kDQK * 2;
            Ring ring;
            for (int w = w_begin; w < w_end; ++w) {
                const dsa_v32_work_info wi = p.works[w];
                const Part pt = part_of(wi, half, p.H);
                const int seq = wi.q_row / p.s_q;
                const int32_t* idx_row = p.indices + (size_t)wi.q_row * p.topk;
                const int pool_split = (!kFp8 && p.pool_split != nullptr) ? __ldg(p.pool_split + wi.q_row) : 0x7FFFFFFF;
                auto load_slot = [&](int t) -> int {
                    const int k = pt.k_begin + t * kSlots + r;
                    return (k < pt.k_end) ? __ldg(idx_row + k) : -1;
                };
                // physical row of a slot (second pool: -2 - row); -1: nothing to read
                auto resolve = [&](int idx, int phys, int t) -> int {
                    if (!kFp8 && p.kv2 != nullptr && pt.k_begin + t * kSlots + r >= pool_split)
                        return (idx >= 0 && idx < p.num_kv2_rows) ? -2 - idx : -1;
                    return row_of(idx, phys, seq, p);
                };
                auto address = [&](int row) -> const uint8_t* {
                    return row >= -1 ? kv_bytes + (size_t)(row < 0 ? 0 : row) * row_bytes
                                     : reinterpret_cast<const uint8_t*>(p.kv2) + (size_t)(-2 - row) * row_bytes;
                };
                // A row's block number is loaded a step before its address is needed and its slot two steps before, so no load is
                // consumed in the step that issues it.  fp8 cache: three tiles ahead of its use the row is asked into L2 (without it
                // 205 instead of 189 us on 128 sequences of 2 x 16 heads); the bf16 copies of two tiles are in flight anyway, and
                // asking made them slower (prefill of 2048 tokens with 16 heads 406 -> 414 us).
                auto ask = [&](int row) {
                    if (kFp8 && oc == 0 && row != -1) bulk_prefetch_l2(address(row), row_bytes);
                };
                int row0, row1, row2, idx3 = load_slot(3), idx4 = load_slot(4), phys3;
                {
                    const int i0 = load_slot(0), i1 = load_slot(1), i2 = load_slot(2);
                    const int b0 = block_of(i0, seq, p), b1 = block_of(i1, seq, p), b2 = block_of(i2, seq, p);
                    phys3 = block_of(idx3, seq, p);
                    row0 = resolve(i0, b0, 0);
                    row1 = resolve(i1, b1, 1);
                    row2 = resolve(i2, b2, 2);
                    ask(row1);
                    ask(row2);
                }
                auto advance = [&](int t) {   // row0 .. row2: the rows of tiles t + 1 .. t + 3 afterwards
                    const int idx5 = load_slot(t + 5);
                    const int phys4 = block_of(idx4, seq, p);
                    const int row3 = resolve(idx3, phys3, t + 3);
                    ask(row3);
                    row0 = row1;
                    row1 = row2;
                    row2 = row3;
                    idx3 = idx4;
                    idx4 = idx5;
                    phys3 = phys4;
                };
                if (kFp8) {
                    struct Row {
                        uint4 raw[4], rope;
                        float sc;   // lanes oc < 4: scale oc of the row
                        bool ok;
                    };
                    auto load_row = [&](int row) -> Row {
                        Row x;
                        x.ok = row >= 0;
                        const uint8_t* src = address(row);
                        x.sc = 0.0f;
                        if (x.ok) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) x.raw[k] = ldg_stream_16(src + (oc + 8 * k) * 16);
                            x.rope = ldg_stream_16(src + kDV + 16 + oc * 16);
                            if (oc < 4) x.sc = __ldg(reinterpret_cast<const float*>(src + kDV) + oc);
                        } else {
#pragma unroll
                            for (int k = 0; k < 4; ++k) x.raw[k] = make_uint4(0u, 0u, 0u, 0u);
                            x.rope = make_uint4(0u, 0u, 0u, 0u);
                        }
                        return x;
                    };
                    Row next = load_row(row0);
                    for (int t = 0; t < pt.n_tiles; ++t, ring.next()) {
                        Row cur = next;
                        advance(t);
                        next = load_row(row0);   // a whole tile ahead
                        // e4m3 -> bf16 before the wait for a stage: a stage is the scarce resource
                        uint32_t o[32], codes = 0u;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t wv[4] = {cur.raw[k].x, cur.raw[k].y, cur.raw[k].z, cur.raw[k].w};
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                codes |= nan_codes(wv[q]);
                                o[8 * k + 2 * q + 0] = e4m3x2_to_bf16x2(__byte_perm(wv[q], 0u, 0x1404u));
                                o[8 * k + 2 * q + 1] = e4m3x2_to_bf16x2(__byte_perm(wv[q], 0u, 0x3424u));
                            }
                        }
                        if (!wait_on(&ctl->kv_empty[ring.s], ring.ph ^ 1u, abort_flag)) goto done;
                        uint8_t* tile = sKV + ring.s * kTileBytes + r * 128;
                        if (oc < 4) reinterpret_cast<float*>(&ctl->row_scale[ring.s][r])[oc] = cur.sc;
                        if (oc == 0) ctl->ok[ring.s][r] = cur.ok;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int j = oc + 8 * k;   // raw chunk -> 64-column block j / 4, its 16-byte chunks 2 c and 2 c + 1
                            const int c = j & 3;
                            uint8_t* dst_row = tile + (j >> 2) * kKvBlock;
                            // lanes 4-7 of a row store their two chunks in the other order: the eight lanes then hit eight different bank groups
                            const int h0 = (oc >> 2) & 1;
                            const uint4 lo = make_uint4(o[8 * k], o[8 * k + 1], o[8 * k + 2], o[8 * k + 3]);
                            const uint4 hi = make_uint4(o[8 * k + 4], o[8 * k + 5], o[8 * k + 6], o[8 * k + 7]);
                            *reinterpret_cast<uint4*>(dst_row + (((2 * c + h0) ^ (r & 7)) * 16)) = h0 ? hi : lo;
                            *reinterpret_cast<uint4*>(dst_row + (((2 * c + (h0 ^ 1)) ^ (r & 7)) * 16)) = h0 ? lo : hi;
                        }
                        // (an e4m3 NaN makes the row's scores NaN by the rope, and with them out and lse of its queries, as in paired_fp8.cu; the conversion
                        // gives 480.  64 rows of 16 heads x 2048 slots 49.5 -> 50.7 us; a vote and a second conversion of such rows: 52.6)
                        if (codes & 0x80808080u) cur.rope.x |= 0x7FFF7FFFu;
                        *reinterpret_cast<uint4*>(tile + 8 * kKvBlock + ((oc ^ (r & 7)) * 16)) = cur.rope;
                        fence_proxy_async_smem();
                        warp_arrive(&ctl->kv_full[ring.s], lane);
                    }
                } else {
                    for (int t = 0; t < pt.n_tiles; ++t, ring.next()) {
                        const int row = row0;
                        advance(t);
                        if (!wait_on(&ctl->kv_empty[ring.s], ring.ph ^ 1u, abort_flag)) goto done;
                        const uint8_t* src = address(row) + oc * 16;
                        const uint32_t n = row != -1 ? 16u : 0u;   // padding and out-of-range rows: nothing is read, the row is zeros
                        const uint32_t dst = smem_u32(sKV + ring.s * kTileBytes) + r * 128 + ((oc ^ (r & 7)) << 4);
#pragma unroll
                        for (int j = 0; j < kBlocks; ++j) cp_async_16(dst + j * kKvBlock, src + j * 128, n);
                        cp_async_mbar_arrive_noinc(smem_u32(&ctl->kv_full[ring.s]));
                        if (oc == 0) ctl->ok[ring.s][r] = row != -1;
                        warp_arrive(&ctl->kv_full[ring.s], lane);
                    }
                }
            }
        }
    }

done:
    if (ctl->abort_flag) st_cluster_u32(peer_abort, 1u);   // let the peer stop waiting for us
    tc_fence_before();
    __syncthreads();
    if (ctl->abort_flag) {   // a wait gave up; nothing more is issued here, and the peer stays at the barrier below meanwhile
        if (tid == 0) atomicExch(p.status, DSA_V32_ERR_DEVICE_WAIT);
        settle_in_flight();
    }
    cluster_sync_all();   // nothing is on its way to either CTA any more: every send has been waited for by its receiver
    if (warp == 4) {
        tc_fence_after();
        tmem_dealloc(tmem, C::kTmemCols);
    }
}

// The opt-in for more than 48 KB of dynamic shared memory is a per-device attribute of the kernel.
template <bool kFp8, int kN>
static cudaError_t launch(int num_lists, const CUtensorMap& tq, const AttnParams& p, cudaStream_t stream) {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> guard(mu);
        if (dev < 0 || dev >= 64 || !done[dev]) {
            e = cudaFuncSetAttribute(small_heads_kernel<kFp8, kN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<kN>::kSmemBytes);
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) done[dev] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cfg.gridDim = dim3(2 * num_lists, 1, 1);
    cfg.blockDim = dim3(32 * kWarps, 1, 1);
    cfg.dynamicSmemBytes = Cfg<kN>::kSmemBytes;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, small_heads_kernel<kFp8, kN>, tq, p);
}

}  // namespace small

// tile_rows: the most rows an item of the plan has, at most 16 with an fp8 cache
cudaError_t launch_small_heads(bool fp8, int tile_rows, int num_lists, const CUtensorMap& tq, const AttnParams& p, cudaStream_t stream) {
    if (fp8) return tile_rows <= 16 ? small::launch<true, 16>(num_lists, tq, p, stream) : cudaErrorInvalidValue;
    return tile_rows <= 16 ? small::launch<false, 16>(num_lists, tq, p, stream) : small::launch<false, 32>(num_lists, tq, p, stream);
}

}  // namespace dsa
