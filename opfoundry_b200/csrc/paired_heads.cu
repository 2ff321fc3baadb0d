// Sparse MLA attention on a bf16 cache for more than 32 tile rows (heads): one tcgen05 pair MMA over the two CTAs of a cluster.
//
// A work item = one query row (or the stacked rows of an MTP group) x up to 128 heads x a slice of its top-k list, as planned in
// plan.h: an online-softmax attention over the gathered latent rows, K = all 576 columns of a row, V = its first 512 columns
// (opus_attn/dsa_v32/gfx950/mla_decode_a16w16_16mx4_64nx1_template.hpp:815-926).
//
// CTA c of the pair owns tile rows (heads) [64 c, 64 c + 64) and, of every tile of 64 slots, gathers slots [32 c, 32 c + 32).
//       S [128 x 64]   = Q K^T   cta_group::2, M = 128, N = 64: A = each CTA's 64 rows of Q, B = each CTA's 32 gathered rows
//       O [128 x 512] += P V     cta_group::2, M = 128, N = 256, twice: A = each CTA's 64 rows of P, B = each CTA's 256 columns
//                                of all 64 gathered rows
// so a CTA holds the whole softmax of its heads: scores, maxima, P and output rows never cross to the other SM.  Per 64 slots the
// tensor pipe needs 1 088 clocks (measured with these operands: 1 295).
//
// Where the operands lie.  A tile has nine 64-column blocks of 32 rows x 128 bytes in this order: X0 (the column blocks CTA 0
// owns for P V), X1 (those of CTA 1), the rope.  For S a CTA needs its 32 rows whole.  For P V it needs its own column blocks
// of all 64 rows, and a pair MMA reads both CTAs' operands at the same offsets: X0 has to hold rows of CTA 0's slots and X1
// rows of CTA 1's slots in both.  CTA c's own rows already are in X_c; the other X region holds columns that it needs no more
// once the scores of the tile are complete, and the late loaders then put the other CTA's rows (own columns) there.  So the
// second read of a row half costs L2 bandwidth (832 bytes per slot and CTA instead of 576) but no shared memory.
//
// S in TMEM: lanes 0-63 = the CTA's 64 rows x slots of CTA 0, lanes 64-127 = the same rows x slots of CTA 1.
// O in TMEM: lanes 0-63 = the rows x columns of X0's blocks, lanes 64-127 = the rows x columns of X1's blocks.
//
// Warp roles (28 warps = seven warpgroups):
//   warps 0-7    softmax: two teams of four warps on alternate tiles; thread = (row, half of the tile's slots).  A row's two
//                threads post their maxima; its reference maximum is a function of the posted maxima that every thread follows
//                by itself: it moves when a tile's maximum exceeds it by more than the lazy margin of 8 (the
//                reference's threshold: ..16mx4_64nx1_template.hpp:700-725).  P goes to shared memory
//   warps 8-11   the next item's Q rows: by TMA into shared memory, three column blocks where the score MMAs read them and six into
//                two stages of the tile ring ahead of the item's first tile, from there into TMEM (both lane halves); then the
//                epilogue of the item before, while the softmax warps are already at this one
//   warps 12, 13 CTA 0: score issuers on alternate tiles
//   warp 14      CTA 0: P V issuer; CTA 1: tells it that its late rows have landed
//   warp 15      tells the issuers that the CTA's rows of a tile have landed
//   warps 16-23  row loaders, four rows of every tile each
//   warps 24-27  late loaders
//
// What bounds it (cycle stamps of an instrumented copy, prefill of 4096 tokens): a tile of 64 slots every 1 390 cycles, the pace of
// its MMAs; a change of item costs 7 800 more (the score MMAs of the next item wait 2 700 for its Q, its first product 4 900 for the
// stores of O), a sixth of an item of 32 tiles.  One score issuer instead of two: 2 050 cycles a tile.  Arrivals at the issuing CTA with a
// release at cluster scope: 2 970.  Q by 32-byte loads into TMEM instead of TMA and the ring: 14 000 cycles a change of item.
// Against a pair that splits the 576 columns and sums partial scores over distributed shared memory, in
// long runs (the power cap): prefill of 4096 tokens x 128 heads 2260 -> 1656 us, 1268 tokens x 64 heads after 1733 642 -> 483, 1024
// tokens with sink and second pool, 640 slots, 293 -> 215.
//
// Every mbarrier wait is bounded; on expiry the CTA raises its own and its peer's abort flag, records DSA_V32_ERR_DEVICE_WAIT in
// the workspace status word and both drain to the normal exit.  A parity wait is only issued on a barrier whose previous phase
// the waiting warp knows to be complete, and that cannot complete its next one before that warp has looked (tests/test_paired_protocol.py:
// a model of the barriers in which any one role may be held back for as long as the others can run).
#include <cuda_bf16.h>
#include <cfloat>
#include <cstddef>
#include <mutex>
#include "defs.h"
#include "ptx.cuh"
#include "rows.cuh"

namespace dsa {
namespace paired {

constexpr int kRows = 64;                          // tile rows (heads) of a CTA
constexpr int kOwn = 32;                           // slots of a tile that one CTA gathers
constexpr int kSlots = 2 * kOwn;
constexpr int kBlocks = kDQK / 64;                 // nine 64-column blocks
constexpr int kKvBlock = kOwn * 128;               // 4 096
constexpr int kTileBytes = kBlocks * kKvBlock;     // 36 864
constexpr int kQBlock = kRows * 128;               // 8 192
constexpr int kPBytes = kRows * kSlots * 2;        // 8 192
constexpr int kScoreWarp = 12, kPvWarp = 14, kReadyWarp = 15, kLoadWarp0 = 16, kLateWarp0 = 24, kWarps = 28;
constexpr int kSoftmaxWarps = 8, kQWarp0 = 8, kQWarps = 4, kLoadWarps = 8;
constexpr int kMaxRing = 4;                        // tiles whose posted maxima are kept: a team posts tile i + 4 after it has seen the other's of
                                                   // tile i + 3, so that team has done with the maxima of tile i
constexpr int kCtlBytes = 6144;
// Registers per thread after the role split: 2 x softmax + Q + issuers + 2 x loaders + late loaders <= 7 x the launch's 72
constexpr int kRegsSoftmax = 112, kRegsQ = 88, kRegsIssuers = 48, kRegsLoaders = 48, kRegsLate = 48;
static_assert(2 * kRegsSoftmax + kRegsQ + kRegsIssuers + 2 * kRegsLoaders + kRegsLate <= 7 * 72, "more registers than the launch has");

constexpr int kStages = 5;
constexpr int kQTmemBlocks = 6;                    // column blocks of Q in TMEM (both lane halves); the others in shared memory
constexpr int kQStages = 2;                        // ring stages that hold an item's TMEM blocks of Q on their way, ahead of its tiles
constexpr int kQPerStage = kTileBytes / kQBlock;   // four blocks fit one
static_assert(kQStages * kQPerStage >= kQTmemBlocks && kQStages < kStages, "Q fits the stages it passes through");
// An item takes at least kQStages + 1 stages, so the first stage of the Q of item n + 2 is free only after the last one of item n
// has been given back: two landing barriers, by item parity, are enough.
static_assert(2 * (kQStages + 1) - kStages >= kQStages - 1, "a landing barrier of Q is not armed twice");
constexpr int kOffQ = 0;
constexpr int kOffKv = (kBlocks - kQTmemBlocks) * kQBlock;
constexpr int kOffP = kOffKv + kStages * kTileBytes;
constexpr int kOffCtl = kOffP + 2 * kPBytes;
constexpr int kSmemBytes = kOffCtl + kCtlBytes + 1024;   // + slack for 1024-byte alignment
static_assert(kSmemBytes <= 232448, "227 KB per CTA");
// TMEM columns: O 256 | Q 32 per block | S 2 x 32
constexpr uint32_t kColO = 0, kColQ = 256, kColS = kColQ + 32 * kQTmemBlocks, kTmemCols = 512;
static_assert(kColS + 2 * 32 <= kTmemCols, "TMEM");

struct Ctl {
    float post[kMaxRing][2][kRows];      // per tile of the ring and half of its slots: the rows' maxima (log2 domain)
    float l_part[2][2][kRows];           // row sums of an item by [team][half]
    float m_fin[kRows];                  // and its reference maxima
    int32_t late_row[kStages][kOwn];     // rows of the tile that the other CTA gathers
    uint8_t tile_mask[kStages][2][8];    // which slots of CTA 0 / CTA 1 hold a row, four slots a byte
    uint64_t kv_full[kStages], kv_empty[kStages];      // own rows landed | P V of the tile complete (a stage with Q: it has been copied)
    uint64_t tile_ready[2][kStages];                   // CTA 0: both CTAs' rows have landed, by the score issuer (tile number mod 2) that takes the tile
    uint64_t dead[kStages], late_full[kStages];        // scores complete: the other X region may be overwritten | late rows landed
    uint64_t peer_late[kStages];                       // CTA 0: late rows of CTA 1 landed
    uint64_t s_full[2], s_empty[2], p_full[2], pv_done[2];
    uint64_t m_bar[kMaxRing][2];         // a tile's maxima of rows [32 i, 32 i + 32) are posted
    uint64_t q_stage[2];                 // by item parity: every row loader has found the stages free and the blocks on their way to TMEM have landed
    uint64_t q_smem, q_copied, q_full, q_empty, o_full, o_free, e_bar, l_free;
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(Ctl) <= kCtlBytes && offsetof(Ctl, tile_mask) % 8 == 0, "control block");

// Position in the ring of stages.  Every item takes kQStages stages for its Q and then one per tile; of the barriers of a stage
// only kv_empty takes part in the former, so a role keeps the parities of the barriers it follows and flips them as they are used.
struct Ring {
    uint32_t s = 0, bits = 0;
    __device__ __forceinline__ uint32_t ph() const { return (bits >> s) & 1u; }
    __device__ __forceinline__ void skip(uint32_t n) {
        s += n;
        if (s >= kStages) s -= kStages;
    }
    __device__ __forceinline__ void next() {
        bits ^= 1u << s;
        skip(1);
    }
};

__device__ __forceinline__ bool wait_on(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    const uint32_t b = smem_u32(bar);
    if (__all_sync(0xffffffffu, mbar_test_wait(b, parity))) return true;
    return warp_wait(b, parity, abort_flag);
}
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(bar));
}
// on the barrier of the same name in the issuing CTA
__device__ __forceinline__ void warp_arrive_lead(uint64_t* bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(bar), 0));
}

__device__ __forceinline__ int tiles_of(const dsa_v32_work_info& w) { return (w.k_end - w.k_begin + kSlots - 1) / kSlots; }

// `n` column blocks of the item's tile rows [row0, row0 + 64) of Q from block `b0` on: boxes of q_box heads of one query row;
// rows without a head become zeros
__device__ __forceinline__ void load_q(const CUtensorMap& tm_q, const AttnParams& p, const dsa_v32_work_info& w, int row0, uint8_t* dst, uint64_t* bar, int b0, int n) {
    for (int row = 0; row < kRows; row += p.q_box) {
        const RowMap rm = map_row(w, row0 + row, p.H);
        for (int b = 0; b < n; ++b)
            tma_load_3d(smem_u32(dst) + static_cast<uint32_t>(b * kQBlock + row * 128), &tm_q, smem_u32(bar), (b0 + b) * 64, rm.live ? rm.head : p.H, rm.q_row);
    }
}

template <bool kExt>
__global__ void __launch_bounds__(32 * kWarps, 1) paired_heads_kernel(const __grid_constant__ CUtensorMap tm_q, const AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // the same offset in both CTAs of a pair
    uint8_t* sQ = smem + kOffQ;
    uint8_t* sKV = smem + kOffKv;
    uint8_t* sP = smem + kOffP;
    Ctl* ctl = reinterpret_cast<Ctl*>(smem + kOffCtl);
    volatile int* abort_flag = &ctl->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int list = blockIdx.x >> 1;
    const int rank = (int)cluster_ctarank(), peer = rank ^ 1;
    const int w_begin = __ldg(p.list_indptr + list), w_end = __ldg(p.list_indptr + list + 1);

    if (tid < kStages) {
        mbar_init(smem_u32(&ctl->kv_full[tid]), kLoadWarps * 33);   // the lanes (their copies) and one plain arrival per warp (mask, rows)
        mbar_init(smem_u32(&ctl->kv_empty[tid]), 1);
        mbar_init(smem_u32(&ctl->tile_ready[0][tid]), 2);
        mbar_init(smem_u32(&ctl->tile_ready[1][tid]), 2);
        mbar_init(smem_u32(&ctl->peer_late[tid]), 1);
        mbar_init(smem_u32(&ctl->dead[tid]), 1);
        mbar_init(smem_u32(&ctl->late_full[tid]), 4 * 32);
        fence_mbar_init();
    } else if (tid >= 32 && tid < 34) {
        const int i = tid - 32;
        mbar_init(smem_u32(&ctl->s_full[i]), 1);
        mbar_init(smem_u32(&ctl->s_empty[i]), 8);    // one team of either CTA
        mbar_init(smem_u32(&ctl->p_full[i]), 8);
        mbar_init(smem_u32(&ctl->pv_done[i]), 1);
        fence_mbar_init();
    } else if (tid >= 64 && tid < 64 + 2 * kMaxRing) {
        mbar_init(smem_u32(&ctl->m_bar[0][0]) + 8 * (tid - 64), 2);
        fence_mbar_init();
    } else if (tid == 96) {
        mbar_init(smem_u32(&ctl->q_stage[0]), kLoadWarps);
        mbar_init(smem_u32(&ctl->q_stage[1]), kLoadWarps);
        mbar_init(smem_u32(&ctl->q_smem), 1);
        mbar_init(smem_u32(&ctl->q_copied), kQWarps);
        mbar_init(smem_u32(&ctl->q_full), 2 * kQWarps);   // of either CTA
        mbar_init(smem_u32(&ctl->q_empty), 2);            // two score issuers
        mbar_init(smem_u32(&ctl->o_full), 1);
        mbar_init(smem_u32(&ctl->o_free), 2 * kQWarps);
        mbar_init(smem_u32(&ctl->e_bar), kSoftmaxWarps);
        mbar_init(smem_u32(&ctl->l_free), kQWarps);
        ctl->abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == kScoreWarp) {
        tmem_alloc_pair(smem_u32(&ctl->tmem_base), kTmemCols);
        tmem_relinquish_pair();
        if (lane == 0) prefetch_tensormap(&tm_q);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer's barriers exist before anything is sent to it
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    grid_dependency_wait();   // everything above may overlap the tail of the kernel before this one
    const uint32_t peer_abort = map_to_cta(smem_u32(&ctl->abort_flag), peer);

    if (warp < kSoftmaxWarps) {
        // ============================================================ softmax
        setmaxnreg_inc<kRegsSoftmax>();
        const int team = warp >> 2, quad = warp & 3;
        const int h = quad >> 1, rq = quad & 1;        // half of the tile's slots (and of the output columns), half of the CTA's rows
        const int r = 32 * rq + lane;                  // row of the CTA's 64
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(quad * 32) << 16);
        const uint32_t p_row = smem_u32(sP) + r * 128;
        uint32_t it_base = 0;
        int item_n = 0;
        Ring ring;
        for (int w = w_begin; w < w_end; ++w, ++item_n) {
            const uint32_t it_end = it_base + tiles_of(p.works[w]);
            ring.skip(kQStages);
            float m_ref = -INFINITY;   // reference maximum after the last tile this thread looked at
            float l = 0.0f;            // this thread's share of the row sum, against l_ref
            float l_ref = -INFINITY;
            // reference after tile `it` from the one before it: the posted maxima of the row's two halves
            auto follow = [&](float m, uint32_t it) -> float {
                const float mt = fmaxf(ctl->post[it % kMaxRing][0][r], ctl->post[it % kMaxRing][1][r]);
                return mt > m + 8.0f ? mt : m;
            };
            for (uint32_t it = it_base; it < it_end; ++it, ring.next()) {
                if ((it & 1u) != static_cast<uint32_t>(team)) continue;
                const uint32_t ph2 = (it >> 1) & 1u;            // phase of the per-team barriers
                const bool first = it == it_base;
                // the tile's mask.  (The stage's phase before is complete: its tile was at least three earlier, and this team has
                // seen the maxima of the tile three earlier, whose team has read the scores of every tile of its own before.)
                if (!wait_on(&ctl->kv_full[ring.s], ring.ph(), abort_flag)) goto done;
                uint32_t mask;
                {
                    const uint2 n = *reinterpret_cast<const uint2*>(ctl->tile_mask[ring.s][h]);
                    uint32_t a = (n.x | (n.x >> 4)) & 0x00FF00FFu, b = (n.y | (n.y >> 4)) & 0x00FF00FFu;
                    a = (a | (a >> 8)) & 0xFFFFu;
                    b = (b | (b >> 8)) & 0xFFFFu;
                    mask = a | (b << 16);
                }
                if (!wait_on(&ctl->s_full[team], ph2, abort_flag)) goto done;
                tc_fence_after();
                uint32_t sr[32];
                tmem_ld32(lane_base + kColS + 32 * team, sr);
                tmem_wait_ld();
                tc_fence_before();
                warp_arrive_lead(&ctl->s_empty[team], lane);
                if (mask != 0xFFFFFFFFu) {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (!((mask >> j) & 1u)) sr[j] = 0xFF800000u;
                }
                // ---- maximum of this half, posted; the reference before this tile and after it
                float mt;
                {
                    float t[11];
#pragma unroll
                    for (int j = 0; j < 10; ++j) t[j] = max3(__uint_as_float(sr[3 * j]), __uint_as_float(sr[3 * j + 1]), __uint_as_float(sr[3 * j + 2]));
                    t[10] = fmaxf(__uint_as_float(sr[30]), __uint_as_float(sr[31]));
                    const float u0 = max3(t[0], t[1], t[2]), u1 = max3(t[3], t[4], t[5]), u2 = max3(t[6], t[7], t[8]), u3 = fmaxf(t[9], t[10]);
                    mt = fmaxf(max3(u0, u1, u2), u3) * p.scale_log2;
                }
                if (it > 0)
                    if (!wait_on(&ctl->m_bar[(it - 1) % kMaxRing][rq], ((it - 1) / kMaxRing) & 1u, abort_flag)) goto done;
                ctl->post[it % kMaxRing][h][r] = mt;
                warp_arrive(&ctl->m_bar[it % kMaxRing][rq], lane);
                if (!first) m_ref = follow(m_ref, it - 1);
                if (!wait_on(&ctl->m_bar[it % kMaxRing][rq], (it / kMaxRing) & 1u, abort_flag)) goto done;
                const float m_old = m_ref;
                m_ref = follow(m_ref, it);
                // ---- P = 2^(score - reference): at most 2^8; a masked slot gives 0
                const float m_use = m_ref == -INFINITY ? 0.0f : m_ref;
                uint32_t pk[16];
                float lsum;
                {
                    const uint64_t c2 = pack2(p.scale_log2, p.scale_log2), nm2 = pack2(-m_use, -m_use);
                    uint64_t ls2 = pack2(0.0f, 0.0f);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float v0, v1;
                        unpack2(fma2(pack2u(sr[2 * j], sr[2 * j + 1]), c2, nm2), v0, v1);
                        const uint64_t e2 = pack2(ex2_approx(v0), ex2_approx(v1));
                        ls2 = add2(ls2, e2);
                        pk[j] = pack_bf16x2_from2(e2);
                    }
                    float l0, l1;
                    unpack2(ls2, l0, l1);
                    lsum = l0 + l1;
                }
                if (l != 0.0f && l_ref != m_ref) l *= ex2_approx(l_ref - m_ref);
                l += lsum;
                l_ref = m_ref;
                // ---- into the P buffer, once the product that read it last is complete
                if (it >= 2)
                    if (!wait_on(&ctl->pv_done[team], ph2 ^ 1u, abort_flag)) goto done;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint32_t a = p_row + team * kPBytes + (((4 * h + c) ^ (r & 7)) << 4);
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(pk[4 * c]), "r"(pk[4 * c + 1]), "r"(pk[4 * c + 2]), "r"(pk[4 * c + 3]) : "memory");
                }
                fence_proxy_async_smem();
                if (!first && __any_sync(0xffffffffu, m_ref != m_old)) {
                    // the reference moved: O so far (complete once the previous tile's product is) is brought to the new one
                    const float f = m_old == m_ref ? 1.0f : (m_old == -INFINITY ? 0.0f : ex2_approx(m_old - m_ref));
                    if (!wait_on(&ctl->pv_done[team ^ 1], ((it - 1) >> 1) & 1u, abort_flag)) goto done;
                    tc_fence_after();
#pragma unroll 1
                    for (int oc = 0; oc < kDvHalf; oc += 32) {
                        uint32_t o[32];
                        tmem_ld32(lane_base + kColO + oc, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                        tmem_st32(lane_base + kColO + oc, o);
                    }
                    tmem_wait_st();
                }
                tc_fence_before();
                warp_arrive_lead(&ctl->p_full[team], lane);
            }
            // ---- the item's sums and reference, for the epilogue
            {
                const uint32_t last = it_end - 1;
                if ((last & 1u) != static_cast<uint32_t>(team)) {   // the other team had the last tile
                    if (!wait_on(&ctl->m_bar[last % kMaxRing][rq], (last / kMaxRing) & 1u, abort_flag)) goto done;
                    m_ref = follow(m_ref, last);
                }
                if (l != 0.0f && l_ref != m_ref) l *= ex2_approx(l_ref - m_ref);
                if (item_n > 0)   // the epilogue has read those of the item before
                    if (!wait_on(&ctl->l_free, (item_n - 1) & 1, abort_flag)) goto done;
                ctl->l_part[team][h][r] = l;
                if (team == 0 && h == 0) ctl->m_fin[r] = m_ref;
                warp_arrive(&ctl->e_bar, lane);
            }
            it_base = it_end;
        }
    } else if (warp < kScoreWarp) {
        // ============================================================ Q, epilogue
        setmaxnreg_inc<kRegsQ>();
        const int quad = warp & 3;
        const int h = quad >> 1, r = 32 * (quad & 1) + lane;   // half of the output columns, row of the CTA's 64
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(quad * 32) << 16);
        uint32_t q_s = 0;   // first stage of the item's Q
        for (int w = w_begin, n = 0; w <= w_end; ++w, ++n) {
            if (w < w_end) {
                // ---- Q of item n
                const dsa_v32_work_info wi = p.works[w];
                if (n > 0)   // the score MMAs of the item before have read theirs
                    if (!wait_on(&ctl->q_empty, (n - 1) & 1, abort_flag)) goto done;
                if (warp == kQWarp0 && lane == 0) {
                    mbar_arrive_expect_tx(smem_u32(&ctl->q_smem), (kBlocks - kQTmemBlocks) * kQBlock);
                    load_q(tm_q, p, wi, kRows * rank, sQ, &ctl->q_smem, kQTmemBlocks, kBlocks - kQTmemBlocks);
                }
                __syncwarp();
                if (!wait_on(&ctl->q_stage[n & 1], (n >> 1) & 1, abort_flag)) goto done;
                tc_fence_after();
                uint32_t s = q_s;
#pragma unroll 1
                for (int b = 0; b < kQTmemBlocks; ++b) {
                    const uint8_t* src = sKV + s * kTileBytes + (b % kQPerStage) * kQBlock + r * 128;
                    uint32_t v[32];
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const uint4 x = *reinterpret_cast<const uint4*>(src + ((c ^ (r & 7)) << 4));
                        v[4 * c] = x.x;
                        v[4 * c + 1] = x.y;
                        v[4 * c + 2] = x.z;
                        v[4 * c + 3] = x.w;
                    }
                    tmem_st32(lane_base + kColQ + 32 * b, v);
                    if (b % kQPerStage == kQPerStage - 1 && ++s == kStages) s = 0;
                }
                tmem_wait_st();   // (the stages have been read: their bytes are in TMEM)
                tc_fence_before();
                warp_arrive(&ctl->q_copied, lane);
                if (warp == kQWarp0) {   // hand the stages back before the item's scores can start
                    if (!wait_on(&ctl->q_copied, n & 1, abort_flag)) goto done;
                    if (lane < kQStages) mbar_arrive(smem_u32(&ctl->kv_empty[(q_s + lane) % kStages]));
                    __syncwarp();
                }
                q_s = (q_s + kQStages + tiles_of(wi)) % kStages;
                if (!wait_on(&ctl->q_smem, n & 1, abort_flag)) goto done;
                warp_arrive_lead(&ctl->q_full, lane);
            }
            if (n > 0) {
                // ---- epilogue of item n - 1
                const dsa_v32_work_info wi = p.works[w - 1];
                const RowMap rm = map_row(wi, kRows * rank + r, p.H);
                if (!wait_on(&ctl->e_bar, (n - 1) & 1, abort_flag)) goto done;
                float ls = (ctl->l_part[0][0][r] + ctl->l_part[0][1][r]) + (ctl->l_part[1][0][r] + ctl->l_part[1][1][r]);
                float m_ref = ctl->m_fin[r];
                warp_arrive(&ctl->l_free, lane);
                if (kExt && p.attn_sink != nullptr) {
                    // attention sink (opus_attn/dsa_v4/common/mla_v4_host.cc:469-472): one more term exp(sink - m) in the
                    // denominator, counted once per query row and head: in the piece that starts the list
                    const float sink2 = rm.live ? __ldg(p.attn_sink + rm.head) * 1.4426950408889634f : -INFINITY;
                    if (m_ref == -INFINITY) m_ref = sink2;                      // no valid score in this piece: the sink is the reference
                    const float d = sink2 - m_ref;   // (a NaN is no term, nor an infinite sink where there is no score)
                    if (wi.k_begin == 0 && sink2 > -INFINITY && d == d) ls += ex2_approx(d);
                }
                const float inv = ls == 0.0f ? 0.0f : 1.0f / ls;   // (a NaN stays one, in lse too)
                const float lse_nat = ls == 0.0f ? INFINITY : (m_ref + __log2f(ls)) * 0.69314718055994531f;
                if (!wait_on(&ctl->o_full, (n - 1) & 1, abort_flag)) goto done;
                tc_fence_after();
                // this thread's 256 columns of the row
                if (wi.partial_slot < 0) {
                    const size_t off = (size_t)rm.q_row * p.stride_o_row + (size_t)rm.head * p.stride_o_head + 256 * h;
                    const int n_dst = kExt && p.n_peers > 0 ? p.n_peers : 1;
#pragma unroll 1
                    for (int oc = 0; oc < kDvHalf; oc += 32) {
                        uint32_t o[32];
                        tmem_ld32(lane_base + kColO + oc, o);
                        tmem_wait_ld();
                        if (oc + 32 == kDvHalf) {   // the next item's products may overwrite O
                            tc_fence_before();
                            warp_arrive_lead(&ctl->o_free, lane);
                        }
                        if (rm.live) {
                            // thread = row, so a store touches 32 lines whatever its width: 32-byte stores
                            uint32_t u[16];
#pragma unroll
                            for (int v = 0; v < 16; ++v) u[v] = pack_bf16x2(__uint_as_float(o[2 * v]) * inv, __uint_as_float(o[2 * v + 1]) * inv);
#pragma unroll 1
                            for (int d = 0; d < n_dst; ++d) {
                                __nv_bfloat16* o_dst = reinterpret_cast<__nv_bfloat16*>(kExt && p.n_peers > 0 ? p.out_peers[d] : p.out) + off + oc;
                                stg_32<kExt>(o_dst, u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7], p.wide);
                                stg_32<kExt>(o_dst + 16, u[8], u[9], u[10], u[11], u[12], u[13], u[14], u[15], p.wide);
                            }
                        }
                    }
                    if (rm.live && h == 0) {
                        const size_t l_off = (size_t)rm.q_row * p.lse_stride_row + rm.head;
                        if (kExt && p.n_peers > 0) {
                            for (int d = 0; d < p.n_peers; ++d)
                                if (p.lse_peers[d] != nullptr) p.lse_peers[d][l_off] = lse_nat;
                        } else if (p.lse != nullptr) {
                            p.lse[l_off] = lse_nat;
                        }
                    }
                } else {
                    float* o_dst = p.o_accum + ((size_t)wi.partial_slot * kHeadsPerBlock + kRows * rank + r) * kDV + 256 * h;
#pragma unroll 1
                    for (int oc = 0; oc < kDvHalf; oc += 32) {
                        uint32_t o[32];
                        tmem_ld32(lane_base + kColO + oc, o);
                        tmem_wait_ld();
                        if (oc + 32 == kDvHalf) {
                            tc_fence_before();
                            warp_arrive_lead(&ctl->o_free, lane);
                        }
                        if (rm.live) {
#pragma unroll
                            for (int v = 0; v < 4; ++v)
                                stg_256(o_dst + oc + 8 * v, __float_as_uint(__uint_as_float(o[8 * v + 0]) * inv), __float_as_uint(__uint_as_float(o[8 * v + 1]) * inv),
                                        __float_as_uint(__uint_as_float(o[8 * v + 2]) * inv), __float_as_uint(__uint_as_float(o[8 * v + 3]) * inv),
                                        __float_as_uint(__uint_as_float(o[8 * v + 4]) * inv), __float_as_uint(__uint_as_float(o[8 * v + 5]) * inv),
                                        __float_as_uint(__uint_as_float(o[8 * v + 6]) * inv), __float_as_uint(__uint_as_float(o[8 * v + 7]) * inv));
                        }
                    }
                    if (h == 0) p.lse_accum[(size_t)wi.partial_slot * kHeadsPerBlock + kRows * rank + r] = ls == 0.0f ? -FLT_MAX : lse_nat;
                }
            }
        }
    } else if (warp < kLoadWarp0) {
        setmaxnreg_dec<kRegsIssuers>();
        if (warp < kPvWarp && rank == 0) {
            // ======================================================== score issuers, alternate tiles
            // (An issuer's turn - barriers, proxy fence, 36 instructions, commits - takes 2 000 cycles, most of it latency.)
            const uint32_t par = warp - kScoreWarp;
            const uint32_t el = elect_one() ? 1u : 0u;
            constexpr uint32_t idesc = make_idesc_bf16(128, kSlots, false);
            const uint64_t q_desc = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
            const uint64_t k_desc0 = make_smem_desc_sw128(smem_u32(sKV), 16, 1024);
            const uint32_t q_lo = static_cast<uint32_t>(q_desc), q_hi = static_cast<uint32_t>(q_desc >> 32);
            uint32_t it = 0;
            Ring ring;
            int item_n = 0;
            for (int w = w_begin; w < w_end; ++w, ++item_n) {
                const int n_tiles = tiles_of(p.works[w]);
                ring.skip(kQStages);
                if (!wait_on(&ctl->q_full, item_n & 1, abort_flag)) goto done;
                for (int t = 0; t < n_tiles; ++t, ++it) {
                    const uint32_t sb = it & 1u;
                    if (sb != par) {   // the other issuer's.  (It has its own barriers: on common ones this warp would have to look at every
                        ring.skip(1);  // phase, and nothing keeps a stage from its next tile until a warp that is not needed for this one has looked.)
                        continue;
                    }
                    if (!wait_on(&ctl->tile_ready[par][ring.s], ring.ph(), abort_flag)) goto done;
                    if (it >= 2)
                        if (!wait_on(&ctl->s_empty[sb], ((it >> 1) & 1u) ^ 1u, abort_flag)) goto done;
                    tc_fence_after();
                    const uint64_t k_desc = k_desc0 + static_cast<uint64_t>((ring.s * kTileBytes) >> 4);
                    const uint32_t k_lo = static_cast<uint32_t>(k_desc), k_hi = static_cast<uint32_t>(k_desc >> 32);
                    const uint32_t d0 = tmem + kColS + 32 * sb;
#pragma unroll
                    for (int kb = 0; kb < kBlocks; ++kb) {
                        const uint32_t b_lo = k_lo + ((kb * kKvBlock) >> 4);
                        if (kb < kQTmemBlocks) umma_pair_ts_x4_el(d0, tmem + kColQ + 32 * kb, b_lo, k_hi, idesc, kb ? 1u : 0u, el);
                        else umma_pair_ss_x4_el(d0, q_lo + (((kb - kQTmemBlocks) * kQBlock) >> 4), q_hi, b_lo, k_hi, idesc, 1u, el);
                    }
                    tc_commit_pair_el(smem_u32(&ctl->s_full[sb]), el);
                    tc_commit_pair_el(smem_u32(&ctl->dead[ring.s]), el);
                    ring.next();
                }
                tc_commit_pair_el(smem_u32(&ctl->q_empty), el);
            }
        } else if (warp == kPvWarp && rank == 0) {
            // ======================================================== P V issuer
            const uint32_t el = elect_one() ? 1u : 0u;
            constexpr uint32_t idesc = make_idesc_bf16(128, 256, true);
            const uint64_t v_desc0 = make_smem_desc_sw128(smem_u32(sKV), kKvBlock, 1024);   // MN-major: 64-column blocks kKvBlock apart
            const uint64_t p_desc0 = make_smem_desc_sw128(smem_u32(sP), 16, 1024);
            uint32_t it = 0;
            uint32_t ready_bits = 0;   // parities of tile_ready
            Ring ring;
            int item_n = 0;
            for (int w = w_begin; w < w_end; ++w, ++item_n) {
                const int n_tiles = tiles_of(p.works[w]);
                ring.skip(kQStages);
                for (int t = 0; t < n_tiles; ++t, ++it, ring.next()) {
                    const uint32_t sb = it & 1u, rb = sb * kStages + ring.s;
                    if (!wait_on(&ctl->tile_ready[0][0] + rb, (ready_bits >> rb) & 1u, abort_flag)) goto done;
                    ready_bits ^= 1u << rb;
                    if (!wait_on(&ctl->late_full[ring.s], ring.ph(), abort_flag)) goto done;
                    fence_proxy_async_smem();   // written by cp.async (generic proxy)
                    if (!wait_on(&ctl->peer_late[ring.s], ring.ph(), abort_flag)) goto done;
                    if (t == 0 && item_n > 0)   // the previous item's O has been read out
                        if (!wait_on(&ctl->o_free, (item_n - 1) & 1, abort_flag)) goto done;
                    if (!wait_on(&ctl->p_full[sb], (it >> 1) & 1u, abort_flag)) goto done;
                    tc_fence_after();
                    const uint64_t v_desc = v_desc0 + static_cast<uint64_t>((ring.s * kTileBytes) >> 4);
                    const uint64_t p_desc = p_desc0 + static_cast<uint64_t>((sb * kPBytes) >> 4);
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
                        for (int j = 0; j < 2; ++j)
                            umma_pair_ss_el(tmem + kColO + 128 * j, p_desc + static_cast<uint64_t>(ks * 2),
                                            v_desc + static_cast<uint64_t>((((ks >> 1) * 4 + 2 * j) * kKvBlock + (ks & 1) * 2048) >> 4), idesc,
                                            (t > 0 || ks > 0) ? 1u : 0u, el);
                    tc_commit_pair_el(smem_u32(&ctl->kv_empty[ring.s]), el);
                    tc_commit_pair_el(smem_u32(&ctl->pv_done[sb]), el);
                    if (t + 1 == n_tiles) tc_commit_pair_el(smem_u32(&ctl->o_full), el);
                }
            }
        } else if (warp == kReadyWarp || (rank == 1 && warp == kPvWarp)) {
            // ======================================================== this CTA's rows' (late rows') arrival, passed on to the issuers
            uint64_t* const from = warp == kReadyWarp ? ctl->kv_full : ctl->late_full;
            uint64_t* const to0 = warp == kReadyWarp ? ctl->tile_ready[0] : ctl->peer_late;   // for even and odd tiles
            uint64_t* const to1 = warp == kReadyWarp ? ctl->tile_ready[1] : ctl->peer_late;
            uint32_t it = 0;
            Ring ring;
            for (int w = w_begin; w < w_end; ++w) {
                const int n_tiles = tiles_of(p.works[w]);
                ring.skip(kQStages);
                for (int t = 0; t < n_tiles; ++t, ++it, ring.next()) {
                    if (!wait_on(&from[ring.s], ring.ph(), abort_flag)) goto done;
                    fence_proxy_async_smem();   // written by cp.async (generic proxy)
                    warp_arrive_lead((it & 1u ? to1 : to0) + ring.s, lane);
                }
            }
        }
    } else if (warp < kLateWarp0) {
        // ============================================================ row loaders: four rows of every tile per warp, eight lanes per row
        setmaxnreg_dec<kRegsLoaders>();
        const int lw = warp - kLoadWarp0;
        const int r = 4 * lw + (lane >> 3), c8 = lane & 7;
        const uint8_t* kv_bytes = reinterpret_cast<const uint8_t*>(p.kv);
        // lanes 0-3 of a row follow its slot among the CTA's own 32, lanes 4-7 the same slot of the other CTA
        const int slot = kOwn * (c8 < 4 ? rank : peer) + r;
        int item_n = 0;
        Ring ring;   // of kv_empty
        ring.bits = (1u << kStages) - 1u;
        for (int w = w_begin; w < w_end; ++w) {
            const dsa_v32_work_info wi = p.works[w];
            const int n_tiles = tiles_of(wi);
            const int seq = wi.q_row / p.s_q;
            const int32_t* idx_row = p.indices + (size_t)wi.q_row * p.topk;
            const int pool_split = (kExt && p.pool_split != nullptr) ? __ldg(p.pool_split + wi.q_row) : 0x7FFFFFFF;
            auto load_slot = [&](int u) -> int {
                const int k = wi.k_begin + u * kSlots + slot;
                return (k < wi.k_end) ? __ldg(idx_row + k) : -1;
            };
            // block numbers are loaded two tiles ahead, slots four
            int idx_a = load_slot(0), idx_b = load_slot(1), idx_c = load_slot(2), idx_d = load_slot(3);
            int phys_a = block_of(idx_a, seq, p), phys_b = block_of(idx_b, seq, p);
            // the stages that the item's Q takes on its way into TMEM
            for (int i = 0; i < kQStages; ++i, ring.next()) {
                if (!wait_on(&ctl->kv_empty[ring.s], ring.ph(), abort_flag)) goto done;
                if (lw == 0 && lane == 0) {
                    const int b0 = i * kQPerStage, nb = min(kQTmemBlocks - b0, kQPerStage);
                    if (i == 0) mbar_expect_tx(smem_u32(&ctl->q_stage[item_n & 1]), kQTmemBlocks * kQBlock);
                    load_q(tm_q, p, wi, kRows * rank, sKV + ring.s * kTileBytes, &ctl->q_stage[item_n & 1], b0, nb);
                }
            }
            warp_arrive(&ctl->q_stage[item_n & 1], lane);
            ++item_n;
            for (int u = 0; u < n_tiles; ++u, ring.next()) {
                int row = row_of(idx_a, phys_a, seq, p);
                if (kExt && p.kv2 != nullptr && wi.k_begin + u * kSlots + slot >= pool_split)   // row of the second pool: -2 - row
                    row = (idx_a >= 0 && idx_a < p.num_kv2_rows) ? -2 - idx_a : -1;
                {
                    const int phys_n = block_of(idx_c, seq, p);
                    const int idx_n = load_slot(u + 4);
                    idx_a = idx_b; phys_a = phys_b;
                    idx_b = idx_c; phys_b = phys_n;
                    idx_c = idx_d; idx_d = idx_n;
                }
                const uint32_t used = __ballot_sync(0xffffffffu, row != -1);   // bit 8 i: own row i of the warp's four, bit 8 i + 4: the other CTA's
                const int own = __shfl_sync(0xffffffffu, row, lane & ~7);
                if (!wait_on(&ctl->kv_empty[ring.s], ring.ph(), abort_flag)) goto done;
                if (c8 == 4) ctl->late_row[ring.s][r] = row;
                if (lane < 2) {
                    const uint32_t b = used >> (4 * lane);
                    ctl->tile_mask[ring.s][lane ? peer : rank][lw] = static_cast<uint8_t>((b & 1u) | ((b >> 7) & 2u) | ((b >> 14) & 4u) | ((b >> 21) & 8u));
                }
                // padding and out-of-range rows: nothing is read, the row is zeros
                const uint8_t* src = (kExt && own < -1) ? reinterpret_cast<const uint8_t*>(p.kv2) + (size_t)(-2 - own) * (kDQK * 2)
                                                        : kv_bytes + (size_t)(own < 0 ? 0 : own) * (kDQK * 2);
                const uint32_t nbytes = own != -1 ? 16u : 0u;
                const uint32_t dst = smem_u32(sKV) + ring.s * kTileBytes + r * 128 + ((c8 ^ (r & 7)) << 4);
#pragma unroll
                for (int j = 0; j < kBlocks; ++j) cp_async_16(dst + j * kKvBlock, src + j * 128 + c8 * 16, nbytes);
                cp_async_mbar_arrive_noinc(smem_u32(&ctl->kv_full[ring.s]));
                warp_arrive(&ctl->kv_full[ring.s], lane);
            }
        }
    } else {
        // ============================================================ late loaders: this CTA's output columns of the other CTA's rows
        setmaxnreg_dec<kRegsLate>();
        const int r = 8 * (warp - kLateWarp0) + (lane >> 2), c4 = lane & 3;
        const uint8_t* kv_bytes = reinterpret_cast<const uint8_t*>(p.kv);
        Ring ring;
        for (int w = w_begin; w < w_end; ++w) {
            const int n_tiles = tiles_of(p.works[w]);
            ring.skip(kQStages);
            for (int t = 0; t < n_tiles; ++t, ring.next()) {
                if (!wait_on(&ctl->kv_full[ring.s], ring.ph(), abort_flag)) goto done;   // the tile's rows are known
                const int row = ctl->late_row[ring.s][r];
                const uint8_t* src = (kExt && row < -1) ? reinterpret_cast<const uint8_t*>(p.kv2) + (size_t)(-2 - row) * (kDQK * 2)
                                                        : kv_bytes + (size_t)(row < 0 ? 0 : row) * (kDQK * 2);
                src += rank * (kDvHalf * 2);
                const uint32_t nbytes = row != -1 ? 16u : 0u;
                const uint32_t dst = smem_u32(sKV) + ring.s * kTileBytes + 4 * peer * kKvBlock + r * 128;
                if (!wait_on(&ctl->dead[ring.s], ring.ph(), abort_flag)) goto done;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int cc = c4 + 4 * j;
                    cp_async_16(dst + (cc >> 3) * kKvBlock + (((cc & 7) ^ (r & 7)) << 4), src + cc * 16, nbytes);
                }
                cp_async_mbar_arrive_noinc(smem_u32(&ctl->late_full[ring.s]));
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
    cluster_sync_all();   // nothing is on its way to either CTA any more
    if (warp == kScoreWarp) {
        tc_fence_after();
        tmem_dealloc_pair(tmem, kTmemCols);
    }
}

// The opt-in for more than 48 KB of dynamic shared memory is a per-device attribute of the kernel.
template <bool kExt>
static cudaError_t configure() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> guard(mu);
    if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(paired_heads_kernel<kExt>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) done[dev] = true;
    return cudaSuccess;
}

static void fill_launch(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int num_lists, cudaStream_t stream) {
    cfg->gridDim = dim3(2 * num_lists, 1, 1);
    cfg->blockDim = dim3(32 * kWarps, 1, 1);
    cfg->dynamicSmemBytes = kSmemBytes;
    cfg->stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 2;
}

template <bool kExt>
static cudaError_t launch(int num_lists, const CUtensorMap& tq, const AttnParams& p, cudaStream_t stream) {
    cudaError_t e = configure<kExt>();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    fill_launch(&cfg, attr, num_lists, stream);
    return cudaLaunchKernelEx(&cfg, paired_heads_kernel<kExt>, tq, p);
}

}  // namespace paired

int max_resident_pairs_paired(int* out) {
    cudaError_t e = paired::configure<false>();
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    int n = 0;
    paired::fill_launch(&cfg, attr, 1, nullptr);
    e = cudaOccupancyMaxActiveClusters(&n, paired::paired_heads_kernel<false>, &cfg);
    if (e != cudaSuccess) return (int)e;
    *out = n;
    return 0;
}

// ext: a sink, second pool or peers are given, or rows of out are aligned to 16 bytes only; tq: boxes of 64 columns x p.q_box heads of one query row
cudaError_t launch_paired_heads(bool ext, int num_lists, const CUtensorMap& tq, const AttnParams& p, cudaStream_t stream) {
    return ext ? paired::launch<true>(num_lists, tq, p, stream) : paired::launch<false>(num_lists, tq, p, stream);
}

}  // namespace dsa
