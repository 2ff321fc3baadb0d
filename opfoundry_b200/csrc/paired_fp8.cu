// Sparse MLA attention on an fp8 cache for more than 32 tile rows (heads): pair MMAs over the two CTAs of a cluster, the cache's
// bytes as they are for the scores, dequantised to f16 for the second product.
//
// A work item = one query row (or the stacked rows of an MTP group) x up to 128 heads x a slice of its top-k list, as planned in
// plan.h: an online-softmax attention over the gathered latent rows, K = all 576 columns of a row, V = its first 512 columns
// (opus_attn/dsa_v32/gfx950/mla_decode_mxfp8_16mx8_32nx1_template.hpp:1362-1490).
//
// CTA c of the pair owns tile rows (heads) [64 c, 64 c + 64), or [32 c, 32 c + 32) where no item has more than 64, and, of every tile of 64 slots, gathers slots [32 c, 32 c + 32).
//       S_g [128 x 64]  = Q_g K_g^T  cta_group::2, M = 128, N = 64, kind::f8f6f4, one accumulator per 128-column scale group g: B = the
//                                    gathered e4m3 bytes, A = Q as the sum of an e5m2 and an e4m3 number (below); the rope with bf16 operands
//       O [128 x 512] += P V         cta_group::2, M = 128, N = 256, twice, kind::f16 on f16: A = each CTA's 64 rows of P, B = each
//                                    CTA's 256 columns of all 64 gathered rows, scale x byte rounded once to f16
// so a CTA holds the whole softmax of its heads: scores, maxima, P and output rows never cross to the other SM.
//
// Numbers.  Scores: an element of Q has 8 significant bits, so after a power-of-two factor per row (largest magnitude into
// [2^11, 2^12)) it is hi + lo with hi in e5m2 (3 bits and the sign of what is left) and lo in e4m3 (4), exact down to 2^-13 of the row's largest magnitude
// and to 2^-22 of that magnitude below; products and sums are those of the bytes themselves, and the scales (fp32) multiply the finished group
// sums.  A row with more than kWideElements, zeros aside, below that line has a few far above the others, which the cache may answer with
// zeros: there the softmax warps add what hi + lo leave out (residual_group), so the row is as exact as with bf16 operands.  (With an element X times the rest in a
// column where the cache holds zeros, the error of lse is 2e-6 to 1.4e-5, the most at X = 2^8; the kernel before this one had 2.5e-5 to 6e-5 for any X.  A row of
// normal numbers needs one of 2^9 for that; if all rows have one, 64 sequences of 128 heads take 392 us instead of 57, one 40 instead of 17.)
// P and V in f16 (11 significant bits, where P in bf16 has 8): P = 2^(s - reference + 7), at most 2^15 (a weight of less than 2^-32 of the reference's is
// lost, which shows only where all larger weights meet zeros); V = byte x scale 2^-e, rounded once,
// with one e per scale group for the tile's 64 rows, so that the largest |V| stays below 2^16.  e starts at the exponent of the group's largest
// scale in an item's first tile and moves up when a scale exceeds it by 2^7, down when a tile's scales all lie 2^24 below; the group's columns of O are then
// brought to the new e like they are to a new reference maximum.  A row whose scales all lie more than 2^16 below their e lends V the difference, x = 20
// octaves at most, and P takes it back (V 2^x, P 2^-x): f16 alone would lose bits of a row at 2^-21 of a large row's scale and less.  What is lost then lies at
// 2^-41 of the tile's largest V at full weight (a group of a row that is small only beside another group of the same row: 2^-21).  The scale of a group of zeros
// does not count where a row would lose bits by it (the cache writer gives such a group 1).
//
// S in TMEM: lanes 0-63 = the CTA's 64 rows x slots of CTA 0, lanes 64-127 = the same rows x slots of CTA 1.
// O in TMEM: lanes 0-63 = the rows x columns of CTA 0, lanes 64-127 = the rows x columns of CTA 1.
//
// Warp roles (32 warps = eight warpgroups):
//   warps 0-15   softmax: two teams of eight warps on alternate tiles; thread = (row, quarter of the tile's slots).  A row's four
//                threads post their maxima; its reference maximum moves, tile after tile, when a tile's maximum exceeds it by more than the
//                lazy margin of 8 (the reference's threshold: ..16mx4_64nx1_template.hpp:700-725).  P goes to shared memory.  At the change
//                of an item all sixteen fetch the next one's Q (global -> hi and lo -> shared memory) and read out O
//   warps 16, 17 CTA 0: score issuers on alternate tiles
//   warp 18      CTA 0: P V issuer
//   warp 19      tells the issuers that the CTA's rows of a tile have landed, and follows e; watches that the CTA moves on
//   warps 20-23  row loaders: 16-byte cp.async copies into the swizzled tile, eight rows of every tile each
//   warps 24-31  converters: e4m3 -> f16, eight of a tile's rows each; four of them fetch the own output columns of the other CTA's rows
//
// What bounds it (cycle stamps of an instrumented copy, 64 sequences x 128 heads x 2048 slots): a tile of 64 slots every 2 300 cycles.  Its MMAs
// take 1 430 (measured alone; the scores' 25 an instruction are the rate of shared memory, 3 KB of operands each), all its traffic in shared
// memory 2 000; what is in flight - four raw tiles, one and a half converted ones - over the 10 000 cycles from a load to the end of P V gives the rest:
// landing 1 900, scores 1 500, softmax 3 100, a converter's turn 2 200.  Every role pays for the number of its instructions, 6 700 a tile and SM (before V had an exponent per group):
// eight warps of a scheduler on five loops miss the instruction cache (4.7 of 19.6 cycles an instruction in a form of 85 KB; a warp number known
// to be uniform, short waits and rolled loops brought 81 us to 61).  Tried: four teams of four warps with 32 slots a thread (fewer instructions, but
// a tile takes 5 000 cycles from scores to P: 2 880 a tile where two teams of eight took 2 780), two teams of four (2 750, and 1.5 us more for one
// sequence), a converter on both units of a tile (3 240).  The other CTA's rows in the raw tiles, three of 28 KB: 60.6 us instead of 56.5.
// Against the kernel before it (the 576 columns split over the pair, partial scores summed through distributed shared memory in 16 bits, four tile
// stages of 32 slots, rows converted to bf16), 128 heads x 2048 slots, 32768 positions each, other inputs every pass: one sequence 19.4 -> 16.7 us with its merge,
// 16 35.6 -> 31.2, 64 84.0 -> 63.9.  (Of these 0.5, 1.0 and 1.7 us are what keeps Q and V exact beside elements, rows and groups that are far larger, in
// instructions here and there: an exponent per group looked at only where a tile asks for it, and one register more a group, gave nothing back.)  Items of
// one tile are slower than they were: 1184 rows of 64 heads x 32 slots 104 -> 130.
// Against 64 bits, nine shapes of 24 to 128 heads: out 1.67e-3 to 1.69e-3 (2-norm, of which the output's own rounding 1.66e-3; the kernel before 2.11e-3 to
// 2.30e-3), lse at most 1.7e-6 (7e-5; the few-heads kernel that took 17 to 32 rows before 1.4e-6).
//
// Every mbarrier wait is bounded: warp 19 of either CTA, which sees every tile and stays until the other warps have finished, waits by time, the
// others end by the abort flag that it raises.  On expiry the CTA raises its own and its peer's abort flag, records DSA_V32_ERR_DEVICE_WAIT in
// the workspace status word and both drain to the normal exit.  A parity wait is only issued on a barrier whose previous phase
// the waiting warp knows to be complete, and that cannot complete its next one before that warp has looked.
#include <cuda_bf16.h>
#include <cfloat>
#include <cstddef>
#include <mutex>
#include <type_traits>
#include "defs.h"
#include "ptx.cuh"
#include "rows.cuh"

namespace dsa {
namespace paired_fp8 {

constexpr int kRows = 64;                          // tile rows (heads) of a CTA
constexpr int kOwn = 32;                           // slots of a tile that one CTA gathers
constexpr int kSlots = 2 * kOwn;
constexpr int kGroups = 4;                         // 128-column scale groups
constexpr int kBlock = kOwn * 128;                 // 4 096: 128 bytes of 32 rows
constexpr int kRawBytes = (kGroups + 1) * kBlock;  // own rows: the four groups, the rope
constexpr int kStages = 4;                         // raw tiles
constexpr int kVUnit = 4 * kBlock;                 // 32 slots x 256 columns of f16
constexpr int kVUnits = 3;                         // a tile takes two
constexpr int kQBlock = kRows * 128;               // 8 192
constexpr int kPBytes = kRows * kSlots * 2;        // 8 192
constexpr int kSoftmaxWarps = 16, kTeamWarps = 8, kScoreWarp = 16, kPvWarp = 18, kReadyWarp = 19, kLoadWarp0 = 20, kLoadWarps = 4;
constexpr int kConvWarp0 = 24, kConvWarps = 8, kWarps = 32;
// Registers per thread after the role split: 4 x softmax + issuers + loaders + converters of own and of the other CTA's rows <= 8 x the launch's 64
constexpr int kRegsSoftmax = 80, kRegsIssuers = 40, kRegsLoaders = 40, kRegsConv = 48, kRegsLate = 56;
static_assert(4 * kRegsSoftmax + kRegsIssuers + kRegsLoaders + kRegsConv + kRegsLate <= 8 * 64, "more registers than the launch has");
constexpr float kPShift = 7.0f;                    // P = 2^(score - reference + 7) <= 2^15

constexpr int kOffQ = 0;                           // hi of the four groups, lo of the four groups, rope
constexpr int kOffRaw = 9 * kQBlock;
constexpr int kOffV = kOffRaw + kStages * kRawBytes;
constexpr int kOffP = kOffV + kVUnits * kVUnit;
constexpr int kOffCtl = kOffP + 2 * kPBytes;
constexpr int kCtlBytes = 10240;
constexpr int kSmemBytes = kOffCtl + kCtlBytes;
static_assert(kSmemBytes <= 232448, "227 KB per CTA");
// TMEM columns: O 256 | S: groups 0-2 of even tiles, of odd tiles, group 3, rope, 32 columns each
constexpr uint32_t kColO = 0, kColS = 256, kColS3 = kColS + 6 * 32, kColRope = kColS3 + 32, kTmemCols = 512;

struct Ctl {
    float scale[kStages][kGroups][kSlots];   // row scales of a tile (0 where the slot holds no row)
    float post[2][4][kRows];                 // by team and quarter of a tile's slots: the rows' maxima (in the scores' units); at the end of an item its row sums
    float m_ref[2][kRows];                   // by tile number mod 2: the rows' reference maxima after the tile (scores' units)
    uint16_t q_exp[kRows];                   // biased exponent of 2^a, Q = 2^a (hi + lo), 255: a row with an infinity or a NaN; 256 more: hi + lo leave out too much
    int32_t late_row[kStages][kOwn];         // rows of the tile that the other CTA gathers
    uint32_t tile_mask[kStages][2];          // which slots of CTA 0 / CTA 1 hold a row
    alignas(8) float2 v_move[kStages][kGroups];          // 2^(e of the tile before - e), 2^e
    alignas(8) float2 v_mul[kStages][kGroups];           // 2^-e, and 1 where some group of a row needs more than that, else 0
    float v_lent[kStages][kSlots];           // then: 2^x of the rows
    alignas(16) uint16_t p_back[kStages][kSlots];        // and 2^-x in f16
    float v_fin[kGroups];                    // 2^e of the item's last tile
    uint64_t late_known[kStages];                      // late_row is written
    uint64_t kv_full[kStages], raw_empty[kStages];     // rows landed | scores complete, rows converted, scales read
    uint64_t prep[kStages];                            // ... and e known
    uint64_t tile_ready[2][kStages];                   // CTA 0: both CTAs' rows have landed, by the score issuer (tile number mod 2) that takes the tile
    uint64_t v_full[kVUnits], v_empty[kVUnits];        // CTA 0: both CTAs have converted the unit | its products are complete
    uint64_t s_full[2], s_empty[2], s3_empty, p_full[2], pv_done[2];   // s3: group 3 and the rope
    uint64_t posted[2][2], moved[2][2];      // by team and half of the rows: a tile's maxima are posted | its reference maxima are written and those before it read
    uint64_t q_here;                         // this CTA's Q and q_exp are written; what the item before left in post, m_ref and v_fin has been read
    uint64_t q_full, q_empty, o_full, o_free, e_bar;
    uint64_t finished;                       // the other warps have come to their end
    uint64_t residual_here[2];               // by half of the rows: the residuals of an item that has some are written
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(Ctl) <= kCtlBytes && offsetof(Ctl, scale) % 16 == 0, "control block");

// Position in a ring of kN: index and the parity of its current use
template <int kN>
struct Ring {
    uint32_t s = 0, ph = 0;
    __device__ __forceinline__ void next() {
        if (++s == kN) {
            s = 0;
            ph ^= 1u;
        }
    }
};

__device__ __forceinline__ bool wait_on(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    return warp_wait_short(smem_u32(bar), parity, abort_flag);
}
__device__ __forceinline__ bool wait_on2(uint64_t* a, uint32_t parity_a, uint64_t* b, uint32_t parity_b, volatile int* abort_flag) {
    return warp_wait_short2(smem_u32(a), parity_a, smem_u32(b), parity_b, abort_flag);
}
__device__ __forceinline__ bool wait_on3(uint64_t* a, uint32_t parity_a, uint64_t* b, uint32_t parity_b, uint64_t* c, uint32_t parity_c, volatile int* abort_flag) {
    return warp_wait_short3(smem_u32(a), parity_a, smem_u32(b), parity_b, smem_u32(c), parity_c, abort_flag);
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

__device__ __forceinline__ int rows_of(const dsa_v32_work_info& w, int H) { return w.stacked_rows > 1 ? w.stacked_rows * H : H - w.head_block * kHeadsPerBlock; }
__device__ __forceinline__ int tiles_of(const dsa_v32_work_info& w) { return (w.k_end - w.k_begin + kSlots - 1) / kSlots; }

// ------------------------------------------------------------------ Q as a sum of an e5m2 and an e4m3 number
constexpr int kWideElements = 16;   // elements of a row that may lie below what hi + lo hold exactly
// Two elements of Q in f16 (after the row's factor) -> hi = e5m2(x) and lo = e4m3(x - hi), in the low halves
__device__ __forceinline__ void split_q(uint32_t u, uint32_t& hi, uint32_t& lo) {
    hi = f16x2_to_e5m2x2(u);
    lo = f16x2_to_e4m3x2(sub_f16x2(u, __byte_perm(hi, 0, 0x1404)));   // (e5m2 is the upper byte of f16)
}
// Eight bf16 elements times the power of two `mul` -> eight bytes each of hi and lo
__device__ __forceinline__ void split_q8(const uint4& x, float mul, uint2& hi, uint2& lo) {
    const uint32_t in[4] = {x.x, x.y, x.z, x.w};
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float u0, u1;
        unpack2(mul2(pack2u(in[i] << 16, in[i] & 0xFFFF0000u), pack2(mul, mul)), u0, u1);
        split_q(pack_f16x2(u0, u1), h[i], l[i]);   // exact where hi or lo resolve anything
    }
    hi = make_uint2(__byte_perm(h[0], h[1], 0x5410), __byte_perm(h[2], h[3], 0x5410));
    lo = make_uint2(__byte_perm(l[0], l[1], 0x5410), __byte_perm(l[2], l[3], 0x5410));
}

// What hi + lo leave out of eight elements, in the same units: exact in bf16
__device__ __forceinline__ uint4 residual8(const uint4& x, float mul) {
    const uint32_t in[4] = {x.x, x.y, x.z, x.w};
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float u0 = __uint_as_float(in[i] << 16) * mul, u1 = __uint_as_float(in[i] & 0xFFFF0000u) * mul;
        uint32_t hi, lo;
        split_q(pack_f16x2(u0, u1), hi, lo);
        float h0, h1, l0, l1;
        unpack_f16x2(__byte_perm(hi, 0, 0x1404), h0, h1);
        unpack_f16x2(e4m3x2_to_f16x2(lo), l0, l1);
        r[i] = pack_bf16x2((u0 - h0) - l0, (u1 - h1) - l1);
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
}
// Where a row's residual waits while its item runs: the row of the output that the item's end overwrites
__device__ __forceinline__ __nv_bfloat16* residual_row(const AttnParams& p, const dsa_v32_work_info& wi, int row, const RowMap& rm) {
    if (wi.partial_slot >= 0) return reinterpret_cast<__nv_bfloat16*>(p.o_accum + ((size_t)wi.partial_slot * kHeadsPerBlock + row) * kDV);
    return reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)rm.q_row * p.stride_o_row + (size_t)rm.head * p.stride_o_head;
}
// Residuals of sixteen rows (q: rows lane / 4 and that + 8; null: zeros) times 16 rows of the cache (k: the same), 128 columns: bf16 operands, sums in fp32.
// By mma.sync, operands from L2: rows that need it are rare.
__device__ __forceinline__ void residual_group(const __nv_bfloat16* q0, const __nv_bfloat16* q1, const uint8_t* k0, const uint8_t* k1, int lane, float (&acc)[2][4]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j >> 2][j & 3] = 0.0f;
#pragma unroll 2
    for (int c = 8 * (lane & 3); c < 128; c += 32) {   // eight columns a lane; which one the MMA takes for which is the same in Q and the cache
        uint4 x[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
        uint2 y[2] = {make_uint2(0u, 0u), make_uint2(0u, 0u)};
        if (q0) x[0] = *reinterpret_cast<const uint4*>(q0 + c);
        if (q1) x[1] = *reinterpret_cast<const uint4*>(q1 + c);
        if (k0) y[0] = __ldg(reinterpret_cast<const uint2*>(k0 + c));
        if (k1) y[1] = __ldg(reinterpret_cast<const uint2*>(k1 + c));
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            uint32_t b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float lo, hi;
                unpack_f16x2(e4m3x2_to_f16x2((j < 2 ? y[n].x : y[n].y) >> (16 * (j & 1))), lo, hi);
                b[j] = pack_bf16x2(lo, hi);
            }
            mma_bf16_16816(acc[n], x[0].x, x[1].x, x[0].y, x[1].y, b[0], b[1]);
            mma_bf16_16816(acc[n], x[0].z, x[1].z, x[0].w, x[1].w, b[2], b[3]);
        }
    }
}

// kShare: tile rows that a CTA owns, 64, or 32 for plans without items of more than 64: softmax warps without a live row only take part in the
// barriers (128 sequences of 2 x 16 heads 144 -> 134 us), and with 32 that is half of either CTA's (64 sequences of 64 heads 55.5 -> 52.5 us; decided
// at run time it costs 0.4 us a launch).
// kExt: a sink, peers, or rows of out on 16-byte boundaries (stacked rows need nothing of it, but come with it, as they do on the bf16 kernel)
template <bool kExt, int kShare>
__global__ void __launch_bounds__(32 * kWarps, 1) paired_fp8_kernel(const AttnParams p) {
    extern __shared__ __align__(1024) uint8_t smem_paired_fp8[];   // the same offset in both CTAs of a pair
    uint8_t* smem = smem_paired_fp8;
    uint8_t* sQ = smem + kOffQ;
    uint8_t* sRaw = smem + kOffRaw;
    uint8_t* sV = smem + kOffV;
    uint8_t* sP = smem + kOffP;
    Ctl* ctl = reinterpret_cast<Ctl*>(smem + kOffCtl);
    volatile int* abort_flag = &ctl->abort_flag;
    // the warp's number by a shuffle: what depends on it is then known to be the same in all lanes, and loop counters, barrier addresses and
    // descriptors stay in uniform registers (a score MMA takes 10 instructions instead of 20)
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int list = blockIdx.x >> 1;
    const int rank = (int)cluster_ctarank(), peer = rank ^ 1;
    const int w_begin = __ldg(p.list_indptr + list), w_end = __ldg(p.list_indptr + list + 1);

    if (tid < kStages) {
        mbar_init(smem_u32(&ctl->kv_full[tid]), kLoadWarps * 33);   // the lanes (their copies) and one plain arrival per warp (mask)
        mbar_init(smem_u32(&ctl->raw_empty[tid]), 1 + kConvWarps + kTeamWarps);   // the scores, the converters, the softmax team
        mbar_init(smem_u32(&ctl->prep[tid]), 1);
        mbar_init(smem_u32(&ctl->tile_ready[0][tid]), 2);
        mbar_init(smem_u32(&ctl->tile_ready[1][tid]), 2);
        mbar_init(smem_u32(&ctl->late_known[tid]), kLoadWarps);
        if (tid < kVUnits) {
            mbar_init(smem_u32(&ctl->v_full[tid]), kConvWarps);   // half of either CTA's converters
            mbar_init(smem_u32(&ctl->v_empty[tid]), 1);
        }
        fence_mbar_init();
    } else if (tid >= 32 && tid < 34) {
        const int i = tid - 32;
        mbar_init(smem_u32(&ctl->s_full[i]), 1);
        mbar_init(smem_u32(&ctl->s_empty[i]), 2 * kTeamWarps);    // one team of either CTA
        mbar_init(smem_u32(&ctl->p_full[i]), 2 * kTeamWarps);
        mbar_init(smem_u32(&ctl->pv_done[i]), 1);
        for (int rq = 0; rq < 2; ++rq) {
            mbar_init(smem_u32(&ctl->posted[i][rq]), kTeamWarps / 2);
            mbar_init(smem_u32(&ctl->moved[i][rq]), kTeamWarps / 2);
        }
        fence_mbar_init();
    } else if (tid == 96) {
        mbar_init(smem_u32(&ctl->s3_empty), 2 * kTeamWarps);
        mbar_init(smem_u32(&ctl->q_full), 2 * kSoftmaxWarps);   // of either CTA
        mbar_init(smem_u32(&ctl->q_here), kSoftmaxWarps);
        mbar_init(smem_u32(&ctl->q_empty), 2);                  // two score issuers
        mbar_init(smem_u32(&ctl->o_full), 1);
        mbar_init(smem_u32(&ctl->o_free), 2 * kSoftmaxWarps);
        mbar_init(smem_u32(&ctl->e_bar), kSoftmaxWarps);
        mbar_init(smem_u32(&ctl->finished), kWarps - 1);
        mbar_init(smem_u32(&ctl->residual_here[0]), kSoftmaxWarps / 2);
        mbar_init(smem_u32(&ctl->residual_here[1]), kSoftmaxWarps / 2);
        ctl->abort_flag = 0;
        fence_mbar_init();
    }
    static_assert(kVUnits <= kStages, "one thread per stage and unit");
    if (warp == kScoreWarp) {
        tmem_alloc_pair(smem_u32(&ctl->tmem_base), kTmemCols);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer's barriers exist before anything is sent to it
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    grid_dependency_wait();   // everything above may overlap the tail of the kernel before this one
    const uint32_t peer_abort = map_to_cta(smem_u32(&ctl->abort_flag), peer);

    if (warp < kSoftmaxWarps) {
        // ============================================================ Q, softmax, epilogue
        setmaxnreg_inc<kRegsSoftmax>();
        const int team = warp >> 3, cs = (warp >> 2) & 1, quad = warp & 3;
        const int h = quad >> 1, rq = quad & 1;        // half of the tile's slots (and of the output columns), half of the CTA's rows
        const int r = 32 * rq + lane;                  // row of the CTA's 64
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(quad * 32) << 16);
        const uint32_t p_lo = smem_u32(sP) + team * kPBytes + r * 128 + (((4 * h + 2 * cs) ^ (r & 7)) << 4);   // 16 slots: this chunk and its neighbour
        // Q of an item: four rows per warp; lane = columns [8 lane, 8 lane + 8) and the same of the upper 256, of the rope eight lanes a row
        auto store_q = [&](const dsa_v32_work_info& wi) {
            const int row0 = 4 * warp;
            uint4 x[4][2], xr = make_uint4(0u, 0u, 0u, 0u);
            auto row_ptr = [&](int row, bool& live) {
                const RowMap rm = map_row(wi, kShare * rank + row, p.H);
                live = rm.live && row < kShare;
                return reinterpret_cast<const __nv_bfloat16*>(p.q) + (size_t)(live ? rm.q_row : wi.q_row) * p.stride_q_row + (size_t)(live ? rm.head : 0) * p.stride_q_head;
            };
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                bool live;
                const __nv_bfloat16* src = row_ptr(row0 + i, live) + 8 * lane;
                x[i][0] = x[i][1] = make_uint4(0u, 0u, 0u, 0u);
                if (live) {
                    x[i][0] = __ldg(reinterpret_cast<const uint4*>(src));
                    x[i][1] = __ldg(reinterpret_cast<const uint4*>(src + 256));
                }
            }
            {
                bool live;
                const __nv_bfloat16* src = row_ptr(row0 + (lane >> 3), live) + kDV + 8 * (lane & 7);
                if (live) xr = __ldg(reinterpret_cast<const uint4*>(src));
            }
            float rope_mul = 1.0f;
            uint2 hi[4][2];
            int maybe = 0;   // rows that may have elements below what hi and lo hold: those that are not all zeros, nor have an infinity or a NaN
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = row0 + i;
                uint32_t m = 0u;
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    m = max_u16x2(max_u16x2(max_u16x2(x[i][k].x & 0x7FFF7FFFu, x[i][k].y & 0x7FFF7FFFu),
                                            max_u16x2(x[i][k].z & 0x7FFF7FFFu, x[i][k].w & 0x7FFF7FFFu)), m);
                m = __reduce_max_sync(0xffffffffu, max(m >> 16, m & 0xFFFFu));
                // the largest magnitude into [2^11, 2^12)
                const uint32_t e = max(m >> 7, 64u);
                const float mul = __uint_as_float((265u - min(e, 254u)) << 23);
                if ((lane >> 3) == i) rope_mul = mul;
                if (m != 0u && e < 255u) maybe |= 1 << i;
                if (lane == 0) ctl->q_exp[row] = static_cast<uint16_t>(e == 255u ? 255u : e - 11u);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    uint2 lo;
                    split_q8(x[i][k], mul, hi[i][k], lo);
                    uint8_t* dst = sQ + (2 * k + (lane >> 4)) * kQBlock + row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4) + 8 * (lane & 1);
                    *reinterpret_cast<uint2*>(dst) = hi[i][k];
                    *reinterpret_cast<uint2*>(dst + kGroups * kQBlock) = lo;
                }
            }
            {
                const int row = row0 + (lane >> 3);
                *reinterpret_cast<uint4*>(sQ + 2 * kGroups * kQBlock + row * 128 + (((lane & 7) ^ (row & 7)) << 4)) =
                    make_uint4(scale_bf16x2(xr.x, rope_mul), scale_bf16x2(xr.y, rope_mul), scale_bf16x2(xr.z, rope_mul), scale_bf16x2(xr.w, rope_mul));
            }
            fence_proxy_async_smem();
            warp_arrive_lead(&ctl->q_full, lane);
            // The scores may start; meanwhile, rows with more than kWideElements below 2^-2 (with the row's factor): two lanes hold such an element, or a 0, by their
            // bytes of hi ...
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t large = 0xFFFFFFFFu;   // bit 7 of a byte: magnitudes of 2^-2 and more only
#pragma unroll
                for (int k = 0; k < 2; ++k) large &= ((hi[i][k].x & 0x7F7F7F7Fu) + 0x4C4C4C4Cu) & ((hi[i][k].y & 0x7F7F7F7Fu) + 0x4C4C4C4Cu);
                const uint32_t lanes = __ballot_sync(0xffffffffu, (large & 0x80808080u) != 0x80808080u);
                if ((lanes & (lanes - 1u)) == 0u) maybe &= ~(1 << i);
            }
            // ... and then they are counted: their magnitudes' bits less 1 (a 0 becomes the largest), cut off to line - 2 or line - 1, two halves in 32-bit sums,
            // from which line - 2 is taken at the end (a 0 in the lower half lends its neighbour's last bit, which may cost an element its place on the line)
            __syncwarp();
#pragma unroll 1
            for (; maybe != 0; maybe &= maybe - 1) {
                const int row = row0 + __ffs(maybe) - 1;
                bool live;
                const uint4* src = reinterpret_cast<const uint4*>(row_ptr(row, live)) + lane;
                const uint4 y[2] = {__ldg(src), __ldg(src + 32)};
                const uint32_t e = ctl->q_exp[row], line = ((e - 2u) << 7) * 0x10001u;
                uint32_t n = 0u;
#pragma unroll
                for (int k = 0; k < 2; ++k)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t w = (j == 0 ? y[k].x : j == 1 ? y[k].y : j == 2 ? y[k].z : y[k].w) & 0x7FFF7FFFu;
                        n += max_u16x2(min_u16x2(w - 0x10001u, line - 0x10001u), line - 0x20002u);
                    }
                n -= 8u * (line - 0x20002u);
                const uint32_t below = 512u - __reduce_add_sync(0xffffffffu, (n & 0xFFFFu) + (n >> 16));
                if (lane == 0 && below > kWideElements) ctl->q_exp[row] = static_cast<uint16_t>(e + 256u);
            }
            warp_arrive(&ctl->q_here, lane);
        };
        uint32_t it_base = 0;
        int item_n = 0;
        Ring<kStages> ring;   // of this team's tiles: every other one
        if (team) ring.next();
        float ls = 0.0f, m_out = 0.0f, v_unit = 1.0f;   // of the last item: its row sum, last reference and 2^e of the columns that this thread reads out
        // The list's items.  Two forms, one after the other: the first leaves with `true` at the first item with rows for residual_group, and the second goes
        // on from there, so that the registers of the first are given out as if the second were not there (both in one loop: 128 sequences of 2 x 16 heads
        // 140 -> 149 us; the residual as a function that is called: 156).
        int w = w_begin;
        auto items = [&](auto residual, bool resume) -> bool {
            constexpr bool kResidual = decltype(residual)::value;
            int n_wide = 0;
#pragma unroll 1
            for (; w <= w_end; ++w, ++item_n, resume = false) {
                if (!resume) {
                    // ---- Q of this item, so that its scores can start; then the output of the one before
                    if (w < w_end) {
                        if (item_n > 0)
                            if (!wait_on(&ctl->q_empty, (item_n - 1) & 1, abort_flag)) return false;
                        store_q(p.works[w]);
                    }
                    if (item_n > 0) {
                        const dsa_v32_work_info wi = p.works[w - 1];
                        const int row = kShare * rank + r;   // of the item's tile
                        const RowMap rm = map_row(wi, row, p.H);
                        if (kExt && p.attn_sink != nullptr) {
                            // attention sink (opus_attn/dsa_v4/common/mla_v4_host.cc:469-472): one more term exp(sink - m) in the
                            // denominator, counted once per query row and head: in the piece that starts the list
                            const float sink2 = rm.live ? __ldg(p.attn_sink + rm.head) * 1.4426950408889634f : -INFINITY;
                            if (m_out == -INFINITY) m_out = sink2;                      // no valid score in this piece: the sink is the reference
                            const float d = sink2 - m_out;
                            if (wi.k_begin == 0 && sink2 > -INFINITY && d == d) {   // (a NaN is no term, nor an infinite sink where there is no score)
                                if (d > 0.0f) {   // a sink above the scores is the reference, so that nothing overflows
                                    const float f = ex2_approx(-d);
                                    ls *= f;
                                    v_unit *= f;
                                    m_out = sink2;
                                }
                                ls += ex2_approx(fminf(d, 0.0f) + kPShift);
                            }
                        }
                        const float inv = ls == 0.0f ? 0.0f : v_unit / ls;   // (a NaN stays one, in lse too)
                        const float lse_nat = ls == 0.0f ? INFINITY : (m_out - kPShift + __log2f(ls)) * 0.69314718055994531f;
                        if (!wait_on(&ctl->o_full, (item_n - 1) & 1, abort_flag)) return false;
                        tc_fence_after();
                        // this thread's 64 columns of the row
                        const int col0 = 64 * (warp >> 2);   // of the 256 in its lane
                        if (32 * rq >= kShare) {   // none of the warp's rows is live
                            tc_fence_before();
                            warp_arrive_lead(&ctl->o_free, lane);
                        } else if (wi.partial_slot < 0) {
                            const size_t off = (size_t)rm.q_row * p.stride_o_row + (size_t)rm.head * p.stride_o_head + 256 * h;
                            const int n_dst = kExt && p.n_peers > 0 ? p.n_peers : 1;
#pragma unroll 1
                            for (int oc = col0; oc < col0 + 64; oc += 32) {
                                uint32_t o[32];
                                tmem_ld32(lane_base + kColO + oc, o);
                                tmem_wait_ld();
                                if (oc != col0) {   // the next item's products may overwrite O
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
                            if (rm.live && warp < 2) {   // the rows' first quarter of the left half
                                const size_t l_off = (size_t)rm.q_row * p.lse_stride_row + rm.head;
                                if (kExt && p.n_peers > 0) {
                                    for (int d = 0; d < p.n_peers; ++d)
                                        if (p.lse_peers[d] != nullptr) p.lse_peers[d][l_off] = lse_nat;
                                } else if (p.lse != nullptr) {
                                    p.lse[l_off] = lse_nat;
                                }
                            }
                        } else {
                            float* o_dst = p.o_accum + ((size_t)wi.partial_slot * kHeadsPerBlock + row) * kDV + 256 * h;
#pragma unroll 1
                            for (int oc = col0; oc < col0 + 64; oc += 32) {
                                uint32_t o[32];
                                tmem_ld32(lane_base + kColO + oc, o);
                                tmem_wait_ld();
                                if (oc != col0) {
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
                            if (rm.live && warp < 2) p.lse_accum[(size_t)wi.partial_slot * kHeadsPerBlock + row] = ls == 0.0f ? -FLT_MAX : lse_nat;
                        }
                    }
                }
                if (w == w_end) break;
                const uint32_t it_end = it_base + tiles_of(p.works[w]);
                float m_ref = -INFINITY;   // reference maximum after this team's last tile
                float l = 0.0f;            // this thread's share of the row sum, against m_ref
                const bool idle = 32 * rq >= kShare || kShare * rank + 32 * rq >= rows_of(p.works[w], p.H);   // none of the warp's rows is live
                if (!resume)
                    if (!wait_on(&ctl->q_here, item_n & 1, abort_flag)) return false;
                const uint32_t q_exp = ctl->q_exp[r] & 255u;
                const bool any_wide = __any_sync(0xffffffffu, ctl->q_exp[r] >= 256u);
                if (!kResidual && any_wide) return true;
                if (kResidual && any_wide) {
                    // four of the 32 rows for each of the warps that share them
                    const dsa_v32_work_info& wi = p.works[w];
#pragma unroll 1
                    for (int row = 32 * rq + 4 * (4 * team + 2 * cs + h), end = row + 4; row < end; ++row) {
                        const uint32_t e = ctl->q_exp[row];
                        if (e < 256u) continue;
                        const RowMap rm = map_row(wi, kShare * rank + row, p.H);   // (a live row)
                        const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.q) + (size_t)rm.q_row * p.stride_q_row + (size_t)rm.head * p.stride_q_head);
                        uint4* dst = reinterpret_cast<uint4*>(residual_row(p, wi, kShare * rank + row, rm));
                        const float mul = __uint_as_float((254u - (e & 255u)) << 23);
#pragma unroll 1
                        for (int k = lane; k < kDV / 8; k += 32) dst[k] = residual8(__ldg(src + k), mul);
                    }
                    warp_arrive(&ctl->residual_here[rq], lane);
                    if (!wait_on(&ctl->residual_here[rq], n_wide & 1, abort_flag)) return false;
                    ++n_wide;
                }
                const float c_log2 = p.scale_log2 * __uint_as_float(q_exp == 255u ? 0x7FC00000u : q_exp << 23);   // of scores in units of 2^a
                uint32_t it = it_base + ((it_base ^ team) & 1u);
                if (idle) {   // the warp's part in the barriers; what P holds for such rows is used for such rows of O only
#pragma unroll 1
                    for (; it < it_end; it += 2, ring.next(), ring.next()) {
                        const uint32_t ph2 = (it >> 1) & 1u;
                        if (!wait_on(&ctl->s_full[team], ph2, abort_flag)) return false;
                        warp_arrive_lead(&ctl->s3_empty, lane);
                        warp_arrive_lead(&ctl->s_empty[team], lane);
                        warp_arrive(&ctl->raw_empty[ring.s], lane);
                        if (it >= 2)   // every warp of the team has come to the end of its last tile
                            if (!wait_on(&ctl->pv_done[team], ph2 ^ 1u, abort_flag)) return false;
                        warp_arrive(&ctl->posted[team][rq], lane);
                        warp_arrive(&ctl->moved[team][rq], lane);
                        warp_arrive_lead(&ctl->p_full[team], lane);
                    }
                }
#pragma unroll 1
                for (; it < it_end; it += 2, ring.next(), ring.next()) {
                    const uint32_t ph2 = (it >> 1) & 1u;            // phase of the per-team barriers
                    const bool first = it == it_base;
                    // the tile's mask, scales and e, and its scores (the stage's phase before is complete: its tile was three earlier, and this team has
                    // seen the references move past that tile); the team has read its last tile's maxima
                    if (!wait_on3(&ctl->prep[ring.s], ring.ph, &ctl->s_full[team], ph2, &ctl->moved[team][rq], ph2 ^ 1u, abort_flag)) return false;
                    tc_fence_after();
                    // ---- scores in units of 2^a: sum_g scale_g S_g + S_rope, in pairs of slots.  Group 3 and the rope, which have one
                    // accumulator for all tiles, first
                    uint64_t sv[8];
                    uint32_t mask;
                    float v_fix;
                    bool lent;
                    {
                        const uint32_t ca = lane_base + kColS + 96 * team + 16 * cs;
                        const float* sc = &ctl->scale[ring.s][0][kOwn * h + 16 * cs];
                        uint32_t x[2][16], sr[16];
                        tmem_ld16(lane_base + kColS3 + 16 * cs, x[1]);
                        tmem_ld16(lane_base + kColRope + 16 * cs, sr);
                        mask = ctl->tile_mask[ring.s][h] >> (16 * cs);
                        const float2 move = ctl->v_move[ring.s][2 * h + cs];
                        v_fix = move.x;
                        v_unit = move.y;
                        lent = __any_sync(0xffffffffu, ctl->v_mul[ring.s][0].y != 0.0f);
                        tmem_wait_ld();
                        tmem_loaded(x[1]);
                        tmem_loaded(sr);
                        tc_fence_before();
                        warp_arrive_lead(&ctl->s3_empty, lane);
#pragma unroll
                        for (int g = kGroups - 1; g >= 0; --g) {   // the next group's scores are on their way while this one's are scaled
                            if (g > 0) tmem_ld16(ca + 32 * (g - 1), x[(g - 1) & 1]);
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                const float4 f = *reinterpret_cast<const float4*>(sc + g * kSlots + 4 * c);
                                const uint32_t* y = x[g & 1] + 4 * c;
                                sv[2 * c] = fma2(pack2(f.x, f.y), pack2u(y[0], y[1]), g == kGroups - 1 ? pack2u(sr[4 * c], sr[4 * c + 1]) : sv[2 * c]);
                                sv[2 * c + 1] = fma2(pack2(f.z, f.w), pack2u(y[2], y[3]), g == kGroups - 1 ? pack2u(sr[4 * c + 2], sr[4 * c + 3]) : sv[2 * c + 1]);
                            }
                            if (g > 0) {
                                tmem_wait_ld();
                                tmem_loaded(x[(g - 1) & 1]);
                            }
                            if (!kResidual && g == 1) {
                                tc_fence_before();
                                warp_arrive_lead(&ctl->s_empty[team], lane);
                            }
                        }
                        if (!kResidual && !lent) warp_arrive(&ctl->raw_empty[ring.s], lane);
                    }
                    if (kResidual && any_wide) {   // what hi + lo leave out of some row of the warp's; meanwhile the scores wait in tensor memory
                        const uint32_t own = lane_base + kColS + 96 * team + 16 * cs;
                        {
                            uint32_t y[16];
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                y[2 * j] = static_cast<uint32_t>(sv[j]);
                                y[2 * j + 1] = static_cast<uint32_t>(sv[j] >> 32);
                            }
                            tmem_st16(own, y);
                            tmem_wait_st();
                        }
                        const dsa_v32_work_info& wi = p.works[w];
                        const uint8_t* rows[2];
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int k = wi.k_begin + static_cast<int>(it - it_base) * kSlots + kOwn * h + 16 * cs + (lane >> 2) + 8 * i;
                            const int row = k < wi.k_end ? translate_row(__ldg(p.indices + (size_t)wi.q_row * p.topk + k), wi.q_row / p.s_q, p) : -1;
                            rows[i] = row < 0 ? nullptr : reinterpret_cast<const uint8_t*>(p.kv) + (size_t)row * kFp8RowBytes;
                        }
#pragma unroll 1
                        for (int m = 0; m < 2; ++m) {   // sixteen rows of Q
                            const __nv_bfloat16* q[2];
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const int row = 32 * rq + 16 * m + 8 * i + (lane >> 2);
                                q[i] = ctl->q_exp[row] < 256u ? nullptr : residual_row(p, wi, kShare * rank + row, map_row(wi, kShare * rank + row, p.H));
                            }
                            float sum[2][4] = {};
#pragma unroll 1
                            for (int g = 0; g < kGroups; ++g) {
                                float acc[2][4];
                                residual_group(q[0] ? q[0] + 128 * g : nullptr, q[1] ? q[1] + 128 * g : nullptr, rows[0] ? rows[0] + 128 * g : nullptr, rows[1] ? rows[1] + 128 * g : nullptr, lane, acc);
                                const float* sc = &ctl->scale[ring.s][g][kOwn * h + 16 * cs + 2 * (lane & 3)];
#pragma unroll
                                for (int j = 0; j < 8; ++j) sum[j >> 2][j & 3] += acc[j >> 2][j & 3] * sc[8 * (j >> 2) + (j & 1)];
                            }
                            // a lane holds rows lane / 4 and that + 8, columns 2 (lane % 4) and the next of either half: a row's go to its own lane
                            uint32_t y[16];
                            tmem_ld16(own, y);
                            tmem_wait_ld();
#pragma unroll
                            for (int n = 0; n < 16; ++n) {
                                const int src = (lane & 7) * 4 + ((n & 7) >> 1);
                                const float lo = __shfl_sync(0xffffffffu, sum[n >> 3][n & 1], src), hi = __shfl_sync(0xffffffffu, sum[n >> 3][2 + (n & 1)], src);
                                if (ctl->q_exp[r] >= 256u && (lane >> 4) == m) y[n] = __float_as_uint(__uint_as_float(y[n]) + (lane & 8 ? hi : lo));
                            }
                            tmem_st16(own, y);
                            tmem_wait_st();
                        }
                        uint32_t y[16];
                        tmem_ld16(own, y);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 8; ++j) sv[j] = pack2u(y[2 * j], y[2 * j + 1]);
                    }
                    if (kResidual) {
                        tc_fence_before();
                        warp_arrive_lead(&ctl->s_empty[team], lane);
                    }
                    if ((mask & 0xFFFFu) != 0xFFFFu) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            float s0, s1;
                            unpack2(sv[j], s0, s1);
                            sv[j] = pack2(((mask >> (2 * j)) & 1u) ? s0 : -INFINITY, ((mask >> (2 * j + 1)) & 1u) ? s1 : -INFINITY);
                        }
                    }
                    // ---- maximum of this quarter, posted
                    {
                        float t[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            float s0, s1;
                            unpack2(sv[j], s0, s1);
                            t[j] = fmaxf(s0, s1);
                        }
                        ctl->post[team][2 * h + cs][r] = fmaxf(max3(max3(t[0], t[1], t[2]), t[3], t[4]), max3(t[5], t[6], t[7]));
                        warp_arrive(&ctl->posted[team][rq], lane);
                    }
                    // ---- P = 2^(score - reference + 7), the difference taken before it is scaled (rounded products would lie octaves apart from scores of 2^24
                    // on, and P in f16 would overflow; 64 sequences 57.75 -> 58.0 us): at most 2^15; a masked slot gives 0.  Taken against the last reference known while
                    // the other maxima are on their way, and again in the rare case that it has moved
                    const float m_was = m_ref;
                    float m_old = -INFINITY;
                    uint32_t pk[8];
                    float lsum = 0.0f;
                    bool settled = false;
#pragma unroll 1
                    while (true) {
                        if (settled || !first) {
                            const float n = m_ref == -INFINITY ? 0.0f : -m_ref;
                            const uint64_t c2 = pack2(c_log2, c_log2), n2 = pack2(n, n), s2 = pack2(kPShift, kPShift);
                            uint64_t ls2 = pack2(0.0f, 0.0f);
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                float e0, e1;
                                unpack2(fma2(add2(sv[j], n2), c2, s2), e0, e1);
                                e0 = ex2_approx(e0);
                                e1 = ex2_approx(e1);
                                ls2 = add2(ls2, pack2(e0, e1));
                                pk[j] = pack_f16x2(e0, e1);
                            }
                            float l0, l1;
                            unpack2(ls2, l0, l1);
                            lsum = l0 + l1;
                        }
                        if (settled) break;
                        // the row's reference after the tile before this one, and after this one: it moves when the tile's maximum exceeds it by
                        // more than the lazy margin
                        // (before tile 0 the second barrier's phase -1 passes)
                        if (!wait_on2(&ctl->posted[team][rq], ph2, &ctl->moved[team ^ 1][rq], ((it - 1) >> 1) & 1u, abort_flag)) return false;
                        const float mt = fmaxf(fmaxf(ctl->post[team][0][r], ctl->post[team][1][r]), fmaxf(ctl->post[team][2][r], ctl->post[team][3][r]));
                        if (!first) m_old = ctl->m_ref[team ^ 1][r];
                        m_ref = (mt - m_old) * c_log2 > 8.0f ? mt : m_old;
                        if (h == 0 && cs == 0) ctl->m_ref[team][r] = m_ref;
                        warp_arrive(&ctl->moved[team][rq], lane);
                        if (!first && !__any_sync(0xffffffffu, m_ref != m_was)) break;
                        settled = true;
                    }
                    if (l != 0.0f && m_was != m_ref) l *= ex2_approx((m_was - m_ref) * c_log2);
                    l += lsum;
                    if (lent) {   // what V was lent
                        const uint4* back = reinterpret_cast<const uint4*>(&ctl->p_back[ring.s][kOwn * h + 16 * cs]);
                        const uint4 b0 = back[0], b1 = back[1];
                        const uint32_t b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                        for (int j = 0; j < 8; ++j) pk[j] = mul_f16x2(pk[j], b[j]);
                    }
                    if (kResidual || lent) warp_arrive(&ctl->raw_empty[ring.s], lane);
                    // ---- into the P buffer, once the product that read it last is complete
                    if (it >= 2)
                        if (!wait_on(&ctl->pv_done[team], ph2 ^ 1u, abort_flag)) return false;
                    sts_16(p_lo, pk[0], pk[1], pk[2], pk[3]);
                    sts_16(p_lo ^ 16u, pk[4], pk[5], pk[6], pk[7]);
                    fence_proxy_async_smem();
                    if (!first && __any_sync(0xffffffffu, m_ref != m_old || v_fix != 1.0f)) {
                        // the reference or e moved: O so far (complete once the previous tile's product is) is brought to the new ones
                        const float f = (m_old == m_ref ? 1.0f : (m_old == -INFINITY ? 0.0f : ex2_approx((m_old - m_ref) * c_log2))) * v_fix;
                        if (!wait_on(&ctl->pv_done[team ^ 1], ((it - 1) >> 1) & 1u, abort_flag)) return false;
                        tc_fence_after();
#pragma unroll 1
                        for (int oc = 128 * cs; oc < 128 * cs + 128; oc += 16) {
                            uint32_t o[16];
                            tmem_ld16(lane_base + kColO + oc, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                            tmem_st16(lane_base + kColO + oc, o);
                        }
                        tmem_wait_st();
                    }
                    tc_fence_before();
                    warp_arrive_lead(&ctl->p_full[team], lane);
                }
                // ---- the item's sums, last reference and last e
                const uint32_t last = it_end - 1, last_team = last & 1u;
                it_base = it_end;
                if (!wait_on(&ctl->moved[last_team][rq], (last >> 1) & 1u, abort_flag)) return false;   // the posted maxima have been read, too
                const float m_fin = ctl->m_ref[last_team][r];
                if (l != 0.0f && m_ref != m_fin) l *= ex2_approx((m_ref - m_fin) * c_log2);
                ctl->post[team][2 * h + cs][r] = l;
                if (team == static_cast<int>(last_team) && rq == 0 && lane == 0) ctl->v_fin[2 * h + cs] = v_unit;
                warp_arrive(&ctl->e_bar, lane);
                if (!wait_on(&ctl->e_bar, item_n & 1, abort_flag)) return false;
                m_out = m_fin * c_log2;
                ls = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) ls += ctl->post[i >> 2][i & 3][r];
                v_unit = ctl->v_fin[2 * h + team];   // the read-out's 64 columns lie in this group
            }
            return false;
        };
        if (items(std::false_type(), false)) items(std::true_type(), true);
    } else if (warp < kLoadWarp0) {
        setmaxnreg_dec<kRegsIssuers>();
        if (warp < kPvWarp && rank == 0) {
            // ======================================================== score issuers, alternate tiles
            const uint32_t par = warp - kScoreWarp;
            const uint32_t el = elect_one() ? 1u : 0u;
            constexpr uint32_t idesc8 = make_idesc_e4m3(128, kSlots), idesc = make_idesc_bf16(128, kSlots, false);
            const uint64_t q_desc = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
            const uint64_t k_desc0 = make_smem_desc_sw128(smem_u32(sRaw), 16, 1024);
            const uint32_t q_lo = static_cast<uint32_t>(q_desc), q_hi = static_cast<uint32_t>(q_desc >> 32);
            uint32_t it = 0;
            uint32_t ready_bits = 0;   // parities of this issuer's tile_ready
            Ring<kStages> ring;
            int item_n = 0;
            for (int w = w_begin; w < w_end; ++w, ++item_n) {
                const int n_tiles = tiles_of(p.works[w]);
                if (!wait_on(&ctl->q_full, item_n & 1, abort_flag)) goto done;
                for (int t = 0; t < n_tiles; ++t, ++it, ring.next()) {
                    if ((it & 1u) != par) continue;
                    if (!wait_on(&ctl->tile_ready[par][ring.s], (ready_bits >> ring.s) & 1u, abort_flag)) goto done;
                    ready_bits ^= 1u << ring.s;
                    if (it >= 2)
                        if (!wait_on(&ctl->s_empty[par], ((it >> 1) & 1u) ^ 1u, abort_flag)) goto done;
                    tc_fence_after();
                    const uint64_t k_desc = k_desc0 + static_cast<uint64_t>((ring.s * kRawBytes) >> 4);
                    const uint32_t k_lo = static_cast<uint32_t>(k_desc), k_hi = static_cast<uint32_t>(k_desc >> 32);
                    const uint32_t d0 = tmem + kColS + 96 * par;
#pragma unroll 1
                    for (int g = 0; g < kGroups; ++g) {
                        if (g == kGroups - 1) {   // group 3 and the rope have one accumulator each: the tile before has been read
                            if (it >= 1)
                                if (!wait_on(&ctl->s3_empty, (it - 1) & 1u, abort_flag)) goto done;
                            tc_fence_after();
                        }
                        const uint32_t d = g < kGroups - 1 ? d0 + 32 * g : tmem + kColS3;
#pragma unroll
                        for (int v = 0; v < 2; ++v)
                            umma_pair_f8_ss_x4_el(d, q_lo + (((v * kGroups + g) * kQBlock) >> 4), q_hi, k_lo + ((g * kBlock) >> 4), k_hi, v ? idesc8 : idesc8 | kIdescAE5m2, v, el);
                    }
                    umma_pair_ss_x4_el(tmem + kColRope, q_lo + ((2 * kGroups * kQBlock) >> 4), q_hi, k_lo + ((kGroups * kBlock) >> 4), k_hi, idesc, 0u, el);
                    tc_commit_pair_el(smem_u32(&ctl->s_full[par]), el);
                    tc_commit_pair_el(smem_u32(&ctl->raw_empty[ring.s]), el);
                }
                tc_commit_pair_el(smem_u32(&ctl->q_empty), el);
            }
        } else if (warp == kPvWarp && rank == 0) {
            // ======================================================== P V issuer
            const uint32_t el = elect_one() ? 1u : 0u;
            constexpr uint32_t idesc = make_idesc_f16(128, 256, true);
            const uint64_t v_desc0 = make_smem_desc_sw128(smem_u32(sV), kBlock, 1024);   // MN-major: 64-column blocks kBlock apart
            const uint64_t p_desc0 = make_smem_desc_sw128(smem_u32(sP), 16, 1024);
            uint32_t it = 0;
            Ring<kVUnits> unit;
            int item_n = 0;
            for (int w = w_begin; w < w_end; ++w, ++item_n) {
                const int n_tiles = tiles_of(p.works[w]);
                for (int t = 0; t < n_tiles; ++t, ++it) {
                    const uint32_t sb = it & 1u;
                    const uint64_t p_desc = p_desc0 + static_cast<uint64_t>((sb * kPBytes) >> 4);
                    if (t == 0 && item_n > 0)   // the previous item's O has been read out
                        if (!wait_on(&ctl->o_free, (item_n - 1) & 1, abort_flag)) goto done;
                    if (!wait_on(&ctl->p_full[sb], (it >> 1) & 1u, abort_flag)) goto done;
#pragma unroll
                    for (int u = 0; u < 2; ++u, unit.next()) {   // slots of CTA 0, of CTA 1
                        if (!wait_on(&ctl->v_full[unit.s], unit.ph, abort_flag)) goto done;
                        tc_fence_after();
                        const uint64_t v_desc = v_desc0 + static_cast<uint64_t>((unit.s * kVUnit) >> 4);
#pragma unroll
                        for (int ks = 0; ks < 2; ++ks)
#pragma unroll
                            for (int j = 0; j < 2; ++j)
                                umma_pair_ss_el(tmem + kColO + 128 * j, p_desc + static_cast<uint64_t>((2 * u + ks) * 2),
                                                v_desc + static_cast<uint64_t>((2 * j * kBlock + ks * 2048) >> 4), idesc, (t > 0 || u > 0 || ks > 0) ? 1u : 0u, el);
                        tc_commit_pair_el(smem_u32(&ctl->v_empty[unit.s]), el);
                    }
                    tc_commit_pair_el(smem_u32(&ctl->pv_done[sb]), el);
                    if (t + 1 == n_tiles) tc_commit_pair_el(smem_u32(&ctl->o_full), el);
                }
            }
        } else if (warp == kReadyWarp) {
            // ======================================================== this CTA's rows' arrival, passed on to the issuers; e
            uint32_t it = 0;
            Ring<kStages> ring;
            int e = 0, e_most = 0;   // lane: those of group lane % 4; the largest of the item
            for (int w = w_begin; w < w_end; ++w) {
                const int n_tiles = tiles_of(p.works[w]);
                for (int t = 0; t < n_tiles; ++t, ++it, ring.next()) {
                    if (!warp_wait(smem_u32(&ctl->kv_full[ring.s]), ring.ph, abort_flag)) goto done;
                    fence_proxy_async_smem();   // written by cp.async (generic proxy)
                    warp_arrive_lead(&ctl->tile_ready[it & 1u][ring.s], lane);
                    // exponents of the scales of slots 2 lane (low half) and 2 lane + 1 (biased; 0: none that counts)
                    uint32_t a[kGroups];
#pragma unroll
                    for (int g = 0; g < kGroups; ++g) {
                        const float2 s = *reinterpret_cast<const float2*>(&ctl->scale[ring.s][g][2 * lane]);
                        const uint32_t x = (__float_as_uint(s.x) >> 23) & 0xFFu, y = (__float_as_uint(s.y) >> 23) & 0xFFu;
                        a[g] = (x < 255u ? x : 0u) | (y < 255u ? y : 0u) << 16;
                    }
                    const int e_old = e;
                    int x0, x1;   // octaves that the two rows take more than 2^-e
                    bool lent;
#pragma unroll 1
                    for (bool looked = false;; looked = true) {
                        // the largest of the tile's rows (of both CTAs' slots, so both CTAs follow the same e)
                        uint32_t top = 0u;
#pragma unroll
                        for (int g = 0; g < kGroups; ++g) {
                            const uint32_t m = __reduce_max_sync(0xffffffffu, max(a[g] & 0xFFFFu, a[g] >> 16));
                            if ((lane & 3) == g) top = m;
                        }
                        const int em = max(static_cast<int>(top) - 127, -120);
                        // (down only from far, and not so far that O, brought to the new e, could overflow)
                        e = t == 0 || em >= e_old + 7 ? min(em, 126) : top != 0u && em + 24 <= e_old ? min(max(em, e_most - 60), e_old) : e_old;
                        // how far a row's groups lie below their e, 512 added: the least and the most of them
                        uint32_t low = 0xFFFFFFFFu, deep = 0u;
#pragma unroll
                        for (int g = 0; g < kGroups; ++g) {
                            const uint32_t d = __shfl_sync(0xffffffffu, (e + 127 + 512) * 0x10001, g) - a[g];
                            const uint32_t counts = (((a[g] + 0x00FF00FFu) >> 8) & 0x00010001u) * 0xFFFFu;   // (a is not 0)
                            low = min_u16x2(low, d | ~counts);
                            deep = max_u16x2(deep, d & counts);
                        }
                        x0 = (low & 0xFFFFu) == 0xFFFFu ? 0 : min(max(static_cast<int>(low & 0xFFFFu) - (512 + 16), 0), 20);
                        x1 = (low >> 16) == 0xFFFFu ? 0 : min(max(static_cast<int>(low >> 16) - (512 + 16), 0), 20);
                        lent = __any_sync(0xffffffffu, max(deep & 0xFFFFu, deep >> 16) > 520u);
                        if (!lent || looked) break;
                        const int y0 = static_cast<int>(deep & 0xFFFFu) - x0, y1 = static_cast<int>(deep >> 16) - x1;
                        if (!__any_sync(0xffffffffu, max(y0, y1) > 512 + 18)) break;
                        // A group of some row would lose bits.  The reason may be a group of zeros under any scale, in that row or in another (the cache
                        // writer gives it 1): its scale does not count and becomes 0 (f16 may not hold what is left of it).
#pragma unroll 1   // (four at a time: 128 sequences of 2 x 16 heads 142.3 -> 151.3 us, by their code alone)
                        for (int slot = 0; slot < kSlots; ++slot) {
                            // sixteen bytes a lane, eight lanes a group
                            uint4 v = make_uint4(0u, 0u, 0u, 0u);
                            const int late = ctl->late_row[ring.s][slot % kOwn];
                            if (slot / kOwn == rank) v = *reinterpret_cast<const uint4*>(sRaw + ring.s * kRawBytes + (lane >> 3) * kBlock + (slot % kOwn) * 128 + 16 * (lane & 7));
                            else if (late >= 0) v = ldg_stream_16(reinterpret_cast<const uint8_t*>(p.kv) + (size_t)late * kFp8RowBytes + 16 * lane);
                            const uint32_t full = __ballot_sync(0xffffffffu, ((v.x | v.y | v.z | v.w) & 0x7F7F7F7Fu) != 0u), half = slot & 1 ? 0xFFFF0000u : 0xFFFFu;
#pragma unroll
                            for (int g = 0; g < kGroups; ++g)
                                if (((full >> (8 * g)) & 0xFFu) == 0u && lane == slot >> 1 && (a[g] & half) != 0u) {
                                    a[g] &= ~half;
                                    ctl->scale[ring.s][g][slot] = 0.0f;
                                }
                        }
                    }
                    e_most = t == 0 ? e : max(e_most, e);
                    if (lent) {
                        *reinterpret_cast<float2*>(&ctl->v_lent[ring.s][2 * lane]) = make_float2(__uint_as_float((127 + x0) << 23), __uint_as_float((127 + x1) << 23));
                        reinterpret_cast<uint32_t*>(ctl->p_back[ring.s])[lane] = pow2_f16(-x0) | pow2_f16(-x1) << 16;
                    }
                    if (lane < kGroups) {
                        const int d = t == 0 ? 0 : e_old - e;
                        ctl->v_move[ring.s][lane] = make_float2(d < -126 ? 0.0f : __uint_as_float(static_cast<uint32_t>(127 + d) << 23), __uint_as_float(static_cast<uint32_t>(127 + e) << 23));
                        ctl->v_mul[ring.s][lane] = make_float2(__uint_as_float(static_cast<uint32_t>(127 - e) << 23), lent ? 1.0f : 0.0f);
                    }
                    warp_arrive(&ctl->prep[ring.s], lane);
                }
            }
            if (!warp_wait(smem_u32(&ctl->finished), 0, abort_flag)) goto done;
        }
    } else if (warp < kConvWarp0) {
        // ============================================================ row loaders: eight rows of every tile per warp, four lanes per row
        setmaxnreg_dec<kRegsLoaders>();
        const int lw = warp - kLoadWarp0;
        const int r = 8 * lw + (lane >> 2), c4 = lane & 3;   // of the copies
        const uint8_t* kv_bytes = reinterpret_cast<const uint8_t*>(p.kv);
        // lanes 0-7 follow the slots of the warp's own rows in even tiles, 8-15 the same slots of the other CTA, 16-31 those of odd tiles:
        // a slot is translated once, two tiles at a time
        const int slot = kSlots * (lane >> 4) + kOwn * ((lane >> 3 & 1) ? peer : rank) + 8 * lw + (lane & 7);
        const uint32_t d0 = smem_u32(sRaw) + r * 128 + ((c4 ^ (r & 7)) << 4), d1 = d0 ^ 64u;   // chunks 8 j + c4 and 8 j + 4 + c4
        const uint32_t scale_own = smem_u32(&ctl->scale[0][c4][kOwn * rank + r]), scale_late = smem_u32(&ctl->scale[0][c4][kOwn * peer + r]);
        Ring<kStages> ring;   // of raw_empty: one use behind
        ring.ph = 1u;
        for (int w = w_begin; w < w_end; ++w) {
            const dsa_v32_work_info wi = p.works[w];
            const int n_tiles = tiles_of(wi);
            const int seq = wi.q_row / p.s_q;
            const int32_t* idx_row = p.indices + (size_t)wi.q_row * p.topk;
            auto load_slot = [&](int u) -> int {
                const int k = wi.k_begin + u * kSlots + slot;
                return (k < wi.k_end) ? __ldg(idx_row + k) : -1;
            };
            // rows are known two tiles ahead (and asked into L2), block numbers loaded four, slots six
            auto ask = [&](int row) {
                if ((lane & 8) == 0 && row >= 0) bulk_prefetch_l2(kv_bytes + (size_t)row * kFp8RowBytes, kFp8RowBytes);
            };
            int idx_a = load_slot(0), idx_b = load_slot(2), idx_c = load_slot(4);
            int phys_a = block_of(idx_a, seq, p), phys_b = block_of(idx_b, seq, p);
            int row_n = row_of(idx_a, phys_a, seq, p);
#pragma unroll 1
            for (int u = 0; u < n_tiles; u += 2) {
                const int row = row_n;
                row_n = row_of(idx_b, phys_b, seq, p);
                ask(row_n);
                idx_b = idx_c;
                phys_b = block_of(idx_b, seq, p);
                idx_c = load_slot(u + 6);
                const uint32_t used = __ballot_sync(0xffffffffu, row != -1);
#pragma unroll 1
                for (int t = 0; t < 2 && u + t < n_tiles; ++t, ring.next()) {
                    const int own = __shfl_sync(0xffffffffu, row, 16 * t + (lane >> 2)), late = __shfl_sync(0xffffffffu, row, 16 * t + 8 + (lane >> 2));
                    if (!wait_on(&ctl->raw_empty[ring.s], ring.ph, abort_flag)) goto done;
                    if (c4 == 0) ctl->late_row[ring.s][r] = late;
                    warp_arrive(&ctl->late_known[ring.s], lane);
                    if (lane < 2) reinterpret_cast<uint8_t*>(&ctl->tile_mask[ring.s][lane ? peer : rank])[lw] = static_cast<uint8_t>(used >> (16 * t + 8 * lane));
                    // padding and out-of-range rows: nothing is read, the row is zeros
                    const uint32_t st = ring.s * kRawBytes, sc = ring.s * (kGroups * kSlots * 4);
                    {
                        const uint8_t* src = kv_bytes + (size_t)(own < 0 ? 0 : own) * kFp8RowBytes;
                        const uint32_t n = own != -1 ? 16u : 0u;
                        cp_async_4(scale_own + sc, src + kDV + 4 * c4, n >> 2);
                        src += 16 * c4;
#pragma unroll
                        for (int j = 0; j < 5; ++j) {   // four blocks of latent columns; the rope, after 16 bytes of scales
                            cp_async_16(d0 + st + j * kBlock, src + 128 * j + (j == 4 ? 16 : 0), n);
                            cp_async_16(d1 + st + j * kBlock, src + 128 * j + (j == 4 ? 16 : 0) + 64, n);
                        }
                    }
                    cp_async_4(scale_late + sc, kv_bytes + (size_t)(late < 0 ? 0 : late) * kFp8RowBytes + kDV + 4 * c4, late != -1 ? 4u : 0u);
                    cp_async_mbar_arrive_noinc(smem_u32(&ctl->kv_full[ring.s]));
                    warp_arrive(&ctl->kv_full[ring.s], lane);
                }
            }
        }
    } else {
        // ============================================================ converters: this CTA's 256 output columns of all 64 rows, to f16
        // Warps 0-3 take the slots of CTA 0 (unit 0 of a tile), warps 4-7 those of CTA 1, eight rows each.  Own rows lie in shared memory, the
        // other CTA's come from L2 through registers, a tile ahead.  Sixteen columns a lane and step: one 16-byte chunk of a row of the cache, two of a
        // row of V.  A quarter of a warp takes half of a block's columns of one row and the other half of its neighbour's, so that its loads and
        // its stores touch every bank once.
        const int cw = warp - kConvWarp0, u = cw >> 2;
        const int r4 = 2 * (lane >> 4) + ((lane >> 2) & 1), half = ((lane >> 3) ^ (lane >> 2)) & 1, k = lane & 3;
        const int r = 8 * (cw & 3) + r4;   // of the first two steps; the others take the row four further
        const uint32_t v0 = smem_u32(sV) + half * kBlock + r * 128 + (((2 * k) ^ (r & 7)) << 4);
        // lane i < 16 (and i + 16): the scale of block i / 8, row i % 8
        const int sg = 2 * rank + ((lane >> 3) & 1), ss = kOwn * u + 8 * (cw & 3) + (lane & 7);
        // ... times 2^-e as a sum of two f16 with 22 significant bits, and, where that takes more than f16's range, the power of two that the bytes are
        // multiplied with before (exact)
        uint32_t scales = 0u, pre = 0u;
        bool lent = false;
        auto load_scale = [&](uint32_t st) {
            const float2 m = ctl->v_mul[st][sg];
            float f = ctl->scale[st][sg][ss] * m.x;
            lent = __any_sync(0xffffffffu, m.y != 0.0f);   // (a vote, so that it is known to be the same in all lanes)
            if (lent) {
                f *= ctl->v_lent[st][ss];
                const int k = min(max(123 - static_cast<int>((__float_as_uint(f) >> 23) & 0xFFu), 0), 15);
                f *= __uint_as_float((127 + k) << 23);
                pre = pow2_f16(-k) * 0x10001u;
            }
            scales = split_f16(f);
        };
        // one chunk of either block of a row, scaled, to V
        auto convert = [&](const uint4 (&x)[2], int i, uint32_t dst) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const uint32_t s = __shfl_sync(0xffffffffu, scales, 8 * b + 4 * i + r4);
                const uint32_t hi = __byte_perm(s, 0, 0x1010), lo = __byte_perm(s, 0, 0x3232);
                const uint32_t v[4] = {x[b].x, x[b].y, x[b].z, x[b].w};
                uint32_t y[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] = e4m3x2_to_f16x2(v[j >> 1] >> (16 * (j & 1)));
                if (lent) {
                    const uint32_t m = __shfl_sync(0xffffffffu, pre, 8 * b + 4 * i + r4);
#pragma unroll
                    for (int j = 0; j < 8; ++j) y[j] = mul_f16x2(y[j], m);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] = scale_f16x2(y[j], hi, lo);
                sts_16(dst + 2 * b * kBlock, y[0], y[1], y[2], y[3]);
                sts_16((dst ^ 16u) + 2 * b * kBlock, y[4], y[5], y[6], y[7]);
            }
        };
        Ring<kStages> ring;
        Ring<kVUnits> unit;   // of v_empty: one use behind
        unit.ph = 1u;
        if (u) unit.next();
        if (u == rank) {
            setmaxnreg_dec<kRegsConv>();
            const uint32_t raw0 = smem_u32(sRaw) + 2 * rank * kBlock + r * 128 + (((4 * half + k) ^ (r & 7)) << 4);
            for (int w = w_begin; w < w_end; ++w) {
                const int n_tiles = tiles_of(p.works[w]);
#pragma unroll 1
                for (int t = 0; t < n_tiles; ++t, ring.next(), unit.next(), unit.next()) {
                    if (!wait_on2(&ctl->prep[ring.s], ring.ph, &ctl->v_empty[unit.s], unit.ph, abort_flag)) goto done;
                    load_scale(ring.s);
                    uint32_t src = raw0 + ring.s * kRawBytes, dst = v0 + unit.s * kVUnit;
                    uint4 x[2] = {lds_16(src), lds_16(src + kBlock)};
#pragma unroll 1
                    for (int i = 0; i < 2; ++i) {   // row r, row r + 4: a short loop, see warp_wait_short
                        const uint4 cur[2] = {x[0], x[1]};
                        src = (src ^ 64u) + 512u;   // four rows on, and bit 2 of the swizzle flips
                        if (i == 0) {
                            x[0] = lds_16(src);
                            x[1] = lds_16(src + kBlock);
                        } else {
                            warp_arrive(&ctl->raw_empty[ring.s], lane);
                        }
                        convert(cur, i, dst);
                        dst = (dst ^ 64u) + 512u;
                    }
                    fence_proxy_async_smem();
                    warp_arrive_lead(&ctl->v_full[unit.s], lane);
                }
            }
        } else {
            setmaxnreg_dec<kRegsLate>();
            const uint8_t* const kv0 = reinterpret_cast<const uint8_t*>(p.kv) + rank * kDvHalf + (4 * half + k) * 16;
            auto load = [&](uint4 (&x)[2], int row) {
                x[0] = x[1] = make_uint4(0u, 0u, 0u, 0u);
                if (row >= 0) {
                    const uint8_t* src = kv0 + (size_t)row * kFp8RowBytes;
                    x[0] = ldg_stream_16(src);
                    x[1] = ldg_stream_16(src + 128);
                }
            };
            Ring<kStages> known;   // of the tile whose rows are fetched
            for (int w = w_begin; w < w_end; ++w) {
                const int n_tiles = tiles_of(p.works[w]);
                uint4 x[2][2];
                if (!wait_on(&ctl->late_known[known.s], known.ph, abort_flag)) goto done;
                load(x[0], ctl->late_row[known.s][r]);
                load(x[1], ctl->late_row[known.s][r + 4]);
                known.next();
#pragma unroll 1
                for (int t = 0; t < n_tiles; ++t, ring.next(), unit.next(), unit.next()) {
                    int next0 = -1, next1 = -1;
                    if (t + 1 < n_tiles) {
                        if (!wait_on(&ctl->late_known[known.s], known.ph, abort_flag)) goto done;
                        next0 = ctl->late_row[known.s][r];
                        next1 = ctl->late_row[known.s][r + 4];
                        known.next();
                    }
                    if (!wait_on2(&ctl->prep[ring.s], ring.ph, &ctl->v_empty[unit.s], unit.ph, abort_flag)) goto done;
                    load_scale(ring.s);
                    const uint32_t dst = v0 + unit.s * kVUnit;
                    convert(x[0], 0, dst);
                    load(x[0], next0);
                    warp_arrive(&ctl->raw_empty[ring.s], lane);
                    convert(x[1], 1, (dst ^ 64u) + 512u);
                    load(x[1], next1);
                    fence_proxy_async_smem();
                    warp_arrive_lead(&ctl->v_full[unit.s], lane);
                }
            }
        }
    }
    if (warp != kReadyWarp) warp_arrive(&ctl->finished, lane);

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
template <bool kExt, int kShare>
static cudaError_t configure() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> guard(mu);
    if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(paired_fp8_kernel<kExt, kShare>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
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

template <bool kExt, int kShare>
static cudaError_t launch(int num_lists, const AttnParams& p, cudaStream_t stream) {
    cudaError_t e = configure<kExt, kShare>();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    fill_launch(&cfg, attr, num_lists, stream);
    return cudaLaunchKernelEx(&cfg, paired_fp8_kernel<kExt, kShare>, p);
}

}  // namespace paired_fp8

int max_resident_pairs_fp8(int* out) {
    cudaError_t e = paired_fp8::configure<false, paired_fp8::kRows>();
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    int n = 0;
    paired_fp8::fill_launch(&cfg, attr, 1, nullptr);
    e = cudaOccupancyMaxActiveClusters(&n, paired_fp8::paired_fp8_kernel<false, paired_fp8::kRows>, &cfg);
    if (e != cudaSuccess) return (int)e;
    *out = n;
    return 0;
}

// ext: a sink or peers are given, rows are stacked, or rows of out are aligned to 16 bytes only; tile_rows: the most rows an item of the plan has
cudaError_t launch_paired_fp8(bool ext, int tile_rows, int num_lists, const AttnParams& p, cudaStream_t stream) {
    using namespace paired_fp8;
    if (tile_rows > kRows) return ext ? launch<true, kRows>(num_lists, p, stream) : launch<false, kRows>(num_lists, p, stream);
    return ext ? launch<true, kRows / 2>(num_lists, p, stream) : launch<false, kRows / 2>(num_lists, p, stream);
}

}  // namespace dsa
