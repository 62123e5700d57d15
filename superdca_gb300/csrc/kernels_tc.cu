// kernels_tc.cu -- the tensor-core contraction form (tcgen05, sm_103a).
//
// Both contractions of an L-BFGS iteration are one-hot GEMMs, C = A . B^T with
// A the one-hot expansion of the alignment and B the per-slot operand:
//
//   forward   u[i][p*4+a]      = sum_{k=n*4+s} [X_in == s] * D_p[a][k]   (A: N x 4L)
//   backward  G[n*4+s][p*4+a]  = sum_i [X_in == s] * R_p[a][i]           (A: 4L x N)
//
// which are SuperDCA's gather (plmDCA_objective.hpp:86-121) and gradient
// scatter (plmDCA_objective.hpp:153-190) for a batch of target loci.
//
// Data path per CTA (128 x 128 output tile, K in steps of 64):
//   * warps 0 and 2, one thread each: TMA loads of the u8 state tiles (2 KB
//     per 128 rows) and of the fp16 hi and lo tiles of B (128 B swizzle);
//   * warps 3-10: expand the u8 tile to the fp16 one-hot A tile directly in the
//     128-byte-swizzled K-major layout the MMA reads (the one-hot matrix never
//     exists in HBM: 1 byte per locus is read instead of 8), fence to the async
//     proxy, arrive on full_a[s];
//   * warp 1, uniformly, its elected lane issuing: tcgen05.mma kind::f16 (M128
//     K16, N fitted to the live columns, FP32 accumulators in TMEM): A x B_hi and then A x B_lo into the same
//     accumulator (or, with exact fp16 operands, a second N tile in the lo
//     slot); tcgen05.commit frees the stage;
//   * warps 11-14: tcgen05.ld the accumulator and store it, scaled back
//     by the per-slot power of two.
// With hi + lo operands the backward keeps the expanded A tiles in TMEM
// instead (tcgen05.st by the expansion warps, MMAs reading A from TMEM; see
// Cfg below).
// B is split as hi + lo fp16 halves of (value * 2^e) so that the product keeps
// about 22 significant bits; the one-hot A is exact in fp16.
//
// Every mbarrier wait is bounded: on timeout the kernel records an error code
// in *err and skips the remaining work instead of spinning.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "df.cuh"
#include "engine.h"
#include "kdig.cuh"
#include "kernels_common.cuh"
#include "tcgen05.cuh"

namespace sdca {
namespace tc {

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;   // one 128-row one-hot subtile
constexpr int B_BYTES = BN * BK * 2;   // one fp16 half (hi or lo) of the slot operand
constexpr int RAW_BYTES = 2048;        // u8 states behind one subtile
constexpr int B_BOX = 32;              // slot-operand rows per TMA box: a tile loads its live rows only
constexpr int THREADS = 96 + 256 + 128;   // two TMA, one MMA, eight expansion and four epilogue warps

// A CTA owns MSUB consecutive 128-row subtiles and reuses each staged B tile
// for all of them: the slot operand is the traffic that the L2 has to carry,
// once per CTA per k-step.  TMEM holds one 128-column accumulator per subtile
// and N tile.  NT = 2 (slot operands exact in fp16, no lo half): the stage's
// lo slot carries a second N tile, so every expanded one-hot tile feeds two
// MMAs per K16 step, as it does for hi + lo.
//
// AT (backward only): the one-hot A tiles live in TMEM instead of shared
// memory.  The expansion warps write them with tcgen05.st (row m of a
// subtile in TMEM lane m, sequence pairs (2j, 2j+1) in column j as the low
// and high halves) and the MMAs read A from TMEM, so shared memory carries
// only the slot operand and the u8 state tiles: an M128 N128 K16 MMA with
// both operands in shared memory reads 8 KB per 64 cycles, which with the
// expansion's stores and the TMA writes is more than the 128 bytes per
// cycle shared memory delivers.  TMEM then holds the accumulators
// (MSUB x NT x 128 columns) and STG stages of MSUB A subtiles (32 columns
// each: 64 sequences).
// The state tiles have a ring of their own, deeper than the stages of A and
// B: they come from HBM, and a stage that waited for its state tile only
// after the MMAs had released it spent most of its time on that latency (a
// check pass of 8 slots: 24k of 39k cycles a CTA waiting for state tiles).
template <int MSUB, int STG, int NT = 1, bool AT = false> struct Cfg {
    static constexpr int STAGE_BYTES = (AT ? 0 : MSUB * A_BYTES) + 2 * B_BYTES;
    static constexpr int RAW_STG = AT ? 16 : 16 / MSUB;          // state-tile stages
    static constexpr int RAW_STAGE = MSUB * RAW_BYTES;
    static constexpr int BARS = 2 * RAW_STG + 3 * STG + 5;       // barriers and the TMEM address
    static constexpr int SMEM_BYTES = STG * STAGE_BYTES + RAW_STG * RAW_STAGE + 1024 /*align*/ + 8 * BARS + 64;
    static constexpr uint32_t ACC_COLS = MSUB * BN * NT;
    static constexpr uint32_t A_COLS = AT ? MSUB * (BK / 2) * STG : 0;
    static constexpr uint32_t TMEM_COLS = AT ? 512 : ACC_COLS;
    static_assert(STAGE_BYTES % 1024 == 0, "stage must keep 1024-byte alignment");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");
    static_assert(ACC_COLS + A_COLS <= 512, "TMEM holds 512 columns");
    static_assert(NT == 1 || NT == 2, "one or two N tiles per CTA");
};

enum { MODE_FWD = 0, MODE_BWD = 1 };

// instruction descriptor, kind::f16: A = B = F16, D = F32, K-major, M = 128, N = 128
constexpr uint32_t IDESC = (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(BM >> 4) << 24);

// (the elected lane's; descriptors by their low words)
__device__ __forceinline__ void mma_f16(uint32_t lead, uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                        uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 e, %6, 0;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(tmem_d),
        "r"(a_lo), "r"(b_lo), "r"(SMEM_DESC_HI), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}

// the same MMA with A read from TMEM (column tmem_a, lanes 0-127)
__device__ __forceinline__ void mma_f16_ts(uint32_t lead, uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo,
                                           uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 db;\n\t"
        "setp.ne.b32 e, %6, 0;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "r"(b_lo), "r"(SMEM_DESC_HI), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}

// kind::f16 descriptor with N = the live columns of a tile rounded up to 16
// (at most BN): a partly filled last N tile issues only the MMA work it needs
__device__ __forceinline__ uint32_t idesc_fit(int cols)
{
    const int n = cols >= BN ? BN : (cols < 16 ? 16 : (cols + 15) / 16 * 16);
    return (IDESC & ~(0x3Fu << 17)) | ((uint32_t)(n >> 3) << 17);
}

// 32 consecutive TMEM columns of this warp's 32 lanes from 32 registers per thread
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
        "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
        "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

// fp16 1.0 in lane s of four 16-bit lanes
__device__ __forceinline__ uint64_t onehot4(uint32_t s)
{
    return (uint64_t)0x3C00u << (16u * (s & 3u));
}

// forward: raw = 128 rows x 16 loci (u8); A row r = sequence, K = locus*4+state
__device__ __forceinline__ void expand_fwd(const uint8_t *raw, uint32_t a_base, int t)
{
    const uint4 w = *reinterpret_cast<const uint4 *>(raw + t * 16);
    const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const uint32_t wd = words[c >> 1];
        const uint32_t s0 = (wd >> (16 * (c & 1))) & 0xFF, s1 = (wd >> (16 * (c & 1) + 8)) & 0xFF;
        const uint64_t lo = onehot4(s0), hi = onehot4(s1);
        st_shared_v4(sw128(a_base, t, c),
                     make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32)));
    }
}

// four bytes (states 0..3) -> four fp16 lanes holding 1.0 where the byte
// equals s: the byte's two bits against s, 0x3C per equal byte, and each byte
// moved to the high half of its fp16 lane
__device__ __forceinline__ uint2 eq_halves(uint32_t bytes, uint32_t s4)
{
    const uint32_t t = bytes ^ s4;
    const uint32_t m = (~(t | (t >> 1)) & 0x01010101u) * 0x3Cu;
    return make_uint2(__byte_perm(m, 0u, 0x1404), __byte_perm(m, 0u, 0x3424));
}

// backward, A in TMEM: row t's 64 one-hot values as 32 sequence pairs
// (low half: the even sequence), the column order of the TMEM A operand
__device__ __forceinline__ void expand_bwd_regs(const uint8_t *raw, int t, uint32_t (&o)[32])
{
    const int nl = t >> 2;
    const uint32_t s4 = (uint32_t)(t & 3) * 0x01010101u;
    const uint4 *rp = reinterpret_cast<const uint4 *>(raw + nl * 64);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint4 w = rp[q];
        const uint2 e0 = eq_halves(w.x, s4), e1 = eq_halves(w.y, s4);
        const uint2 e2 = eq_halves(w.z, s4), e3 = eq_halves(w.w, s4);
        o[8 * q + 0] = e0.x;
        o[8 * q + 1] = e0.y;
        o[8 * q + 2] = e1.x;
        o[8 * q + 3] = e1.y;
        o[8 * q + 4] = e2.x;
        o[8 * q + 5] = e2.y;
        o[8 * q + 6] = e3.x;
        o[8 * q + 7] = e3.y;
    }
}

// backward: raw = 32 loci x 64 sequences (u8); A row r = locus*4+state, K = sequence
__device__ __forceinline__ void expand_bwd(const uint8_t *raw, uint32_t a_base, int t)
{
    const int nl = t >> 2;
    const uint32_t s4 = (uint32_t)(t & 3) * 0x01010101u;
    const uint4 *rp = reinterpret_cast<const uint4 *>(raw + nl * 64);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint4 w = rp[q];
        const uint2 e0 = eq_halves(w.x, s4), e1 = eq_halves(w.y, s4);
        const uint2 e2 = eq_halves(w.z, s4), e3 = eq_halves(w.w, s4);
        st_shared_v4(sw128(a_base, t, 2 * q), make_uint4(e0.x, e0.y, e1.x, e1.y));
        st_shared_v4(sw128(a_base, t, 2 * q + 1), make_uint4(e2.x, e2.y, e3.x, e3.y));
    }
}

struct GemmArgs {
    int mode;
    int kt_begin_stride;  // k-tiles per split
    int kt_total;
    int m_groups, n_groups, splits;   // tiles: groups of MSUB subtiles x groups of NT N tiles x K splits
    int m_rows;           // valid output rows (N for forward, 4L for backward)
    int nlist;
    const int32_t *list;  // list position -> slot
    const SlotDev *sd;
    float inv_scale_fwd;  // unused when per-slot scales are read from sd
    // forward output: partial[split][slot][Nx] float4
    float4 *partial;
    int Bmax;
    int64_t Nx;
    // backward output: raw gradient into the slot's new-gradient buffer
    float *gpool;
    int64_t Dp;
    float inv_scale_bwd;
    int hi_only;          // the slot operand is exact in fp16 (its lo half is zero): skip the lo MMA
    // backward, max only: instead of writing the gradient, each slot's
    // max |g| over the blocks n != locus goes to gmax_acc[slot * gmax_stride]
    // (non-negative double bits, atomicMax)
    double *gmax_acc;
    int gmax_stride;
    // backward, digit planes: the list holds nslot slots and the B operand
    // planes x nslot virtual columns (plane d of list position s at virtual
    // position d * nslot + s); virtual position P is written to gpool buffer P
    int planes, nslot;
    int *err;
};

template <int MSUB, int STG, int NT, bool AT = false>
__global__ void __launch_bounds__(THREADS, 1)
k_gemm(const __grid_constant__ CUtensorMap tmRaw, const __grid_constant__ CUtensorMap tmBhi,
       const __grid_constant__ CUtensorMap tmBlo, const GemmArgs args)
{
    using C = Cfg<MSUB, STG, NT, AT>;
    constexpr int SB = C::STAGE_BYTES, RST = C::RAW_STG;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase0 = smem_u32(smem_raw);
    const uint32_t sbase = (sbase0 + 1023u) & ~1023u;
    uint8_t *const sgen = smem_raw + (sbase - sbase0);
    const uint32_t raws = sbase + STG * SB, bars = raws + RST * C::RAW_STAGE;
    // stage layout: [A subtiles (not with AT) | B hi | B lo]; then the state-tile ring
    constexpr uint32_t BHI = AT ? 0 : MSUB * A_BYTES, BLO = BHI + B_BYTES;
    // barriers: state tile landed / read, slot operand landed, A expanded,
    // stage free (its MMAs are done), accumulators complete / read; TMEM address
    auto full_raw = [&](int r) { return bars + 8u * r; };
    auto free_raw = [&](int r) { return bars + 8u * (RST + r); };
    auto full_b = [&](int s) { return bars + 8u * (2 * RST + s); };
    auto full_a = [&](int s) { return bars + 8u * (2 * RST + STG + s); };
    auto empty = [&](int s) { return bars + 8u * (2 * RST + 2 * STG + s); };
    auto acc_full = [&](int u) { return bars + 8u * (2 * RST + 3 * STG + u); };
    auto acc_free = [&](int u) { return bars + 8u * (2 * RST + 3 * STG + 2 + u); };
    const uint32_t tmem_slot = bars + 8u * (2 * RST + 3 * STG + 4);
    uint32_t *tmem_slot_gen = reinterpret_cast<uint32_t *>(sgen + (tmem_slot - sbase));

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // (warp: uniform)
    // The CTA's share of the tiles (output subtile group, N tile, K split), in
    // turn.  Every role walks them with its own counters through the rings, so
    // the state tiles of the next tile load and expand while the last one is
    // in its epilogue: with one tile per CTA, 10 us of launch, set-up, first
    // loads and epilogue stood beside each tile's 4 us of work at 616 sequences.
    const int tiles = args.m_groups * args.n_groups * args.splits;
    // live columns of a tile's N tiles (4 per list position) and the TMA
    // boxes that hold them: a check pass of 8 slots (32 columns) loads a
    // quarter of what a full tile takes
    struct Tile {
        int m_group, n_tile, split, kt0, nkt, cols0, cols1, boxes0, boxes1;
    };
    auto tile_at = [&](int i) {
        Tile T;
        T.m_group = i % args.m_groups;
        const int rest = i / args.m_groups;
        T.n_tile = rest % args.n_groups * NT;
        T.split = rest / args.n_groups;
        T.kt0 = T.split * args.kt_begin_stride;
        T.nkt = max(0, min(args.kt_total, T.kt0 + args.kt_begin_stride) - T.kt0);
        T.cols0 = min(BN, 4 * args.nlist - T.n_tile * BN);
        T.cols1 = min(BN, 4 * args.nlist - (T.n_tile + 1) * BN);
        T.boxes0 = max(0, (T.cols0 + B_BOX - 1) / B_BOX);
        T.boxes1 = max(0, (T.cols1 + B_BOX - 1) / B_BOX);
        return T;
    };
    constexpr int BOX_BYTES = B_BOX * BK * 2;
    // with at most 64 live columns a subtile's 128 accumulator columns hold
    // two tiles' sums: the MMAs of one run during the epilogue of the other
    const int nbuf = NT == 1 && 4 * args.nlist <= BN / 2 ? 2 : 1;

    if (threadIdx.x == 0) {
        for (int r = 0; r < RST; ++r) {
            mbar_init(full_raw(r), 1);
            mbar_init(free_raw(r), 8);
        }
        for (int s = 0; s < STG; ++s) {
            mbar_init(full_b(s), 1);
            mbar_init(full_a(s), 256);
            mbar_init(empty(s), 1);
        }
        for (int u = 0; u < 2; ++u) {
            mbar_init(acc_full(u), 1);
            mbar_init(acc_free(u), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot),
                     "r"(C::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot_gen, 0);   // (uniform)
    bool failed = false;

    if (warp == 0) {
        if (lane == 0) {   // state tiles
            int it = 0;
            for (int i = blockIdx.x; i < tiles && !failed; i += gridDim.x) {
                const Tile T = tile_at(i);
                for (int j = 0; j < T.nkt; ++j, ++it) {
                    const int r = it % RST, kt = T.kt0 + j;
                    if (!mbar_wait(free_raw(r), (uint32_t)((it / RST) & 1) ^ 1u)) { failed = true; break; }
                    mbar_expect_tx(full_raw(r), C::RAW_STAGE);
#pragma unroll
                    for (int ms = 0; ms < MSUB; ++ms) {
                        const int mt = T.m_group * MSUB + ms;
                        const uint32_t dst = raws + (uint32_t)(r * C::RAW_STAGE + ms * RAW_BYTES);
                        if (args.mode == MODE_FWD) tma_load_2d(dst, &tmRaw, kt * 16, mt * BM, full_raw(r));
                        else tma_load_2d(dst, &tmRaw, kt * BK, mt * 32, full_raw(r));
                    }
                }
            }
            // loads still in flight land before the block retires
            for (int k = max(0, it - RST); k < it; ++k)
                if (!mbar_wait(full_raw(k % RST), (uint32_t)((k / RST) & 1))) failed = true;
        }
    } else if (warp == 2) {
        if (lane == 0) {   // the slot operand
            int it = 0;
            for (int i = blockIdx.x; i < tiles && !failed; i += gridDim.x) {
                const Tile T = tile_at(i);
                const int lo_boxes = NT == 2 ? T.boxes1 : args.hi_only ? 0 : T.boxes0;
                for (int j = 0; j < T.nkt; ++j, ++it) {
                    const int s = it % STG, kt = T.kt0 + j;
                    if (!mbar_wait(empty(s), (uint32_t)((it / STG) & 1) ^ 1u)) { failed = true; break; }
                    const uint32_t st = sbase + (uint32_t)s * SB;
                    mbar_expect_tx(full_b(s), (T.boxes0 + lo_boxes) * BOX_BYTES);
                    for (int x = 0; x < T.boxes0; ++x)
                        tma_load_2d(st + BHI + x * BOX_BYTES, &tmBhi, kt * BK, T.n_tile * BN + x * B_BOX, full_b(s));
                    // the lo half, or the second N tile
                    for (int x = 0; x < lo_boxes; ++x)
                        tma_load_2d(st + BLO + x * BOX_BYTES, NT == 2 ? &tmBhi : &tmBlo, kt * BK,
                                    (T.n_tile + (NT == 2 ? 1 : 0)) * BN + x * B_BOX, full_b(s));
                }
            }
            for (int k = max(0, it - STG); k < it; ++k)
                if (!mbar_wait(full_b(k % STG), (uint32_t)((k / STG) & 1))) failed = true;
        }
    } else if (warp == 1) {
        const uint32_t lead = elect_lane();
        int it = 0, dr = 0;
        for (int i = blockIdx.x; i < tiles && !failed; i += gridDim.x, ++dr) {
            const Tile T = tile_at(i);
            const uint32_t id0 = idesc_fit(T.cols0), id1 = idesc_fit(T.cols1);
            const int u = nbuf == 2 ? dr & 1 : 0, use = nbuf == 2 ? dr >> 1 : dr;
            const uint32_t acc0 = tmem_base + (uint32_t)(u * (BN / 2));
            // (the sums of the tile before in this buffer have been read)
            if (!mbar_wait_warp(acc_free(u), (uint32_t)(use & 1) ^ 1u)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int j = 0; j < T.nkt; ++j, ++it) {
                const int s = it % STG;
                const uint32_t ph = (uint32_t)((it / STG) & 1);
                if (!mbar_wait_warp(full_b(s), ph) || !mbar_wait_warp(full_a(s), ph)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t st = smem_desc_lo(sbase + (uint32_t)s * SB);
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk) {
                    const uint32_t bh = st + (BHI + kk * 32) / 16, bl = st + (BLO + kk * 32) / 16;
                    const uint32_t more = (j > 0 || kk > 0) ? 1u : 0u;
#pragma unroll
                    for (int ms = 0; ms < MSUB; ++ms) {
                        const uint32_t td = acc0 + (uint32_t)(ms * BN);
                        if (AT) {
                            // K16 step kk: 8 of the subtile's 32 A columns
                            const uint32_t ta =
                                tmem_base + C::ACC_COLS + (uint32_t)((s * MSUB + ms) * (BK / 2) + kk * 8);
                            mma_f16_ts(lead, td, ta, bh, id0, more);
                            if (NT == 2) {
                                if (T.cols1 > 0)   // (a second tile with no live column is not computed)
                                    mma_f16_ts(lead, td + (uint32_t)(MSUB * BN), ta, bl, id1, more);
                            } else if (!args.hi_only) {
                                mma_f16_ts(lead, td, ta, bl, id0, 1u);
                            }
                        } else {
                            const uint32_t ad = st + (uint32_t)(ms * A_BYTES + kk * 32) / 16;
                            mma_f16(lead, td, ad, bh, id0, more);
                            if (NT == 2) {
                                if (T.cols1 > 0) mma_f16(lead, td + (uint32_t)(MSUB * BN), ad, bl, id1, more);
                            } else if (!args.hi_only) {
                                mma_f16(lead, td, ad, bl, id0, 1u);
                            }
                        }
                    }
                }
                mma_commit_if(lead, empty(s));
            }
            // the accumulators are complete (or abandoned) once every issued MMA retired
            mma_commit_if(lead, acc_full(u));
        }
    } else if (warp < 11) {
        // two groups of four warps, each taking every other subtile (with one
        // warp per scheduler the expansion waited on its own latencies and
        // set the pace); a warp writes only its TMEM lane quadrant: row =
        // 32 (warp % 4) + lane
        const int t = 32 * (warp & 3) + lane, group = (warp - 3) >> 2;
        int it = 0;
        for (int i = blockIdx.x; i < tiles && !failed; i += gridDim.x) {
            const Tile T = tile_at(i);
            for (int j = 0; j < T.nkt; ++j, ++it) {
                const int s = it % STG, r = it % RST;
                // the state tile is here, and the MMAs that read this stage's A before are done
                if (!mbar_wait(full_raw(r), (uint32_t)((it / RST) & 1)) ||
                    !mbar_wait(empty(s), (uint32_t)((it / STG) & 1) ^ 1u)) {
                    failed = true;
                    break;
                }
                // (A in TMEM: the stores below follow the MMAs whose completion was waited for)
                if (AT) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t st = sbase + (uint32_t)s * SB;
#pragma unroll
                for (int ms2 = 0; ms2 < MSUB; ms2 += 2) {
                    const int ms = ms2 + group;
                    if (ms >= MSUB) break;
                    const uint8_t *raw = sgen + (raws - sbase) + r * C::RAW_STAGE + ms * RAW_BYTES;
                    if (AT) {
                        uint32_t o[32];
                        expand_bwd_regs(raw, t, o);
                        tmem_st32(tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + C::ACC_COLS +
                                      (uint32_t)((s * MSUB + ms) * (BK / 2)),
                                  o);
                    } else if (args.mode == MODE_FWD) {
                        expand_fwd(raw, st + (uint32_t)(ms * A_BYTES), t);
                    } else {
                        expand_bwd(raw, st + (uint32_t)(ms * A_BYTES), t);
                    }
                }
                if (AT) {
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                } else {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
                mbar_arrive(full_a(s));
                __syncwarp();
                if (lane == 0) mbar_arrive(free_raw(r));
            }
        }
    } else {
        // epilogue: warp = TMEM lane quadrant
        const int q = warp & 3;
        const int r = q * 32 + lane;
        // What a store needs of its slot, one slot of the N tile per lane
        // (lane p: list position 32 n_tile + p), read when the N tile changes
        // and passed round by shuffles: with the slot's list entry and state
        // read at every use, their latency was most of a tile's epilogue.
        int loc[NT], cur = -1;
        int64_t off[NT];
        float sc[NT];
        unsigned top[NT];   // max-only: the slot's largest |g| so far (float bits)
        auto flush = [&]() {   // one atomic per warp and slot
            if (args.gmax_acc)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
                    if (cur >= 0 && top[nt] != 0u)
                        atomicMax(reinterpret_cast<unsigned long long *>(args.gmax_acc + off[nt]),
                                  (unsigned long long)__double_as_longlong((double)__uint_as_float(top[nt])));
        };
        int dr = 0;
        for (int i = blockIdx.x; i < tiles; i += gridDim.x, ++dr) {
            const Tile T = tile_at(i);
            if (T.n_tile != cur) {
                flush();
                cur = T.n_tile;
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const int P = (cur + nt) * (BN / 4) + lane;
                    loc[nt] = -1;
                    off[nt] = 0;
                    sc[nt] = args.inv_scale_bwd;
                    top[nt] = 0u;
                    if (P >= args.nlist) continue;
                    const int b = args.planes > 1 ? args.list[P % args.nslot] : args.list[P];
                    if (args.mode == MODE_FWD) {
                        sc[nt] = (float)args.sd[b].tc_inv_scale;
                        off[nt] = (int64_t)b * args.Nx;
                    } else if (args.gmax_acc) {
                        loc[nt] = args.sd[b].locus;
                        off[nt] = (int64_t)b * args.gmax_stride;
                    } else {
                        off[nt] = (args.planes > 1 ? (int64_t)P : (int64_t)(2 * b + 1 - args.sd[b].gcur)) * args.Dp;
                    }
                }
            }
            const int u = nbuf == 2 ? dr & 1 : 0, use = nbuf == 2 ? dr >> 1 : dr;
            if (!mbar_wait_warp(acc_full(u), (uint32_t)(use & 1))) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int cols = nt == 0 ? T.cols0 : T.cols1;
#pragma unroll 1
                for (int ms = 0; ms < MSUB && T.nkt > 0; ++ms) {
                    const uint32_t tbase =
                        tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(u * (BN / 2) + (nt * MSUB + ms) * BN);
                    const int row = (T.m_group * MSUB + ms) * BM + r;
#pragma unroll 1
                    for (int c0 = 0; c0 < cols; c0 += 32) {
                        float v[32];
                        tmem_ld32(tbase + (uint32_t)c0, v);
#pragma unroll
                        for (int tt = 0; tt < 8; ++tt) {
                            const int p = c0 / 4 + tt;   // the slot's place in the N tile: its lane
                            if (4 * p >= cols) break;
                            if (args.gmax_acc) {
                                const int locus = __shfl_sync(0xffffffffu, loc[nt], p);
                                float mv = 0.f;
                                if (row < args.m_rows && (row >> 2) != locus)
                                    mv = fmaxf(fmaxf(fabsf(v[4 * tt]), fabsf(v[4 * tt + 1])),
                                               fmaxf(fabsf(v[4 * tt + 2]), fabsf(v[4 * tt + 3]))) * args.inv_scale_bwd;
                                const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(mv));
                                if (lane == p) top[nt] = max(top[nt], mb);
                                continue;
                            }
                            const int64_t o = __shfl_sync(0xffffffffu, off[nt], p);
                            const float f = __shfl_sync(0xffffffffu, sc[nt], p);
                            const float4 w = make_float4(v[4 * tt] * f, v[4 * tt + 1] * f, v[4 * tt + 2] * f, v[4 * tt + 3] * f);
                            if (args.mode == MODE_FWD) {
                                if (row < args.Nx) args.partial[(int64_t)T.split * args.Bmax * args.Nx + o + row] = w;
                            } else if (row < args.m_rows) {
                                *reinterpret_cast<float4 *>(args.gpool + o + (int64_t)row * Q) = w;
                            }
                        }
                    }
                }
            }
            // this warp has read the buffer
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_free(u));
        }
        flush();
    }
    __syncwarp();
    if (failed) atomicExch(args.err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::TMEM_COLS)
                     : "memory");
    }
}

// ---------------------------------------------------------------------------
// Exact K rho for the dual form on the tensor cores.
//
// K (agreement counts, 0..L, L < 2^18) less its middle c = (L + 1) / 2 is held
// as three fp16 planes of balanced base-64 digits (|digit| <= 32), rho_q
// (integers, |rho_q| <= 2^27) as three fp16 planes of balanced base-640 digits
// (|digit| <= 320, the top one <= 328).  A product of two digits is an integer
// of at most 32 x 328 = 10,496, so sums over up to 1598 sequences stay below
// 2^24 and are exact in the FP32 TMEM accumulators: the sequences are taken in
// segments of 1536, and after each the epilogue warps add the nine
// accumulators, weighted 64^k 640^p, to 64-bit integers (modulo 2^64: the
// total is below 2^62).  K rho is that plus c times the column's sum of rho_q.
// (Twelve products of unsigned base-64 and base-128 digits, which need no
// second drain, issue a third more MMAs and hold four planes of rho.)
//
// Every row of rho_q sums to zero (k_dual_quant makes it so exactly), so the
// fourth column of K rho is minus the sum of the other three: only three
// columns per slot enter the product.
//
// A pair of CTAs (cta_group::2) takes 256 rows of K, 128 each, and 17 slots:
// 51 columns x 3 planes = 153 of the MMA's N = 160, 3 K digits x 160 = 480 of
// the 512 TMEM columns.  An M128 N160 MMA of one CTA reads 9 KB of shared
// memory per K16 step in the 80 cycles it computes, and the TMA writes about
// as much: shared memory was the bound (0.8 us per 64 sequences against 0.46
// of MMA work).  In the pair each CTA holds half of the rho rows, so an SM
// reads 6.5 KB and receives 4.8 KB per MMA.
// The kernel is persistent over the (row pair, slot group) tiles: the TMA
// loads of the next tile run on while the epilogue warps, which keep their
// sums in registers, store the last one; the MMAs wait only for the
// accumulators to be read.
// 186 us a launch at 512 slots of 3000 x 94,000 (303 with twelve products on
// single CTAs of 13 slots), tensor pipe 63 % active; 64 slots of 1000 x 4001:
// 23 us (26).

constexpr int KD_BM = 128, KD_BK = 64;   // (the digits' layout: kdig.cuh)
constexpr int KD_COLS = KD_S * KD_C;         // 51 live columns per plane
constexpr int KD_SEG = 24;                   // k-steps per segment: 1536 sequences
constexpr int KD_A_BYTES = KD_BM * KD_BK * 2;             // one K digit plane tile, 16 KB
constexpr int KD_B_BYTES = KD_NB / 2 * KD_BK * 2;         // this CTA's half of the rho rows, 10 KB
constexpr int KD_STAGE = KD_KDIG * KD_A_BYTES + KD_B_BYTES;
constexpr int KD_STG = 3;
constexpr int KD_SMEM = KD_STG * KD_STAGE + 1024 + 256;
constexpr int KD_THREADS = 64 + 512, KD_READERS = 32;    // TMA, MMA and 16 epilogue warps
constexpr uint32_t KD_TMEM_COLS = 512;
// kind::f16, D = F32, A = B = F16, K-major, M = 256 over the CTA pair
constexpr uint32_t IDESC_KD = (1u << 4) | ((uint32_t)(KD_NB >> 3) << 17) | ((uint32_t)(2 * KD_BM >> 4) << 24);
static_assert(KD_STAGE % 1024 == 0 && KD_B_BYTES % 1024 == 0, "tiles keep 1024-byte alignment");
static_assert(KD_KDIG * KD_NB <= (int)KD_TMEM_COLS, "accumulators fit TMEM");
static_assert(KD_NB % 16 == 0 && KD_NB <= 256, "MMA N for M = 256");
static_assert((KD_RDIG - 1) * KD_PS + KD_COLS <= KD_NB && KD_COLS <= KD_PS && KD_PS % 4 == 0, "planes of a tile");
static_assert(32ll * 328 * KD_SEG * KD_BK < (1ll << 24), "a segment's sums are exact in FP32");

// one MMA of the CTA pair, issued by the leader's elected lane: each CTA's A
// rows and half of the B rows at the same shared-memory offsets
__device__ __forceinline__ void mma_f16_pair(uint32_t lead, uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo,
                                             uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 e, %6, 0;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(tmem_d),
        "r"(a_lo), "r"(b_lo), "r"(SMEM_DESC_HI), "r"(IDESC_KD), "r"(accumulate), "r"(lead)
        : "memory");
}

struct KdArgs {
    int kt_total;        // Nx / 64
    int nk_rows;         // rows per K digit plane (multiple of 256)
    int N;
    int64_t Nx;
    int nlist;
    const int32_t *list;
    const uint8_t *rstate;
    const long long *csum;       // class sums and column sums of rho_q (CSUM per slot)
    long long center;            // c: K = K' + c
    double inv_qscale;
    float2 *KR;                  // K rho / qscale in double-float
    int *err;
    const int *ncount;           // list length in device memory (the grid covers the most slots), or null
    unsigned long long *ts;      // time stamps, or null
};

struct KdEpilogue {
    uint32_t tmem_base, acc_full, lead_read;   // lead_read: the leader's barrier (shared::cluster address)
    int rank, m_pairs, tiles, tile0, tstep, nkt, nlist;
};

// Slots S0 .. S0 + NS - 1 of this CTA pair's tiles: the warp's 32 rows of K.
// The digit products' sums are integers below 2^24 (exact in the FP32
// accumulators): each is converted with a 32-bit conversion; the K digits of
// a plane are combined by shifts and the planes by Horner's rule in 64-bit
// integers (no 64-bit conversion, which runs on GB300's narrow FP64 pipe).
// False when a wait gave up.
template <int S0, int NS>
__device__ __forceinline__ bool kd_epilogue(const KdArgs &args, const KdEpilogue &e, int q, int lane)
{
    constexpr int C0 = S0 * KD_C, NC = NS * KD_C;
    static_assert(C0 % 4 == 0, "columns are read in groups of four");
    const uint32_t tm = e.tmem_base + ((uint32_t)(q * 32) << 16);
    const float2 iq = df_from_d(args.inv_qscale);
    int dr = 0;
    for (int tile = e.tile0; tile < e.tiles; tile += e.tstep) {
        const int row = (tile % e.m_pairs) * 2 * KD_BM + e.rank * KD_BM + q * 32 + lane;
        const int P0 = (tile / e.m_pairs) * KD_S + S0;
        // start from what the products lack: c times the column sums, less the
        // agreement at the slot's own locus (read while the MMAs run)
        long long acc[NC];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const bool live = P0 + s < e.nlist && row < args.N;
            const int b = live ? args.list[P0 + s] : 0;
            const int y = live ? args.rstate[(int64_t)b * args.Nx + row] & 3 : 0;
            const long long *cs = args.csum + (int64_t)b * CSUM;
#pragma unroll
            for (int c = 0; c < KD_C; ++c)
                acc[KD_C * s + c] = live ? args.center * cs[CSUM_ALL + c] - cs[y * 4 + c] : 0ll;
        }
        for (int j0 = 0; j0 < e.nkt; j0 += KD_SEG, ++dr) {
            if (!mbar_wait(e.acc_full, (uint32_t)(dr & 1))) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int c0 = 0; c0 < NC; c0 += 4) {
                long long h[4] = {0ll, 0ll, 0ll, 0ll};
#pragma unroll
                for (int p = KD_RDIG - 1; p >= 0; --p) {
                    float v[KD_KDIG][4];
#pragma unroll
                    for (int k = 0; k < KD_KDIG; ++k)
                        tmem_ld4(tm + (uint32_t)(k * KD_NB + p * KD_PS + C0 + c0), v[k]);
                    tmem_ld_wait<KD_KDIG * 4>(&v[0][0]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int low = __float2int_rn(v[0][c]) + (__float2int_rn(v[1][c]) << 6);   // below 2^31
                        h[c] = h[c] * KD_RBASE + ((long long)__float2int_rn(v[2][c]) * 4096 + low);
                    }
                }
#pragma unroll
                for (int c = 0; c < 4 && c0 + c < NC; ++c) acc[c0 + c] += h[c];
            }
            // this warp has read its accumulators
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(e.lead_read);
        }
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const int P = P0 + s;
            if (P >= e.nlist || row >= args.Nx) continue;
            const int b = args.list[P];
            float2 val[4] = {df_zero(), df_zero(), df_zero(), df_zero()};
            if (row < args.N) {
                long long tot[4];
#pragma unroll
                for (int c = 0; c < KD_C; ++c) tot[c] = acc[KD_C * s + c];
                tot[3] = -(tot[0] + tot[1] + tot[2]);
#pragma unroll
                for (int c = 0; c < 4; ++c) val[c] = df_mul(df_from_ll_fast(tot[c]), iq);
            }
            float4 *o = reinterpret_cast<float4 *>(args.KR + ((int64_t)b * args.Nx + row) * 4);
            o[0] = make_float4(val[0].x, val[0].y, val[1].x, val[1].y);
            o[1] = make_float4(val[2].x, val[2].y, val[3].x, val[3].y);
        }
    }
    return true;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(KD_THREADS, 1)
k_kdig(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmR, const KdArgs args)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase0 = smem_u32(smem_raw);
    const uint32_t sbase = (sbase0 + 1023u) & ~1023u;
    uint8_t *const sgen = smem_raw + (sbase - sbase0);
    const uint32_t bars = sbase + KD_STG * KD_STAGE;
    // full (the leader's: both CTAs' loads), empty (in each CTA: the MMAs have
    // read the stage), accumulators complete (in each CTA), accumulators read
    // (the leader's: both CTAs' epilogue warps), TMEM address
    auto full = [&](int s) { return bars + 8u * s; };
    auto empty = [&](int s) { return bars + 8u * (KD_STG + s); };
    const uint32_t acc_full = bars + 8u * (2 * KD_STG), acc_read = bars + 8u * (2 * KD_STG + 1);
    const uint32_t tmem_slot = bars + 8u * (2 * KD_STG + 2);
    uint32_t *tmem_slot_gen = reinterpret_cast<uint32_t *>(sgen + KD_STG * KD_STAGE + 8 * (2 * KD_STG + 2));
    constexpr uint32_t BOFF = KD_KDIG * KD_A_BYTES;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // (warp: uniform)
    const uint32_t rank = cluster_rank();
    const int nkt = args.kt_total;
    const int nlist = args.ncount ? *args.ncount : args.nlist;
    const int m_pairs = args.nk_rows / (2 * KD_BM);
    const int tiles = m_pairs * ((nlist + KD_S - 1) / KD_S);
    const int tile0 = blockIdx.x >> 1, tstep = gridDim.x >> 1;
    if (tile0 >= tiles) return;   // (both CTAs of the pair, before any barrier or TMEM allocation)
    stamp_begin(args.ts);

    if (threadIdx.x == 0) {
        for (int s = 0; s < KD_STG; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_read, KD_READERS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot),
                     "r"(KD_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();               // the peer's barriers are initialised
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot_gen, 0);   // (uniform)
    bool failed = false;

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t lead_bars = map_to_rank(bars, 0);
            int it = 0;
            for (int tile = tile0; tile < tiles && !failed; tile += tstep) {
                const int m0 = (tile % m_pairs) * 2 * KD_BM + (int)rank * KD_BM;
                const int r0 = (tile / m_pairs) * KD_NB + (int)rank * (KD_NB / 2);
                for (int j = 0; j < nkt; ++j, ++it) {
                    const int s = it % KD_STG;
                    if (!mbar_wait(empty(s), (uint32_t)((it / KD_STG) & 1) ^ 1u)) { failed = true; break; }
                    const uint32_t st = sbase + (uint32_t)s * KD_STAGE;
                    if (rank == 0) mbar_expect_tx(full(s), 2 * KD_STAGE);   // the pair's bytes
#pragma unroll
                    for (int k = 0; k < KD_KDIG; ++k)
                        tma_load_2d_pair(st + k * KD_A_BYTES, &tmK, j * KD_BK, k * args.nk_rows + m0, lead_bars + 8u * s);
                    tma_load_2d_pair(st + BOFF, &tmR, j * KD_BK, r0, lead_bars + 8u * s);
                }
            }
            // loads still in flight (both CTAs') land before the pair leaves
            // its last cluster barrier
            if (rank == 0)
                for (int i = max(0, it - KD_STG); i < it; ++i)
                    if (!mbar_wait(full(i % KD_STG), (uint32_t)((i / KD_STG) & 1))) failed = true;
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t lead = elect_lane();
            int it = 0, dr = 0;
            for (int tile = tile0; tile < tiles && !failed; tile += tstep) {
                for (int j0 = 0; j0 < nkt && !failed; j0 += KD_SEG, ++dr) {
                    const int j1 = min(nkt, j0 + KD_SEG);
                    // (the accumulators of the segment before have been read)
                    if (!mbar_wait_warp(acc_read, (uint32_t)(dr & 1) ^ 1u)) { failed = true; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int j = j0; j < j1; ++j, ++it) {
                        const int s = it % KD_STG;
                        if (!mbar_wait_warp(full(s), (uint32_t)((it / KD_STG) & 1))) { failed = true; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t st = smem_desc_lo(sbase + (uint32_t)s * KD_STAGE);
#pragma unroll
                        for (int kk = 0; kk < KD_BK / 16; ++kk)
#pragma unroll
                            for (int k = 0; k < KD_KDIG; ++k)
                                mma_f16_pair(lead, tmem_base + (uint32_t)(k * KD_NB), st + (k * KD_A_BYTES + kk * 32) / 16,
                                             st + (BOFF + kk * 32) / 16, (j > j0 || kk > 0) ? 1u : 0u);
                        mma_commit_pair_if(lead, empty(s));
                    }
                    mma_commit_pair_if(lead, acc_full);
                }
            }
        }
    } else {
        // four warps per TMEM lane quadrant: slots 0..3, 4..7, 8..11 and 12..16 of the tile
        const KdEpilogue e{tmem_base, acc_full, map_to_rank(acc_read, 0), (int)rank, m_pairs, tiles, tile0, tstep,
                           nkt, nlist};
        const int part = (warp - 2) >> 2, q = warp & 3;
        failed = part == 0   ? !kd_epilogue<0, 4>(args, e, q, lane)
                 : part == 1 ? !kd_epilogue<4, 4>(args, e, q, lane)
                 : part == 2 ? !kd_epilogue<8, 4>(args, e, q, lane)
                             : !kd_epilogue<12, 5>(args, e, q, lane);
    }
    __syncwarp();
    if (failed) atomicExch(args.err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();   // no MMA, load or remote arrival of the pair is left
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(KD_TMEM_COLS)
                     : "memory");
    }
    stamp_end(args.ts, true);
}

// K (int32, Nx x Nx) less c -> three fp16 planes of balanced base-64 digits,
// rows padded to nk_rows (padding sequences hold 0: their rho is 0)
__global__ void k_kdig_split_k(const int32_t *__restrict__ K, int64_t Nx, int N, int center, int nk_rows,
                               __half *__restrict__ Kd)
{
    const int64_t total = (int64_t)nk_rows * Nx;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / Nx, j = t - i * Nx;
        int v = i < N && j < N ? K[t] - center : 0;
        const int d0 = ((v + 32) & 63) - 32;
        v = (v - d0) >> 6;
        const int d1 = ((v + 32) & 63) - 32;
        Kd[t] = __int2half_rn(d0);
        Kd[(int64_t)nk_rows * Nx + t] = __int2half_rn(d1);
        Kd[2 * (int64_t)nk_rows * Nx + t] = __int2half_rn((v - d1) >> 6);
    }
}

// d (engine layout [n][s][a]) -> B rows p*4+a, columns n*4+s, fp16 hi and lo of d*2^e
__global__ void k_split_dir(const SlotDev *__restrict__ sd, const int32_t *__restrict__ list, int64_t L,
                            int64_t Dp, int64_t Kp, const float *__restrict__ vecs, __half *__restrict__ hi,
                            __half *__restrict__ lo)
{
    const int P = blockIdx.y;
    const int b = list[P];
    const float sc = (float)sd[b].tc_scale;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < 4 * L; k += (int64_t)gridDim.x * blockDim.x) {
        const float4 v = *reinterpret_cast<const float4 *>(vecs + (int64_t)b * Dp + k * 4);
        const float vv[4] = {v.x * sc, v.y * sc, v.z * sc, v.w * sc};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const __half h = __float2half_rn(vv[a]);
            const __half l = __float2half_rn(vv[a] - __half2float(h));
            const int64_t o = ((int64_t)P * 4 + a) * Kp + k;
            hi[o] = h;
            lo[o] = l;
        }
    }
}

// R (float4 per sequence) -> B rows p*4+a, columns i, fp16 hi and lo of R*2^e
__global__ void k_split_R(const int32_t *__restrict__ list, int64_t Nx, const float4 *__restrict__ R, float sc,
                          __half *__restrict__ hi, __half *__restrict__ lo, int direct)
{
    const int P = blockIdx.y;
    const int b = direct ? P : list[P];   // direct: R rows by list position (digit planes)
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < Nx; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 v = R[(int64_t)b * Nx + i];
        const float vv[4] = {v.x * sc, v.y * sc, v.z * sc, v.w * sc};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const __half h = __float2half_rn(vv[a]);
            const __half l = __float2half_rn(vv[a] - __half2float(h));
            const int64_t o = ((int64_t)P * 4 + a) * Nx + i;
            hi[o] = h;
            lo[o] = l;
        }
    }
}

} // namespace tc

// ---------------------------------------------------------------------------
// host side

namespace {

using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn()
{
    // initialised once, thread-safely (solver lanes create plans concurrently)
    static const EncodeFn fn = []() -> EncodeFn {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeFn>(p);
        return nullptr;
    }();
    return fn;
}

bool make_map(CUtensorMap *m, CUtensorMapDataType dt, void *base, uint64_t cols, uint64_t rows,
              uint64_t row_bytes, uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle sw)
{
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_cols, box_rows};
    const cuuint32_t es[2] = {1, 1};
    return fn(m, dt, 2, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

} // namespace

struct TcPlan {
    CUtensorMap mX, mXT, mDhi, mDlo, mRhi, mRlo;
    bool has_fwd = false;   // the forward's slot operand (null for the dual form, which has no forward GEMM)
    int64_t Kp = 0;
    int fwd_splits = 1;
};

namespace {

// Subtiles per CTA (MSUB) and pipeline depth: {4, 2} keeps four 128-row
// accumulators (all 512 TMEM columns) and two 104 KB stages; {2, 3} and
// {1, 4} trade L2 reuse of the slot operand for deeper pipelines.
// SDCA_TC_MSUB (1, 2 or 4) overrides the choice for tuning runs.
int msub_choice()
{
    static const int v = []() {
        const char *e = std::getenv("SDCA_TC_MSUB");
        return (e && (e[0] == '1' || e[0] == '2')) ? e[0] - '0' : 4;
    }();
    return v;
}

template <int MSUB, int STG, int NT = 1, bool AT = false>
void launch_gemm(int m_tiles, int n_tiles, int splits, const CUtensorMap &a, const CUtensorMap &bh,
                 const CUtensorMap &bl, tc::GemmArgs args, cudaStream_t st)
{
    args.m_groups = (m_tiles + MSUB - 1) / MSUB;
    args.n_groups = (n_tiles + NT - 1) / NT;
    args.splits = splits;
    // persistent: one CTA per SM (its shared memory allows no second)
    const int64_t tiles = (int64_t)args.m_groups * args.n_groups * splits;
    tc::k_gemm<MSUB, STG, NT, AT>
        <<<(unsigned)std::min<int64_t>(tiles, 152), tc::THREADS, tc::Cfg<MSUB, STG, NT, AT>::SMEM_BYTES, st>>>(a, bh, bl,
                                                                                                        args);
}

// The backward with hi + lo operands (the tensor-core form's gradient, the
// dual form's max-norm checks) keeps its one-hot A in TMEM: two subtiles,
// four stages, the MMAs' N fitted to the live columns.  On the 3000 x 94,000
// workload (ncu, check launches of about 8 slots) it takes 204 us (234 with a
// CTA per tile; 65 against 95 at 616 x 65,563); A in shared memory took
// 426-439 against 337-375 when both fed the MMAs from one lane and the state
// tiles from the same ring.  Exact (hi-only) operands -- the dual form's
// solution digit planes, two N tiles per CTA, 392 us for 21 slots (455 with a
// CTA per tile; 120 against 164 at 616 x 65,563) -- stay with A in shared memory: the TMEM form with one subtile and six
// stages took 689 against 607 us there.  SDCA_TC_BWD_SMEM_A=1 keeps A in
// shared memory everywhere.
bool bwd_tmem_a()
{
    static const bool v = [] {
        const char *e = std::getenv("SDCA_TC_BWD_SMEM_A");
        return !(e && e[0] == '1');
    }();
    return v;
}

void launch_gemm_any(int msub, int m_tiles, int n_tiles, int splits, const CUtensorMap &a, const CUtensorMap &bh,
                     const CUtensorMap &bl, const tc::GemmArgs &args, cudaStream_t st)
{
    if (args.mode == tc::MODE_BWD && !args.hi_only && bwd_tmem_a())
        launch_gemm<2, 4, 1, true>(m_tiles, n_tiles, splits, a, bh, bl, args, st);
    else if (args.hi_only && args.mode == tc::MODE_BWD)
        // exact fp16 operands: two N tiles per CTA, two subtiles, three stages
        launch_gemm<2, 3, 2>(m_tiles, n_tiles, splits, a, bh, bl, args, st);
    else if (msub == 4)
        launch_gemm<4, 2>(m_tiles, n_tiles, splits, a, bh, bl, args, st);
    else if (msub == 2)
        launch_gemm<2, 3>(m_tiles, n_tiles, splits, a, bh, bl, args, st);
    else
        launch_gemm<1, 4>(m_tiles, n_tiles, splits, a, bh, bl, args, st);
}

} // namespace

int tc_fwd_splits(const Problem &P, int nlist)
{
    // split K so that the CTAs fill whole waves of 152 SMs (one CTA per SM)
    const int msub = msub_choice();
    const int mt = (int)((P.Nx + tc::BM - 1) / tc::BM);
    const int mg = (mt + msub - 1) / msub;
    const int nt = (4 * nlist + tc::BN - 1) / tc::BN;
    const int kt = (int)((4 * P.L + tc::BK - 1) / tc::BK);
    int best = 1;
    double best_t = 1e30;
    for (int s = 1; s <= (int)P.C; ++s) {
        const double waves = std::ceil((double)mg * nt * s / 152.0);
        const double t = waves * std::ceil((double)kt / s) + 8.0 * waves;
        if (t < best_t) {
            best_t = t;
            best = s;
        }
    }
    // no empty split: every launched split owns at least one k-tile
    const int stride = (kt + best - 1) / best;
    return (kt + stride - 1) / stride;
}

TcPlan *tc_plan_create(const Problem &P, const uint8_t *X, const uint8_t *XT, __half *Dhi, __half *Dlo,
                       __half *Rhi, __half *Rlo, int64_t Kp)
{
    TcPlan *p = new TcPlan();
    p->Kp = Kp;
    bool ok = true;
    ok &= make_map(&p->mX, CU_TENSOR_MAP_DATA_TYPE_UINT8, const_cast<uint8_t *>(X), (uint64_t)P.Lx,
                   (uint64_t)P.N, (uint64_t)P.Lx, 16, 128, CU_TENSOR_MAP_SWIZZLE_NONE);
    ok &= make_map(&p->mXT, CU_TENSOR_MAP_DATA_TYPE_UINT8, const_cast<uint8_t *>(XT), (uint64_t)P.Nx,
                   (uint64_t)P.L, (uint64_t)P.Nx, 64, 32, CU_TENSOR_MAP_SWIZZLE_NONE);
    p->has_fwd = Dhi && Dlo;
    if (p->has_fwd) {
        ok &= make_map(&p->mDhi, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, Dhi, (uint64_t)Kp, (uint64_t)4 * P.Bmax,
                       (uint64_t)Kp * 2, 64, tc::B_BOX, CU_TENSOR_MAP_SWIZZLE_128B);
        ok &= make_map(&p->mDlo, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, Dlo, (uint64_t)Kp, (uint64_t)4 * P.Bmax,
                       (uint64_t)Kp * 2, 64, tc::B_BOX, CU_TENSOR_MAP_SWIZZLE_128B);
    }
    ok &= make_map(&p->mRhi, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, Rhi, (uint64_t)P.Nx, (uint64_t)4 * P.Bmax,
                   (uint64_t)P.Nx * 2, 64, tc::B_BOX, CU_TENSOR_MAP_SWIZZLE_128B);
    ok &= make_map(&p->mRlo, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, Rlo, (uint64_t)P.Nx, (uint64_t)4 * P.Bmax,
                   (uint64_t)P.Nx * 2, 64, tc::B_BOX, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!ok) {
        delete p;
        return nullptr;
    }
    return p;
}

void tc_plan_destroy(TcPlan *p) { delete p; }

struct KdPlan {
    CUtensorMap mK, mR;   // K digit planes; the tiles' rho digit rows
    int nk_rows = 0;
};

int kd_nk_rows(const Problem &P) { return (int)((P.Nx + 2 * tc::KD_BM - 1) / (2 * tc::KD_BM) * (2 * tc::KD_BM)); }
// rho digit rows: whole tiles of 17 slots
int kd_nr_rows(const Problem &P) { return (int)((P.Bmax + tc::KD_S - 1) / tc::KD_S * tc::KD_NB); }

namespace {
int kd_center(const Problem &P) { return (int)((P.L + 1) / 2); }
} // namespace

KdPlan *tc_kdig_plan_create(const Problem &P, __half *Kd, __half *Rd)
{
    KdPlan *p = new KdPlan();
    p->nk_rows = kd_nk_rows(P);
    bool ok = make_map(&p->mK, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, Kd, (uint64_t)P.Nx, (uint64_t)tc::KD_KDIG * p->nk_rows,
                       (uint64_t)P.Nx * 2, tc::KD_BK, tc::KD_BM, CU_TENSOR_MAP_SWIZZLE_128B);
    ok &= make_map(&p->mR, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, Rd, (uint64_t)P.Nx, (uint64_t)kd_nr_rows(P),
                   (uint64_t)P.Nx * 2, tc::KD_BK, tc::KD_NB / 2, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!ok) {
        delete p;
        return nullptr;
    }
    return p;
}

void tc_kdig_plan_destroy(KdPlan *p) { delete p; }

void tc_kdig_fill_k(const KdPlan *pl, const Problem &P, const int32_t *K, __half *Kd, cudaStream_t st)
{
    const int64_t total = (int64_t)pl->nk_rows * P.Nx;
    tc::k_kdig_split_k<<<(unsigned)std::min<int64_t>((total + 255) / 256, 8192), 256, 0, st>>>(
        K, P.Nx, (int)P.N, kd_center(P), pl->nk_rows, Kd);
}

cudaError_t tc_launch_kdig(const KdPlan *pl, const Problem &P, const int32_t *list, int n, const uint8_t *rstate,
                           const long long *csum, double inv_qscale, float2 *KR, int *err, cudaStream_t st, const int *cnt,
                           unsigned long long *ts)
{
    if (n <= 0) return cudaSuccess;
    tc::KdArgs a{};
    a.kt_total = (int)(P.Nx / tc::KD_BK);
    a.nk_rows = pl->nk_rows;
    a.N = (int)P.N;
    a.Nx = P.Nx;
    a.nlist = n;
    a.list = list;
    a.rstate = rstate;
    a.csum = csum;
    a.center = kd_center(P);
    a.inv_qscale = inv_qscale;
    a.KR = KR;
    a.err = err;
    a.ncount = cnt;
    a.ts = ts;
    // persistent: at most one CTA pair per two of the 152 SMs
    const int64_t tiles = (int64_t)(pl->nk_rows / (2 * tc::KD_BM)) * ((n + tc::KD_S - 1) / tc::KD_S);
    const unsigned pairs = (unsigned)std::min<int64_t>(tiles, 76);
    tc::k_kdig<<<2 * pairs, tc::KD_THREADS, tc::KD_SMEM, st>>>(pl->mK, pl->mR, a);
    return cudaGetLastError();
}

cudaError_t tc_launch_fwd(const TcPlan *pl, const Problem &P, const SlotDev *sd, const int32_t *list, int n,
                          const float *vecs, __half *Dhi, __half *Dlo, float *partial, int splits, int *err,
                          cudaStream_t st)
{
    if (!pl->has_fwd) return cudaErrorInvalidValue;   // a plan without the forward's operand
    if (n <= 0) return cudaSuccess;
    {
        dim3 g((unsigned)std::min<int64_t>((4 * P.L + 255) / 256, 1024), (unsigned)n);
        tc::k_split_dir<<<g, 256, 0, st>>>(sd, list, P.L, P.Dp, pl->Kp, vecs, Dhi, Dlo);
    }
    tc::GemmArgs a{};
    a.mode = tc::MODE_FWD;
    a.kt_total = (int)((4 * P.L + tc::BK - 1) / tc::BK);
    a.kt_begin_stride = (a.kt_total + splits - 1) / splits;
    a.m_rows = (int)P.N;
    a.nlist = n;
    a.list = list;
    a.sd = sd;
    a.partial = reinterpret_cast<float4 *>(partial);
    a.Bmax = P.Bmax;
    a.Nx = P.Nx;
    a.err = err;
    launch_gemm_any(msub_choice(), (int)((P.Nx + tc::BM - 1) / tc::BM), (4 * n + tc::BN - 1) / tc::BN, splits,
                    pl->mX, pl->mDhi, pl->mDlo, a, st);
    return cudaGetLastError();
}

cudaError_t tc_launch_bwd(const TcPlan *pl, const Problem &P, const SlotDev *sd, const int32_t *list, int n,
                          const float *R, float r_scale, __half *Rhi, __half *Rlo, float *gpool, int *err,
                          cudaStream_t st, bool exact_fp16, double *gmax_acc, int gmax_stride, int planes)
{
    if (n <= 0) return cudaSuccess;
    const int nslot = n;
    if (planes > 1) {
        if ((int64_t)planes * n > P.Bmax) return cudaErrorInvalidValue;   // B operand rows and gpool buffers
        n *= planes;
    }
    {
        dim3 g((unsigned)std::min<int64_t>((P.Nx + 255) / 256, 64), (unsigned)n);
        tc::k_split_R<<<g, 256, 0, st>>>(list, P.Nx, reinterpret_cast<const float4 *>(R), r_scale, Rhi, Rlo,
                                          planes > 1 ? 1 : 0);
    }
    tc::GemmArgs a{};
    a.mode = tc::MODE_BWD;
    a.kt_total = (int)(P.Nx / tc::BK);
    a.kt_begin_stride = a.kt_total;
    a.m_rows = (int)(4 * P.L);
    a.nlist = n;
    a.list = list;
    a.sd = sd;
    a.gpool = gpool;
    a.Dp = P.Dp;
    a.inv_scale_bwd = 1.0f / r_scale;
    a.hi_only = exact_fp16 ? 1 : 0;
    a.gmax_acc = gmax_acc;
    a.gmax_stride = gmax_stride;
    a.planes = planes > 1 ? planes : 1;
    a.nslot = nslot;
    a.Nx = P.Nx;
    a.err = err;
    launch_gemm_any(msub_choice(), (int)((4 * P.L + tc::BM - 1) / tc::BM), (4 * n + tc::BN - 1) / tc::BN, 1,
                    pl->mXT, pl->mRhi, pl->mRlo, a, st);
    return cudaGetLastError();
}

cudaError_t tc_configure()
{
    cudaError_t e = cudaFuncSetAttribute(tc::k_gemm<4, 2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         tc::Cfg<4, 2>::SMEM_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(tc::k_gemm<2, 3, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 tc::Cfg<2, 3, 2>::SMEM_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(tc::k_gemm<2, 3, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 tc::Cfg<2, 3>::SMEM_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(tc::k_gemm<1, 4, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 tc::Cfg<1, 4>::SMEM_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(tc::k_gemm<2, 4, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 tc::Cfg<2, 4, 1, true>::SMEM_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(tc::k_kdig, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::KD_SMEM);
    return e;
}

} // namespace sdca
