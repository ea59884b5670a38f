// Binary64 products of a real and a complex operand on the bf16 tensor cores,
// for the binary64 form's contractions:
//   V-build     V (W x n^2)    = x~ (W x G) . L (G x n^2)      (prop/chol_afqmc_ops.py:70-74)
//   force bias  fb (W x G)     = 2 G_half (W x o n) . L~^T     (meas/rhf.py:27-33)
//   exchange    f_g (o x o)    = L~_g G_half^T                 (meas/rhf.py:36-50)
//   Taylor      T_k            = (i sqrt_dt / k) V_w T_{k-1}   (prop/utils.py:20-31)
// and the adjoint's GEMMs.  GB300's binary64 pipe gives two FMAs a clock an
// SM (1.2 TFLOP/s a GPU), the bf16 tensor cores 2 PFLOP/s: cutting both
// operands into exact integer digits (the integer slicing of Ozaki, Ogita,
// Oishi and Rump, 2012) costs 34 bf16 products a binary64 one and is still
// tens of times faster.
//
// Digits.  Each operand row r (K contiguous) is scaled by a power of two E_r
// above its largest entry and rounded to 55 bits: X = x 2^(7 - E_r) is
// seven signed base-256 digits X = sum_s a_s 2^(-8 s), |a_s| <= 128, stored as
// bf16 (a_s 2^(-8 s), exact).  A digit array is stored as the MMAs read it: for
// each 32 k and digit a (rows x 64 bytes) plane with the 64-byte swizzle, so
// that a tile is one contiguous bulk copy and rows past the end are never
// copied.  The product of two rows is
// sum_{s,t} 2^(-8 (s + t)) sum_k a_s b_t; the pairs s + t <= 7 are kept.  What
// is dropped is below the rounding to 55 bits (with s + t <= 6 it is eight
// times that, and the error of a force bias passes the binary64 chain's).
// Pairs of one s + t = d share a tensor-memory accumulator (d = 5, 6, 7 share
// one): their sum is an integer multiple of 2^(-8 d), at most 2^14 (d + 1) of
// them a product, which the fp32 accumulator holds exactly below 2^24, that is
// for 256 products at d = 2, 3 and 512 at d = 0, 1, where it is drained.  d =
// 4 and the last one (drained every 512) pass 2^24 only in sums of hundreds of
// extremal digits of one sign; what truncation loses there is below 2^-45 of
// such a sum's value and nothing otherwise.  The drained values are summed in
// 64-bit integers (d <= 4; units of 2^-46 of the largest product, which
// leave room for the 2^62 of fewer than 2^16 of them, OZ_KMAX) and in fp32
// (the last accumulator), and converted once to binary64.
//
// A product is held to its operands' largest entries, where a binary64 chain's
// error goes with the terms.  So each is checked by its results (oz_lost in
// oz_digits.cuh) and, where those are too small for that (or with inf and nan),
// formed again on the binary64 pipe: k_zgemm_lost's tiles, the walkers marked for
// k_trotter, k_green and the adjoint's kernels, k_oz_exchange's blocks by itself.
// Where all is sound, which the first 32 results mostly tell, that costs a launch
// of 3-4 us a product: a step of 30 orbitals and 200 walkers 144 -> 153 us, of 120 x
// 20, 600 vectors and 2048 walkers 5.43 -> 5.51 ms.
//
// Kernel: persistent CTAs with 128 x 64 tiles, so that all six accumulators
// stay in tensor memory and each digit tile is read once for its 34 products.
// The digit tiles of a 32-k stage arrive as seven units (A_{6-j}, B_j) in the
// order in which the rows of products A_s B_0 .. A_s B_{6-s}, s = 6 .. 0,
// need them (s + t = 7 included); an A tile is released after its row, the B
// tiles after the stage, so that one stage is refilled while the other is
// multiplied (three stages of B gained nothing).  A row's MMAs keep A_s in the
// tensor core's collector buffer: 35 clocks an MMA of 128 x 64 x 16 against 48
// (the operands' shared-memory reads), as issued from resident operands.  The
// whole MMA warp runs the issue loop and elects a lane in each instruction:
// descriptors then stay in uniform registers (recomputed ones cost 77 clocks an
// MMA).  In long products the MMAs bound it (V-build of 200 orbitals, 1000
// vectors, 1024 walkers: 3.0 ms for 2.4 of MMAs), in short ones the drains and
// the conversion of six accumulators a tile, in single tiles the chain of both
// (18-25 us).
#include "afq_internal.cuh"
#include "copy_ring.h"
#include "oz_digits.cuh"
#include "sym_blocks.cuh"
#include "tc_common.cuh"

namespace afq {

namespace {

using namespace tc;

constexpr int OZ_ROWS = 128;              // real-operand rows a tile (tensor-memory lanes)
constexpr int OZ_BK = 32;                 // K a stage: one 64-byte swizzle row
constexpr int OZ_TN = 64;                 // complex-operand digit rows a tile
constexpr int OZ_CHUNK = 8;               // stages (256 k) between drains of d = 2, 3 (16 for the others)
constexpr int OZ_EW = 16;                 // epilogue warps
constexpr int OZ_GT = 64 + 32 * OZ_EW;    // threads
constexpr int OZ_CW = OZ_TN * 4 / OZ_EW;  // columns an epilogue thread
constexpr int OZ_STG = 2;                 // stages in shared memory
constexpr int OZ_A_SL = OZ_ROWS * OZ_BK * 2, OZ_B_SL = OZ_TN * OZ_BK * 2;
constexpr int OZ_GSMEM = OZ_STG * OZ_S * (OZ_A_SL + OZ_B_SL) + 1024 + 512;
// tensor-memory slot of an accumulator; d = 2 and 3 alternate between two
enum { OZ_D5, OZ_D4, OZ_D1, OZ_D0, OZ_D3, OZ_D2 = 6, OZ_SLOTS = 8 };
constexpr uint32_t OZ_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_TN >> 3) << 17) |
                              ((uint32_t)(OZ_ROWS >> 4) << 24);
static_assert(OZ_GSMEM <= 227 * 1024, "digit GEMM shared memory");

__device__ __forceinline__ void oz_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"((unsigned long long)src), "r"(bytes), "r"(bar)
                 : "memory");
}

// K-major tile of 64-byte rows, 64-byte swizzle: 8-row atoms 512 bytes apart.
__device__ __forceinline__ uint64_t desc_k64(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

// Where output (row r, complex column m) of batch b goes: C[b bs + (m / md)
// ms1 + (m % md) ms0 + r rs], times 2^aexp, plus the same entry of add.
struct OzOut {
    double2* C;
    long long bs, ms1, ms0, rs;
    int md, aexp;
    const double2* add;
    const int* skip;  // blocks m / md whose walker (m / md / sd) % sm it marks are not written
    int sd, sm;
};

struct OzArgs {
    const uint8_t *da, *db;   // digit arrays of the real and the complex operand
    int r8a, r8b;             // their plane rows
    int rows, cols, K;        // cols: digit rows of the complex operand (re, im interleaved)
    int batch, adiv;          // batch b takes real-operand plane b / adiv (adiv 0: the one plane)
    int gn;                   // column tiles a group of the tile order
    int splits, cps;          // K splits, 256-k chunks a split
    const int *ea, *eb;       // row scales
    long long* raw;           // splits > 1: integer sums (splits x cols x rows), and the tails
    float* rawt;
    int* err;
    OzOut out;
    SymRows sym;
};

__device__ __forceinline__ void oz_tile(const OzArgs& a, int t, int mt, int nt, int& z, int& mb, int& nb) {
    z = t / (mt * nt);
    const int r = t - z * (mt * nt), g = r / (a.gn * mt), rr = r - g * a.gn * mt, gs = min(a.gn, nt - g * a.gn);
    mb = rr / gs;
    nb = g * a.gn + rr % gs;
}

// One MMA, issued by the warp's elected lane (the whole warp calls, so that
// descriptors stay warp-uniform).  H: 0 no collector hint, 1 A is read into
// the collector, 2 used from it, 3 used for the last time.
template <int H>
__device__ __forceinline__ void oz_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
#define AFQ_OZ_MMA(HINT)                                                                                      \
    asm volatile(                                                                                             \
        "{\n\t.reg .pred p, q;\n\t"                                                                           \
        "elect.sync _|q, 0xffffffff;\n\t"                                                                     \
        "setp.ne.b32 p, %4, 0;\n\t"                                                                           \
        "@q tcgen05.mma.cta_group::1.kind::f16" HINT " [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),                 \
        "l"(a), "l"(b), "r"(OZ_IDESC), "r"(acc)                                                               \
        : "memory")
    if (H == 0) AFQ_OZ_MMA("");
    else if (H == 1) AFQ_OZ_MMA(".collector::a::fill");
    else if (H == 2) AFQ_OZ_MMA(".collector::a::use");
    else AFQ_OZ_MMA(".collector::a::lastuse");
#undef AFQ_OZ_MMA
}
__device__ __forceinline__ void oz_commit(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(bar)
        : "memory");
}
// accumulator slot of digit pairs s + t = d, `buf` the copy of d = 2, 3 in use
__device__ __forceinline__ constexpr int oz_slot(int d, int buf) {
    return d >= 5 ? OZ_D5 : d == 4 ? OZ_D4 : d == 1 ? OZ_D1 : d == 0 ? OZ_D0 : (d == 3 ? OZ_D3 : OZ_D2) + buf;
}
// products A_s B_0 .. A_s B_{min(6, 7-s)} of one k step; acc0 = 0: the row's new accumulator (d = s) begins
template <int S>
__device__ __forceinline__ void oz_row(uint32_t tmem, uint64_t ad, uint64_t bd, int buf, uint32_t acc0) {
    constexpr int N = S == 0 ? OZ_S : OZ_S + 1 - S;
#pragma unroll
    for (int t = 0; t < N; ++t) {
        const uint32_t d = tmem + oz_slot(S + t, buf) * OZ_TN;
        const uint64_t b = bd + (uint64_t)((t * OZ_B_SL) >> 4);
        const uint32_t acc = t == 0 ? acc0 : 1u;
        if (t == 0) oz_mma<1>(d, ad, b, acc);
        else if (t < N - 1) oz_mma<2>(d, ad, b, acc);
        else oz_mma<3>(d, ad, b, acc);
    }
}

// Wait of the MMA warp: expiry raises the CTA's abort flag and the error word,
// and the warp carries on (its sums are lost, nothing is out of bounds), so
// that the issue loop stays free of divergent exits and its descriptors in
// uniform registers (recomputed ones cost 77 clocks an MMA).
__device__ __noinline__ void oz_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err) {
    if (!mbar_wait_inl(bar, parity, abort_flag)) {
        atomicExch(err, 1);
        *abort_flag = 1;
    }
}
__device__ __forceinline__ void oz_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err) {
    if (!mbar_try_wait(bar, parity)) oz_wait_slow(bar, parity, abort_flag, err);
    __syncwarp();
}

// the whole warp gives up where one of its lanes does: what follows a wait is the warp's together
__device__ __forceinline__ bool oz_all(bool ok) { return __all_sync(0xffffffffu, ok); }

// shared-memory offsets of the barriers (8 bytes each) after the tiles
constexpr int OZ_BAR0 = OZ_STG * OZ_S * (OZ_A_SL + OZ_B_SL);
enum {
    OZB_FA = 0,                      // an A tile landed
    OZB_FB = OZB_FA + OZ_STG * OZ_S, // a B tile landed
    OZB_EA = OZB_FB + OZ_STG * OZ_S, // an A tile's row of MMAs finished
    OZB_EB = OZB_EA + OZ_STG * OZ_S, // a stage's MMAs finished
    OZB_TFS = OZB_EB + OZ_STG,       // the single accumulators hold their sums
    OZB_TFD = OZB_TFS + 1,           // a copy of the double ones does
    OZB_TE = OZB_TFD + 2,            // a slot has been drained
    OZB_DRAIN = OZB_TE + OZ_SLOTS,
    OZB_N = OZB_DRAIN + 1
};
static_assert(OZB_N * 8 + 8 <= 512, "barrier area");

struct OzMmaState {
    unsigned c, ns, nd;  // stages, drains of the single and of the double accumulators so far
};
// row S of the stage in buffer P
template <int S>
__device__ __forceinline__ void oz_stage_row(int P, uint32_t smem, uint32_t tmem, int k2, bool sd, bool ss, const OzMmaState& m,
                                             int buf, volatile int* abort_flag, int* err) {
    constexpr int J = OZ_S - 1 - S;
    const uint32_t bars = smem + OZ_BAR0, par = (m.c >> 1) & 1;
    // the row's last B tile: row 6 takes B_0 and B_1, every later one a further tile
    if (S == 6) oz_wait(bars + 8 * (OZB_FB + P * OZ_S), par, abort_flag, err);
    if (S > 0) oz_wait(bars + 8 * (OZB_FB + P * OZ_S + J + 1), par, abort_flag, err);
    oz_wait(bars + 8 * (OZB_FA + P * OZ_S + J), par, abort_flag, err);
    constexpr bool dbl = S == 2 || S == 3;
    const bool st = S == 5 ? false : dbl ? sd : ss;
    if (st) {
        const uint32_t slot = dbl ? (S == 3 ? OZ_D3 : OZ_D2) + buf : oz_slot(S, 0);
        oz_wait(bars + 8 * (OZB_TE + slot), ((dbl ? m.nd >> 1 : m.ns) & 1) ^ 1, abort_flag, err);
    }
    tc_fence_after();
    const uint64_t ad = desc_k64(smem + (P * OZ_S + J) * OZ_A_SL);
    const uint64_t bd = desc_k64(smem + OZ_STG * OZ_S * OZ_A_SL + P * OZ_S * OZ_B_SL);
    oz_row<S>(tmem, ad, bd, buf, st ? 0u : 1u);
    if (k2 > 1) oz_row<S>(tmem, ad + 2, bd + 2, buf, 1u);
    oz_commit(bars + 8 * (OZB_EA + P * OZ_S + J));
}
__device__ __forceinline__ void oz_stage(int P, uint32_t smem, uint32_t tmem, int k2, bool sd, bool ss, const OzMmaState& m,
                                         volatile int* abort_flag, int* err) {
    const int buf = (int)(m.nd & 1);
    oz_stage_row<6>(P, smem, tmem, k2, sd, ss, m, buf, abort_flag, err);
    oz_stage_row<5>(P, smem, tmem, k2, sd, ss, m, buf, abort_flag, err);
    oz_stage_row<4>(P, smem, tmem, k2, sd, ss, m, buf, abort_flag, err);
    oz_stage_row<3>(P, smem, tmem, k2, sd, ss, m, buf, abort_flag, err);
    oz_stage_row<2>(P, smem, tmem, k2, sd, ss, m, buf, abort_flag, err);
    oz_stage_row<1>(P, smem, tmem, k2, sd, ss, m, buf, abort_flag, err);
    oz_stage_row<0>(P, smem, tmem, k2, sd, ss, m, buf, abort_flag, err);
    oz_commit(smem + OZ_BAR0 + 8 * (OZB_EB + P));
}

// SYM: the real operand's rows may be those of symmetric vectors (sym_blocks.cuh).  SKIP: out.skip is looked at.
template <bool SYM, bool SKIP>
__global__ void __launch_bounds__(OZ_GT, 1) k_ozgemm(const OzArgs a) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = smem + OZ_BAR0;
    uint32_t* tmem_slot = (uint32_t*)(smem_raw + (bars + 8 * OZB_N - smem_u32(smem_raw)));
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const bool sym = SYM && sym_on(a.sym);
    const int rows = SYM ? sym_rows(a.sym, sym, a.rows) : a.rows;
    const int mt = (rows + OZ_ROWS - 1) / OZ_ROWS, nt = (a.cols + OZ_TN - 1) / OZ_TN;
    const int ntiles = mt * nt * a.batch * a.splits, kst = (a.K + OZ_BK - 1) / OZ_BK;
    if (SYM && (int)blockIdx.x >= ntiles) return;  // the symmetric rows take fewer CTAs

    if (threadIdx.x == 0) {
        for (int i = 0; i < OZB_N; ++i)  // one arrival an epilogue warp on a drained slot
            mbar_init(bars + 8 * i, i >= OZB_TE && i < OZB_TE + OZ_SLOTS ? OZ_EW : 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    if (warp == 0) {
        if (lane == 0) {
            unsigned c = 0;  // stages issued
            int na = 0;      // A tiles issued of the next one
            bool ok = true;
            for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x) {
                int z, mb, nb;
                oz_tile(a, t, mt, nt, z, mb, nb);
                const int b = z / a.splits, sp = z - b * a.splits;
                const int k0 = sp * a.cps * OZ_CHUNK, k1 = min(kst, k0 + a.cps * OZ_CHUNK);
                const uint32_t ab = 64u * min(OZ_ROWS, a.r8a - mb * OZ_ROWS), bb = 64u * min(OZ_TN, a.r8b - nb * OZ_TN);
                const long long pa = 64LL * a.r8a, pb = 64LL * a.r8b;  // plane bytes
                const uint8_t* ga = a.da + ((long long)(a.adiv ? b / a.adiv : 0) * kst + k0) * OZ_S * pa + mb * OZ_ROWS * 64LL;
                const uint8_t* gb = a.db + ((long long)(a.adiv ? b : 0) * kst + k0) * OZ_S * pb + nb * OZ_TN * 64LL;
                for (int ks = k0; ks < k1; ++ks, ++c) {
                    const uint32_t p = c & 1, par = ((c >> 1) & 1) ^ 1;
                    // A_{6-j} as its row of two stages ago finishes, then the B tiles after that stage's end
                    for (int j = 0; j < OZ_S; ++j) {
                        const uint32_t i = p * OZ_S + j, fa = bars + 8 * (OZB_FA + i);
                        if (!mbar_wait_inl(bars + 8 * (OZB_EA + i), par, abort_flag)) { ok = false; break; }
                        mbar_expect_tx(fa, ab);
                        oz_copy(smem + i * OZ_A_SL, ga + (OZ_S - 1 - j) * pa, ab, fa);
                        na = j + 1;
                    }
                    if (!ok || !mbar_wait_inl(bars + 8 * (OZB_EB + p), par, abort_flag)) { ok = false; break; }
                    for (int j = 0; j < OZ_S; ++j) {
                        const uint32_t i = p * OZ_S + j, fb = bars + 8 * (OZB_FB + i);
                        mbar_expect_tx(fb, bb);
                        oz_copy(smem + OZ_STG * OZ_S * OZ_A_SL + i * OZ_B_SL, gb + j * pb, bb, fb);
                    }
                    na = 0;
                    ga += OZ_S * pa;
                    gb += OZ_S * pb;
                }
            }
            if (!ok) {
                atomicExch(a.err, 1);
                *abort_flag = 1;
            }
            // every copy this thread issued lands before the CTA exits, also where it gave up in the middle of a stage
            // (a stage's B tiles are issued together, with its last A tile behind them)
            static_assert(OZ_STG == 2, "ring_last");
            for (int p = 0; p < OZ_STG; ++p)
                for (int j = 0; j < OZ_S; ++j) {
                    const int va = ring_last(c, na, j, p), vb = ring_last(c, 0, j, p);
                    if (va >= 0) mbar_wait(bars + 8 * (OZB_FA + p * OZ_S + j), (va >> 1) & 1, nullptr);
                    if (vb >= 0) mbar_wait(bars + 8 * (OZB_FB + p * OZ_S + j), (vb >> 1) & 1, nullptr);
                }
        }
    } else if (warp == 1) {
        OzMmaState m = {0, 0, 0};
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
            const int sp = (t / (mt * nt)) % a.splits;
            const int k0 = sp * a.cps * OZ_CHUNK, n = min(kst, k0 + a.cps * OZ_CHUNK) - k0;
            for (int i = 0; i < n; ++i, ++m.c) {
                const bool sd = i % OZ_CHUNK == 0, ss = i % (2 * OZ_CHUNK) == 0;  // accumulators that begin here
                const bool ed = i % OZ_CHUNK == OZ_CHUNK - 1 || i == n - 1;       // and that end
                const bool es = i % (2 * OZ_CHUNK) == 2 * OZ_CHUNK - 1 || i == n - 1;
                const int k2 = a.K - (k0 + i) * OZ_BK > 16 ? 2 : 1;
                oz_stage((int)(m.c & 1), smem, tmem, k2, sd, ss, m, abort_flag, a.err);
                if (es) {
                    oz_commit(bars + 8 * OZB_TFS);
                    ++m.ns;
                }
                if (ed) {
                    oz_commit(bars + 8 * (OZB_TFD + (m.nd & 1)));
                    ++m.nd;
                }
            }
        }
        // every MMA issued finishes before the tensor memory is freed
        oz_commit(bars + 8 * OZB_DRAIN);
        mbar_wait(bars + 8 * OZB_DRAIN, 0, nullptr);
    } else {
        const int q = warp & 3, cb = ((warp - 2) >> 2) * OZ_CW;
        unsigned ns = 0, nd = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x) {
            int z, mb, nb;
            oz_tile(a, t, mt, nt, z, mb, nb);
            const int b = z / a.splits, sp = z - b * a.splits;
            const int k0 = sp * a.cps * OZ_CHUNK, ni = min(kst, k0 + a.cps * OZ_CHUNK) - k0;
            const int row = mb * OZ_ROWS + 32 * q + lane, c0 = nb * OZ_TN + cb;
            long long acc[OZ_CW];
#pragma unroll
            for (int j = 0; j < OZ_CW; ++j) acc[j] = 0;
            float tail[OZ_CW];
#pragma unroll
            for (int j = 0; j < OZ_CW; ++j) tail[j] = 0.f;
            // D_d 2^(-8 d), an integer multiple of 2^(-8 d) for d <= 4, into 2^-32 units; the last accumulator is summed
            // in fp32 (its value is below 2^-22 of a sum's largest terms, its rounding below 2^-59 of the largest product)
            auto take = [&](int d, int slot) {
                const float sc = __int_as_float((127 + 8 * d) << 23);
                uint32_t r[OZ_CW];
                tmem_ld16(tmem + slot * OZ_TN + cb + ((uint32_t)(32 * q) << 16), r);
#pragma unroll
                for (int j = 0; j < OZ_CW; ++j) {
                    const float x = __uint_as_float(r[j]);
                    if (d == 5) tail[j] += x;
                    else acc[j] += (long long)((unsigned long long)(long long)__float2int_rn(x * sc) << (32 - 8 * d));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bars + 8 * (OZB_TE + slot));
            };
            for (int i = OZ_CHUNK; ok; i += OZ_CHUNK) {
                const bool end = i >= ni;
                if (end || i % (2 * OZ_CHUNK) == 0) {
                    if (!oz_all(mbar_wait_inl(bars + 8 * OZB_TFS, ns & 1, abort_flag))) { ok = false; break; }
                    tc_fence_after();
                    take(5, OZ_D5);
                    take(4, OZ_D4);
                    take(1, OZ_D1);
                    take(0, OZ_D0);
                    ++ns;
                }
                if (!oz_all(mbar_wait_inl(bars + 8 * (OZB_TFD + (nd & 1)), (nd >> 1) & 1, abort_flag))) { ok = false; break; }
                tc_fence_after();
                take(3, OZ_D3 + (int)(nd & 1));
                take(2, OZ_D2 + (int)(nd & 1));
                ++nd;
                if (end) break;
            }
            if (!ok) {
                atomicExch(a.err, 1);
                *abort_flag = 1;
                break;
            }
            if (row >= rows) continue;
            if (a.splits > 1) {
                const long long at = (long long)sp * a.cols * a.rows + row;
#pragma unroll
                for (int j = 0; j < OZ_CW; ++j)
                    if (c0 + j < a.cols) {
                        a.raw[at + (long long)(c0 + j) * a.rows] = acc[j];
                        a.rawt[at + (long long)(c0 + j) * a.rows] = tail[j];
                    }
                continue;
            }
            const int* eb = a.eb + (a.adiv ? (long long)b * a.cols : 0) + c0;
            const int ea = a.ea[(a.adiv ? b / a.adiv * a.rows : 0) + row];
            long long at = (long long)b * a.out.bs + (long long)row * a.out.rs, mirror = 0;
            if (sym) {
                int i, j;
                if (!sym_at(a.sym, row, i, j)) continue;
                at = (long long)i * a.sym.n + j;
                if (i >> 3 != j >> 3) mirror = (long long)j * a.sym.n + i - at;
            } else if (SYM) {
                at += a.sym.r0;
            }
            const int ex = ea - 14 + a.out.aexp;
#pragma unroll
            for (int j = 0; j < OZ_CW; j += 2) {
                if (c0 + j < a.cols) {
                    const int e0 = eb[j], e1 = eb[j + 1], m = (c0 + j) >> 1;
                    double2 v = make_double2(oz_to_double(acc[j], tail[j], ex + e0),
                                             oz_to_double(acc[j + 1], tail[j + 1], ex + e1));
                    if (ea == OZ_NAN || e0 == OZ_NAN) v.x = __longlong_as_double(0x7ff8000000000000ll);
                    if (ea == OZ_NAN || e1 == OZ_NAN) v.y = __longlong_as_double(0x7ff8000000000000ll);
                    const int mh = a.out.md == 1 ? m : m / a.out.md;
                    const long long e = at + (long long)mh * a.out.ms1 + (long long)(m - mh * a.out.md) * a.out.ms0;
                    if (a.out.add) v = cadd(v, a.out.add[e]);
                    if (SKIP && a.out.skip[mh / a.out.sd % a.out.sm]) continue;
                    a.out.C[e] = v;
                    if (SYM && mirror) a.out.C[e + mirror] = v;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// The K splits' sums added (the integers exactly, the tails in order) and converted.
__global__ void k_oz_finish(const OzArgs a) {
    const bool sym = sym_on(a.sym);
    const int rows = sym_rows(a.sym, sym, a.rows);
    const long long total = (long long)rows * (a.cols >> 1);
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int m = (int)(e / rows), row = (int)(e - (long long)m * rows);
        int i = 0, j = 0;
        if (sym && !sym_at(a.sym, row, i, j)) continue;
        long long re = 0, im = 0;
        float tr = 0.f, ti = 0.f;
        for (int z = 0; z < a.splits; ++z) {
            const long long at = ((long long)z * a.cols + 2 * m) * a.rows + row;
            re += a.raw[at];
            im += a.raw[at + a.rows];
            tr += a.rawt[at];
            ti += a.rawt[at + a.rows];
        }
        const int ea = a.ea[row], e0 = a.eb[2 * m], e1 = a.eb[2 * m + 1], ex = ea - 14 + a.out.aexp;
        double2 v = make_double2(oz_to_double(re, tr, ex + e0), oz_to_double(im, ti, ex + e1));
        if (ea == OZ_NAN || e0 == OZ_NAN) v.x = __longlong_as_double(0x7ff8000000000000ll);
        if (ea == OZ_NAN || e1 == OZ_NAN) v.y = __longlong_as_double(0x7ff8000000000000ll);
        const int mh = m / a.out.md;
        const long long am = (long long)mh * a.out.ms1 + (long long)(m - mh * a.out.md) * a.out.ms0;
        const long long at = am + (sym ? (long long)i * a.sym.n + j : (long long)row * a.out.rs + a.sym.r0);
        if (a.out.add) v = cadd(v, a.out.add[at]);
        a.out.C[at] = v;
        if (sym && i >> 3 != j >> 3) a.out.C[am + (long long)j * a.sym.n + i] = v;
    }
}

// *asym |= the G matrices (n x n) are not all symmetric, bit for bit: 32 x 32 blocks I <= J against their mirrors.
__global__ void __launch_bounds__(256) k_oz_asym(int n, int G, const double* __restrict__ L, int* asym) {
    __shared__ unsigned long long tile[2][32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    int J = 0, I = blockIdx.x;
    while (I > J) I -= ++J;
    const int i = 32 * I, j = 32 * J;
    bool bad = false;
    for (int g = 2 * blockIdx.y; g < G; g += 2 * gridDim.y) {  // two matrices at a time: bytes in flight
        unsigned long long a[2][4], b[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const unsigned long long* x = (const unsigned long long*)L + (size_t)(g + h) * n * n;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = ty + 8 * q;
                a[h][q] = g + h < G && i + r < n && j + tx < n ? x[(size_t)(i + r) * n + j + tx] : 0ull;
                b[h][q] = g + h < G && j + r < n && i + tx < n ? x[(size_t)(j + r) * n + i + tx] : 0ull;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q) tile[h][ty + 8 * q][tx] = a[h][q];
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q) bad |= b[h][q] != tile[h][tx][ty + 8 * q];
        if (__syncthreads_or(bad || *(volatile int*)asym)) break;
    }
    if (bad) *asym = 1;
}

// ------------------------------------------------------------------ digits --
// A digit array: [batch][32 k][digit] planes of r8 rows x 64 bytes.
struct OzDst {
    uint8_t* d;
    int nks, r8;
};
// eight consecutive k (k a multiple of 8) of row r of batch b into the seven planes
__device__ __forceinline__ void oz_store8(const OzDst& o, long long b, int r, int k, const long long (&y)[8]) {
    const long long plane = 64LL * o.r8;
    uint8_t* d = o.d + (b * o.nks + (k >> 5)) * OZ_S * plane + r * 64LL + ((((k >> 3) ^ (r >> 1)) & 3) << 4);
    *(uint4*)(d) = oz_pack8<0>(y);
    *(uint4*)(d + plane) = oz_pack8<1>(y);
    *(uint4*)(d + 2 * plane) = oz_pack8<2>(y);
    *(uint4*)(d + 3 * plane) = oz_pack8<3>(y);
    *(uint4*)(d + 4 * plane) = oz_pack8<4>(y);
    *(uint4*)(d + 5 * plane) = oz_pack8<5>(y);
    *(uint4*)(d + 6 * plane) = oz_pack8<6>(y);
}
// The largest of the values of the LN threads that share a row (LN <= 32 lanes of a warp, or the CTA's 256).
template <int LN>
__device__ __forceinline__ int row_max(int e, int* s_max) {
#pragma unroll
    for (int o = (LN < 32 ? LN : 32) / 2; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    if (LN <= 32) return e;
    __syncthreads();  // the last row's values have been read
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = e;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) e = max(e, s_max[i]);
    return e;
}

// Real rows with K contiguous (row r at src + r ld), LN threads a row: a lane
// cuts eight entries, so a warp takes four rows of up to 64 entries, and a CTA
// takes one where rows are few and long.  `per` rows a batch; one: minus the
// identity.  Every split writes zeros from K up to a multiple of 32.  AMAX: of
// one batch, whose largest scale amax is raised to.
template <int LN, bool AMAX>
__global__ void __launch_bounds__(256) k_oz_rows(long long rows, int per, int K, const double* __restrict__ src,
                                                 long long ld, int one, OzDst dst, int* __restrict__ ex, int* amax) {
    __shared__ int s_max[8];
    const int t = threadIdx.x % LN;  // place in the row's threads
    constexpr int RC = 256 / LN;     // rows a CTA
    int most = OZ_EMPTY;
    // every thread of a warp stays for the shuffles
    for (long long r0 = (long long)blockIdx.x * RC; r0 < rows; r0 += (long long)gridDim.x * RC) {
        const long long r = r0 + threadIdx.x / LN;
        const bool in = r < rows;
        const double* x = src + (in ? r : 0) * ld;
        const long long rd = one ? r : -1;  // the diagonal entry to lower by one
        int e = 0;
        if (in) {
#pragma unroll 4
            for (int k = t; k < K; k += LN) e = max(e, oz_key(k == rd ? x[k] - 1.0 : x[k]));
        }
        const int E = oz_scale(row_max<LN>(e, s_max));
        if (!in) continue;
        if (t == 0) ex[r] = E;
        if (AMAX) most = max(most, E);
        const long long b = r / per;
        for (int k = 8 * t; k < 32 * dst.nks; k += 8 * LN) {
            long long y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = oz_fix(k + i < K ? (k + i == rd ? x[k + i] - 1.0 : x[k + i]) : 0.0, E);
            oz_store8(dst, b, (int)(r - b * per), k, y);
        }
    }
    if (AMAX) {
        most = __reduce_max_sync(0xffffffffu, most);
        if ((threadIdx.x & 31) == 0) atomicMax(amax, most);
    }
}

// Complex rows with K contiguous: digit rows 2 r (real parts) and 2 r + 1.
// amax (optional): set for the other operand's cut to raise; arrived, one a 64 rows, too (k_zgemm_lost).
template <int LN>
__global__ void __launch_bounds__(256) k_oz_crows(long long rows, int K, const double2* __restrict__ src, long long ld,
                                                  OzDst dst, int* __restrict__ ex, int* __restrict__ amax,
                                                  int* __restrict__ arrived) {
    __shared__ int s_max[2][8];
    const int t = threadIdx.x % LN;
    if (amax && blockIdx.x == 0 && threadIdx.x == 0) *amax = OZ_EMPTY;
    for (long long r = (long long)blockIdx.x * (256 / LN) + threadIdx.x / LN; r < rows;
         r += (long long)gridDim.x * (256 / LN)) {
        const double2* x = src + r * ld;
        int e0 = 0, e1 = 0;
#pragma unroll 4
        for (int k = t; k < K; k += LN) {
            const double2 v = x[k];
            e0 = max(e0, oz_key(v.x));
            e1 = max(e1, oz_key(v.y));
        }
        const int E0 = oz_scale(row_max<LN>(e0, s_max[0])), E1 = oz_scale(row_max<LN>(e1, s_max[1]));
        if (t == 0) {
            ex[2 * r] = E0;
            ex[2 * r + 1] = E1;
            if (amax && r % 64 == 0) arrived[r / 64] = 0;
        }
        for (int k = 8 * t; k < 32 * dst.nks; k += 8 * LN) {
            long long y[8], w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const double2 v = k + i < K ? x[k + i] : make_double2(0.0, 0.0);
                y[i] = oz_fix(v.x, E0);
                w[i] = oz_fix(v.y, E1);
            }
            oz_store8(dst, 0, (int)(2 * r), k, y);
            oz_store8(dst, 0, (int)(2 * r + 1), k, w);
        }
    }
}

// Real rows with K strided: row r's entry k at src[k ld + r es] (or at the
// place of symmetric vectors' row r); RB rows a CTA (32, or 8 where few rows
// would leave SMs idle), transposed through shared memory.
template <int RB>
__global__ void __launch_bounds__(256) k_oz_cols(int nrows, int K, const double* __restrict__ src, long long ld, int es,
                                                 OzDst dst, int* __restrict__ ex, SymRows sym, int* amax) {
    constexpr int TY = 256 / RB, KT = 8 * TY;  // threads a row; k at a time
    __shared__ double tile[RB][KT + 1];
    __shared__ int se[RB], s_most;
    const int tx = threadIdx.x % RB, ty = threadIdx.x / RB, r0 = blockIdx.x * RB;
    const bool sy = sym_on(sym);
    const int rows = sym_rows(sym, sy, nrows);
    if (r0 >= rows) return;
    bool in = r0 + tx < rows;
    long long at = (long long)(r0 + tx) * es;
    if (sy) {
        int i, j;
        in = sym_at(sym, r0 + tx, i, j) && in;
        at = (long long)i * sym.n + j;
    } else {
        at += sym.r0;
    }
    if (threadIdx.x < RB) se[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_most = OZ_EMPTY;
    __syncthreads();
    int e = 0;
    if (in) {
#pragma unroll 8
        for (int k = ty; k < K; k += TY) e = max(e, oz_key(src[(long long)k * ld + at]));
    }
    atomicMax(&se[tx], e);
    __syncthreads();
    const int rr = threadIdx.x / TY, kq = (threadIdx.x % TY) * 8, E = oz_scale(se[rr]);
    if (threadIdx.x % TY == 0 && r0 + rr < rows) {
        ex[r0 + rr] = E;
        atomicMax(&s_most, E);
    }
    for (int k0 = 0; k0 < 32 * dst.nks; k0 += KT) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int k = k0 + ty + TY * i;
            tile[tx][ty + TY * i] = in && k < K ? src[(long long)k * ld + at] : 0.0;
        }
        __syncthreads();
        if (r0 + rr < rows && k0 + kq < 32 * dst.nks) {
            long long y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = oz_fix(tile[rr][kq + i], E);
            oz_store8(dst, 0, r0 + rr, k0 + kq, y);
        }
    }
    if (amax && threadIdx.x == 0) atomicMax(amax, s_most);  // every row's is in: the loop above has barriers
}

// Walker-shaped blocks (j, c), c fastest, `ws` entries apart, eight columns c
// a CTA.  Two blocks `ss` apart may be taken as one of 2 `on` columns (the two
// spins, or halves, that share a V: their products fill one tile's columns):
//   WALK  digits of the block's columns over j, rows (w, c, part)
//   PLAIN digits of T = Y as the right operand of V T
//   INIT  T = W + Y; U = T; digits of T as the right operand of V T
//   TERM  T = i s Y; U += T; digits of T as the right operand of V T
//   LAST  T = i s Y; U += T; digits of U as WALK's
// The right operand of V T (V's rows hold Re, Im interleaved): rows (c, Re)
// [Tr, -Ti] and (c, Im) [Ti, Tr] over (j, part), a batch a walker.
//   COLS  as WALK, a batch a walker (both operands of its Gram matrix)
//   BACK  T = U - i s Y; digits of T as the right operand of V T
//   BACKL T = U = U - i s Y; digits of U as WALK's
// tp (optional): T also there, tw entries a walker apart.  mx.p (optional):
// raised, at the walker (w / mx.div) % mx.mod, to the largest scale of the cut
// entries times 2^mx.add.
struct OzMax {
    int *p, div, mod, add;
};
enum { OZ_WALK, OZ_PLAIN, OZ_INIT, OZ_TERM, OZ_LAST, OZ_COLS, OZ_BACK, OZ_BACKL };
constexpr int OZ_CB = 8;
template <int MODE>
__global__ void __launch_bounds__(256, MODE == OZ_WALK || MODE == OZ_LAST || MODE == OZ_COLS || MODE == OZ_BACKL ? 4 : 3)
    k_oz_term(int n, int o, int on, long long ws, long long ss, int ncg, double s, const double2* __restrict__ Y,
                                                 const double2* __restrict__ W, double2* __restrict__ U, OzDst dst, int* __restrict__ ex,
                                                 double2* __restrict__ tp, long long tw, OzMax mx) {
    constexpr bool SERIES = MODE == OZ_INIT || MODE == OZ_TERM || MODE == OZ_LAST || MODE == OZ_BACK || MODE == OZ_BACKL;
    extern __shared__ double2 sh[];  // OZ_CB x (n + 1)
    __shared__ int se[2 * OZ_CB];
    const int w = blockIdx.x / ncg, c0 = (blockIdx.x - w * ncg) * OZ_CB, tid = threadIdx.x;
    const int c = tid & (OZ_CB - 1), pitch = n + 1;
    if (tid < 2 * OZ_CB) se[tid] = 0;
    __syncthreads();
    int e0 = 0, e1 = 0;
    if (c0 + c < o) {
        const int spin = c0 + c >= on;
        for (int j = tid / OZ_CB; j < n; j += 256 / OZ_CB) {
            const long long at = w * ws + (long long)j * on + (c0 + c - spin * on) + spin * ss;
            double2 t = Y[at];
            if (MODE == OZ_TERM || MODE == OZ_LAST) {
                t = make_double2(-s * t.y, s * t.x);
                const double2 u = cadd(U[at], t);
                U[at] = u;
                if (MODE == OZ_LAST) t = u;
            }
            if (MODE == OZ_INIT) U[at] = t = cadd(W[at], t);
            if (MODE == OZ_BACK || MODE == OZ_BACKL) {
                const double2 u = U[at];
                t = make_double2(fma(s, t.y, u.x), fma(-s, t.x, u.y));
                if (MODE == OZ_BACKL) U[at] = t;
            }
            if (SERIES && MODE != OZ_LAST && tp) tp[w * tw + (long long)j * on + c0 + c] = t;
            sh[c * pitch + j] = t;
            e0 = max(e0, oz_key(t.x));
            e1 = max(e1, oz_key(t.y));
        }
    }
    atomicMax(&se[2 * c], e0);
    atomicMax(&se[2 * c + 1], e1);
    __syncthreads();
    const int cn = min(OZ_CB, o - c0);
    if (MODE != OZ_COLS && MODE != OZ_PLAIN && mx.p && tid < 32) {
        const int E = oz_scale(__reduce_max_sync(0xffffffffu, tid < 2 * cn ? se[tid] : 0));
        if (tid == 0) atomicMax(mx.p + w / mx.div % mx.mod, E == OZ_NAN || E == OZ_ZERO ? E : E + mx.add);
    }
    if (MODE == OZ_WALK || MODE == OZ_LAST || MODE == OZ_COLS || MODE == OZ_BACKL) {
        const int nq = 4 * dst.nks;
        for (int it = tid; it < cn * nq; it += 256) {
            const int cc = it / nq, j = (it - cc * nq) * 8;
            const int E0 = oz_scale(se[2 * cc]), E1 = oz_scale(se[2 * cc + 1]);
            long long y[8], x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const double2 t = j + i < n ? sh[cc * pitch + j + i] : make_double2(0.0, 0.0);
                y[i] = oz_fix(t.x, E0);
                x[i] = oz_fix(t.y, E1);
            }
            const int b = MODE == OZ_COLS ? w : 0, row = 2 * ((w - b) * o + c0 + cc);
            oz_store8(dst, b, row, j, y);
            oz_store8(dst, b, row + 1, j, x);
            if (j == 0) {
                ex[(long long)b * 2 * o + row] = E0;
                ex[(long long)b * 2 * o + row + 1] = E1;
            }
        }
    } else {
        const int nq = 4 * dst.nks;
        for (int it = tid; it < cn * nq; it += 256) {
            const int cc = it / nq, j = (it - cc * nq) * 4;
            const int E = oz_scale(max(se[2 * cc], se[2 * cc + 1]));
            long long y[8], x[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 t = j + i < n ? sh[cc * pitch + j + i] : make_double2(0.0, 0.0);
                y[2 * i] = oz_fix(t.x, E);
                y[2 * i + 1] = oz_fix(-t.y, E);
                x[2 * i] = oz_fix(t.y, E);
                x[2 * i + 1] = y[2 * i];
            }
            const int row = 2 * (c0 + cc);
            oz_store8(dst, w, row, 2 * j, y);
            oz_store8(dst, w, row + 1, 2 * j, x);
            if (j == 0) {
                ex[(long long)w * 2 * o + row] = E;
                ex[(long long)w * 2 * o + row + 1] = E;
            }
        }
    }
}

__device__ __forceinline__ void cfma2(double& re, double& im, double2 a, double2 b) {
    re = fma(a.x, b.x, re);
    im = fma(a.x, b.y, im);
    re = fma(-a.y, b.y, re);
    im = fma(a.y, b.x, im);
}

// The adjoint's outer products: row i of walker w over (k, c, part) is
// conj(i sqrt_dt / k) tb_k[i, c] = (sqrt_dt / k) (tb.y, -tb.x), k = 1 .. K (A); the right
// operand's rows (j, Re) [Re, Im] and (j, Im) [-Im, Re] of t_{k-1}[j, c] give
// sum a conj(t).  LN lanes a row, eight entries a lane.
template <int LN>
__global__ void __launch_bounds__(256) k_oz_vbar(int W, int n, int o, int K, double sqrt_dt,
                                                 const double2* __restrict__ tbar, const double2* __restrict__ terms,
                                                 OzDst A, int* __restrict__ ea, OzDst B, int* __restrict__ eb) {
    constexpr int RC = 256 / LN;  // rows a CTA
    const int t = threadIdx.x % LN, no = n * o, L = K * o;
    const long long rows = (long long)W * n;
    // every thread of a warp stays for the shuffles
    for (long long r0 = (long long)blockIdx.x * RC; r0 < 2 * rows; r0 += (long long)gridDim.x * RC) {
        const long long r = r0 + threadIdx.x / LN;
        const bool in = r < 2 * rows, right = in && r >= rows;
        const long long x = !in ? 0 : right ? r - rows : r;
        const int w = (int)(x / n), i = (int)(x - (long long)w * n);
        // entry l = (k - 1) o + c of the row
        const double2* src = right ? terms + (long long)w * K * no + (long long)i * o
                                   : tbar + ((long long)w * (K + 1) + 1) * no + (long long)i * o;
        auto at = [&](int l) {
            const int k = l / o;
            double2 v = src[(long long)k * no + (l - k * o)];
            if (!right) {
                const double c = sqrt_dt / (k + 1);
                v = make_double2(c * v.y, -c * v.x);
            }
            return v;
        };
        int e = 0;
        for (int l = t; in && l < L; l += LN) {
            const double2 v = at(l);
            e = max(e, max(oz_key(v.x), oz_key(v.y)));
        }
        const int E = oz_scale(row_max<LN>(e, nullptr));
        if (!in) continue;
        if (t == 0) {
            if (right) eb[2 * x] = eb[2 * x + 1] = E;
            else ea[x] = E;
        }
        for (int k = 8 * t; k < 32 * A.nks; k += 8 * LN) {
            long long y[8], z[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int l = k / 2 + q;
                const double2 v = l < L ? at(l) : make_double2(0.0, 0.0);
                y[2 * q] = oz_fix(v.x, E);
                y[2 * q + 1] = oz_fix(v.y, E);
                z[2 * q] = oz_fix(-v.y, E);
                z[2 * q + 1] = y[2 * q];
            }
            if (right) {
                oz_store8(B, w, 2 * i, k, y);
                oz_store8(B, w, 2 * i + 1, k, z);
            } else {
                oz_store8(A, w, i, k, y);
            }
        }
    }
}

__device__ __forceinline__ int warp_max(const int* x, int n) {
    int m = OZ_EMPTY;
    for (int i = threadIdx.x & 31; i < n; i += 32) m = max(m, x[i]);
    return __reduce_max_sync(0xffffffffu, m);
}

// Coulomb and exchange partials of a chunk of ng Cholesky vectors from F
// (rows (w, k), columns (g, i): f_g[i, k]), as launch_energy_partial's:
// partial[w, chunk] = (sum_g (tr f_g)^2, sum_g sum_ik f_g[i, k] f_g[k, i]).
// Its floor is the binary64 pipe: four FMAs a pair i < k.  F's blocks are
// checked (oz_lost; scales ea of L~'s rows (g, i) and eb of G_half's) and, where
// they have lost too much, formed here from L~ and G_half.
__global__ void __launch_bounds__(256) k_oz_exchange(int n, int o, int G, int NG, const double2* __restrict__ F,
                                                     double2* __restrict__ partial, const int* __restrict__ ea,
                                                     const int* __restrict__ eb,
                                                     const double* __restrict__ rot, const double2* __restrict__ green) {
    extern __shared__ double2 sh[];  // NG blocks of o x (o + 1)
    const int nchunk = gridDim.x, w = blockIdx.y, g0 = blockIdx.x * NG, ng = min(NG, G - g0), tid = threadIdx.x;
    const int lane = tid & 31, wid = tid >> 5;
    const int pitch = o + 1, gi = ng * o;
    const double2* Fw = F + (long long)w * o * G * o + (long long)g0 * o;
    const float io = 1.0f / o;  // quotients of small integers below: (x + 0.5) / o is never within rounding of an integer
    __shared__ int s_max[2];
    if (wid == 7) {  // which mostly has no column below
        const int am = warp_max(ea + g0 * o, gi), bm = warp_max(eb + (long long)w * 2 * o, 2 * o);
        if (lane == 0) {
            s_max[0] = am;
            s_max[1] = bm;
        }
    }
    for (int x = tid; x < gi; x += 256) {
        const int g = (int)((x + 0.5f) * io), i = x - g * o;
        const double2* src = Fw + x;
        double2* dst = sh + g * o * pitch + i;
#pragma unroll 8
        for (int k = 0; k < o; ++k) dst[k * pitch] = src[(long long)k * G * o];
    }
    __syncthreads();
    const int am = s_max[0], bm = s_max[1];
    const int reach = oz_reach(am, bm);
    bool lost = oz_lost(am, bm, oz_scan(sh, pitch - 1, reach));  // a row of the first block tells enough, mostly
    if (lost) {
        bool any = false;
        for (int x = tid; x < gi; x += 256)
            for (int k = 0; k < o; ++k) any |= oz_key_expo(oz_key(sh[(x / o * o + k) * pitch + x % o])) >= reach;
        lost = oz_lost(am, bm, __syncthreads_or(any));
    }
    if (lost) {
        for (int e = tid; e < gi * o; e += 256) {
            const int k = e / gi, x = e - k * gi, g = x / o;
            const double* l = rot + ((long long)g0 * o + x) * n;
            const double2* gk = green + ((long long)w * o + k) * n;
            double2 f = make_double2(0.0, 0.0);
            for (int j = 0; j < n; ++j) rfma(f, l[j], gk[j]);
            sh[(g * o + k) * pitch + x - g * o] = f;
        }
        __syncthreads();
    }
    double cr = 0.0, ci = 0.0, xr = 0.0, xi = 0.0;
    // sum over i < k of f[i, k] f[k, i], doubled below, a warp a vector: rows k = r and o - 1 - r hold o - 1 such pairs
    // together (the middle row of an odd o half of that)
    const int half = (o + 1) / 2, per = o > 1 ? o - 1 : 1, mid = o & 1 ? half - 1 : -1;
    const float ip = 1.0f / per;
    for (int g = wid; g < ng; g += 8) {
        const double2* f = sh + g * o * pitch;
        for (int e = lane; e < half * per; e += 32) {
            const int r = (int)((e + 0.5f) * ip), c = e - r * per, hi = o - 1 - r;
            const int k = c < hi ? hi : r, i = c < hi ? c : c - hi;
            if (i >= k || (r == mid && c >= hi)) continue;
            cfma2(xr, xi, f[k * pitch + i], f[i * pitch + k]);
        }
    }
    xr *= 2.0;
    xi *= 2.0;
    for (int e = tid; e < gi; e += 256) {
        const double2 f = sh[e * pitch + (e - (int)((e + 0.5f) * io) * o)];
        cfma2(xr, xi, f, f);
    }
    for (int g = tid; g < ng; g += 256) {
        double2 c = make_double2(0.0, 0.0);
        for (int i = 0; i < o; ++i) c = cadd(c, sh[(g * o + i) * pitch + i]);
        cfma2(cr, ci, c, c);
    }
    cr = warp_sum(cr); ci = warp_sum(ci); xr = warp_sum(xr); xi = warp_sum(xi);
    __shared__ double red[8][4];
    if (lane == 0) {
        red[wid][0] = cr; red[wid][1] = ci; red[wid][2] = xr; red[wid][3] = xi;
    }
    __syncthreads();
    if (tid == 0) {
        for (int i = 1; i < 8; ++i) {
            cr += red[i][0]; ci += red[i][1]; xr += red[i][2]; xi += red[i][3];
        }
        partial[((size_t)w * nchunk + blockIdx.x) * 2] = make_double2(cr, ci);
        partial[((size_t)w * nchunk + blockIdx.x) * 2 + 1] = make_double2(xr, xi);
    }
}

// flag[w]: one of walker w's two products (at most) has lost too much (oz_lost): scales of its `rows` rows (shared: of
// all) and `cols` columns, its `results` results.  A warp a walker.
struct OzWalk {
    const int *a, *b;
    const double2* c;
    int results, rows, cols, shared;
};
__global__ void __launch_bounds__(128) k_oz_flags(int W, OzWalk g, OzWalk h, int* __restrict__ flag) {
    const int w = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (w >= W) return;
    auto lost = [&](const OzWalk& p) {
        if (!p.c) return false;
        const int a = warp_max(p.a + (p.shared ? 0 : (long long)w * p.rows), p.rows);
        const int b = warp_max(p.b + (long long)w * p.cols, p.cols);
        return oz_lost(a, b, oz_scan(p.c + (long long)w * p.results, p.results, oz_reach(a, b)));
    };
    const bool l = lost(g) || lost(h);
    if ((threadIdx.x & 31) == 0) flag[w] = l;
}

// The same of a Taylor series, whose products are to be judged by its sum U (E_half X and its last product are X + (E -
// I) X): largest scales of E - I (e) and X, of the terms times their coefficients (t), of U (u), and those of V's n rows.
struct OzSeries {
    int *e, *x, *t, *u, *flag;
};
__global__ void __launch_bounds__(128) k_oz_series_flags(int W, int n, OzSeries g, const int* __restrict__ v) {
    const int w = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (w >= W) return;
    const int a = warp_max(v + (long long)w * n, n);
    if ((threadIdx.x & 31) != 0) return;
    auto lost = [&](int a, int b) { return oz_lost(a, b, g.u[w] - 1 >= oz_reach(a, b)); };
    g.flag[w] = lost(*g.e, g.x[w]) || lost(a, g.t[w]);
}

constexpr int OZ_XSMEM = 96 * 1024;  // the exchange kernel's F blocks
DeviceOnce g_ozterm[8], g_ozx;
template <bool SYM, bool SKIP>
int run_ozgemm(const OzArgs& a, int grid, cudaStream_t s) {
    static DeviceOnce once;
    AFQ_TRY(raise_smem_once(once, k_ozgemm<SYM, SKIP>, OZ_GSMEM));
    k_ozgemm<SYM, SKIP><<<grid, OZ_GT, OZ_GSMEM, s>>>(a);
    AFQ_LAUNCHED("k_ozgemm");
    return AFQ_OK;
}

int nks_of(int K) { return (K + OZ_BK - 1) / OZ_BK; }
long long digit_row_bytes(int K) { return 64LL * OZ_S * nks_of(K); }

// Digit arrays of one operand.
struct OzDigits {
    uint8_t* d;
    int* ex;
};

// K splits (and 256-k chunks a split) so that few tiles still fill the GPU.
void oz_splits(long long tiles, int K, int sms, int& splits, int& cps) {
    const int nch = (K + OZ_BK * OZ_CHUNK - 1) / (OZ_BK * OZ_CHUNK);
    int z = (int)(sms / (tiles > 0 ? tiles : 1));
    if (z > nch) z = nch;
    if (z < 1) z = 1;
    cps = (nch + z - 1) / z;
    splits = (nch + cps - 1) / cps;
}

int oz_launch(int rows, int cols, int K, int batch, int adiv, const OzDigits& A, const OzDigits& B, const OzOut& out,
              int splits, int cps, long long* raw, int* err, cudaStream_t s, const SymRows& sym = {}) {
    OzArgs a = {};
    a.sym = sym;
    a.da = A.d; a.db = B.d;
    a.r8a = (int)round_up(rows, 8); a.r8b = (int)round_up(cols, 8);
    a.rows = rows; a.cols = cols; a.K = K; a.batch = batch; a.adiv = adiv;
    a.splits = splits; a.cps = cps;
    a.ea = A.ex; a.eb = B.ex; a.raw = raw; a.err = err; a.out = out;
    a.rawt = (float*)(raw + (long long)splits * cols * rows);
    const int mt = (rows + OZ_ROWS - 1) / OZ_ROWS, nt = (cols + OZ_TN - 1) / OZ_TN;
    // column tiles fastest in groups whose digits take at most 40 MB of L2
    const long long tb = OZ_TN * digit_row_bytes(K);
    long long gn = (40LL << 20) / (tb > 0 ? tb : 1);
    if (gn < 1) gn = 1;
    if (gn > nt) gn = nt;
    a.gn = (int)gn;
    int sms = 0;
    AFQ_TRY(device_sms(&sms));
    const long long tiles = (long long)mt * nt * batch * splits;
    if (tiles > 0x7fffffffLL) return fail(AFQ_E_UNSUPPORTED, "digit GEMM: %lld tiles", tiles);
    const int grid = tiles < sms ? (int)tiles : sms;
    if (sym.asym) AFQ_TRY((run_ozgemm<true, false>(a, grid, s)));
    else if (out.skip) AFQ_TRY((run_ozgemm<false, true>(a, grid, s)));
    else AFQ_TRY((run_ozgemm<false, false>(a, grid, s)));
    if (splits > 1) {
        long long blocks = ((long long)rows * (cols >> 1) + 255) / 256;
        if (blocks > 152 * 16) blocks = 152 * 16;
        k_oz_finish<<<(unsigned)blocks, 256, 0, s>>>(a);
        AFQ_LAUNCHED("k_oz_finish");
    }
    return AFQ_OK;
}

OzDst dst_of(const OzDigits& D, long long rows, int K) { return {D.d, nks_of(K), (int)round_up(rows, 8)}; }

unsigned row_blocks(long long rows, int per_cta = 8) {
    const long long b = (rows + per_cta - 1) / per_cta;
    return (unsigned)(b > 152 * 64 ? 152 * 64 : b);
}
// A warp a row leaves SMs idle below some 16 warps an SM; a row of a few hundred k is short for a CTA.
bool row_cta(long long rows, int K) { return rows < 16 * 152 && K >= 512; }
int split_rows(long long rows, int per, int K, const double* src, long long ld, const OzDigits& D, cudaStream_t s,
               int* amax = nullptr, int one = 0) {
    const OzDst dst = dst_of(D, per, K);
#define AFQ_OZR(LN, BLOCKS)                                                                                       \
    do {                                                                                                          \
        if (amax) k_oz_rows<LN, true><<<BLOCKS, 256, 0, s>>>(rows, per, K, src, ld, one, dst, D.ex, amax);        \
        else k_oz_rows<LN, false><<<BLOCKS, 256, 0, s>>>(rows, per, K, src, ld, one, dst, D.ex, nullptr);         \
    } while (0)
    if (row_cta(rows, K)) AFQ_OZR(256, row_blocks(rows, 1));
    else if (K <= 64) AFQ_OZR(8, row_blocks(rows, 32));
    else if (K <= 128) AFQ_OZR(16, row_blocks(rows, 16));
    else AFQ_OZR(32, row_blocks(rows));
#undef AFQ_OZR
    AFQ_LAUNCHED("k_oz_rows");
    return AFQ_OK;
}
int split_crows(long long rows, int K, const double2* src, long long ld, const OzDigits& D, cudaStream_t s,
                int* amax = nullptr, int* arrived = nullptr) {
    const OzDst dst = dst_of(D, 2 * rows, K);
    if (row_cta(rows, K)) k_oz_crows<256><<<row_blocks(rows, 1), 256, 0, s>>>(rows, K, src, ld, dst, D.ex, amax, arrived);
    else k_oz_crows<32><<<row_blocks(rows), 256, 0, s>>>(rows, K, src, ld, dst, D.ex, amax, arrived);
    AFQ_LAUNCHED("k_oz_crows");
    return AFQ_OK;
}
int split_cols(int rows, int K, const double* src, long long ld, const OzDigits& D, cudaStream_t s, int* amax, int es = 1,
               const SymRows& sym = {}) {
    const OzDst dst = dst_of(D, rows, K);
    if (rows <= 32 * 152) k_oz_cols<8><<<(rows + 7) / 8, 256, 0, s>>>(rows, K, src, ld, es, dst, D.ex, sym, amax);
    else k_oz_cols<32><<<(rows + 31) / 32, 256, 0, s>>>(rows, K, src, ld, es, dst, D.ex, sym, amax);
    AFQ_LAUNCHED("k_oz_cols");
    return AFQ_OK;
}
OzDigits take_digits(Arena& a, size_t rows, int K, size_t batch = 1) {
    OzDigits D;
    D.d = a.take<uint8_t>(batch * round_up(rows, 8) * digit_row_bytes(K));
    D.ex = a.take<int>(batch * rows);
    return D;
}

// Digit scratch is bounded: operands whose digits take more than this are
// processed in row chunks (but the energy's rotated vectors, cut whole).
constexpr long long OZ_CAP = 1LL << 30;
int cap_rows(long long rows, long long bytes_per_row) {
    long long c = OZ_CAP / (bytes_per_row > 0 ? bytes_per_row : 1) / OZ_ROWS * OZ_ROWS;
    if (c < OZ_ROWS) c = OZ_ROWS;
    return (int)(c < rows ? c : rows);
}

// W walkers in equal chunks of at most `most`
int even_chunk(int W, long long most) {
    if (most < 1) most = 1;
    const long long n = (W + most - 1) / most;
    return (int)((W + n - 1) / n);
}

// a call's layout in the region that it was given
int oz_room(const Arena& a) {
    if (!a.base || !a.ok()) return fail(AFQ_E_WORKSPACE, "digit scratch of %zu bytes < %zu needed", a.cap, a.used);
    return AFQ_OK;
}

constexpr int OZ_TILE_SMS = 152;

constexpr int OZ_LOST = 64;  // rows a tile of k_zgemm_lost
struct ZLayout {
    int mc, nc;
    OzDigits A, B;
    long long* raw;
    int *asym, *amax, *arrived;
};
ZLayout z_layout(Arena& a, int M, int N, int K) {
    ZLayout z;
    const long long rb = digit_row_bytes(K);
    z.mc = cap_rows(M, 2 * rb);
    z.nc = cap_rows(N, rb);
    z.A = take_digits(a, z.nc, K);
    z.B = take_digits(a, 2 * (size_t)z.mc, K);
    // K splits: at most one tile an SM, at most one split a 256-k chunk
    const size_t nch = (K + 255) / 256, most = (size_t)OZ_TILE_SMS * OZ_ROWS * OZ_TN, all = nch * 2 * z.mc * z.nc;
    z.raw = a.take<long long>((nch > 1 ? (all < most ? all : most) : 0) * 3 / 2);  // 64-bit sums, 32-bit tails
    z.asym = a.take<int>(64);
    z.amax = a.take<int>(1);
    z.arrived = a.take<int>((z.mc + OZ_LOST - 1) / OZ_LOST);
    return z;
}

}  // namespace

// Routes.  The binary64 kernels' own limits stay (a call past them is theirs
// to refuse).  Measured in captured graphs, binary64 pipe -> digits:
//   GEMM     wins over k_zgemm from the smallest (M x N x K 5 x 7 x 1: 36 -> 21 us with launches; 64 x 144 x 48: 103 ->
//            28; 1024 x 600 x 2400: 9.6 -> 0.32 ms; 1024 x 1000 x 6000: 24 -> 0.78 ms); below that k_zgemm_small
//            (zgemm_small_pays).
//   Taylor   one kernel a walker (k_trotter_oz.cu) against the binary64 kernel: n = 5, o = 2: 21 -> 24 us at 200
//            walkers, 117 -> 33 at 2048; n = 8, o = 2: 26 -> 23 at 8; n = 30, o = 7: 66 -> 36 at 8, 120 -> 44 at 200,
//            817 -> 191 at 2048.  Tiles of all walkers (16 launches at least) against one kernel a walker: n = 45, o =
//            9: 218 / 94 at 200, 1177 / 649 at 2048; n = 60, o = 10: 168 / 92 at 8, 1317 / 1289 at 2048; n = 61, o =
//            18: 170 / 136 at 8, 270 / 272 at 200, 1671 / 1935 at 2048 (mma.sync runs at a ninth of tcgen05's rate).
//   green    m and G_half cost 6 n o^2 binary64 FMAs a walker against a 128 x 64 tile each, the factorisation is the
//            same: n = 60, o = 10 (n o^2 = 6000): 230 -> 401 us at 2048 walkers; 60, 20 (24000): 107 -> 99 at 8, 790 ->
//            724 at 2048; 120, 20 (48000): 154 -> 105 at 8, 1287 -> 891 at 2048; 200, 30: 467 -> 176 at 8, 4526 -> 1863.
//   QR       nine launches against one kernel a walker, whose work goes as n o^2 where the digits' goes as n o: 24 x 24
//            138 -> 114 us at 8 walkers, 2097 -> 1503 at 4096; 64 x 17 113 -> 109 at 64, 1806 -> 1537 at 4096; 61 x 18
//            125 -> 102 at 8, 2028 -> 1327 at 4096; 120 x 20 224 -> 121, 4379 -> 1757; 200 x 30 535 -> 165, 12.4 -> 3.3
//            ms; 400 x 50 3178 -> 407 us, 114 -> 13.5 ms.  But 20 x 16 80 -> 93 at 8; 75 x 13 121 -> 139 at 200; 200 x
//            10 140 -> 193 at 200, 1595 -> 2469 at 4096.
//   energy   n = 8, o = 2, 40 vectors: 12 -> 24 us at 200 walkers, 64 -> 55 at 2048; n = 12, o = 6, 60 vectors: 27 ->
//            29 at 8, 51 -> 34 at 200; n = 20, o = 5, 100 vectors: 41 -> 30 at 8, 547 -> 185 at 2048.
bool zgemm_oz_pays(int M, int N, int K) { return M > 0 && N > 0 && K >= 1 && K <= OZ_KMAX && M <= 65535 * 64; }
int launch_asym(int n, int G, const double* chol, int* asym, cudaStream_t s) {
    AFQ_CUDA(cudaMemsetAsync(asym, 0, sizeof(int), s));
    const int nt = (n + 31) / 32, pairs = nt * (nt + 1) / 2, gy = (152 * 8 + pairs - 1) / pairs;
    k_oz_asym<<<dim3(pairs, gy < G ? gy : G), 256, 0, s>>>(n, G, chol, asym);
    AFQ_LAUNCHED("k_oz_asym");
    return AFQ_OK;
}

// Symmetric vectors' half V-build: where the whole one is more than a wave of tiles (a smaller one takes the same time)
// and the 8 x 8 blocks cover at most four fifths of n^2 (from n = 29 on).  n = 120, 600 vectors, 2048 walkers: 1.46 ->
// 0.87 ms with the cut; 200, 1000, 1024: 3.34 -> 1.95; 400, 2000, 128: 5.01 -> 3.22 (0.4 of it the vectors' check, which
// a block makes once and which stops at the first pair that differs).
static bool vbuild_sym_pays(int W, int n) {
    const long long n2 = (long long)n * n;
    return 5LL * sym_total(n) <= 4 * n2 && ((n2 + OZ_ROWS - 1) / OZ_ROWS) * ((2LL * W + OZ_TN - 1) / OZ_TN) > 152;
}
bool qr_oz_pays(int W, int n, int o) { return W > 0 && n <= 512 && n >= o && o <= 64 && o >= 17 && n * o * o >= 13000; }
bool green_oz_pays(int n, int o) { return n <= 512 && n * o * o >= 24000; }
bool trotter_oz_pays(int W, int n, int n_terms) { return W <= 65535 && n > 32 && n <= 512 && n_terms >= 1; }
// W walkers, oc columns each
bool trotter_small_pays(int W, int n, int oc, int n_terms) {
    return W <= 65535 && trotter_small_fits(n, oc, n_terms) && (n <= 48 || oc <= 10 || W <= 152) && (n >= 8 || W > 256);
}
bool energy_oz_pays(int W, int n, int o, int G) {
    const int nchunk = energy_partial_chunks(o, G), ng = (G + nchunk - 1) / nchunk;
    return W <= 65535 && energy_partial_fits(o, G, 1) && ng * o * (o + 1) * (int)sizeof(double2) <= OZ_XSMEM &&
           (n >= 16 || (double)W * G * o * o * n >= 1 << 20);
}

size_t zgemm_oz_scratch(int M, int N, int K) {
    if (!zgemm_oz_pays(M, N, K)) return 0;
    Arena a;
    z_layout(a, M, N, K);
    return a.used + 256;
}

// Digits of a real operand kept by the caller (a block's steps share theirs): bytes, 0 where they would take more
// than OZ_KEEP.
constexpr long long OZ_KEEP = 640LL << 20;
struct ZKept {
    OzDigits D;
    int* amax;
};
static ZKept kept_layout(Arena& a, int N, int K) {
    ZKept k;
    k.D = take_digits(a, N, K);
    k.amax = a.take<int>(1);
    return k;
}
size_t oz_real_bytes(int N, int K) {
    if (!zgemm_oz_pays(1, N, K) || round_up(N, 8) * digit_row_bytes(K) > OZ_KEEP) return 0;
    Arena a;
    kept_layout(a, N, K);
    return a.used + 256;
}

static int oz_real_split(int N, int K, const double* B, int64_t ldb, bool b_trans, void* real, cudaStream_t s,
                         const SymRows& sym = {}) {
    Arena a(real, (size_t)-1);
    const ZKept k = kept_layout(a, N, K);
    AFQ_CUDA(cudaMemsetAsync(k.amax, 0x80, sizeof(int), s));
    return b_trans ? split_rows(N, N, K, B, ldb, k.D, s, k.amax) : split_cols(N, K, B, ldb, k.D, s, k.amax, 1, sym);
}

// sn > 0: the V-build over sn orbitals, whose symmetric vectors' rows are in SymRows's order (asym: the flag of `real`)
static int zgemm_oz(int M, int N, int K, double alpha, const double2* A, int64_t lda, const double* B, int64_t ldb,
                    bool b_trans, double2* C, int64_t ldc, const OzScratch& oz, cudaStream_t s, const void* real,
                    int sn, const int* asym) {
    if (M <= 0 || N <= 0) return AFQ_OK;
    int ae = 0;
    if (frexp(alpha, &ae) != 0.5) return fail(AFQ_E_UNSUPPORTED, "digit GEMM: alpha=%g is no power of two", alpha);
    Arena ar(oz.p, oz.bytes);
    ZLayout z = z_layout(ar, M, N, K);
    AFQ_TRY(oz_room(ar));
    const int* amax = z.amax;
    if (real) {
        Arena a((void*)real, (size_t)-1);
        const ZKept k = kept_layout(a, N, K);
        z.A = k.D;
        amax = k.amax;
        z.nc = N;
    } else if (sn) {
        AFQ_TRY(launch_asym(sn, K, B, z.asym, s));
        asym = z.asym;
    }
    int sms = 0;
    AFQ_TRY(device_sms(&sms));
    for (int m0 = 0; m0 < M; m0 += z.mc) {
        const int mc = M - m0 < z.mc ? M - m0 : z.mc;
        AFQ_TRY(split_crows(mc, K, A + (int64_t)m0 * lda, lda, z.B, s, z.amax, z.arrived));
        for (int n0 = 0; n0 < N; n0 += z.nc) {
            const int nc = N - n0 < z.nc ? N - n0 : z.nc;
            const SymRows sym = {sn ? asym : nullptr, sn, n0};  // the chunk's first row
            if (real) {}
            else if (b_trans) AFQ_TRY(split_rows(nc, nc, K, B + (int64_t)n0 * ldb, ldb, z.A, s, z.amax));
            else AFQ_TRY(split_cols(nc, K, B, ldb, z.A, s, z.amax, 1, sym));
            const OzOut out = {C + (int64_t)m0 * ldc + (sn ? 0 : n0), 0, ldc, 0, 1, 1, ae - 1, nullptr};
            const long long tiles = (long long)((nc + OZ_ROWS - 1) / OZ_ROWS) * ((2 * mc + OZ_TN - 1) / OZ_TN);
            int splits, cps;
            oz_splits(tiles, K, sms < OZ_TILE_SMS ? sms : OZ_TILE_SMS, splits, cps);
            AFQ_TRY(oz_launch(nc, 2 * mc, K, 1, 0, z.A, z.B, out, splits, cps, z.raw, oz.err, s, sn ? sym : SymRows{}));
            // a chunk's columns of C, or all where its rows are symmetric vectors' blocks
            const bool all = sn != 0;
            AFQ_TRY(launch_zgemm_lost(mc, all ? N : nc, K, alpha, A + (int64_t)m0 * lda, lda,
                                      all ? B : b_trans ? B + (int64_t)n0 * ldb : B + n0, ldb, b_trans,
                                      C + (int64_t)m0 * ldc + (all ? 0 : n0), ldc, amax, z.B.ex, ae - 1, z.arrived,
                                      oz.err, s));
            if (n0 + nc < N) {  // the next is judged by itself
                AFQ_CUDA(cudaMemsetAsync(z.amax, 0x80, sizeof(int), s));
                AFQ_CUDA(cudaMemsetAsync(z.arrived, 0, (size_t)(mc + OZ_LOST - 1) / OZ_LOST * sizeof(int), s));
            }
        }
    }
    return AFQ_OK;
}

int launch_zgemm_oz(int M, int N, int K, double alpha, const double2* A, int64_t lda, const double* B, int64_t ldb,
                    bool b_trans, double2* C, int64_t ldc, const OzScratch& oz, cudaStream_t s, const void* real) {
    return zgemm_oz(M, N, K, alpha, A, lda, B, ldb, b_trans, C, ldc, oz, s, real, 0, nullptr);
}

// ---------------------------------------------------------------- Taylor --
namespace {
struct TrLayout {
    int wc;
    OzDigits E, V, T, X;  // E_half, V rows, right operands of V T, walker columns
    double2 *Y, *U;
    OzSeries g;
};
// a chunk's scales and marks (x, t, u and flag), and that of E - I
constexpr int OZ_SERIES = 4;
OzSeries take_series(Arena& a, int wc) {
    int* p = a.take<int>(OZ_SERIES * (size_t)wc + 1);
    if (!p) return {};
    return {p + OZ_SERIES * (size_t)wc, p, p + wc, p + 2 * (size_t)wc, p + 3 * (size_t)wc};
}
// all maxima of nothing yet
int clear_series(const OzSeries& g, cudaStream_t s) {
    AFQ_CUDA(cudaMemsetAsync(g.x, 0x80, (size_t)(g.flag - g.x) * sizeof(int), s));
    return AFQ_OK;
}
int series_flags(const OzSeries& g, int wc, int n, const OzDigits& V, cudaStream_t s) {
    k_oz_series_flags<<<(wc + 3) / 4, 128, 0, s>>>(wc, n, g, V.ex);
    AFQ_LAUNCHED("k_oz_series_flags");
    return AFQ_OK;
}
// the power of two above a coefficient
int coef(double s) { return s == 0.0 ? -1100 : ilogb(s) + 1; }
// walkers of ns blocks (n x o) each in a chunk: their digits and blocks take at most OZ_CAP
long long tr_most(int n, int o, int ns) {
    const long long per = (round_up(n, 8) + round_up(2 * ns * o, 8)) * digit_row_bytes(2 * n) +
                          2LL * ns * o * (digit_row_bytes(n) + 16LL * n) + 4 * OZ_SERIES;
    return OZ_CAP / per > 1 ? OZ_CAP / per : 1;
}
// a chunk of wc walkers
TrLayout tr_layout(Arena& a, int wc, int n, int o, int ns) {
    TrLayout t;
    t.wc = wc;
    const size_t nb = (size_t)t.wc * ns;
    t.E = take_digits(a, n, n);
    t.V = take_digits(a, n, 2 * n, t.wc);
    t.T = take_digits(a, 2 * ns * o, 2 * n, t.wc);
    t.X = take_digits(a, nb * 2 * o, n);
    t.Y = a.take<double2>(nb * n * o);
    t.U = a.take<double2>(nb * n * o);
    t.g = take_series(a, t.wc);
    return t;
}
// W blocks of o columns, ns of them taken together (block strides ws, ss)
template <int MODE>
int launch_term(int W, int n, int o, double s, const double2* Y, const double2* X, double2* U, const OzDigits& D,
                cudaStream_t st, OzMax mx = {nullptr, 1, 1, 0}, int ns = 1, long long ws = 0, long long ss = 0,
                double2* tp = nullptr, long long tw = 0) {
    const int oc = o * ns, ncg = (oc + OZ_CB - 1) / OZ_CB, smem = OZ_CB * (n + 1) * (int)sizeof(double2);
    if (ns == 1) ws = (long long)n * o;
    AFQ_TRY(raise_smem_once(g_ozterm[MODE], k_oz_term<MODE>, OZ_CB * 513 * (int)sizeof(double2)));
    const OzDst dst = MODE == OZ_WALK || MODE == OZ_LAST || MODE == OZ_BACKL ? dst_of(D, 2LL * W * oc, n)
                      : MODE == OZ_COLS                                      ? dst_of(D, 2 * oc, n)
                                                                             : dst_of(D, 2 * oc, 2 * n);
    k_oz_term<MODE><<<(unsigned)W * ncg, 256, smem, st>>>(n, oc, o, ws, ss, ncg, s, Y, X, U, dst, D.ex, tp, tw, mx);
    AFQ_LAUNCHED("k_oz_term");
    return AFQ_OK;
}
}  // namespace

// The largest chunk of up to W walkers, not the even one that a call of W takes: where W walkers are two chunks of half
// of them, W - 1 can be one.
size_t trotter_oz_scratch(int W, int n, int o, int ns) {
    size_t most = 0;
    for (int k = 1; k <= ns; ++k) {  // the spins together, or one at a time
        Arena a;
        const long long m = tr_most(n, o, k);
        tr_layout(a, W < m ? W : (int)m, n, o, k);
        most = std::max(most, a.used);
    }
    return most + 256;
}
bool trotter_oz_whole(int W, int n, int o, int ns) { return W <= tr_most(n, o, ns); }

// E_half . sum_{k <= K} (i sqrt_dt V)^k / k! . E_half . X, n_terms >= 1, of the
// ns blocks X of each walker, which share its V: block p of walker w is n x o at
// w ws + p ss (ns = 2: ws = 2 n o, ss = n o, or ws = n o, ss = W n o where
// trotter_oz_whole).
// E_half X is formed as X + (E_half - I) X: E_half is close to the identity,
// and a digit product's error scales with its operands' largest entries.
int launch_trotter_oz(int W, int n, int o, int n_terms, double sqrt_dt, const double* E, const double2* V,
                      const double2* win, double2* wout, int ns, long long ws, long long ss, const OzScratch& oz,
                      cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    Arena ar(oz.p, oz.bytes);
    const TrLayout t = tr_layout(ar, even_chunk(W, tr_most(n, o, ns)), n, o, ns);
    AFQ_TRY(oz_room(ar));
    int* err = oz.err;
    AFQ_CUDA(cudaMemsetAsync(t.g.e, 0x80, sizeof(int), s));
    AFQ_TRY(split_rows(n, n, n, E, n, t.E, s, t.g.e, 1));
    const size_t no = (size_t)n * o;
    for (int w0 = 0; w0 < W; w0 += t.wc) {
        const int wc = W - w0 < t.wc ? W - w0 : t.wc, nb = wc * ns;  // the chunk's blocks are contiguous
        const int bd = ws == (long long)no ? 1 : ns;                 // block b is walker b / bd % wc's
        const double2* x = win + (size_t)w0 * ns * no;
        AFQ_TRY(clear_series(t.g, s));
        AFQ_TRY(split_rows((long long)wc * n, n, 2 * n, (const double*)(V + (size_t)w0 * n * n), 2 * n, t.V, s));
        AFQ_TRY(launch_term<OZ_WALK>(nb, n, o, 0.0, x, nullptr, nullptr, t.X, s, {t.g.x, bd, wc, 0}));
        const OzOut xo = {t.Y, 0, (long long)no, 1, o, o, 0, nullptr};
        AFQ_TRY(oz_launch(n, 2 * nb * o, n, 1, 0, t.E, t.X, xo, 1, (n + 255) / 256, nullptr, err, s));
        AFQ_TRY(launch_term<OZ_INIT>(wc, n, o, 0.0, t.Y, x, t.U, t.T, s, {t.g.t, 1, wc, coef(sqrt_dt)}, ns, ws, ss));
        for (int k = 1; k <= n_terms; ++k) {
            const OzOut to = {t.Y, ns == 1 ? (long long)no : ws, ss, 1, o, o, 0, nullptr};
            AFQ_TRY(oz_launch(n, 2 * ns * o, 2 * n, wc, 1, t.V, t.T, to, 1, (2 * n + 255) / 256, nullptr, err, s));
            if (k < n_terms)
                AFQ_TRY(launch_term<OZ_TERM>(wc, n, o, sqrt_dt / k, t.Y, nullptr, t.U, t.T, s,
                                             {t.g.t, 1, wc, coef(sqrt_dt / (k + 1))}, ns, ws, ss));
            else AFQ_TRY(launch_term<OZ_LAST>(nb, n, o, sqrt_dt / k, t.Y, nullptr, t.U, t.X, s, {t.g.u, bd, wc, 0}));
        }
        AFQ_TRY(series_flags(t.g, wc, n, t.V, s));
        double2* y = wout + (size_t)w0 * ns * no;
        const OzOut wo = {y, 0, (long long)no, 1, o, o, 0, t.U, t.g.flag, bd, wc};
        AFQ_TRY(oz_launch(n, 2 * nb * o, n, 1, 0, t.E, t.X, wo, 1, (n + 255) / 256, nullptr, err, s));
        // the marked walkers, whose input is still in place where wout is win
        const double2* v = V + (size_t)w0 * n * n;
        if (bd == ns) {
            AFQ_TRY(launch_trotter(nb, n, o, n_terms, sqrt_dt, E, v, x, y, s, ns, t.g.flag));
        } else {
            for (int p = 0; p < ns; ++p)
                AFQ_TRY(launch_trotter(wc, n, o, n_terms, sqrt_dt, E, v, x + p * ss, y + p * ss, s, 1, t.g.flag));
        }
    }
    return AFQ_OK;
}

// ------------------------------------------ Taylor series with its terms --
// The differentiated step's series (k_adjoint.cu has the formulas) where a walker does not fit k_trotter_oz.cu's kernel:
// launch_trotter_oz's products with every term kept, and its reverse with V^H and E^T.  Five steps forward and back, the
// two by k_adjoint.cu's binary64 kernels -> by digits: 66 x 8, 8 walkers 10.9 -> 9.9 ms; 80 x 16, 64 walkers 19.0 ->
// 14.2; 100 x 20, 200 walkers 56.6 -> 33.8; 120 x 32, 100 walkers 67.3 -> 38.9.
namespace {
// out[w][i][j] = conj(in[w][j][i]) (double2), or the transpose (double)
__device__ __forceinline__ double oz_conj(double x) { return x; }
__device__ __forceinline__ double2 oz_conj(double2 x) { return make_double2(x.x, -x.y); }
template <typename T>
__global__ void __launch_bounds__(256) k_oz_adjoint(int n, const T* __restrict__ in, T* __restrict__ out) {
    __shared__ T tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, i0 = 32 * blockIdx.x, j0 = 32 * blockIdx.y;
    const size_t b = (size_t)blockIdx.z * n * n;
    for (int r = ty; r < 32; r += 8)
        if (j0 + r < n && i0 + tx < n) tile[r][tx] = in[b + (size_t)(j0 + r) * n + i0 + tx];
    __syncthreads();
    for (int r = ty; r < 32; r += 8)
        if (i0 + r < n && j0 + tx < n) out[b + (size_t)(i0 + r) * n + j0 + tx] = oz_conj(tile[tx][r]);
}
struct TgLayout {
    int wc;
    OzDigits E, V, T, X;
    double2 *Y, *U, *vh;
    double* et;
    OzSeries g;
};
TgLayout tg_layout(Arena& a, int W, int n, int o) {
    TgLayout t;
    const long long n2 = (long long)n * n, per = (round_up(n, 8) + round_up(2 * o, 8)) * digit_row_bytes(2 * n) + 16 * n2 +
                                                 2LL * o * (digit_row_bytes(n) + 16LL * n) + 4 * OZ_SERIES;
    const long long most = OZ_CAP / per;
    t.wc = even_chunk(W, most < 65535 ? most : 65535);
    t.E = take_digits(a, n, n);
    t.V = take_digits(a, n, 2 * n, t.wc);
    t.T = take_digits(a, 2 * o, 2 * n, t.wc);
    t.X = take_digits(a, (size_t)t.wc * 2 * o, n);
    t.Y = a.take<double2>((size_t)t.wc * n * o);
    t.U = a.take<double2>((size_t)t.wc * n * o);
    t.vh = a.take<double2>(t.wc * n2);
    t.et = a.take<double>(n2);
    t.g = take_series(a, t.wc);
    return t;
}
}  // namespace

size_t taylor_grad_oz_scratch(int W, int n, int o) {
    Arena a;
    tg_layout(a, W, n, o);
    return a.used + 256;
}

int launch_taylor_tape_oz(int W, int n, int o, int K, double sqrt_dt, const double* E, const double2* V,
                          const double2* win, double2* terms, double2* w2, const OzScratch& oz, cudaStream_t s) {
    Arena ar(oz.p, oz.bytes);
    const TgLayout t = tg_layout(ar, W, n, o);
    AFQ_TRY(oz_room(ar));
    int* err = oz.err;
    const size_t no = (size_t)n * o;
    AFQ_CUDA(cudaMemsetAsync(t.g.e, 0x80, sizeof(int), s));
    AFQ_TRY(split_rows(n, n, n, E, n, t.E, s, t.g.e, 1));
    const OzOut xo = {t.Y, 0, (long long)no, 1, o, o, 0, nullptr}, to = {t.Y, (long long)no, 0, 1, o, o, 0, nullptr};
    for (int w0 = 0; w0 < W; w0 += t.wc) {
        const int wc = W - w0 < t.wc ? W - w0 : t.wc;
        const double2* x = win + w0 * no;
        double2 *u = w2 + w0 * no, *tp = terms + w0 * K * no;
        AFQ_TRY(clear_series(t.g, s));
        AFQ_TRY(split_rows((long long)wc * n, n, 2 * n, (const double*)(V + (size_t)w0 * n * n), 2 * n, t.V, s));
        AFQ_TRY(launch_term<OZ_WALK>(wc, n, o, 0.0, x, nullptr, nullptr, t.X, s, {t.g.x, 1, wc, 0}));
        AFQ_TRY(oz_launch(n, 2 * wc * o, n, 1, 0, t.E, t.X, xo, 1, (n + 255) / 256, nullptr, err, s));
        AFQ_TRY(launch_term<OZ_INIT>(wc, n, o, 0.0, t.Y, x, u, t.T, s, {t.g.t, 1, wc, coef(sqrt_dt)}, 1, 0, 0, tp, K * no));
        for (int k = 1; k <= K; ++k) {
            AFQ_TRY(oz_launch(n, 2 * o, 2 * n, wc, 1, t.V, t.T, to, 1, (2 * n + 255) / 256, nullptr, err, s));
            if (k < K)
                AFQ_TRY(launch_term<OZ_TERM>(wc, n, o, sqrt_dt / k, t.Y, nullptr, u, t.T, s,
                                             {t.g.t, 1, wc, coef(sqrt_dt / (k + 1))}, 1, 0, 0, tp + k * no, K * no));
            else AFQ_TRY(launch_term<OZ_LAST>(wc, n, o, sqrt_dt / k, t.Y, nullptr, u, t.X, s, {t.g.u, 1, wc, 0}));
        }
        AFQ_TRY(series_flags(t.g, wc, n, t.V, s));
        AFQ_TRY(launch_taylor_tape_plain(wc, n, o, K, sqrt_dt, E, V + (size_t)w0 * n * n, x, tp, u, t.g.flag, s));
    }
    return AFQ_OK;
}

int launch_taylor_adj_oz(int W, int n, int o, int K, double sqrt_dt, const double* E, const double2* V,
                         const double2* wbar_post, double2* tbar, double2* wbar_pre, const OzScratch& oz,
                         cudaStream_t s) {
    Arena ar(oz.p, oz.bytes);
    const TgLayout t = tg_layout(ar, W, n, o);
    AFQ_TRY(oz_room(ar));
    int* err = oz.err;
    const size_t no = (size_t)n * o;
    const unsigned nt = (n + 31) / 32;
    k_oz_adjoint<double><<<dim3(nt, nt, 1), 256, 0, s>>>(n, E, t.et);
    AFQ_LAUNCHED("k_oz_adjoint");
    AFQ_CUDA(cudaMemsetAsync(t.g.e, 0x80, sizeof(int), s));
    AFQ_TRY(split_rows(n, n, n, t.et, n, t.E, s, t.g.e, 1));
    const OzOut xo = {t.Y, 0, (long long)no, 1, o, o, 0, nullptr}, to = {t.Y, (long long)no, 0, 1, o, o, 0, nullptr};
    for (int w0 = 0; w0 < W; w0 += t.wc) {
        const int wc = W - w0 < t.wc ? W - w0 : t.wc;
        const double2* x = wbar_post + w0 * no;
        double2* tp = tbar + w0 * (K + 1) * no;
        k_oz_adjoint<double2><<<dim3(nt, nt, wc), 256, 0, s>>>(n, V + (size_t)w0 * n * n, t.vh);
        AFQ_LAUNCHED("k_oz_adjoint");
        AFQ_TRY(clear_series(t.g, s));
        AFQ_TRY(split_rows((long long)wc * n, n, 2 * n, (const double*)t.vh, 2 * n, t.V, s));
        AFQ_TRY(launch_term<OZ_WALK>(wc, n, o, 0.0, x, nullptr, nullptr, t.X, s, {t.g.x, 1, wc, 0}));
        AFQ_TRY(oz_launch(n, 2 * wc * o, n, 1, 0, t.E, t.X, xo, 1, (n + 255) / 256, nullptr, err, s));
        AFQ_TRY(launch_term<OZ_INIT>(wc, n, o, 0.0, t.Y, x, t.U, t.T, s, {t.g.t, 1, wc, coef(sqrt_dt / K)}, 1, 0, 0,
                                     tp + K * no, (K + 1) * no));
        for (int k = K - 1; k >= 0; --k) {
            AFQ_TRY(oz_launch(n, 2 * o, 2 * n, wc, 1, t.V, t.T, to, 1, (2 * n + 255) / 256, nullptr, err, s));
            const double c = sqrt_dt / (k + 1);
            if (k > 0)
                AFQ_TRY(launch_term<OZ_BACK>(wc, n, o, c, t.Y, nullptr, t.U, t.T, s, {t.g.t, 1, wc, coef(sqrt_dt / k)}, 1, 0,
                                             0, tp + k * no, (K + 1) * no));
            else AFQ_TRY(launch_term<OZ_BACKL>(wc, n, o, c, t.Y, nullptr, t.U, t.X, s, {t.g.u, 1, wc, 0}, 1, 0, 0, tp,
                                               (K + 1) * no));
        }
        AFQ_TRY(series_flags(t.g, wc, n, t.V, s));
        const OzOut wo = {wbar_pre + w0 * no, 0, (long long)no, 1, o, o, 0, t.U, t.g.flag, 1, wc};
        AFQ_TRY(oz_launch(n, 2 * wc * o, n, 1, 0, t.E, t.X, wo, 1, (n + 255) / 256, nullptr, err, s));
        AFQ_TRY(launch_taylor_adj_plain(wc, n, o, K, sqrt_dt, E, V + (size_t)w0 * n * n, x, tp, wbar_pre + w0 * no, t.g.flag,
                                        s));
    }
    return AFQ_OK;
}

// ----------------------------------------------------------------- green --
namespace {
struct GrLayout {
    int wc;
    OzDigits C, X, A, B;  // trial columns, walker columns, walker rows, right operands W^T m^-1
    double2 *m, *inv;
    int* flag;  // walkers whose product has lost too much
};
GrLayout gr_layout(Arena& a, int W, int n, int o) {
    GrLayout g;
    const long long per = 2LL * o * digit_row_bytes(n) + round_up(n, 8) * digit_row_bytes(2 * o) +
                          round_up(2 * o, 8) * digit_row_bytes(2 * o) + 32LL * o * o + 4;
    long long wc = OZ_CAP / per;
    g.wc = even_chunk(W, wc);
    g.C = take_digits(a, o, n);
    g.X = take_digits(a, (size_t)g.wc * 2 * o, n);
    g.A = take_digits(a, n, 2 * o, g.wc);
    g.B = take_digits(a, 2 * o, 2 * o, g.wc);
    g.m = a.take<double2>((size_t)g.wc * o * o);
    g.inv = a.take<double2>((size_t)g.wc * o * o);
    g.flag = a.take<int>(g.wc);
    return g;
}
}  // namespace

size_t green_oz_scratch(int W, int n, int o) {
    Arena a;
    gr_layout(a, W, n, o);
    return a.used + 256;
}

// m = C^T W of all walkers as one product, its factorisations, and G_half[b, i] = sum_a W[i, a] m^-1[a, b] a walker
int launch_green_oz(int W, int n, int o, const double2* mo, const double2* walkers, double2* ovlp_out,
                    double2* green_out, int ov_square, const OzScratch& oz, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    Arena ar(oz.p, oz.bytes);
    const GrLayout g = gr_layout(ar, W, n, o);
    AFQ_TRY(oz_room(ar));
    int* err = oz.err;
    const size_t no = (size_t)n * o;
    AFQ_TRY(split_cols(o, n, (const double*)mo, 2LL * o, g.C, s, nullptr, 2));
    for (int w0 = 0; w0 < W; w0 += g.wc) {
        const int wc = W - w0 < g.wc ? W - w0 : g.wc;
        const double2* w = walkers + w0 * no;
        double2 *ov = ovlp_out ? ovlp_out + w0 : nullptr, *gr = green_out ? green_out + w0 * no : nullptr;
        AFQ_TRY(launch_term<OZ_WALK>(wc, n, o, 0.0, w, nullptr, nullptr, g.X, s));
        const OzOut mout = {g.m, 0, (long long)o * o, 1, o, o, 0, nullptr};
        AFQ_TRY(oz_launch(o, 2 * wc * o, n, 1, 0, g.C, g.X, mout, 1, (n + 255) / 256, nullptr, err, s));
        AFQ_TRY(launch_lu(wc, o, g.m, ov, gr ? g.inv : nullptr, ov_square, s));
        if (gr) {
            AFQ_TRY(split_rows((long long)wc * n, n, 2 * o, (const double*)w, 2 * o, g.A, s));
            AFQ_TRY(launch_term<OZ_PLAIN>(wc, o, o, 0.0, g.inv, nullptr, nullptr, g.B, s));
            const OzOut gout = {gr, (long long)no, 0, n, 1, 2 * o, 0, nullptr};
            AFQ_TRY(oz_launch(n, 2 * o, 2 * o, wc, 1, g.A, g.B, gout, 1, (2 * o + 255) / 256, nullptr, err, s));
        }
        const OzWalk gm = {g.C.ex, g.X.ex, g.m, o * o, o, 2 * o, 1}, gg = {g.A.ex, g.B.ex, gr, (int)no, n, 2 * o, 0};
        k_oz_flags<<<(wc + 3) / 4, 128, 0, s>>>(wc, gm, gg, g.flag);
        AFQ_LAUNCHED("k_oz_flags");
        AFQ_TRY(launch_green_sq(wc, n, o, mo, 1, w, ov, gr, ov_square, s, g.flag));
    }
    return AFQ_OK;
}

// -------------------------------------------------------------------- QR --
// What bounds it is the factorisation's chain of steps and the tiles' fill (2 nocc of 128 rows), so a chunk holds as
// many walkers as the scratch allows: 4096 walkers of 200 x 30 took 3.7 ms in chunks of 256 MiB, 3.3 in 1 GiB.
namespace {
struct QrLayout {
    int wc;
    OzDigits X, A, B;  // walker columns, walker rows, right operands R1^-1
    double2 *q1, *gram, *tinv;
    double* det;
    int *flag, *err;
};
QrLayout qr_layout(Arena& a, int W, int n, int o) {
    QrLayout g;
    const long long per = round_up(2 * o, 8) * (digit_row_bytes(n) + digit_row_bytes(2 * o)) +
                          round_up(n, 8) * digit_row_bytes(2 * o) + 16LL * n * o + 48LL * o * o;
    g.wc = even_chunk(W, OZ_CAP / per);
    g.X = take_digits(a, 2 * o, n, g.wc);
    g.A = take_digits(a, n, 2 * o, g.wc);
    g.B = take_digits(a, 2 * o, 2 * o, g.wc);
    g.q1 = a.take<double2>((size_t)g.wc * n * o);
    g.gram = a.take<double2>((size_t)g.wc * 2 * o * o);
    g.tinv = a.take<double2>((size_t)g.wc * o * o);
    g.det = a.take<double>(g.wc);
    g.flag = a.take<int>(W);
    g.err = a.take<int>(64);
    return g;
}
}  // namespace

size_t qr_oz_scratch(int W, int n, int o) {
    if (!qr_oz_pays(W, n, o)) return 0;
    Arena a;
    qr_layout(a, W, n, o);
    return a.used + 256;
}

int launch_qr_oz(int W, int n, int o, const double2* win, double2* wout, double2* det_r, const OzScratch& oz,
                 cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    Arena ar(oz.p, oz.bytes);
    const QrLayout g = qr_layout(ar, W, n, o);
    AFQ_TRY(oz_room(ar));
    const size_t no = (size_t)n * o;
    const OzOut gout = {g.gram, 2LL * o * o, 2 * o, 0, 1, 1, 0, nullptr};      // gram[b][2 a + part]
    const OzOut qout = {g.q1, (long long)no, 1, 0, o, 1, 0, nullptr};          // q1[i][c]
    AFQ_CUDA(cudaMemsetAsync(g.err, 0, sizeof(int), s));
    for (int w0 = 0; w0 < W; w0 += g.wc) {
        const int wc = W - w0 < g.wc ? W - w0 : g.wc;
        const double2* w = win + w0 * no;
        AFQ_TRY(launch_term<OZ_COLS>(wc, n, o, 0.0, w, nullptr, nullptr, g.X, s));
        AFQ_TRY(oz_launch(2 * o, 2 * o, n, wc, 1, g.X, g.X, gout, 1, (n + 255) / 256, nullptr, g.err, s));
        AFQ_TRY(launch_qr_factor(wc, o, g.gram, g.tinv, g.det, g.flag + w0, s));
        AFQ_TRY(split_rows((long long)wc * n, n, 2 * o, (const double*)w, 2 * o, g.A, s));
        AFQ_TRY(launch_term<OZ_PLAIN>(wc, o, o, 0.0, g.tinv, nullptr, nullptr, g.B, s));
        AFQ_TRY(oz_launch(n, 2 * o, 2 * o, wc, 1, g.A, g.B, qout, 1, (2 * o + 255) / 256, nullptr, g.err, s));
        AFQ_TRY(launch_term<OZ_COLS>(wc, n, o, 0.0, g.q1, nullptr, nullptr, g.X, s));
        AFQ_TRY(oz_launch(2 * o, 2 * o, n, wc, 1, g.X, g.X, gout, 1, (n + 255) / 256, nullptr, g.err, s));
        AFQ_TRY(launch_qr_finish(wc, n, o, g.q1, g.gram, g.det, g.err, wout + w0 * no, det_r ? det_r + w0 : nullptr,
                                 g.flag + w0, s));
    }
    return launch_qr(W, n, o, win, wout, det_r, s, g.flag);
}

int launch_qr_auto(int W, int n, int o, const double2* win, double2* wout, double2* det_r, const OzScratch& oz,
                   cudaStream_t s) {
    if (oz.p && qr_oz_pays(W, n, o)) return launch_qr_oz(W, n, o, win, wout, det_r, oz, s);
    return launch_qr(W, n, o, win, wout, det_r, s);
}

// ------------------------------------------------- adjoint outer products --
namespace {
struct VbLayout {
    int wc;
    OzDigits A, B;
    int* flag;
};
VbLayout vb_layout(Arena& a, int W, int n, int o, int K) {
    VbLayout v;
    const int k2 = 2 * K * o;
    v.wc = even_chunk(W, OZ_CAP / (3 * round_up(n, 8) * digit_row_bytes(k2)));
    v.A = take_digits(a, n, k2, v.wc);
    v.B = take_digits(a, 2 * n, k2, v.wc);
    v.flag = a.take<int>(v.wc);
    return v;
}
}  // namespace

// Where the sums are too long for the digits the adjoint's binary64 kernel (k_adjoint.cu) forms them.
bool vbar_oz_pays(int o, int K) { return K >= 1 && 2LL * K * o <= OZ_KMAX; }
size_t vbar_oz_scratch(int W, int n, int o, int K) {
    if (!vbar_oz_pays(o, K)) return 0;
    Arena a;
    vb_layout(a, W, n, o, K);
    return a.used + 256;
}

// Vb_w = sum_{k = 1 .. K} conj(i sqrt_dt / k) tb_k t_{k-1}^H
int launch_vbar_oz(int W, int n, int o, int K, double sqrt_dt, const double2* tbar, const double2* terms,
                   double2* vbar, const OzScratch& oz, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    if (!vbar_oz_pays(o, K)) return launch_vbar(W, n, o, K, sqrt_dt, tbar, terms, vbar, nullptr, s);
    Arena ar(oz.p, oz.bytes);
    const VbLayout v = vb_layout(ar, W, n, o, K);
    AFQ_TRY(oz_room(ar));
    const int k2 = 2 * K * o;
    const long long no = (long long)n * o, n2 = (long long)n * n;
    for (int w0 = 0; w0 < W; w0 += v.wc) {
        const int wc = W - w0 < v.wc ? W - w0 : v.wc;
        // eight lanes a row of up to 64 entries, sixteen of 128 (60 orbitals, 120 entries, 256 walkers: 106 -> 65 us)
        const int lanes = k2 <= 64 ? 8 : k2 <= 128 ? 16 : 32;
        const auto cut = lanes == 8 ? k_oz_vbar<8> : lanes == 16 ? k_oz_vbar<16> : k_oz_vbar<32>;
        const double2 *tb = tbar + (long long)w0 * (K + 1) * no, *tm = terms + (long long)w0 * K * no;
        cut<<<row_blocks(2LL * wc * n, 256 / lanes), 256, 0, s>>>(wc, n, o, K, sqrt_dt, tb, tm, dst_of(v.A, n, k2), v.A.ex,
                                                                  dst_of(v.B, 2 * n, k2), v.B.ex);
        AFQ_LAUNCHED("k_oz_vbar");
        const OzOut out = {vbar + w0 * n2, n2, 0, 1, n, n, 0, nullptr};
        AFQ_TRY(oz_launch(n, 2 * n, k2, wc, 1, v.A, v.B, out, 1, (k2 + 255) / 256, nullptr, oz.err, s));
        k_oz_flags<<<(wc + 3) / 4, 128, 0, s>>>(wc, {v.A.ex, v.B.ex, out.C, (int)n2, n, 2 * n, 0}, {}, v.flag);
        AFQ_LAUNCHED("k_oz_flags");
        AFQ_TRY(launch_vbar(wc, n, o, K, sqrt_dt, tb, tm, vbar + w0 * n2, v.flag, s));
    }
    return AFQ_OK;
}

// ---------------------------------------------------------------- energy --
namespace {
struct EnLayout {
    int wc;
    OzDigits L, X;
    double2* F;
};
EnLayout en_layout(Arena& a, int W, int n, int o, int G) {
    EnLayout e;
    long long wc = OZ_CAP / ((long long)o * G * o * 16);
    e.wc = even_chunk(W, wc);
    e.L = take_digits(a, (size_t)G * o, n);
    e.X = take_digits(a, (size_t)e.wc * 2 * o, n);
    e.F = a.take<double2>((size_t)e.wc * o * G * o);
    return e;
}
}  // namespace

size_t energy_oz_scratch(int W, int n, int o, int G) {
    Arena a;
    en_layout(a, W, n, o, G);
    return a.used + 256;
}

int launch_energy_partial_oz(int W, int n, int o, int G, const double2* green, const double* rot_chol,
                             double* partial_d, const OzScratch& oz, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    Arena ar(oz.p, oz.bytes);
    const EnLayout e = en_layout(ar, W, n, o, G);
    AFQ_TRY(oz_room(ar));
    const int nchunk = energy_partial_chunks(o, G), ng = (G + nchunk - 1) / nchunk;
    const int smem = ng * o * (o + 1) * (int)sizeof(double2);
    if (smem > OZ_XSMEM || W > 65535) return fail(AFQ_E_UNSUPPORTED, "digit energy: nocc=%d W=%d", o, W);
    AFQ_TRY(raise_smem_once(g_ozx, k_oz_exchange, OZ_XSMEM));
    AFQ_TRY(split_rows((long long)G * o, G * o, n, rot_chol, n, e.L, s));
    for (int w0 = 0; w0 < W; w0 += e.wc) {
        const int wc = W - w0 < e.wc ? W - w0 : e.wc;
        const double2* g = green + (size_t)w0 * o * n;
        AFQ_TRY(split_crows((long long)wc * o, n, g, n, e.X, s));
        const OzOut out = {e.F, 0, (long long)G * o, 0, 1, 1, 0, nullptr};
        AFQ_TRY(oz_launch(G * o, 2 * wc * o, n, 1, 0, e.L, e.X, out, 1, (n + 255) / 256,
                          nullptr, oz.err, s));
        k_oz_exchange<<<dim3(nchunk, wc), 256, smem, s>>>(n, o, G, ng, e.F, (double2*)partial_d + (size_t)w0 * nchunk * 2,
                                                          e.L.ex, e.X.ex, rot_chol, g);
        AFQ_LAUNCHED("k_oz_exchange");
    }
    return AFQ_OK;
}

void take_oz_block(Arena& a, const afq_dims* d, OzScratch& oz) {
    const int n2 = d->norb * d->norb, on = d->nocc * d->norb;
    const int W = d->n_walkers;  // (parts of the walkers take the small product where all of them do)
    const size_t c = zgemm_small_pays(W, n2, d->nchol) ? 0 : oz_real_bytes(n2, d->nchol);
    const size_t r = !d->trial_is_real || zgemm_small_pays(W, d->nchol, on) ? 0 : oz_real_bytes(d->nchol, on);
    oz.chol = c ? a.take<char>(c) : nullptr;
    oz.asym = c && vbuild_sym_pays(d->n_walkers, d->norb) ? a.take<int>(64) : nullptr;
    oz.rot = r ? a.take<char>(r) : nullptr;
}

int split_oz_block(const afq_dims* d, const double* chol, const double* rot_chol, const OzScratch& oz, cudaStream_t s) {
    const int n2 = d->norb * d->norb, on = d->nocc * d->norb;
    if (oz.asym) AFQ_TRY(launch_asym(d->norb, d->nchol, chol, oz.asym, s));
    if (oz.chol) AFQ_TRY(oz_real_split(n2, d->nchol, chol, n2, false, oz.chol, s, {oz.asym, d->norb, 0}));
    if (oz.rot) AFQ_TRY(oz_real_split(d->nchol, on, rot_chol, on, true, oz.rot, s));
    return AFQ_OK;
}

// ---------------------------------------------------------------- routes --
int launch_zgemm_auto(int M, int N, int K, double alpha, const double2* A, int64_t lda, const void* B, int64_t ldb,
                      bool b_complex, bool b_trans, double2* C, int64_t ldc, const OzScratch& oz, cudaStream_t s,
                      const void* real) {
    if (!b_complex && zgemm_small_pays(M, N, K))
        return launch_zgemm_small(M, N, K, alpha, A, lda, (const double*)B, ldb, b_trans, C, ldc, s);
    if (!b_complex && zgemm_oz_pays(M, N, K))
        return launch_zgemm_oz(M, N, K, alpha, A, lda, (const double*)B, ldb, b_trans, C, ldc, oz, s, real);
    return launch_zgemm(M, N, K, alpha, A, lda, B, ldb, b_complex, b_trans, C, ldc, s);
}

int launch_vbuild(int W, int n, int G, const double2* xs, const double* chol, double2* V, const OzScratch& oz,
                  cudaStream_t s) {
    const int n2 = n * n, sn = (oz.chol ? oz.asym != nullptr : vbuild_sym_pays(W, n)) ? n : 0;
    if (zgemm_small_pays(W, n2, G)) return launch_zgemm_small(W, n2, G, 1.0, xs, G, chol, n2, false, V, n2, s);
    if (zgemm_oz_pays(W, n2, G))
        return zgemm_oz(W, n2, G, 1.0, xs, G, chol, n2, false, V, n2, oz, s, oz.chol, sn, oz.asym);
    return launch_zgemm(W, n2, G, 1.0, xs, G, chol, n2, false, false, V, n2, s);
}

int launch_trotter_auto(int W, int n, int o, int n_terms, double sqrt_dt, const double* E, const double2* V,
                        const double2* win, double2* wout, int vdiv, const OzScratch& oz, cudaStream_t s) {
    const long long no = (long long)n * o;
    const int wp = W / vdiv;  // walkers (blocks that share a V)
    if (trotter_small_pays(wp, n, o * vdiv, n_terms))
        return launch_trotter_small(wp, n, o, n_terms, sqrt_dt, E, V, win, wout, vdiv, vdiv * no, no, s);
    if (trotter_oz_pays(W, n, n_terms))
        return launch_trotter_oz(wp, n, o, n_terms, sqrt_dt, E, V, win, wout, vdiv, vdiv * no, no, oz, s);
    return launch_trotter(W, n, o, n_terms, sqrt_dt, E, V, win, wout, s, vdiv);
}

int launch_trotter_spins(int W, int n, int o, int n_terms, double sqrt_dt, const double* E, const double2* V,
                         const double2* win, double2* wout, size_t half, const OzScratch& oz, cudaStream_t s) {
    const long long no = (long long)n * o;
    if (trotter_small_pays(W, n, 2 * o, n_terms))
        return launch_trotter_small(W, n, o, n_terms, sqrt_dt, E, V, win, wout, 2, no, (long long)half, s);
    if (trotter_oz_pays(W, n, n_terms) && (long long)half == W * no && trotter_oz_whole(W, n, o, 2))
        return launch_trotter_oz(W, n, o, n_terms, sqrt_dt, E, V, win, wout, 2, no, W * no, oz, s);
    for (int spin = 0; spin < 2; ++spin)
        AFQ_TRY(launch_trotter_auto(W, n, o, n_terms, sqrt_dt, E, V, win + spin * half, wout + spin * half, 1, oz, s));
    return AFQ_OK;
}

int launch_energy_partial_auto(int W, int n, int o, int G, const double2* green, const void* rot_chol, int trial_real,
                               double* partial, const OzScratch& oz, cudaStream_t s) {
    if (trial_real && energy_oz_pays(W, n, o, G))
        return launch_energy_partial_oz(W, n, o, G, green, (const double*)rot_chol, partial, oz, s);
    return launch_energy_partial(W, n, o, G, green, rot_chol, trial_real, partial, s);
}

}  // namespace afq
