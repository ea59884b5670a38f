// Binary64 GEMM with a complex left operand and a real or complex right
// operand.  Used by the FP64 step for
//   V-build     V (W x n^2) = x~ (W x G) . L (G x n^2)     (prop/chol_afqmc_ops.py:70-74)
//   force bias  fb (W x G)  = 2 G_half (W x o n) . L~^T    (meas/rhf.py:27-33)
// On GB300 binary64 runs on the SM's scalar FP64 pipe (no FP64 tensor path),
// so the kernel is a register-blocked SIMT GEMM: 64x64 tile, 4x4 complex
// outputs per thread, K staged through shared memory 16 at a time.
#include "afq_internal.cuh"
#include "oz_digits.cuh"

namespace afq {

namespace {
constexpr int BM = 64, BN = 64, BK = 16;

template <bool BC>
struct BElem;
template <>
struct BElem<false> { using T = double; };
template <>
struct BElem<true> { using T = double2; };

__device__ __forceinline__ double2 zero2() { return make_double2(0.0, 0.0); }
__device__ __forceinline__ void load_b(double& dst, const double* p, bool ok) { dst = ok ? *p : 0.0; }
__device__ __forceinline__ void load_b(double2& dst, const double2* p, bool ok) { dst = ok ? *p : zero2(); }
__device__ __forceinline__ void mac(double2& acc, double2 a, double b) { rfma(acc, b, a); }
__device__ __forceinline__ void mac(double2& acc, double2 a, double2 b) { cfma(acc, a, b); }

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// One 64 x 64 tile by 256 threads, sums over k in [kbeg, kend).
template <bool BC, bool BT>
__device__ __forceinline__ void zgemm_tile(int M, int N, int kbeg, int kend, double alpha, const double2* __restrict__ A,
                                           int64_t lda, const typename BElem<BC>::T* __restrict__ B, int64_t ldb,
                                           double2* __restrict__ C, int64_t ldc, int m0, int n0) {
    using TB = typename BElem<BC>::T;
    __shared__ double2 As[BK][BM + 1];
    __shared__ TB Bs[BK][BN + 1];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;

    double2 acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = zero2();

    for (int k0 = kbeg; k0 < kend; k0 += BK) {
        // A tile: 64 rows x 16 k, k fastest for coalescing
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            int mm = (tid >> 4) + 16 * r, kk = tid & 15;
            int gm = m0 + mm, gk = k0 + kk;
            As[kk][mm] = (gm < M && gk < kend) ? A[(int64_t)gm * lda + gk] : zero2();
        }
        if (!BT) {
            // B(k, n) = B[k*ldb + n], n fastest
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                int kk = (tid >> 6) + 4 * r, nn = tid & 63;
                int gk = k0 + kk, gn = n0 + nn;
                bool ok = gk < kend && gn < N;
                load_b(Bs[kk][nn], B + (ok ? (int64_t)gk * ldb + gn : 0), ok);
            }
        } else {
            // B(k, n) = B[n*ldb + k], k fastest
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                int nn = (tid >> 4) + 16 * r, kk = tid & 15;
                int gk = k0 + kk, gn = n0 + nn;
                bool ok = gk < kend && gn < N;
                load_b(Bs[kk][nn], B + (ok ? (int64_t)gn * ldb + gk : 0), ok);
            }
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            double2 a[4];
            TB b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) mac(acc[i][j], a[i], b[j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int gm = m0 + ty + 16 * i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int gn = n0 + tx + 16 * j;
            if (gn < N) C[(int64_t)gm * ldc + gn] = cscale(acc[i][j], alpha);
        }
    }
}
}  // namespace

// grid.z > 1 (split K): CTA layer z sums k in [z kc, min(K, (z + 1) kc)) into
// C + z cs (the caller adds the layers in a fixed order).
template <bool BC, bool BT>
__global__ void __launch_bounds__(256) k_zgemm(int M, int N, int K, double alpha,
                                               const double2* __restrict__ A, int64_t lda,
                                               const void* __restrict__ Bv, int64_t ldb,
                                               double2* __restrict__ C, int64_t ldc, int kc, int64_t cs) {
    const int kbeg = blockIdx.z * kc;
    zgemm_tile<BC, BT>(M, N, kbeg, min(K, kbeg + kc), alpha, A, lda, (const typename BElem<BC>::T*)Bv, ldb,
                       C + (int64_t)blockIdx.z * cs, ldc, blockIdx.y * BM, blockIdx.x * BN);
}

// The rows of C (tiles of 64) among which the digits (scales ex of the rows' parts) lost too much (oz_lost).  A tile's
// CTAs all check its rows and, mostly, end.  Otherwise they all see it, and wait for one another (arrived[tile], a
// cooperative launch) before the first of them writes what another one may still be reading.
template <bool BT>
__global__ void __launch_bounds__(256) k_zgemm_lost(int M, int N, int K, double alpha, const double2* __restrict__ A,
                                                    int64_t lda, const double* __restrict__ B, int64_t ldb,
                                                    double2* __restrict__ C, int64_t ldc, const int* __restrict__ amax,
                                                    const int* __restrict__ ex, int aexp, int* arrived, int* err) {
    const int m0 = blockIdx.y * BM, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // eight rows a warp: mostly one of a row's first 32 results tells that it is sound
    constexpr int R = BM / 8;
    int key[R], bmax[R];
    bool lost = false;
    const int am = *amax;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int m = min(m0 + R * wid + r, M - 1);
        key[r] = lane < N ? oz_key(C[(int64_t)m * ldc + lane]) : 0;
        bmax[r] = max(ex[2 * m], ex[2 * m + 1]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int m = min(m0 + R * wid + r, M - 1), bm = bmax[r], to = oz_reach(am, bm);
        const bool any = __any_sync(0xffffffffu, oz_key_expo(key[r]) - aexp >= to);
        lost = lost || oz_lost(am, bm, any || oz_scan(C + (int64_t)m * ldc, N, to == OZ_NAN ? to : to + aexp));
    }
    if (!__syncthreads_or(lost)) return;
    if (gridDim.x > 1) {
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(arrived + blockIdx.y, 1);
            const unsigned long long t0 = now_ns();
            while (*(volatile int*)(arrived + blockIdx.y) < (int)gridDim.x)
                if (now_ns() - t0 > 1000000000ull) {
                    atomicExch(err, AFQ_STATUS_WAIT_EXPIRED);
                    break;
                }
        }
        __syncthreads();
    }
    for (int n0 = blockIdx.x * BN; n0 < N; n0 += gridDim.x * BN)
        zgemm_tile<false, BT>(M, N, 0, K, alpha, A, lda, B, ldb, C, ldc, m0, n0);
}

int launch_zgemm_lost(int M, int N, int K, double alpha, const double2* A, int64_t lda, const double* B, int64_t ldb,
                      bool b_trans, double2* C, int64_t ldc, const int* amax, const int* ex, int aexp, int* arrived,
                      int* err, cudaStream_t s) {
    int sms = 0;
    AFQ_TRY(device_sms(&sms));
    const int mt = (M + BM - 1) / BM, nt = (N + BN - 1) / BN, per = sms / mt;  // at most a CTA an SM where they wait
    const dim3 grid(per < 1 ? 1 : per < nt ? per : nt, mt);
    void* args[] = {&M, &N, &K, &alpha, &A, &lda, &B, &ldb, &C, &ldc, &amax, &ex, &aexp, &arrived, &err};
    const void* kernel = b_trans ? (const void*)k_zgemm_lost<true> : (const void*)k_zgemm_lost<false>;
    AFQ_CUDA(grid.x > 1 ? cudaLaunchCooperativeKernel(kernel, grid, dim3(256), args, 0, s)
                        : cudaLaunchKernel(kernel, grid, dim3(256), args, 0, s));
    AFQ_LAUNCHED("k_zgemm_lost");
    return AFQ_OK;
}

int launch_zgemm(int M, int N, int K, double alpha, const double2* A, int64_t lda, const void* B,
                 int64_t ldb, bool b_complex, bool b_trans, double2* C, int64_t ldc,
                 cudaStream_t s) {
    if (M <= 0 || N <= 0) return AFQ_OK;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535u) return fail(AFQ_E_UNSUPPORTED, "zgemm: M=%d too large", M);
    if (b_complex) {
        if (b_trans) k_zgemm<true, true><<<grid, 256, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, C, ldc, K, 0);
        else k_zgemm<true, false><<<grid, 256, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, C, ldc, K, 0);
    } else {
        if (b_trans) k_zgemm<false, true><<<grid, 256, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, C, ldc, K, 0);
        else k_zgemm<false, false><<<grid, 256, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, C, ldc, K, 0);
    }
    AFQ_LAUNCHED("k_zgemm");
    return AFQ_OK;
}

// C (M x N, ldc = N) = sum_z part[z] in order z = 0 .. splits-1
__global__ void k_zsum_layers(long long count, int splits, const double2* __restrict__ part,
                              double2* __restrict__ C) {
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < count;
         e += (long long)gridDim.x * blockDim.x) {
        double2 a = part[e];
        for (int z = 1; z < splits; ++z) a = cadd(a, part[(long long)z * count + e]);
        C[e] = a;
    }
}

int zgemm_splits(int M, int N, int K) {
    const long long ctas = (long long)((N + BN - 1) / BN) * ((M + BM - 1) / BM);
    int z = 1;
    while (ctas * z < 2 * 152 && K / (z * 2) >= 4 * BK && z < 8) z *= 2;
    return z;
}

int launch_zgemm_splitk(int M, int N, int K, double alpha, const double2* A, int64_t lda, const void* B,
                        int64_t ldb, bool b_complex, bool b_trans, double2* C, double2* part, cudaStream_t s) {
    if (M <= 0 || N <= 0) return AFQ_OK;
    const int z = zgemm_splits(M, N, K);
    if (z == 1) return launch_zgemm(M, N, K, alpha, A, lda, B, ldb, b_complex, b_trans, C, N, s);
    const int kc = ((K + z - 1) / z + BK - 1) / BK * BK;  // z layers of kc cover K
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, z);
    if (grid.y > 65535u) return fail(AFQ_E_UNSUPPORTED, "zgemm: M=%d too large", M);
    const int64_t cs = (int64_t)M * N;
    if (b_complex) {
        if (b_trans) k_zgemm<true, true><<<grid, 256, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, part, N, kc, cs);
        else k_zgemm<true, false><<<grid, 256, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, part, N, kc, cs);
    } else {
        if (b_trans) k_zgemm<false, true><<<grid, 256, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, part, N, kc, cs);
        else k_zgemm<false, false><<<grid, 256, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, part, N, kc, cs);
    }
    AFQ_LAUNCHED("k_zgemm(split k)");
    long long blocks = (cs + 255) / 256;
    if (blocks > 152 * 32) blocks = 152 * 32;
    k_zsum_layers<<<(unsigned)blocks, 256, 0, s>>>(cs, z, part, C);
    AFQ_LAUNCHED("k_zsum_layers");
    return AFQ_OK;
}

// ------------------------------------------------------------ few products --
// Products of a few million multiplies, real right operand: a CTA of 128
// threads takes TM x 16 outputs, TM / 8 a thread, so that the binary64 pipe of
// every SM has the same share; the next 32 k are loaded while these are
// multiplied (one warp a quarter: nothing else hides the loads).
template <int TM, bool BT>
__global__ void __launch_bounds__(128) k_zgemm_small(int M, int N, int K, double alpha, const double2* __restrict__ A,
                                                     int64_t lda, const double* __restrict__ B, int64_t ldb,
                                                     double2* __restrict__ C, int64_t ldc) {
    constexpr int KS = 32, TN = 16, R = TM / 8;
    __shared__ double2 As[TM][KS + 1];
    __shared__ double Bs[KS][TN + 1];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    double2 acc[R], pa[2 * R];
    double pb[4];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = make_double2(0.0, 0.0);
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < 2 * R; ++q) {
            const int m = m0 + (tid >> 5) + 4 * q, k = k0 + (tid & 31);
            pa[q] = m < M && k < K ? A[m * lda + k] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = k0 + (BT ? tid & 31 : (tid >> 4) + 8 * q), n = n0 + (BT ? (tid >> 5) + 4 * q : tid & 15);
            pb[q] = k < K && n < N ? (BT ? B[n * ldb + k] : B[k * ldb + n]) : 0.0;
        }
    };
    load(0);
    for (int k0 = 0; k0 < K; k0 += KS) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 2 * R; ++q) As[(tid >> 5) + 4 * q][tid & 31] = pa[q];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (BT) Bs[tid & 31][(tid >> 5) + 4 * q] = pb[q];
            else Bs[(tid >> 4) + 8 * q][tid & 15] = pb[q];
        }
        __syncthreads();
        if (k0 + KS < K) load(k0 + KS);
        const int kn = min(KS, K - k0);
#pragma unroll 4
        for (int k = 0; k < kn; ++k) {
            const double b = Bs[k][tx];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const double2 a = As[ty + 8 * r][k];
                acc[r].x = fma(a.x, b, acc[r].x);
                acc[r].y = fma(a.y, b, acc[r].y);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int m = m0 + ty + 8 * r;
        if (m < M && n0 + tx < N) C[m * ldc + n0 + tx] = make_double2(alpha * acc[r].x, alpha * acc[r].y);
    }
}

// rows a CTA: the least work on the fullest SM, the larger tile at a tie; work: products a thread there and k
static int small_rows(int M, int N, long long* work) {
    int tm = 0;
    for (int t = 32; t >= 8; t /= 2) {
        const long long ctas = (long long)((M + t - 1) / t) * ((N + 15) / 16), w = (ctas + 151) / 152 * (t / 8);
        if (tm && w >= *work) continue;
        tm = t;
        *work = w;
    }
    return tm;
}

// A product and k costs a thread 128 clocks (two operations of a warp on the binary64 pipe), the digits 20-30 us of
// launches and a tile's chain whatever the size.  In captured graphs, small -> digits: M x N x K 256 x 144 x 48 9.0 ->
// 21.9 us, 256 x 48 x 72 7.5 -> 23.4, 8 x 150 x 210 18.5 -> 28.7, 400 x 100 x 100 (work 300) 21.3 -> 26.3; 500 x 500 x
// 20 (280) 20.8 -> 21.2; 200 x 150 x 210 (420) 34.0 -> 31.1, 8 x 301 x 549 (549) 45.9 -> 28.7.
bool zgemm_small_pays(int M, int N, int K) {
    if (M <= 0 || N <= 0) return false;
    long long work = 0;
    small_rows(M, N, &work);
    return work * K <= 300;
}

int launch_zgemm_small(int M, int N, int K, double alpha, const double2* A, int64_t lda, const double* B, int64_t ldb,
                       bool b_trans, double2* C, int64_t ldc, cudaStream_t s) {
    if (M <= 0 || N <= 0) return AFQ_OK;
    long long work = 0;
    const int tm = small_rows(M, N, &work);
    const dim3 grid((N + 15) / 16, (M + tm - 1) / tm);
    if (grid.y > 65535) return fail(AFQ_E_UNSUPPORTED, "small gemm: M=%d", M);
#define AFQ_ZS(TM)                                                                                          \
    do {                                                                                                    \
        if (b_trans) k_zgemm_small<TM, true><<<grid, 128, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, C, ldc);  \
        else k_zgemm_small<TM, false><<<grid, 128, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, C, ldc);         \
    } while (0)
    if (tm == 32) AFQ_ZS(32);
    else if (tm == 16) AFQ_ZS(16);
    else AFQ_ZS(8);
#undef AFQ_ZS
    AFQ_LAUNCHED("k_zgemm_small");
    return AFQ_OK;
}

}  // namespace afq
