// Overlap matrix, determinant and half-rotated Green's function of each
// walker in binary64:  m = C^H W (o x o), overlap = det(m)^2 (meas/rhf.py:22-24),
// G_half = solve(m^T, W^T) = (W m^-1)^T (meas/rhf.py:15-19).
//
// The binary64 pipe of this GPU starts two lane operations a clock an SM (a
// warp instruction occupies its quarter for 64 clocks), so what counts is the
// number of binary64 warp instructions, also the redundant ones.  One CTA of
// four warps (one a quarter) takes a walker; m is held one element a thread
// and register, and an in-place Gauss-Jordan with implicit row pivoting (rows
// stay where they are, the pivot order is undone in the last indexing) turns
// it into m^-1 with four FMAs an element and step.  Pivots are chosen by
// integer comparisons of max(|Re|, |Im|); one warp a step, another one in
// every CTA, forms the pivot's reciprocal and the scaled pivot row.
//
// k_green<., INV = false> (overlaps only) skips the rows that are done.
// Where m and G_half are large products of their own they go by digits on
// the tensor cores (launch_green_oz) and this kernel only factorises.  only
// (optional): the walkers it marks.
#include "afq_internal.cuh"

namespace afq {

namespace {

constexpr int GR_T = 128;       // threads
constexpr int GR_IC = 32;       // walker rows staged at a time
// m is summed in blocks of 8 orbitals: the determinant and the inverse carry its error on, and that goes with the longest
// chain.  Off from a 113-bit evaluation, one chain -> blocks: overlaps of 30 x 7 1.31e-15 -> 0.93e-15, of 120 x 20 3.8e-15 ->
// 2.2e-15, G_half 3.3e-16 -> 2.6e-16 and 5.5e-16 -> 4.2e-16 (a Gauss-Jordan of the whole [m, I], one chain: 1.22e-15,
// 3.3e-15, 3.0e-16, 4.9e-16).  A block of ten steps of 12 orbitals takes 1 % longer, of 30 and more the same time.
constexpr int GR_IB = 8;

__device__ __forceinline__ unsigned long long gr_key(double2 v) {
    const unsigned long long a = (unsigned long long)__double_as_longlong(v.x) & 0x7fffffffffffffffull;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v.y) & 0x7fffffffffffffffull;
    const unsigned long long k = a > b ? a : b;
    return k > 0x7ff0000000000000ull ? 0ull : k;  // nan is never chosen over a number
}

// 1 / b = conj(b) / |b|^2 with b first scaled by a power of two near its
// magnitude, so that |b|^2 neither overflows nor underflows: one division
// where Smith's method takes three.
__device__ __forceinline__ double2 gr_recip(double2 b) {
    const int eb = (int)((gr_key(b) >> 52) & 0x7ffu);
    // scale 2^(1023 - eb), within the normal range (0 and subnormal b give inf or nan as a division does)
    const double sc = __longlong_as_double((long long)min(max(2046 - eb, 1), 2046) << 52);
    const double x = b.x * sc, y = b.y * sc;
    const double r = 1.0 / fma(x, x, y * y);
    return make_double2(x * r * sc, -(y * r) * sc);
}

// NE: elements of m a thread (NE x 128 >= o x o).  m_in (optional): m of every
// walker, else it is formed from the walker and the trial mo (n x o).  Outputs
// that are null are left out; green_out and inv_out need INV.
template <int NE, bool CR, bool INV>
__global__ void __launch_bounds__(GR_T) k_green(int n, int o, const double2* __restrict__ mo,
                                                const double2* __restrict__ walkers, const double2* __restrict__ m_in,
                                                double2* __restrict__ ovlp_out, double2* __restrict__ green_out,
                                                double2* __restrict__ inv_out, int ov_square,
                                                const int* __restrict__ only) {
    if (only && !only[blockIdx.x]) return;
    extern __shared__ double2 sm[];
    __shared__ double2 s_col[2][64], s_row[64], s_piv[64];
    __shared__ unsigned long long s_key[2][64];
    __shared__ int s_perm[64], s_iperm[64];
    const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const double2* Wp = walkers + (size_t)w * n * o;
    const int oo = o * o, wp = o | 1;  // staged rows are wp apart
    double2 a[NE];
    int er[NE], ej[NE];
#pragma unroll
    for (int q = 0; q < NE; ++q) {
        const int e = tid + GR_T * q;
        er[q] = e < oo ? e / o : 64;
        ej[q] = e < oo ? e - er[q] * o : 64;
        a[q] = make_double2(0.0, 0.0);
    }
    if (m_in) {
#pragma unroll
        for (int q = 0; q < NE; ++q)
            if (er[q] < 64) a[q] = m_in[(size_t)w * oo + tid + GR_T * q];
    } else {
        // m[r, j] = sum_i conj(C[i, r]) W[i, j], GR_IC rows of W and C at a time in shared memory
        double2* Ws = sm;
        double2* Cc = sm + GR_IC * wp;
        double* Cs = (double*)Cc;
        for (int i0 = 0; i0 < n; i0 += GR_IC) {
            const int in = min(GR_IC, n - i0);
            __syncthreads();
            for (int e = tid; e < in * o; e += GR_T) {
                const int i = e / o, j = e - i * o;
                Ws[i * wp + j] = Wp[(size_t)i0 * o + e];
                const double2 c = mo[(size_t)i0 * o + e];
                if (CR) Cs[i * wp + j] = c.x;
                else Cc[i * wp + j] = c;
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < NE; ++q) {
                if (er[q] >= 64) continue;
                for (int i1 = 0; i1 < in; i1 += GR_IB) {
                    double2 b = make_double2(0.0, 0.0);
                    for (int i = i1; i < min(in, i1 + GR_IB); ++i) {
                        const double2 x = Ws[i * wp + ej[q]];
                        if (CR) {
                            rfma(b, Cs[i * wp + er[q]], x);
                        } else {
                            const double2 c = Cc[i * wp + er[q]];
                            b.x = fma(c.x, x.x, b.x); b.x = fma(c.y, x.y, b.x);
                            b.y = fma(c.x, x.y, b.y); b.y = fma(-c.y, x.x, b.y);
                        }
                    }
                    a[q] = cadd(a[q], b);
                }
            }
        }
    }
    __syncthreads();

    unsigned long long used = 0;  // rows that have been pivots
    int swaps = 0;
    for (int k = 0; k < o; ++k) {
        const int buf = k & 1;
#pragma unroll
        for (int q = 0; q < NE; ++q)
            if (ej[q] == k) {
                s_col[buf][er[q]] = a[q];
                s_key[buf][er[q]] = gr_key(a[q]);
            }
        __syncthreads();
        // the unused row with the largest entry in column k, the lowest such row
        int p;
        {
            const unsigned long long k0 = lane < o && !((used >> lane) & 1) ? s_key[buf][lane] + 1 : 0;
            const unsigned long long k1 = lane + 32 < o && !((used >> (lane + 32)) & 1) ? s_key[buf][lane + 32] + 1 : 0;
            const unsigned long long km = k0 >= k1 ? k0 : k1;
            const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(km >> 32));
            const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(km >> 32) == hi ? (unsigned)km : 0u);
            const unsigned long long top = ((unsigned long long)hi << 32) | lo;
            const unsigned b0 = __ballot_sync(0xffffffffu, k0 == top), b1 = __ballot_sync(0xffffffffu, k1 == top);
            p = b0 ? __ffs(b0) - 1 : __ffs(b1) + 31;
        }
        // moving row p to the front of the unused rows passes the unused ones before it
        swaps += __popcll(~used & ((1ull << p) - 1));
        used |= 1ull << p;
#pragma unroll
        for (int q = 0; q < NE; ++q)
            if (er[q] == p) s_row[ej[q]] = a[q];
        __syncthreads();
        if (wid == ((k + w) & 3)) {
            const double2 piv = s_row[k];
            const double2 rp = gr_recip(piv);
            __syncwarp();
            for (int j = lane; j < o; j += 32) s_row[j] = j == k ? rp : cmul(s_row[j], rp);
            if (lane == 0) {
                s_piv[k] = piv;
                s_perm[k] = p;
                s_iperm[p] = k;
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NE; ++q) {
            const int r = er[q], j = ej[q];
            if (r >= 64) continue;
            if (r == p) {
                a[q] = s_row[j];
            } else if (INV || (j > k && !((used >> r) & 1))) {
                const double2 f = s_col[buf][r], s = s_row[j];
                double2 v = j == k ? make_double2(0.0, 0.0) : a[q];
                cfma(v, make_double2(-f.x, -f.y), s);
                a[q] = v;
            }
        }
    }
    // det(m): the pivots' product.  An exactly zero pivot (the rest of its column is zero too: m is singular)
    // makes it exactly 0, as LAPACK's LU gives it; the division by it has made the inverse, and so the Green's
    // function, non-finite, as the reference's solve does.
    if (ovlp_out && wid == (w & 3)) {
        double2 d = lane < o ? s_piv[lane] : make_double2(1.0, 0.0);
        const double2 d2 = lane + 32 < o ? s_piv[lane + 32] : make_double2(1.0, 0.0);
        const bool zero = (d.x == 0.0 && d.y == 0.0) || (d2.x == 0.0 && d2.y == 0.0);
        if (o > 32) d = cmul(d, d2);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            if (off >= o) continue;
            const double2 t = make_double2(__shfl_xor_sync(0xffffffffu, d.x, off), __shfl_xor_sync(0xffffffffu, d.y, off));
            d = cmul(d, t);
        }
        const bool sing = __any_sync(0xffffffffu, zero);
        if (lane == 0) {
            if (swaps & 1) d = make_double2(-d.x, -d.y);
            ovlp_out[w] = sing ? make_double2(0.0, 0.0) : ov_square ? cmul(d, d) : d;
        }
    }
    if (!INV) return;
    // row p_k of the reduced matrix is row k of the inverse, its column l belongs to row p_l of m
    if (inv_out) {
#pragma unroll
        for (int q = 0; q < NE; ++q)
            if (er[q] < 64) inv_out[(size_t)w * oo + s_iperm[er[q]] * o + s_perm[ej[q]]] = a[q];
    }
    if (!green_out) return;
    double2* inv = sm;                    // o x o
    double2* Ws = sm + oo;                // GR_IC rows of W
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NE; ++q)
        if (er[q] < 64) inv[s_iperm[er[q]] * o + s_perm[ej[q]]] = a[q];
    // G_half[b, i] = sum_a W[i, a] inv[a, b]
    double2* Gp = green_out + (size_t)w * o * n;
    for (int i0 = 0; i0 < n; i0 += GR_IC) {
        const int in = min(GR_IC, n - i0);
        __syncthreads();
        for (int e = tid; e < in * o; e += GR_T) {
            const int i = e / o;
            Ws[i * wp + (e - i * o)] = Wp[(size_t)i0 * o + e];
        }
        __syncthreads();
        for (int e = tid; e < in * o; e += GR_T) {
            const int b = e / in, i = e - b * in;
            double2 acc = make_double2(0.0, 0.0);
            for (int x = 0; x < o; ++x) cfma(acc, Ws[i * wp + x], inv[x * o + b]);
            Gp[(size_t)b * n + i0 + i] = acc;
        }
    }
}

template <int NE, bool CR, bool INV>
int run(int W, int n, int o, const double2* mo, const double2* walkers, const double2* m_in, double2* ovlp_out,
        double2* green_out, double2* inv_out, int ov_square, cudaStream_t s, const int* only) {
    static DeviceOnce once;
    const size_t wp = o | 1, stage = m_in ? 0 : GR_IC * wp * (sizeof(double2) + (CR ? sizeof(double) : sizeof(double2)));
    const size_t gsm = green_out ? ((size_t)o * o + GR_IC * wp) * sizeof(double2) : 0;
    const size_t smem = stage > gsm ? stage : gsm;
    AFQ_TRY(raise_smem_once(once, k_green<NE, CR, INV>, (64 * 64 + GR_IC * 65) * (int)sizeof(double2)));
    k_green<NE, CR, INV><<<W, GR_T, smem, s>>>(n, o, mo, walkers, m_in, ovlp_out, green_out, inv_out, ov_square, only);
    AFQ_LAUNCHED("k_green");
    return AFQ_OK;
}
template <bool CR, bool INV>
int run_ne(int W, int n, int o, const double2* mo, const double2* walkers, const double2* m_in, double2* ovlp_out,
           double2* green_out, double2* inv_out, int ov_square, cudaStream_t s, const int* only = nullptr) {
    const int ne = (o * o + GR_T - 1) / GR_T;
#define AFQ_GR(NE) \
    if (ne <= NE) return run<NE, CR, INV>(W, n, o, mo, walkers, m_in, ovlp_out, green_out, inv_out, ov_square, s, only)
    AFQ_GR(1);
    AFQ_GR(2);
    AFQ_GR(4);
    AFQ_GR(8);
    AFQ_GR(13);
    AFQ_GR(20);
    AFQ_GR(32);
#undef AFQ_GR
    return fail(AFQ_E_UNSUPPORTED, "green: nocc=%d > 64", o);
}

}  // namespace

// Factorisation of given m (W x o x o): determinants and, with inv_out, inverses.
int launch_lu(int W, int o, const double2* m, double2* ovlp_out, double2* inv_out, int ov_square, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    if (inv_out) return run_ne<true, true>(W, 0, o, nullptr, nullptr, m, ovlp_out, nullptr, inv_out, ov_square, s);
    return run_ne<true, false>(W, 0, o, nullptr, nullptr, m, ovlp_out, nullptr, nullptr, ov_square, s);
}

int launch_green_sq(int W, int n, int o, const double2* mo, int trial_real, const double2* walkers, double2* ovlp_out,
                    double2* green_out, int ov_square, cudaStream_t s, const int* only) {
    if (W <= 0) return AFQ_OK;
    if (trial_real) {
        if (green_out) return run_ne<true, true>(W, n, o, mo, walkers, nullptr, ovlp_out, green_out, nullptr, ov_square, s, only);
        return run_ne<true, false>(W, n, o, mo, walkers, nullptr, ovlp_out, nullptr, nullptr, ov_square, s, only);
    }
    if (green_out) return run_ne<false, true>(W, n, o, mo, walkers, nullptr, ovlp_out, green_out, nullptr, ov_square, s, only);
    return run_ne<false, false>(W, n, o, mo, walkers, nullptr, ovlp_out, nullptr, nullptr, ov_square, s, only);
}

int launch_green(int W, int n, int o, const double2* mo, int trial_real, const double2* walkers, double2* ovlp_out,
                 double2* green_out, cudaStream_t s) {
    return launch_green_sq(W, n, o, mo, trial_real, walkers, ovlp_out, green_out, 1, s);
}

int launch_green_auto(int W, int n, int o, const double2* mo, int trial_real, const double2* walkers,
                      double2* ovlp_out, double2* green_out, int ov_square, const OzScratch& oz, cudaStream_t s) {
    if (trial_real && oz.p && green_oz_pays(n, o))
        return launch_green_oz(W, n, o, mo, walkers, ovlp_out, green_out, ov_square, oz, s);
    return launch_green_sq(W, n, o, mo, trial_real, walkers, ovlp_out, green_out, ov_square, s);
}

}  // namespace afq
