// The small kernels of the binary64 QR by digits (launch_qr_oz in
// k_ozgemm.cu; walkers.py:169-211: the unique Q with diag(R) real and > 0).
//
//   G = W^H W;  G = R1^H R1;  Q1 = W R1^-1;  I + E = Q1^H Q1;
//   Q = Q1 - Q1 U, U the strict upper triangle of E plus half its diagonal,
// with W^H W, Q1^H Q1 and W R1^-1 as digit products.  E is of the order of
// cond(W)^2 1e-16 and the next order, E^2, is dropped where every |E| is below
// 1e-9; Q1 U is then a correction of Q1's last digits and fp32 forms it.
// det R = (1 + sum E_kk / 2) / prod (R1^-1)_kk.
//
// Walkers this does not suit take the Householder form (k_qr), whose input is
// still in place: a pivot of G below 1e-4 of its column's squared norm,
// squared column norms more than 2^6 apart (the rows of W are cut at one scale
// each, so a small column would lose digits), |E| of 1e-9 or more, inf or nan,
// or an expired wait.
#include "afq_internal.cuh"

namespace afq {

namespace {

constexpr int QF_T = 128;

// Entry (a, b) of the Gram matrix from the real products C[b][2 a + part] =
// (<a_part, Re b>, <a_part, Im b>) of a walker's columns.
__device__ __forceinline__ double2 qr_gram(const double2* c, int o, int a, int b) {
    const double2 r = c[(size_t)b * 2 * o + 2 * a], i = c[(size_t)b * 2 * o + 2 * a + 1];
    return make_double2(r.x + i.y, r.y - i.x);
}

// R1^-1 of a walker (30 columns, 342 walkers: 66 us) from its Gram matrix: L D L^H by elimination, one element
// a thread and register; the places below the diagonal take L^-1, and R1^-1 =
// L^-H D^-1/2.  A chain of o steps with two barriers each; the binary64 pipe
// (two lanes a clock an SM) sees o^3 / 3 complex products and one division a
// step, by one warp.
template <int NE>
__global__ void __launch_bounds__(QF_T) k_qr_factor(int o, const double2* __restrict__ gram, double2* __restrict__ tinv,
                                                    double* __restrict__ det, int* __restrict__ flag) {
    __shared__ double2 s_row[2][64], s_f[64];
    __shared__ double s_d[64], s_g[64], s_is[64];
    const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, oo = o * o;
    const double2* c = gram + (size_t)w * 2 * oo;
    double2 a[NE];
    int er[NE], ej[NE];
#pragma unroll
    for (int q = 0; q < NE; ++q) {
        const int e = tid + QF_T * q;
        er[q] = e < oo ? e / o : -1;
        ej[q] = e < oo ? e - er[q] * o : 0;
        a[q] = make_double2(0.0, 0.0);
        if (er[q] < 0) continue;
        if (ej[q] >= er[q]) a[q] = qr_gram(c, o, er[q], ej[q]);
        if (ej[q] == er[q]) s_g[er[q]] = a[q].x;
        if (er[q] == 0) s_row[0][ej[q]] = a[q];
    }
    __syncthreads();
    for (int k = 0; k < o; ++k) {
        const double2* row = s_row[k & 1];
        if (wid == (k & 3)) {
            const double d = row[k].x, rd = 1.0 / d;
            if (lane == 0) s_d[k] = d;
            for (int t = k + 1 + lane; t < o; t += 32) s_f[t] = make_double2(-row[t].x * rd, row[t].y * rd);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NE; ++q) {
            const int i = er[q], j = ej[q];
            if (i <= k || (j < i && j > k)) continue;
            if (j == k) a[q] = s_f[i];
            else cfma(a[q], s_f[i], row[j]);
            if (i == k + 1) s_row[(k + 1) & 1][j] = a[q];
        }
        __syncthreads();
    }
    if (wid == 0) {
        int lo = 0x7fffffff, hi = 0, bad = 0;
        double p = 1.0;
        for (int k = lane; k < o; k += 32) {
            const double d = s_d[k];
            const int x = __double2hiint(s_g[k]) >> 20;  // sign and exponent
            lo = min(lo, x);
            hi = max(hi, x);
            if (!(d > 1e-4 * s_g[k])) bad = 1;
            const double is = 1.0 / sqrt(d);
            s_is[k] = is;
            p *= is;
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        bad = __any_sync(0xffffffffu, bad) || lo <= 0 || hi >= 0x7ff || hi - lo > 6;
#pragma unroll
        for (int t = 16; t > 0; t >>= 1) p *= __shfl_xor_sync(0xffffffffu, p, t);
        if (lane == 0) {
            flag[w] = bad;
            det[w] = 1.0 / p;
        }
    }
    __syncthreads();
    double2* T = tinv + (size_t)w * oo;
#pragma unroll
    for (int q = 0; q < NE; ++q) {
        const int i = er[q], j = ej[q];
        if (i < 0) continue;
        const double is = s_is[i];
        T[j * o + i] = j > i ? make_double2(0.0, 0.0) : j == i ? make_double2(is, 0.0) : make_double2(a[q].x * is, -a[q].y * is);
    }
}

// binary64 <-> fp32 by integer operations (the binary64 pipe converts two a clock an SM); truncates, zero below 2^-126
__device__ __forceinline__ float qr_f32(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int e = (int)((hi >> 20) & 0x7ffu) - 896;
    return e <= 0 ? 0.f : __uint_as_float((hi & 0x80000000u) | (unsigned)min(e, 254) << 23 | (hi & 0xfffffu) << 3 | lo >> 29);
}
__device__ __forceinline__ double qr_f64(float x) {
    const unsigned u = __float_as_uint(x), e = (u >> 23) & 255u;
    return e == 0 ? 0.0 : __hiloint2double((int)((u & 0x80000000u) | (e + 896u) << 20 | (u >> 3 & 0xfffffu)), (int)(u << 29));
}

// Q = Q1 - Q1 U and det R of the walkers that pass.  A thread takes one column
// of four rows, so that an entry of U serves four (200 x 30, 342 walkers: 46
// us, 59 with one row and the conversions on the binary64 pipe).
__global__ void __launch_bounds__(256) k_qr_finish(int n, int o, const double2* __restrict__ q1,
                                                   const double2* __restrict__ gram, const double* __restrict__ det,
                                                   const int* __restrict__ err, double2* __restrict__ out,
                                                   double2* __restrict__ det_out, int* __restrict__ flag) {
    extern __shared__ float2 qfs[];  // U (o x o), then rows of Q1 in fp32
    constexpr int RB = 64;           // rows at a time
    __shared__ double s_e[64];
    const int w = blockIdx.x, tid = threadIdx.x, oo = o * o;
    const double2* c = gram + (size_t)w * 2 * oo;
    float2 *U = qfs, *X = qfs + oo;
    bool bad = flag[w] != 0 || *err != 0;
    for (int e = tid; e < oo; e += 256) {
        const int a = e / o, b = e - a * o;
        float2 u = make_float2(0.f, 0.f);
        if (a <= b) {
            double2 g = qr_gram(c, o, a, b);
            if (a == b) {
                g.x -= 1.0;
                s_e[a] = g.x;
            }
            u = make_float2((float)g.x, (float)g.y);
            if (!(fabsf(u.x) < 1e-9f && fabsf(u.y) < 1e-9f)) bad = true;
            if (a == b) u = make_float2(0.5f * u.x, 0.f);
        }
        U[e] = u;
    }
    bad = __syncthreads_or(bad);
    if (bad) {
        if (tid == 0) flag[w] = 1;
        return;
    }
    const double2* q = q1 + (size_t)w * n * o;
    double2* Q = out + (size_t)w * n * o;
    for (int i0 = 0; i0 < n; i0 += RB) {
        const int m = min(RB, n - i0) * o;
        __syncthreads();
        for (int e = tid; e < m; e += 256) {
            const double2 v = q[(size_t)i0 * o + e];
            X[e] = make_float2(qr_f32(v.x), qr_f32(v.y));
        }
        __syncthreads();
        for (int e = tid; e < RB / 4 * o; e += 256) {
            const int i = e / o * 4, b = e - e / o * o;
            float x[4] = {}, y[4] = {};
            for (int a = 0; a <= b; ++a) {
                const float2 u = U[a * o + b];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float2 p = X[(i + r) * o + a];
                    x[r] = fmaf(p.x, u.x, fmaf(-p.y, u.y, x[r]));
                    y[r] = fmaf(p.x, u.y, fmaf(p.y, u.x, y[r]));
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (i0 + i + r >= n) break;
                const size_t at = (size_t)(i0 + i + r) * o + b;
                const double2 v = q[at];
                Q[at] = make_double2(v.x - qr_f64(x[r]), v.y - qr_f64(y[r]));
            }
        }
    }
    if (det_out && tid == 0) {
        double t = 0.0;
        for (int k = 0; k < o; ++k) t += s_e[k];
        det_out[w] = make_double2(fma(det[w], 0.5 * t, det[w]), 0.0);
    }
}

}  // namespace

int launch_qr_factor(int W, int o, const double2* gram, double2* tinv, double* det, int* flag, cudaStream_t s) {
    if (o > 64) return fail(AFQ_E_UNSUPPORTED, "qr: nocc=%d > 64", o);
    const int ne = (o * o + QF_T - 1) / QF_T;
#define AFQ_QF(NE) k_qr_factor<NE><<<W, QF_T, 0, s>>>(o, gram, tinv, det, flag)
    if (ne <= 2) AFQ_QF(2);
    else if (ne <= 4) AFQ_QF(4);
    else if (ne <= 8) AFQ_QF(8);
    else if (ne <= 16) AFQ_QF(16);
    else AFQ_QF(32);
#undef AFQ_QF
    AFQ_LAUNCHED("k_qr_factor");
    return AFQ_OK;
}

int launch_qr_finish(int W, int n, int o, const double2* q1, const double2* gram, const double* det, const int* err,
                     double2* out, double2* det_out, int* flag, cudaStream_t s) {
    static DeviceOnce once;
    AFQ_TRY(raise_smem_once(once, k_qr_finish, 2 * 64 * 64 * (int)sizeof(float2)));
    k_qr_finish<<<W, 256, (size_t)(o * o + 64 * o) * sizeof(float2), s>>>(n, o, q1, gram, det, err, out, det_out, flag);
    AFQ_LAUNCHED("k_qr_finish");
    return AFQ_OK;
}

}  // namespace afq
