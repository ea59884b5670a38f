// Per-walker binary64 kernels of the AFQMC step and block.
//
// Layouts: walkers (W, n, o) complex, row-major; G_half (W, o, n) complex;
// fields / shifted fields (W, G); chol (G, n, n) real; rot_chol (G, o, n)
// real (real trial) or complex.
#include "afq_internal.cuh"

namespace afq {

template <class K>
static int set_smem(K kernel, size_t bytes) {
    if (bytes > 227 * 1024) return fail(AFQ_E_UNSUPPORTED, "kernel needs %zu bytes of shared memory", bytes);
    if (bytes > 32 * 1024)  // with the kernel's static shared memory the default limit is below 48 KB
        AFQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return AFQ_OK;
}

// =====================================================================
// Trotter propagation  E_half . sum_{k<=K} (i sqrt_dt V)^k / k! . E_half . W
// (prop/chol_afqmc_ops.py:173-183, prop/utils.py:20-31).  Walker columns are
// independent, so a CTA owns (walker, OC columns): the current Taylor term
// lives in shared memory, the running sum in registers, and V / E_half are
// streamed through shared memory BJ columns at a time.
// =====================================================================
constexpr int TR_OC = 8, TR_BJ = 16, TR_THREADS = 256, TR_NRG = TR_THREADS / TR_OC;

template <int NR, bool REAL_M>
__device__ __forceinline__ void tr_matmul(int n, const void* __restrict__ Mg, const double2* __restrict__ T,
                                          double2* __restrict__ Ms, double2 (&acc)[NR], int c, int rg) {
#pragma unroll
    for (int q = 0; q < NR; ++q) acc[q] = make_double2(0.0, 0.0);
    double* Msr = (double*)Ms;
    for (int j0 = 0; j0 < n; j0 += TR_BJ) {
        const int jn = min(TR_BJ, n - j0);
        for (int e = threadIdx.x; e < n * TR_BJ; e += TR_THREADS) {
            int i = e / TR_BJ, jj = e % TR_BJ;
            if (REAL_M) Msr[e] = (jj < jn) ? ((const double*)Mg)[(size_t)i * n + j0 + jj] : 0.0;
            else Ms[e] = (jj < jn) ? ((const double2*)Mg)[(size_t)i * n + j0 + jj] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        for (int jj = 0; jj < jn; ++jj) {
            const double2 t = T[(j0 + jj) * TR_OC + c];
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                const int i = rg + TR_NRG * q;
                if (i < n) {
                    if (REAL_M) rfma(acc[q], Msr[i * TR_BJ + jj], t);
                    else cfma(acc[q], Ms[i * TR_BJ + jj], t);
                }
            }
        }
        __syncthreads();
    }
}

template <int NR>
__global__ void __launch_bounds__(TR_THREADS) k_trotter(int n, int o, int n_terms, double sqrt_dt,
                                                        const double* __restrict__ E,
                                                        const double2* __restrict__ V,
                                                        const double2* win, double2* wout, int vdiv,
                                                        const int* __restrict__ only) {
    if (only && !only[blockIdx.y / vdiv]) return;
    extern __shared__ double2 sm[];
    double2* T = sm;                    // n x OC
    double2* Ms = sm + (size_t)n * TR_OC;  // n x BJ
    const int w = blockIdx.y, c0 = blockIdx.x * TR_OC;
    const int tid = threadIdx.x, c = tid % TR_OC, rg = tid / TR_OC;
    const double2* Wp = win + (size_t)w * n * o;
    const double2* Vw = V + (size_t)(w / vdiv) * n * n;

    for (int e = tid; e < n * TR_OC; e += TR_THREADS) {
        int i = e / TR_OC, cc = e % TR_OC;
        T[e] = (c0 + cc < o) ? Wp[(size_t)i * o + c0 + cc] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    double2 acc[NR], out[NR];
    tr_matmul<NR, true>(n, E, T, Ms, acc, c, rg);
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        const int i = rg + TR_NRG * q;
        out[q] = acc[q];
        if (i < n) T[i * TR_OC + c] = acc[q];
    }
    __syncthreads();
    for (int k = 1; k <= n_terms; ++k) {
        tr_matmul<NR, false>(n, Vw, T, Ms, acc, c, rg);
        const double s = sqrt_dt / k;  // (i sqrt_dt / k) * z = s * (-z.y, z.x)
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            const int i = rg + TR_NRG * q;
            double2 t = make_double2(-s * acc[q].y, s * acc[q].x);
            out[q] = cadd(out[q], t);
            if (i < n) T[i * TR_OC + c] = t;
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        const int i = rg + TR_NRG * q;
        if (i < n) T[i * TR_OC + c] = out[q];
    }
    __syncthreads();
    tr_matmul<NR, true>(n, E, T, Ms, acc, c, rg);
    double2* Wo = wout + (size_t)w * n * o;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        const int i = rg + TR_NRG * q;
        if (i < n && c0 + c < o) Wo[(size_t)i * o + c0 + c] = acc[q];
    }
}

int launch_trotter(int W, int n, int o, int n_terms, double sqrt_dt, const double* E, const double2* V,
                   const double2* win, double2* wout, cudaStream_t s, int vdiv, const int* only) {
    if (W <= 0) return AFQ_OK;
    const int nr = (n + TR_NRG - 1) / TR_NRG;
    size_t smem = (size_t)n * (TR_OC + TR_BJ) * sizeof(double2);
    dim3 grid((o + TR_OC - 1) / TR_OC, W);
    if (W > 65535) return fail(AFQ_E_UNSUPPORTED, "trotter: chunk of %d walkers > 65535", W);
#define AFQ_TR(NRV)                                                                   \
    do {                                                                              \
        AFQ_TRY(set_smem(k_trotter<NRV>, smem));                                      \
        k_trotter<NRV><<<grid, TR_THREADS, smem, s>>>(n, o, n_terms, sqrt_dt, E, V, win, wout, vdiv, only); \
    } while (0)
    if (nr <= 1) AFQ_TR(1);
    else if (nr <= 2) AFQ_TR(2);
    else if (nr <= 4) AFQ_TR(4);
    else if (nr <= 8) AFQ_TR(8);
    else if (nr <= 16) AFQ_TR(16);
    else return fail(AFQ_E_UNSUPPORTED, "trotter: norb=%d > %d", n, 16 * TR_NRG);
#undef AFQ_TR
    AFQ_LAUNCHED("k_trotter");
    return AFQ_OK;
}

// =====================================================================
// Field shifts (prop/afqmc.py:97-101), one warp per walker:
//   fs = -sqrt_dt (i fb - mf);  x~ = x - fs;
//   shift_term = sum_g x~ mf;   fb_term = sum_g (x fs - fs^2 / 2)
// Bound by its 14 binary64 operations a field; few walkers go two warps a CTA
// so that they reach every SM.
// =====================================================================
__global__ void k_field_shift(int W, int G, double sqrt_dt, const double* __restrict__ x,
                              const double2* __restrict__ fb, const double2* __restrict__ mf,
                              double2* __restrict__ xs, double2* __restrict__ shift_term,
                              double2* __restrict__ fb_term) {
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= W) return;
    double sr = 0.0, si = 0.0, br = 0.0, bi = 0.0;
    for (int g = lane; g < G; g += 32) {
        const size_t e = (size_t)w * G + g;
        const double2 f = fb[e], m = mf[g];
        const double xv = x[e];
        // i fb - mf = (-f.y - m.x, f.x - m.y)
        const double2 fs = make_double2(sqrt_dt * (f.y + m.x), sqrt_dt * (m.y - f.x));
        const double2 xt = make_double2(xv - fs.x, -fs.y);
        xs[e] = xt;
        sr = fma(xt.x, m.x, sr);
        sr = fma(-xt.y, m.y, sr);
        si = fma(xt.x, m.y, si);
        si = fma(xt.y, m.x, si);
        // x fs - fs^2 / 2: real part fs.x (x - fs.x / 2) + fs.y^2 / 2, imaginary part fs.y (x - fs.x)
        br = fma(fs.x, fma(-0.5, fs.x, xv), br);
        br = fma(0.5 * fs.y, fs.y, br);
        bi = fma(fs.y, xt.x, bi);
    }
    sr = warp_sum(sr); si = warp_sum(si); br = warp_sum(br); bi = warp_sum(bi);
    if (lane == 0) {
        shift_term[w] = make_double2(sr, si);
        fb_term[w] = make_double2(br, bi);
    }
}

int launch_field_shift(int W, int G, double sqrt_dt, const double* x, const double2* fb, const double2* mf,
                       double2* xs, double2* shift_term, double2* fb_term, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    const int wpb = W < 8 * 152 ? 2 : 8;  // warps (walkers) a CTA
    k_field_shift<<<(W + wpb - 1) / wpb, 32 * wpb, 0, s>>>(W, G, sqrt_dt, x, fb, mf, xs, shift_term, fb_term);
    AFQ_LAUNCHED("k_field_shift");
    return AFQ_OK;
}

// =====================================================================
// Importance weights with the phaseless cut (prop/afqmc.py:116-138): one
// thread a walker and one warp a CTA (a walker's exponential, sincos and
// division are ~150 binary64 operations, of which a quarter of an SM starts one
// warp's in 64 clocks, so warps go to different SMs: 200 walkers 16 -> 7 us), then one CTA reduces the
// mean weight feeding the population-control shift in a fixed order
// (thread t sums walkers t, t + 1024, ...; then the warps and the CTA).
//
// Non-finite walkers: a NaN or infinite new overlap or weight propagates as
// in the reference (its floor and cap comparisons are false for NaN, so the
// weight stays NaN and the mean weight, hence the population shift, turns
// NaN).  With a status word (status != nullptr) every such walker is counted
// into status[1] and status[0] is set to AFQ_STATUS_NONFINITE if it was 0.
// =====================================================================
__global__ void __launch_bounds__(32) k_weight_update(
    int W, double dt, double sqrt_dt, double w_floor, double w_cap, double2 h0_prop,
    const double2* __restrict__ shift_term, const double2* __restrict__ fb_term,
    const double2* __restrict__ ovlp_new, double* __restrict__ weights, double2* __restrict__ overlaps,
    const double* __restrict__ pop_shift, int* __restrict__ status) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= W) return;
    const double ps = pop_shift[0];
    const double2 on = ovlp_new[w];
    double imp_ph = weight_factor<false>(dt, sqrt_dt, ps, h0_prop, shift_term[w], fb_term[w], on, overlaps[w]).imp_ph;
    if (imp_ph < w_floor) imp_ph = 0.0;
    if (imp_ph > w_cap) imp_ph = 0.0;
    double wn = weights[w] * imp_ph;
    if (wn > w_cap) wn = 0.0;
    weights[w] = wn;
    overlaps[w] = on;
    if (status && !(isfinite(wn) && isfinite(on.x) && isfinite(on.y))) {
        atomicAdd(status + 1, 1);
        atomicCAS(status, 0, AFQ_STATUS_NONFINITE);
    }
}

__global__ void __launch_bounds__(1024) k_weight_mean(int W, double dt, double damping,
                                                      const double* __restrict__ weights,
                                                      double* __restrict__ pop_shift,
                                                      const double* __restrict__ e_est) {
    double local = 0.0;
    for (int w = threadIdx.x; w < W; w += blockDim.x) local += weights[w];
    __shared__ double red[32];
    local = warp_sum(local);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0;
        v = warp_sum(v);
        if (threadIdx.x == 0) {
            double avg = v / W;
            avg = (avg < 1.0e-300) ? 1.0e-300 : avg;  // NaN passes through, as with clip
            pop_shift[0] = e_est[0] - damping * (log(avg) / dt);
        }
    }
}

// Overlaps after a QR from those before it: det(C^H Q)^2 = det(C^H W)^2 /
// det(R)^2 for Q = W R^-1 (walkers.py:183-203's restricted normalisation).
__global__ void k_overlap_div_det2(int W, const double2* __restrict__ det_r, double2* __restrict__ overlaps) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= W) return;
    const double2 r = det_r[w];
    overlaps[w] = cdiv(overlaps[w], cmul(r, r));
}

int launch_overlap_div_det2(int W, const double2* det_r, double2* overlaps, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    k_overlap_div_det2<<<(W + 255) / 256, 256, 0, s>>>(W, det_r, overlaps);
    AFQ_LAUNCHED("k_overlap_div_det2");
    return AFQ_OK;
}

int launch_weight_update(int W, const afq_params* p, double sqrt_dt, double dt, double2 h0_prop,
                         const double2* shift_term, const double2* fb_term, const double2* ovlp_new,
                         double* weights, double2* overlaps, double* pop_shift, const double* e_est,
                         cudaStream_t s, int* status) {
    if (W <= 0) return AFQ_OK;
    k_weight_update<<<(W + 31) / 32, 32, 0, s>>>(W, dt, sqrt_dt, p->weight_floor, p->weight_cap, h0_prop,
                                                    shift_term, fb_term, ovlp_new, weights, overlaps, pop_shift,
                                                    status);
    AFQ_LAUNCHED("k_weight_update");
    k_weight_mean<<<1, 1024, 0, s>>>(W, dt, p->pop_control_damping, weights, pop_shift, e_est);
    AFQ_LAUNCHED("k_weight_mean");
    return AFQ_OK;
}

// =====================================================================
// Local energy (meas/rhf.py:36-50).  f_g = L~_g G_half^T (o x o) for a chunk
// of NG Cholesky vectors per CTA; the tile keeps whole o x o blocks so that
// c_g = tr f_g and exc_g = sum_ij f_g[i,j] f_g[j,i] are reduced in the CTA
// and f never reaches global memory.  partial[w, chunk] = (sum c^2, sum exc).
// =====================================================================
constexpr int EN_BJ = 32, EN_R = 16, EN_THREADS = 256;

template <bool CR>
__global__ void __launch_bounds__(EN_THREADS) k_energy_partial(int n, int o, int G, int NG,
                                                               const double2* __restrict__ green,
                                                               const void* __restrict__ rotv,
                                                               double2* __restrict__ partial) {
    extern __shared__ double2 sm[];
    const int nchunk = gridDim.x;
    const int w = blockIdx.y, g0 = blockIdx.x * NG;
    const int ng = min(NG, G - g0);
    const int tid = threadIdx.x;
    const int nout = ng * o * o;
    double2* Gs = sm;                          // o x BJ
    double2* Ls = sm + o * EN_BJ;              // ng*o x BJ (complex or real)
    double* Lsr = (double*)Ls;
    double2* F = sm + o * EN_BJ + (CR ? (NG * o * EN_BJ + 1) / 2 : NG * o * EN_BJ);  // ng x o x o
    const double2* Gw = green + (size_t)w * o * n;

    double2 acc[EN_R];
    int offL[EN_R], offG[EN_R];
#pragma unroll
    for (int r = 0; r < EN_R; ++r) {
        acc[r] = make_double2(0.0, 0.0);
        int e = tid + EN_THREADS * r;
        int g = e / (o * o), rem = e % (o * o), i = rem / o, k = rem % o;
        offL[r] = (g * o + i) * EN_BJ;
        offG[r] = k * EN_BJ;
    }
    for (int j0 = 0; j0 < n; j0 += EN_BJ) {
        const int jn = min(EN_BJ, n - j0);
        for (int e = tid; e < o * EN_BJ; e += EN_THREADS) {
            int k = e / EN_BJ, jj = e % EN_BJ;
            Gs[e] = jj < jn ? Gw[(size_t)k * n + j0 + jj] : make_double2(0.0, 0.0);
        }
        for (int e = tid; e < ng * o * EN_BJ; e += EN_THREADS) {
            int gi = e / EN_BJ, jj = e % EN_BJ;  // gi = g*o + i
            size_t src = ((size_t)g0 * o + gi) * n + j0 + jj;
            if (CR) Lsr[e] = jj < jn ? ((const double*)rotv)[src] : 0.0;
            else Ls[e] = jj < jn ? ((const double2*)rotv)[src] : make_double2(0.0, 0.0);
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < EN_R; ++r) {
            if (tid + EN_THREADS * r < nout) {
                for (int jj = 0; jj < jn; ++jj) {
                    if (CR) rfma(acc[r], Lsr[offL[r] + jj], Gs[offG[r] + jj]);
                    else cfma(acc[r], Ls[offL[r] + jj], Gs[offG[r] + jj]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < EN_R; ++r) {
        int e = tid + EN_THREADS * r;
        if (e < nout) F[e] = acc[r];
    }
    __syncthreads();
    // per g: c = tr f, exc = sum_ik f[i,k] f[k,i]; thread-strided over (g, i, k)
    double cr = 0.0, ci = 0.0, xr = 0.0, xi = 0.0;
    for (int e = tid; e < nout; e += EN_THREADS) {
        int g = e / (o * o), rem = e % (o * o), i = rem / o, k = rem % o;
        double2 a = F[e], b = F[g * o * o + k * o + i];
        double2 p = cmul(a, b);
        xr += p.x; xi += p.y;
    }
    // sum_g c_g^2 : one thread per g
    for (int g = tid; g < ng; g += EN_THREADS) {
        double2 c = make_double2(0.0, 0.0);
        for (int i = 0; i < o; ++i) c = cadd(c, F[g * o * o + i * o + i]);
        double2 c2 = cmul(c, c);
        cr += c2.x; ci += c2.y;
    }
    __shared__ double red[4][EN_THREADS / 32];
    cr = warp_sum(cr); ci = warp_sum(ci); xr = warp_sum(xr); xi = warp_sum(xi);
    if ((tid & 31) == 0) {
        red[0][tid >> 5] = cr; red[1][tid >> 5] = ci; red[2][tid >> 5] = xr; red[3][tid >> 5] = xi;
    }
    __syncthreads();
    if (tid == 0) {
        double s[4] = {0, 0, 0, 0};
        for (int q = 0; q < 4; ++q)
            for (int k = 0; k < EN_THREADS / 32; ++k) s[q] += red[q][k];
        partial[((size_t)w * nchunk + blockIdx.x) * 2 + 0] = make_double2(s[0], s[1]);
        partial[((size_t)w * nchunk + blockIdx.x) * 2 + 1] = make_double2(s[2], s[3]);
    }
}

// energy = h0 + 2 sum G_half * rot_h1 + 2 sum c^2 - exc, one warp per walker
__global__ void k_energy_finish(int W, int n, int o, int nchunk, double h0, const double2* __restrict__ green,
                                const double2* __restrict__ rot_h1, const double2* __restrict__ partial,
                                double2* __restrict__ energy) {
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= W) return;
    const double2* Gw = green + (size_t)w * o * n;
    double er = 0.0, ei = 0.0;
    for (int e = lane; e < o * n; e += 32) {
        double2 p = cmul(Gw[e], rot_h1[e]);
        er += p.x; ei += p.y;
    }
    er = warp_sum(er); ei = warp_sum(ei);
    double cr = 0.0, ci = 0.0, xr = 0.0, xi = 0.0;
    for (int c = lane; c < nchunk; c += 32) {
        double2 a = partial[((size_t)w * nchunk + c) * 2 + 0], b = partial[((size_t)w * nchunk + c) * 2 + 1];
        cr += a.x; ci += a.y; xr += b.x; xi += b.y;
    }
    cr = warp_sum(cr); ci = warp_sum(ci); xr = warp_sum(xr); xi = warp_sum(xi);
    if (lane == 0) energy[w] = make_double2(h0 + 2.0 * er + 2.0 * cr - xr, 2.0 * ei + 2.0 * ci - xi);
}

static int energy_ng(int o, int G) {
    int ng = (EN_R * EN_THREADS) / (o * o);
    if (ng < 1) ng = 1;
    if (ng > G) ng = G;
    return ng;
}

size_t energy_partial_count(int W, int o, int G) {  // number of double2
    int ng = energy_ng(o, G);
    return (size_t)W * ((G + ng - 1) / ng) * 2;
}

int energy_partial_chunks(int o, int G) {
    const int ng = energy_ng(o, G);
    return (G + ng - 1) / ng;
}

static size_t energy_smem(int o, int G, int trial_real) {
    const int ng = energy_ng(o, G);
    const size_t lsz = trial_real ? (size_t)(ng * o * EN_BJ + 1) / 2 : (size_t)ng * o * EN_BJ;
    return ((size_t)o * EN_BJ + lsz + (size_t)ng * o * o) * sizeof(double2);
}

bool energy_partial_fits(int o, int G, int trial_real) {
    return o * o <= EN_R * EN_THREADS && energy_smem(o, G, trial_real) <= 227 * 1024;
}

int launch_energy(int W, int n, int o, int G, double h0, const double2* green, const void* rot_chol,
                  int trial_real, const double2* rot_h1, double* partial_d, double2* energy, const OzScratch& oz,
                  cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    AFQ_TRY(launch_energy_partial_auto(W, n, o, G, green, rot_chol, trial_real, partial_d, oz, s));
    return launch_energy_finish(W, n, o, energy_partial_chunks(o, G), h0, green, rot_h1, (const double2*)partial_d,
                                energy, s);
}

int launch_energy_partial(int W, int n, int o, int G, const double2* green, const void* rot_chol, int trial_real,
                          double* partial_d, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    if (o * o > EN_R * EN_THREADS) return fail(AFQ_E_UNSUPPORTED, "energy: nocc=%d > 64", o);
    const int ng = energy_ng(o, G);
    const int nchunk = (G + ng - 1) / ng;
    double2* partial = (double2*)partial_d;
    const size_t smem = energy_smem(o, G, trial_real);
    dim3 grid(nchunk, W);
    if (W > 65535) return fail(AFQ_E_UNSUPPORTED, "energy: %d walkers > 65535 per call", W);
    if (trial_real) {
        AFQ_TRY(set_smem(k_energy_partial<true>, smem));
        k_energy_partial<true><<<grid, EN_THREADS, smem, s>>>(n, o, G, ng, green, rot_chol, partial);
    } else {
        AFQ_TRY(set_smem(k_energy_partial<false>, smem));
        k_energy_partial<false><<<grid, EN_THREADS, smem, s>>>(n, o, G, ng, green, rot_chol, partial);
    }
    AFQ_LAUNCHED("k_energy_partial");
    return AFQ_OK;
}

int launch_energy_finish(int W, int n, int o, int nchunk, double h0, const double2* green, const double2* rot_h1,
                         const double2* partial, double2* energy, cudaStream_t s) {
    k_energy_finish<<<(W + 7) / 8, 256, 0, s>>>(W, n, o, nchunk, h0, green, rot_h1, partial, energy);
    AFQ_LAUNCHED("k_energy_finish");
    return AFQ_OK;
}

// =====================================================================
// Householder QR with diag(R) real >= 0 (walkers.py:169-180), in place in
// shared memory, column-major with odd leading dimension.  Q is formed in
// place by backward accumulation of the reflectors H_k = I - tau v v^H.
//
// The binary64 pipe bounds it (two lane operations a clock an SM): eight FMAs
// an element of v and column, forward and backward, 1.35 M lane operations a
// walker at 200 x 30.  So v stays unscaled (tau = 1 / (|x| (|x| + |x_0|))
// takes the scale), one warp forms a reflector's scalars, and a warp takes
// up to four columns at a time, whose eight dot products are reduced together
// (nine adds instead of forty).  4096 walkers of 200 x 30: 25.2 ms with scaled
// reflectors, separate multiplies and adds and every thread forming the scalars.
// =====================================================================

// Sums over the warp of NV (2, 4 or 8) values a lane; every lane gets all of them.
template <int NV>
__device__ __forceinline__ void warp_sum_n(double (&v)[NV], int lane) {
    int off = 16;
#pragma unroll
    for (int h = NV / 2; h >= 1; h >>= 1, off >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < NV / 2; ++i) {
            if (i >= h) continue;
            const double send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    // lane bits 4 .. (the log2 NV highest) choose the value; the others still hold partial sums
    double x = v[0];
#pragma unroll
    for (int o2 = 16; o2 >= 1; o2 >>= 1)
        if (o2 * NV < 32) x += __shfl_xor_sync(0xffffffffu, x, o2);
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = __shfl_sync(0xffffffffu, x, i * (32 / NV));
}

// Columns j0 .. j0 + C - 1: y -= tau v (v^H y) over the rows from k on (one warp).
template <int C>
__device__ __forceinline__ void qr_apply(const double2* v, double2* y, int ldy, int rs, int k, int n, double tau, int lane) {
    constexpr int NV = C == 1 ? 2 : C == 2 ? 4 : 8;
    double d[NV];
#pragma unroll
    for (int c = 0; c < NV; ++c) d[c] = 0.0;
    for (int i = k + lane; i < n; i += 32) {
        const double2 x = v[i * rs];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const double2 b = y[c * ldy + i * rs];
            d[2 * c] = fma(x.x, b.x, d[2 * c]);
            d[2 * c + 1] = fma(x.x, b.y, d[2 * c + 1]);
            d[2 * c] = fma(x.y, b.y, d[2 * c]);
            d[2 * c + 1] = fma(-x.y, b.x, d[2 * c + 1]);
        }
    }
    warp_sum_n<NV>(d, lane);
#pragma unroll
    for (int c = 0; c < 2 * C; ++c) d[c] *= -tau;
    for (int i = k + lane; i < n; i += 32) {
        const double2 x = v[i * rs];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            double2 b = y[c * ldy + i * rs];
            cfma(b, x, make_double2(d[2 * c], d[2 * c + 1]));
            y[c * ldy + i * rs] = b;
        }
    }
}
// The columns from j0 to o - 1, spread over the CTA's eight warps.
__device__ __forceinline__ void qr_apply_all(double2* A, int ld, int rs, int k, int j0, int n, int o, double tau, int wid,
                                             int lane) {
    const int c = min(4, (o - j0 + 7) / 8);  // columns a warp takes at a time
    const double2* v = A + k * ld;
    for (int j = j0 + c * wid; j < o; j += 8 * c) {
        const int m = min(c, o - j);
        double2* y = A + j * ld;
        if (m == 4) qr_apply<4>(v, y, ld, rs, k, n, tau, lane);
        else if (m == 3) qr_apply<3>(v, y, ld, rs, k, n, tau, lane);
        else if (m == 2) qr_apply<2>(v, y, ld, rs, k, n, tau, lane);
        else qr_apply<1>(v, y, ld, rs, k, n, tau, lane);
    }
}

// GLOBAL: the walker is factorised in place in wout (element (i, j) at
// A[i o + j], wout already holding the input), for walkers too large for
// shared memory; otherwise A[j ld + i] in shared memory.
template <bool GLOBAL>
__global__ void __launch_bounds__(256) k_qr(int n, int o, const double2* __restrict__ win,
                                            double2* __restrict__ wout, double2* __restrict__ det_out,
                                            const int* __restrict__ flag) {
    if (flag && !flag[blockIdx.x]) return;
    extern __shared__ double2 Asm[];
    __shared__ double2 s_ph[64];             // alpha / |alpha|, the phase that makes diag(R) >= 0
    __shared__ double s_tau[64], s_nx[64];   // reflector scales and |R_kk|
    const int ld = GLOBAL ? 1 : (n | 1);  // column stride
    const int rs = GLOBAL ? o : 1;        // row stride
    const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double2* A = GLOBAL ? wout + (size_t)w * n * o : Asm;
    if (!GLOBAL) {
        const double2* Wp = win + (size_t)w * n * o;
        for (int e = tid; e < n * o; e += blockDim.x) {
            int i = e / o, j = e % o;
            A[j * ld + i] = Wp[e];
        }
    } else if (flag && win != wout) {
        for (int e = tid; e < n * o; e += blockDim.x) A[e] = win[(size_t)w * n * o + e];
    }
    __syncthreads();
    for (int k = 0; k < o; ++k) {
        // one warp, another one in each CTA and step, forms reflector k
        if (wid == ((k + w) & 7)) {
            double2* x = A + k * ld;
            double sg = 0.0;
            for (int i = k + 1 + lane; i < n; i += 32) {
                const double2 t = x[i * rs];
                sg = fma(t.x, t.x, sg);
                sg = fma(t.y, t.y, sg);
            }
            sg = warp_sum(sg);
            const double2 x0 = x[k * rs];
            const double a2 = cabs2(x0), ax0 = sqrt(a2), nx = sqrt(a2 + sg), den = nx * (nx + ax0);
            const double ia = 1.0 / ax0;
            const double2 ph = ax0 == 0.0 ? make_double2(1.0, 0.0) : make_double2(x0.x * ia, x0.y * ia);
            __syncwarp();
            if (lane == 0) {
                x[k * rs] = make_double2(x0.x + ph.x * nx, x0.y + ph.y * nx);  // v_0 = x_0 - alpha, alpha = -ph |x|
                s_tau[k] = den > 0.0 ? 1.0 / den : 0.0;
                s_ph[k] = nx == 0.0 ? make_double2(1.0, 0.0) : make_double2(-ph.x, -ph.y);
                s_nx[k] = nx;
            }
        }
        __syncthreads();
        qr_apply_all(A, ld, rs, k, k + 1, n, o, s_tau[k], wid, lane);
        __syncthreads();
    }
    // backward accumulation of Q: H_k on the later columns, then column k itself is H_k e_k
    for (int k = o - 1; k >= 0; --k) {
        double2* v = A + k * ld;
        const double tau = s_tau[k];
        qr_apply_all(A, ld, rs, k, k + 1, n, o, tau, wid, lane);
        const double2 v0 = v[k * rs];
        __syncthreads();
        const double2 f = make_double2(-tau * v0.x, tau * v0.y);  // -tau conj(v_0)
        for (int i = tid; i < n; i += blockDim.x) {
            if (i < k) v[i * rs] = make_double2(0.0, 0.0);
            else if (i == k) v[i * rs] = make_double2(fma(-tau, cabs2(v0), 1.0), 0.0);
            else v[i * rs] = cmul(f, v[i * rs]);
        }
        __syncthreads();
    }
    // R~_kk = alpha_k is complex here (the reference's LAPACK R has a real
    // diagonal, hence its conj(phase) fix); Q[:, k] *= alpha_k / |alpha_k|
    // gives the same unique Q with diag(R) real and >= 0.
    double2* Wo = wout + (size_t)w * n * o;
    for (int e = tid; e < n * o; e += blockDim.x) {
        int i = e / o, j = e % o;
        Wo[e] = cmul(A[j * ld + i * rs], s_ph[j]);
    }
    if (det_out && tid == 0) {
        double d = 1.0;
        for (int k = 0; k < o; ++k) d *= s_nx[k];
        det_out[w] = make_double2(d, 0.0);
    }
}

int launch_qr(int W, int n, int o, const double2* win, double2* wout, double2* det_r, cudaStream_t s,
              const int* flag) {
    if (W <= 0) return AFQ_OK;
    if (o > 64) return fail(AFQ_E_UNSUPPORTED, "qr: nocc=%d > 64", o);
    size_t smem = (size_t)(n | 1) * o * sizeof(double2);
    if (smem <= 200 * 1024) {
        AFQ_TRY(set_smem(k_qr<false>, smem));
        k_qr<false><<<W, 256, smem, s>>>(n, o, win, wout, det_r, flag);
        AFQ_LAUNCHED("k_qr");
        return AFQ_OK;
    }
    // too large for shared memory: in place in wout
    if (wout != win && !flag)
        AFQ_CUDA(cudaMemcpyAsync(wout, win, sizeof(double2) * (size_t)W * n * o, cudaMemcpyDeviceToDevice, s));
    k_qr<true><<<W, 256, 0, s>>>(n, o, flag ? win : wout, wout, det_r, flag);
    AFQ_LAUNCHED("k_qr(global)");
    return AFQ_OK;
}

// =====================================================================
// Stochastic comb (walkers.py:233-265).  The prefix sum of |w| follows the
// association order of jax.lax.associative_scan, which is what the
// reference's jnp.cumsum lowers to on CPU and GPU: an up-sweep of pairwise
// sums e_{L+1}[k] = e_L[2k] + e_L[2k+1], then a down-sweep
// s_L[2k+1] = s_{L+1}[k], s_L[0] = e_L[0], s_L[2k] = s_{L+1}[k-1] + e_L[2k].
// Each add is one IEEE binary64 add (__dadd_rn: never contracted), so the
// bits are reproducible.  The search repeats jnp.searchsorted's default
// probe sequence (ceil(log2(W+1)) rounds of mid = (lo+hi)/2,
// z <= cw[mid] ? hi = mid : lo = mid; result hi), so even an ulp-level
// inversion of cw is searched identically.  One CTA; levels in `lv`.
// =====================================================================
size_t sr_levels_size(int W) {  // doubles over all levels (<= 2W)
    size_t t = 0;
    for (size_t n = (size_t)(W > 0 ? W : 1);; n >>= 1) {
        t += n;
        if (n < 2) break;
    }
    return t;
}

__global__ void __launch_bounds__(1024) k_sr_scan(int W, const double* __restrict__ weights, double zeta,
                                                  const double* __restrict__ zeta_dev,
                                                  double* __restrict__ lv, int32_t* __restrict__ idx,
                                                  double* __restrict__ cumsum_out, double* __restrict__ avg_out) {
    __shared__ int s_off[40], s_cnt[40], s_top;
    const int tid = threadIdx.x, nt = blockDim.x;
    if (tid == 0) {
        int off = 0, n = W, L = 0;
        for (;;) {
            s_off[L] = off;
            s_cnt[L] = n;
            off += n;
            if (n < 2) break;
            n >>= 1;
            ++L;
        }
        s_top = L;
    }
    for (int i = tid; i < W; i += nt) lv[i] = fabs(weights[i]);
    __syncthreads();
    const int top = s_top;
    for (int L = 0; L < top; ++L) {  // up-sweep
        const double* e = lv + s_off[L];
        double* r = lv + s_off[L + 1];
        for (int k = tid; k < s_cnt[L + 1]; k += nt) r[k] = __dadd_rn(e[2 * k], e[2 * k + 1]);
        __syncthreads();
    }
    for (int L = top - 1; L >= 0; --L) {  // down-sweep, in place
        double* e = lv + s_off[L];
        const double* su = lv + s_off[L + 1];
        const int nL = s_cnt[L];
        for (int k = tid; 2 * k < nL; k += nt) {
            const double ev = (k == 0) ? e[0] : __dadd_rn(su[k - 1], e[2 * k]);
            if (2 * k + 1 < nL) e[2 * k + 1] = su[k];
            e[2 * k] = ev;
        }
        __syncthreads();
    }
    if (cumsum_out)
        for (int i = tid; i < W; i += nt) cumsum_out[i] = lv[i];
    const double tot = lv[W - 1];
    const double zt = zeta_dev ? zeta_dev[0] : zeta;
    if (tid == 0 && avg_out) avg_out[0] = __ddiv_rn(tot, (double)W);
    int rounds = 0;
    while ((1ll << rounds) < (long long)W + 1) ++rounds;
    for (int k = tid; k < W; k += nt) {
        const double z = __ddiv_rn(__dmul_rn(tot, __dadd_rn((double)k, zt)), (double)W);
        int lo = 0, hi = W;
        for (int r = 0; r < rounds; ++r) {
            const int mid = (int)(((unsigned)lo + (unsigned)hi) >> 1);
            const bool left = z <= lv[mid < W ? mid : W - 1];
            lo = left ? lo : mid;
            hi = left ? mid : hi;
        }
        idx[k] = hi < W ? hi : W - 1;
    }
}

int launch_sr_scan(int W, const double* weights, double zeta, double* levels, int32_t* idx, double* cumsum_out,
                   double* avg_out, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    k_sr_scan<<<1, 1024, 0, s>>>(W, weights, zeta, nullptr, levels, idx, cumsum_out, avg_out);
    AFQ_LAUNCHED("k_sr_scan");
    return AFQ_OK;
}

int launch_sr_scan_dev(int W, const double* weights, const double* zeta_dev, double* levels, int32_t* idx,
                       double* avg_out, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    k_sr_scan<<<1, 1024, 0, s>>>(W, weights, 0.0, zeta_dev, levels, idx, nullptr, avg_out);
    AFQ_LAUNCHED("k_sr_scan");
    return AFQ_OK;
}

// dst[k] = src[idx[k]] for rows of `row` complex; weights_out[k] = avg
__global__ void k_gather(int W, int64_t row, const int32_t* __restrict__ idx, const double2* __restrict__ src,
                         double2* __restrict__ dst, const double* __restrict__ avg, double* __restrict__ weights_out) {
    const int k = blockIdx.y;
    const int64_t base = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int j = idx[k];
    for (int64_t e = base; e < row; e += (int64_t)gridDim.x * blockDim.x)
        dst[(size_t)k * row + e] = src[(size_t)j * row + e];
    if (weights_out && blockIdx.x == 0 && threadIdx.x == 0) weights_out[k] = avg[0];
}

int launch_gather(int W, int64_t row, const int32_t* idx, const double2* src, double2* dst, const double* avg,
                  double* weights_out, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    if (W > 65535) return fail(AFQ_E_UNSUPPORTED, "gather: %d walkers > 65535", W);
    int bx = (int)((row + 255) / 256);
    if (bx > 64) bx = 64;
    if (bx < 1) bx = 1;
    k_gather<<<dim3(bx, W), 256, 0, s>>>(W, row, idx, src, dst, avg, weights_out);
    AFQ_LAUNCHED("k_gather");
    return AFQ_OK;
}

// =====================================================================
// Block measurement (prop/blocks.py:59-79): clip |E - e_est| > sqrt(2/dt),
// weighted mean (w_sum == 0 -> e_est), EMA of the population shift.
// =====================================================================
__global__ void __launch_bounds__(1024) k_block_measure(int W, double dt, double alpha,
                                                        const double* __restrict__ weights,
                                                        const double2* __restrict__ energy,
                                                        const double* __restrict__ e_est, double* pop_shift,
                                                        double* block_energy, double* block_weight) {
    const double eref = e_est[0];
    const double thresh = sqrt(2.0 / dt);
    double sw = 0.0, swe = 0.0;
    for (int w = threadIdx.x; w < W; w += blockDim.x) {
        double e = energy[w].x;
        if (fabs(e - eref) > thresh) e = eref;
        const double wt = weights[w];
        sw += wt;
        swe += wt * e;
    }
    __shared__ double r0[32], r1[32];
    sw = warp_sum(sw); swe = warp_sum(swe);
    if ((threadIdx.x & 31) == 0) { r0[threadIdx.x >> 5] = sw; r1[threadIdx.x >> 5] = swe; }
    __syncthreads();
    if (threadIdx.x < 32) {
        const bool ok = threadIdx.x < (blockDim.x >> 5);
        double a = ok ? r0[threadIdx.x] : 0.0, b = ok ? r1[threadIdx.x] : 0.0;
        a = warp_sum(a); b = warp_sum(b);
        if (threadIdx.x == 0) {
            const double safe = (a == 0.0) ? 1.0 : a;
            double eb = b / safe;
            if (a == 0.0) eb = eref;
            block_energy[0] = eb;
            block_weight[0] = a;
            pop_shift[0] = (1.0 - alpha) * pop_shift[0] + alpha * eb;
        }
    }
}

// Files one block's energy and weight at the run's next index and advances
// the run's Philox counter (the tail of a captured block).
__global__ void k_run_record(const double* __restrict__ e, const double* __restrict__ w, double* __restrict__ es,
                             double* __restrict__ ws, int* __restrict__ idx, uint64_t* __restrict__ counter,
                             uint64_t inc) {
    const int b = idx[0];
    es[b] = e[0];
    ws[b] = w[0];
    idx[0] = b + 1;
    counter[0] += inc;
}

int launch_run_record(const double* e, const double* w, double* es, double* ws, int* idx, uint64_t* counter,
                      uint64_t inc, cudaStream_t s) {
    k_run_record<<<1, 1, 0, s>>>(e, w, es, ws, idx, counter, inc);
    AFQ_LAUNCHED("k_run_record");
    return AFQ_OK;
}

int launch_block_measure(int W, double dt, double shift_ema, const double* weights, const double2* energy,
                         const double* e_est, double* pop_shift, double* block_energy, double* block_weight,
                         cudaStream_t s) {
    k_block_measure<<<1, 1024, 0, s>>>(W, dt, shift_ema, weights, energy, e_est, pop_shift, block_energy,
                                       block_weight);
    AFQ_LAUNCHED("k_block_measure");
    return AFQ_OK;
}

// =====================================================================
// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) counter-based RNG.
// Call e uses counter (lo(e), hi(e), lo(counter), hi(counter)) and key
// (lo(seed), hi(seed)); its four words give two 53-bit uniforms u, v.
// Normals: Box-Muller, r = sqrt(-2 log(1-u)), (r cos 2 pi v, r sin 2 pi v),
// evaluated in fp32 from x = fp32(1 - u) and fp32(v) (the binary64
// transcendentals cost ~80 binary64 operations a pair at 1/64 of the fp32
// rate); each normal carries fp32 rounding, ~1e-7 relative.
// =====================================================================
__device__ __forceinline__ uint4 philox10(uint4 c, uint2 k) {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r > 0) { k.x += W0; k.y += W1; }
        const uint32_t hi0 = __umulhi(M0, c.x), lo0 = M0 * c.x;
        const uint32_t hi1 = __umulhi(M1, c.z), lo1 = M1 * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    }
    return c;
}

__device__ __forceinline__ double u53(uint32_t a, uint32_t b) {
    return ((double)(a >> 5) * 67108864.0 + (double)(b >> 6)) * (1.0 / 9007199254740992.0);
}

__global__ void k_philox(int64_t count, uint64_t seed, uint64_t counter0, int normal, double* __restrict__ out,
                         const uint64_t* __restrict__ cbase) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * e >= count) return;
    const uint64_t counter = counter0 + (cbase ? cbase[0] : 0ull);
    const uint4 r = philox10(make_uint4((uint32_t)e, (uint32_t)((uint64_t)e >> 32), (uint32_t)counter,
                                        (uint32_t)(counter >> 32)),
                             make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
    const double u = u53(r.x, r.y), v = u53(r.z, r.w);
    double a = u, b = v;
    if (normal) {
        const float rad = sqrtf(-2.0f * logf((float)(1.0 - u)));
        float sn, cs;
        sincospif(2.0f * (float)v, &sn, &cs);
        a = (double)(rad * cs);
        b = (double)(rad * sn);
    }
    out[2 * e] = a;
    if (2 * e + 1 < count) out[2 * e + 1] = b;
}

// Counter base read on the device, set for the duration of a captured block
// loop (afq_run_blocks) on the calling thread; null otherwise.
thread_local const uint64_t* t_counter_base = nullptr;

int launch_philox(int64_t count, uint64_t seed, uint64_t counter, int normal, double* out, cudaStream_t s) {
    if (count <= 0) return AFQ_OK;
    int64_t pairs = (count + 1) / 2;
    k_philox<<<(unsigned)((pairs + 255) / 256), 256, 0, s>>>(count, seed, counter, normal, out, t_counter_base);
    AFQ_LAUNCHED("k_philox");
    return AFQ_OK;
}

}  // namespace afq
