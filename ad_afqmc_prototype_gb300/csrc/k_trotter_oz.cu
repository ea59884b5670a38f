// The binary64 Taylor series of small walkers, E_half . sum_{k <= K} (i sqrt_dt
// V)^k / k! . E_half . W (prop/utils.py:20-31, prop/chol_afqmc_ops.py:173-183),
// in one kernel a walker: up to 64 orbitals, whose V fits shared memory as
// digits.
//
// Each complex product Y = A T (A = V or E_half - I, n x n) is one real
// product with the K index (j, part): rows of A hold Re, Im interleaved, the
// column pair of T's column c holds [Tr, -Ti] and [Ti, Tr].  Both are cut
// into the seven exact base-256 digits of k_ozgemm.cu; the 34 digit products
// run on mma.sync m16n8k16 (a tcgen05 tile has 128 rows: a walker of 30
// orbitals fills a quarter of it, and the 128-row tile of V's digits would not
// fit beside T's at 60), with the six sums of each 16 x 8 tile in registers:
// K <= 128, so every sum d <= 4 is an exact integer below 2^24 units.  The
// accumulator's column pairs are complex entries, so a thread keeps its part of
// the running sum U in registers, turns its Y into the next T and writes T's
// digits back to shared memory; between the walker's read and its write no
// term leaves the SM.  The binary64 kernel (k_trotter) needs 28 n^2 o FMAs a
// walker at two a clock an SM, the tensor-core path of larger walkers
// (launch_trotter_oz) 16 launches and a 128 x 64 tile a walker and product.
#include "afq_internal.cuh"
#include "oz_digits.cuh"

namespace afq {

namespace {

constexpr int TS_NMAX = 64;  // orbitals

__device__ __forceinline__ uint32_t sm_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldm_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void ldm_x2(uint32_t& a, uint32_t& b, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Shared memory: A digits [7][16 mt][pitch], B digits [7][8 nt][pitch] (bf16,
// pitch = K + 8: ldmatrix rows 16 bytes apart modulo 128), row scales of A.
struct TsGeo {
    int mt, nt, kp, pitch;  // 16-row and 8-column tiles, K (a multiple of 16), row pitch in elements
    size_t a_bytes, b_bytes;
    __host__ __device__ TsGeo(int n, int oc)
        : mt((n + 15) / 16), nt((2 * oc + 7) / 8), kp((2 * n + 15) / 16 * 16), pitch(kp + 8),
          a_bytes((size_t)OZ_S * 16 * mt * pitch * 2), b_bytes((size_t)OZ_S * 8 * nt * pitch * 2) {}
};

// Digits of A's rows: eight k a lane, GL lanes a row, the scale from a max over
// the row's lanes.  ONE: A = E - I with E real (its Im parts zero).  ADJ: of
// the conjugate transpose.  s_amax is raised to the largest scale.
template <bool ONE, bool ADJ>
__device__ void ts_load_a(const TsGeo& g, int n, const void* __restrict__ src, __nv_bfloat16* As, int* s_ea, int* s_amax) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int l8 = g.kp / 8, gl = l8 <= 2 ? 2 : l8 <= 4 ? 4 : l8 <= 8 ? 8 : 16;  // lanes a row
    const int rw = 32 / gl, sub = lane / gl, k = 8 * (lane % gl);
    for (int r0 = rw * wid; r0 < 16 * g.mt; r0 += rw * nw) {
        const int r = r0 + sub;
        double x[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = k / 2 + i;
            double2 v = make_double2(0.0, 0.0);
            if (r < n && j < n) {
                const int at = ADJ ? j * n + r : r * n + j;
                if (ONE) v.x = ((const double*)src)[at] - (r == j ? 1.0 : 0.0);
                else v = ((const double2*)src)[at];
                if (ADJ) v.y = -v.y;
            }
            x[2 * i] = v.x;
            x[2 * i + 1] = v.y;
        }
        int e = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) e = max(e, oz_key(x[i]));
        for (int o = gl / 2; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
        const int E = oz_scale(e);
        if (k == 0 && r < 16 * g.mt) {
            s_ea[r] = E;
            atomicMax(s_amax, E);
        }
        if (k < g.kp && r < 16 * g.mt) {
            long long y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = oz_fix(x[i], E);
            __nv_bfloat16* d = As + (size_t)r * g.pitch + k;
            const size_t plane = (size_t)16 * g.mt * g.pitch;
            *(uint4*)d = oz_pack8<0>(y);
            *(uint4*)(d + plane) = oz_pack8<1>(y);
            *(uint4*)(d + 2 * plane) = oz_pack8<2>(y);
            *(uint4*)(d + 3 * plane) = oz_pack8<3>(y);
            *(uint4*)(d + 4 * plane) = oz_pack8<4>(y);
            *(uint4*)(d + 5 * plane) = oz_pack8<5>(y);
            *(uint4*)(d + 6 * plane) = oz_pack8<6>(y);
        }
    }
}

template <int S>
__device__ __forceinline__ void ts_put(uint32_t* d, size_t plane, int pw, long long y, long long z) {
    const float a = oz_dig<S>(y), b = oz_dig<S>(z);
    d[S * plane] = oz_pack(a, -b);      // row (c, Re): Tr, -Ti
    d[S * plane + pw] = oz_pack(b, a);  // row (c, Im): Ti, Tr
}

// NT: 8-column tiles a warp; warps = mt x (column groups).  Block p of walker w
// (ns of them, o columns each) is at w ws + p ss; V of the walker at w n^2.
// MODE:
//   TS_STEP  wout = E sum_k t_k, t_0 = E W, t_k = (i sqrt_dt / k) V t_{k-1}
//   TS_TAPE  the terms t_0 .. t_{K-1} to `terms` (W, K, n, o), wout = sum_k t_k
//   TS_ADJ   the reverse: b = E^T W, t_K = b, t_k = b + conj(i sqrt_dt / (k + 1)) V^H
//            t_{k+1} to `terms` (W, K + 1, n, o), wout = E^T t_0
enum { TS_STEP, TS_TAPE, TS_ADJ };

// The walker's series on the binary64 pipe, for the one that the digits cannot be left to (oz_lost): its input is still
// in place, the digits' shared memory (at least 28 n (n + 4 oc) bytes) holds two terms and the sum.
template <int MODE>
__device__ __forceinline__ void ts_plain(int n, int o, int oc, long long ws, long long ss, int n_terms, double sqrt_dt,
                                      const double* E, const double2* V, const double2* win, double2* wout, double2* terms,
                                      double2* sm) {
    const int w = blockIdx.x, no = n * oc;
    const double2* Vw = V + (size_t)w * n * n;
    double2 *cur = sm, *nxt = sm + no, *sum = sm + 2 * no;
    auto at = [&](int e) {
        const int i = e / oc, c = e - i * oc, p = c >= o;
        return w * ws + (long long)i * o + (c - p * o) + p * ss;
    };
    auto keep = [&](int slot, int e, double2 t) {  // ns = 1: oc = o
        if (MODE != TS_STEP) terms[((size_t)w * (MODE == TS_ADJ ? n_terms + 1 : n_terms) + slot) * no + e] = t;
    };
    auto e_times = [&](const double2* x, int e) {  // (E x)[e], E^T in the adjoint
        const int i = e / oc, c = e - i * oc;
        double2 a = make_double2(0.0, 0.0);
        for (int j = 0; j < n; ++j) rfma(a, E[MODE == TS_ADJ ? j * n + i : i * n + j], x[j * oc + c]);
        return a;
    };
    for (int e = threadIdx.x; e < no; e += blockDim.x) nxt[e] = win[at(e)];
    __syncthreads();
    for (int e = threadIdx.x; e < no; e += blockDim.x) {
        cur[e] = sum[e] = e_times(nxt, e);
        keep(MODE == TS_ADJ ? n_terms : 0, e, cur[e]);
    }
    __syncthreads();
    for (int k = 1; k <= n_terms; ++k) {
        const double s = sqrt_dt / (MODE == TS_ADJ ? n_terms + 1 - k : k);
        for (int e = threadIdx.x; e < no; e += blockDim.x) {
            const int i = e / oc, c = e - i * oc;
            double2 a = make_double2(0.0, 0.0);
            for (int j = 0; j < n; ++j) {
                const double2 v = Vw[MODE == TS_ADJ ? (size_t)j * n + i : (size_t)i * n + j];
                cfma(a, MODE == TS_ADJ ? make_double2(v.x, -v.y) : v, cur[j * oc + c]);
            }
            if (MODE == TS_ADJ) {
                nxt[e] = make_double2(sum[e].x + s * a.y, sum[e].y - s * a.x);
                keep(n_terms - k, e, nxt[e]);
            } else {
                nxt[e] = make_double2(-s * a.y, s * a.x);
                sum[e] = cadd(sum[e], nxt[e]);
                if (k < n_terms) keep(k, e, nxt[e]);
            }
        }
        __syncthreads();
        double2* t = cur;
        cur = nxt;
        nxt = t;
    }
    for (int e = threadIdx.x; e < no; e += blockDim.x)
        wout[at(e)] = MODE == TS_TAPE ? sum[e] : e_times(MODE == TS_ADJ ? cur : sum, e);
}

template <int NT, int MODE>
__global__ void __launch_bounds__(256) k_trotter_oz(int n, int o, int ns, long long ws, long long ss, int n_terms,
                                                    double sqrt_dt, const double* __restrict__ E,
                                                    const double2* __restrict__ V, const double2* win, double2* wout,
                                                    double2* __restrict__ terms) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int oc = o * ns;
    const TsGeo g(n, oc);
    __nv_bfloat16* As = (__nv_bfloat16*)smem_raw;
    __nv_bfloat16* Bs = (__nv_bfloat16*)(smem_raw + g.a_bytes);
    __shared__ int s_ea[TS_NMAX], s_eb[2][TS_NMAX], s_amax[2], s_most[2];  // s_amax: of E - I, V
    const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int mt = wid % g.mt, n0 = wid / g.mt * NT;  // this warp's row tile and first column tile
    const int r0 = 16 * mt + (lane >> 2), q = lane & 3;
    const int pw = g.pitch / 2;                        // row pitch in 32-bit words
    const size_t plane_b = (size_t)8 * g.nt * pw;      // words a digit plane

    for (int e = tid; e < 2 * TS_NMAX; e += blockDim.x) s_eb[0][e] = 0;
    if (tid == 0) {
        s_amax[0] = s_amax[1] = s_most[0] = OZ_EMPTY;
        s_most[1] = 0;
    }
    for (int e = tid; e < (int)(g.b_bytes / 16); e += blockDim.x) ((uint4*)Bs)[e] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    ts_load_a<true, MODE == TS_ADJ>(g, n, E, As, s_ea, &s_amax[0]);

    // entry (t, h): row r0 + 8 h, column c = 4 (n0 + t) + q
    double2 U[NT][2], T[NT][2];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = r0 + 8 * h, c = 4 * (n0 + t) + q, p = c >= o;
            U[t][h] = r < n && c < oc ? win[w * ws + (long long)r * o + (c - p * o) + p * ss] : make_double2(0.0, 0.0);
            T[t][h] = U[t][h];
        }
    __syncthreads();

    const size_t no = (size_t)n * o;
    auto keep = [&](size_t slot) {  // T to terms[slot]
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + 8 * h, c = 4 * (n0 + t) + q;
                if (r < n && c < oc) terms[slot * no + (size_t)r * o + c] = T[t][h];
            }
    };
    int buf = 0;
    // T's digits into Bs (after every warp has read the last ones); the product to come is A's (s_amax[v]) by a
    // coefficient below 2^ce
    auto put = [&](int v, int ce) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            int e = max(max(oz_key(T[t][0].x), oz_key(T[t][0].y)), max(oz_key(T[t][1].x), oz_key(T[t][1].y)));
            e = max(e, __shfl_xor_sync(0xffffffffu, e, 4));
            e = max(e, __shfl_xor_sync(0xffffffffu, e, 8));
            e = max(e, __shfl_xor_sync(0xffffffffu, e, 16));
            const int c = 4 * (n0 + t) + q;
            if (lane < 4 && c < oc) atomicMax(&s_eb[buf][c], e);
        }
        __syncthreads();
        if (tid < oc) {
            const int Ea = s_amax[v], Eb = oz_scale(s_eb[buf][tid]);
            if (Ea == OZ_NAN || Eb == OZ_NAN) atomicMax(&s_most[0], OZ_NAN);
            else if (Ea > OZ_ZERO && Eb > OZ_ZERO) atomicMax(&s_most[0], Ea + Eb + ce);
        }
        for (int e = tid; e < TS_NMAX; e += blockDim.x) s_eb[buf ^ 1][e] = 0;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int c = 4 * (n0 + t) + q;
            if (c >= oc) continue;
            const int Eb = oz_scale(s_eb[buf][c]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + 8 * h;
                if (r >= n) continue;
                const long long y = oz_fix(T[t][h].x, Eb), z = oz_fix(T[t][h].y, Eb);
                uint32_t* d = (uint32_t*)Bs + (size_t)(2 * c) * pw + r;
                ts_put<0>(d, plane_b, pw, y, z);
                ts_put<1>(d, plane_b, pw, y, z);
                ts_put<2>(d, plane_b, pw, y, z);
                ts_put<3>(d, plane_b, pw, y, z);
                ts_put<4>(d, plane_b, pw, y, z);
                ts_put<5>(d, plane_b, pw, y, z);
                ts_put<6>(d, plane_b, pw, y, z);
            }
        }
        __syncthreads();
    };
    // T = A T from the digits
    auto mul = [&]() {
        const uint32_t a0 = sm_addr(As) + ((16 * mt + (lane & 15)) * g.pitch + 8 * (lane >> 4)) * 2;
        const uint32_t plane_a = 16 * g.mt * g.pitch * 2;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            if (n0 + t >= g.nt) break;
            // lanes 0-15 address a digit's 8 x 16 block, lanes 16-31 the next digit's
            const uint32_t b0 = sm_addr(Bs) + ((8 * (n0 + t) + (lane & 7)) * g.pitch + 8 * ((lane >> 3) & 1)) * 2 +
                                (lane >> 4) * (uint32_t)(plane_b * 4);
            const uint32_t b6 = b0 - (lane >> 4) * (uint32_t)(plane_b * 4) + 6 * (uint32_t)(plane_b * 4);
            float acc[6][4];
#pragma unroll
            for (int d = 0; d < 6; ++d)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[d][i] = 0.f;
            for (int k = 0; k < g.kp; k += 16) {
                uint32_t b[4][4];
#pragma unroll
                for (int s = 0; s < 3; ++s) ldm_x4(b[s], b0 + 2 * s * (uint32_t)(plane_b * 4) + 2 * k);
                ldm_x2(b[3][0], b[3][1], b6 + 2 * k);
#pragma unroll
                for (int s = 0; s < OZ_S; ++s) {
                    uint32_t a[4];
                    ldm_x4(a, a0 + s * plane_a + 2 * k);
#pragma unroll
                    for (int x = 0; x < OZ_S; ++x)
                        if (s + x <= OZ_S) mma_bf16(acc[s + x < 5 ? s + x : 5], a, b[x / 2][2 * (x & 1)], b[x / 2][2 * (x & 1) + 1]);
                }
            }
            const int c = 4 * (n0 + t) + q, Eb = c < oc ? oz_scale(s_eb[buf][c]) : 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + 8 * h, Ea = s_ea[r];
                double v[2];
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    long long m = 0;
#pragma unroll
                    for (int d = 0; d < 5; ++d)
                        m += (long long)((unsigned long long)(long long)__float2int_rn(acc[d][2 * h + p] *
                                                                                       (float)(1ull << (8 * d)))
                                         << (32 - 8 * d));
                    v[p] = Ea == OZ_NAN || Eb == OZ_NAN ? __longlong_as_double(0x7ff8000000000000ll)
                                                        : oz_to_double(m, acc[5][2 * h + p], Ea + Eb - 14);
                }
                T[t][h] = make_double2(v[0], v[1]);
            }
        }
        buf ^= 1;
    };

    put(0, 0);
    mul();
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) U[t][h] = T[t][h] = cadd(U[t][h], T[t][h]);
    __syncthreads();
    ts_load_a<false, MODE == TS_ADJ>(g, n, V + (size_t)w * n * n, As, s_ea, &s_amax[1]);
    if (MODE == TS_TAPE) keep((size_t)w * n_terms);
    if (MODE == TS_ADJ) keep((size_t)w * (n_terms + 1) + n_terms);
    for (int k = 1; k <= n_terms; ++k) {
        // (i sqrt_dt / k) z = s (-z.y, z.x); the adjoint's coefficient is conj(i sqrt_dt / (K + 1 - k))
        const double s = sqrt_dt / (MODE == TS_ADJ ? n_terms + 1 - k : k);
        put(1, oz_scale(oz_key(s)));
        mul();
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (MODE == TS_ADJ) {
                    T[t][h] = make_double2(fma(s, T[t][h].y, U[t][h].x), fma(-s, T[t][h].x, U[t][h].y));
                } else {
                    T[t][h] = make_double2(-s * T[t][h].y, s * T[t][h].x);
                    U[t][h] = cadd(U[t][h], T[t][h]);
                }
            }
        if (MODE == TS_TAPE && k < n_terms) keep((size_t)w * n_terms + k);
        if (MODE == TS_ADJ) keep((size_t)w * (n_terms + 1) + n_terms - k);
    }
    if (MODE != TS_TAPE) {
        __syncthreads();
        ts_load_a<true, MODE == TS_ADJ>(g, n, E, As, s_ea, &s_amax[0]);
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (MODE == TS_ADJ) U[t][h] = T[t][h];
                else T[t][h] = U[t][h];
            }
        put(0, -4000);  // judged with the first one, by the same E
        mul();
    }
    // the products' scales against the sum's (oz_lost)
    int top = 0;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (r0 + 8 * h < n && 4 * (n0 + t) + q < oc) top = max(top, max(oz_key(U[t][h].x), oz_key(U[t][h].y)));
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) atomicMax(&s_most[1], top);
    __syncthreads();
    if (s_most[0] != OZ_EMPTY && oz_lost(s_most[0], 0, (s_most[1] >> 20) - 1023 >= oz_reach(s_most[0], 0))) {
        ts_plain<MODE>(n, o, oc, ws, ss, n_terms, sqrt_dt, E, V, win, wout, terms, (double2*)smem_raw);
        return;
    }
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = r0 + 8 * h, c = 4 * (n0 + t) + q, p = c >= o;
            if (r < n && c < oc)
                wout[w * ws + (long long)r * o + (c - p * o) + p * ss] =
                    MODE == TS_TAPE ? U[t][h] : cadd(U[t][h], T[t][h]);
        }
}

constexpr size_t TS_SMEM = 226 * 1024 - 1024;

// Column groups (warps a row tile) and column tiles a warp.
void ts_split(const TsGeo& g, int& groups, int& per) {
    groups = 8 / g.mt < g.nt ? 8 / g.mt : g.nt;
    per = (g.nt + groups - 1) / groups;
    groups = (g.nt + per - 1) / per;
}

template <int NT, int MODE>
int ts_run(int W, int n, int o, int ns, long long ws, long long ss, int n_terms, double sqrt_dt, const double* E,
           const double2* V, const double2* win, double2* wout, double2* terms, int warps, size_t smem, cudaStream_t s) {
    static DeviceOnce once;
    AFQ_TRY(raise_smem_once(once, k_trotter_oz<NT, MODE>, (int)TS_SMEM));
    k_trotter_oz<NT, MODE><<<W, 32 * warps, smem, s>>>(n, o, ns, ws, ss, n_terms, sqrt_dt, E, V, win, wout, terms);
    AFQ_LAUNCHED("k_trotter_oz");
    return AFQ_OK;
}

template <int MODE>
int ts_launch(int W, int n, int o, int n_terms, double sqrt_dt, const double* E, const double2* V, const double2* win,
              double2* wout, double2* terms, int ns, long long ws, long long ss, cudaStream_t s) {
    if (W <= 0) return AFQ_OK;
    if (!trotter_small_fits(n, o * ns, n_terms)) return fail(AFQ_E_UNSUPPORTED, "small trotter: norb=%d nocc=%d", n, o * ns);
    const TsGeo g(n, o * ns);
    int groups, per;
    ts_split(g, groups, per);
#define AFQ_TS(NT)                                                                                                       \
    if (per <= NT)                                                                                                       \
    return ts_run<NT, MODE>(W, n, o, ns, ws, ss, n_terms, sqrt_dt, E, V, win, wout, terms, g.mt * groups,                \
                            g.a_bytes + g.b_bytes, s)
    AFQ_TS(1);
    AFQ_TS(2);
    AFQ_TS(3);
    AFQ_TS(4);
    AFQ_TS(6);
#undef AFQ_TS
    return fail(AFQ_E_UNSUPPORTED, "small trotter: %d column tiles a warp", per);
}

}  // namespace

bool trotter_small_fits(int n, int oc, int n_terms) {
    if (n > TS_NMAX || oc > TS_NMAX || n_terms < 1) return false;
    const TsGeo g(n, oc);
    int groups, per;
    ts_split(g, groups, per);
    return per <= 6 && g.a_bytes + g.b_bytes <= TS_SMEM;
}

int launch_trotter_small(int W, int n, int o, int n_terms, double sqrt_dt, const double* E, const double2* V,
                         const double2* win, double2* wout, int ns, long long ws, long long ss, cudaStream_t s) {
    return ts_launch<TS_STEP>(W, n, o, n_terms, sqrt_dt, E, V, win, wout, nullptr, ns, ws, ss, s);
}

int launch_taylor_tape_small(int W, int n, int o, int K, double sqrt_dt, const double* E, const double2* V,
                             const double2* win, double2* terms, double2* w2, cudaStream_t s) {
    return ts_launch<TS_TAPE>(W, n, o, K, sqrt_dt, E, V, win, w2, terms, 1, (long long)n * o, 0, s);
}

int launch_taylor_adj_small(int W, int n, int o, int K, double sqrt_dt, const double* E, const double2* V,
                            const double2* wbar_post, double2* tbar, double2* wbar_pre, cudaStream_t s) {
    return ts_launch<TS_ADJ>(W, n, o, K, sqrt_dt, E, V, wbar_post, wbar_pre, tbar, 1, (long long)n * o, 0, s);
}

}  // namespace afq
