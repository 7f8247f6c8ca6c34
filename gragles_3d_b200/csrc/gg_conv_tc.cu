// gg_conv_tc.cu -- mixed-precision per-axis circulant convolution (FP32 storage).
//
// See gg_conv_tc.cuh.  Two batched passes over all boxes:
//   xy: one CTA per (grain, z-plane): x then y contraction of the plane with C_n
//   z:  one CTA per (grain, y-row):   z contraction of the [z][x] slab, in place
#include <algorithm>
#include <cmath>

#include "gg_common.cuh"
#include "gg_conv_tc.cuh"

namespace gg {

void circulant_matrix(int n, int N, double time_step, float* out) {
    // per-axis factor of box.cpp:760-761: exp(-sqrt(2/pi) 4 dt N^2 pi^2 / n^2 * f^2), f = min(k, n-k)
    const double pi = 3.14159265358979323846;
    const double dt = time_step / double(N * N);
    const double c = std::sqrt(2 / pi) * 4.0 * dt * double(N * N) / double(n * n) * pi * pi;
    std::vector<long double> factor(n);
    for (int f = 0; f < n; f++) {
        const int ff = f < n - f ? f : n - f;
        factor[f] = std::exp(-(long double)c * ff * ff);
    }
    std::vector<float> col(n);
    for (int d = 0; d < n; d++) {
        long double acc = 0;
        for (int f = 0; f < n; f++) acc += factor[f] * std::cos(2.0L * (long double)pi * f * d / n);
        col[d] = (float)(acc / n);
    }
    for (int p = 0; p < n; p++)
        for (int q = 0; q < n; q++) out[(size_t)p * n + q] = col[(p - q + n) % n];
}

void circulant_tables(int N, double time_step, int lo, int hi, const std::vector<char>* need, std::vector<float>& out,
                      std::vector<long long>& off) {
    long long total = 0;
    for (int n = lo; n <= hi; n++) {
        off[n] = total;
        if (!need || (*need)[n]) total += (long long)n * n;
    }
    out.resize(total);
    for_sides(lo, hi, [&](int n) {
        if (!need || (*need)[n]) circulant_matrix(n, N, time_step, out.data() + off[n]);
    });
}

namespace {

constexpr int kThreads = 384;
constexpr int kR = 8;        // output rows per thread
constexpr int kMaxNB = 5;    // 32-wide column groups of the largest side (139)

// Pitch of the shared-memory matrices: even, for the two-element reads, and 2 modulo 4, so that
// the 32 lanes that read one column of 32 rows fall on 16 banks.
__host__ __device__ constexpr int pitch_of(int n) { return (n + 1) / 4 * 4 + 2; }
// Rows of the plane that pass xy stages at a time: all, or half where all would not fit.
__host__ __device__ constexpr int plane_rows(int n) {
    return 3 * n * pitch_of(n) * (int)sizeof(float) <= 227 * 1024 ? n : (n + 1) / 2;
}

// out(a, b) = sum_m A[a][m] B(m, b), a < na, b < n, one fma per m in order.  A warp takes kR
// rows a and all columns b = lane + 32 j; A's rows are read two m at a time, the same
// address for all lanes.  TRANS: B(m, b) = Bs[b][m], else Bs[m][b].  A warp's shared-memory
// reads per two m are kR + 2 NB for 2 kR NB fma.
template <int NB, bool TRANS, typename F>
__device__ __forceinline__ void product(const float* __restrict__ A, const float* __restrict__ Bs, int pitch, int n,
                                        int na, F&& store) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int at[NB];
#pragma unroll
    for (int j = 0; j < NB; j++) {
        const int b = min(lane + 32 * j, n - 1);
        at[j] = TRANS ? b * pitch : b;
    }
    for (int a0 = warp * kR; a0 < na; a0 += kThreads / 32 * kR) {
        const float* rows[kR];
#pragma unroll
        for (int r = 0; r < kR; r++) rows[r] = A + min(a0 + r, na - 1) * pitch;
        float acc[kR][NB];
#pragma unroll
        for (int r = 0; r < kR; r++)
#pragma unroll
            for (int j = 0; j < NB; j++) acc[r][j] = 0.f;
        auto step = [&](int m, const float (&av)[kR]) {
#pragma unroll
            for (int j = 0; j < NB; j++) {
                const float bv = Bs[at[j] + (TRANS ? m : m * pitch)];
#pragma unroll
                for (int r = 0; r < kR; r++) acc[r][j] = fmaf(av[r], bv, acc[r][j]);
            }
        };
        int m = 0;
        for (; m + 2 <= n; m += 2) {
            float2 v[kR];
            float av[kR];
#pragma unroll
            for (int r = 0; r < kR; r++) v[r] = *reinterpret_cast<const float2*>(rows[r] + m);
#pragma unroll
            for (int r = 0; r < kR; r++) av[r] = v[r].x;
            step(m, av);
#pragma unroll
            for (int r = 0; r < kR; r++) av[r] = v[r].y;
            step(m + 1, av);
        }
        for (; m < n; m++) {
            float av[kR];
#pragma unroll
            for (int r = 0; r < kR; r++) av[r] = rows[r][m];
            step(m, av);
        }
#pragma unroll
        for (int r = 0; r < kR; r++)
#pragma unroll
            for (int j = 0; j < NB; j++)
                if (a0 + r < na && lane + 32 * j < n) store(a0 + r, lane + 32 * j, acc[r][j]);
    }
}

template <bool TRANS, typename F>
__device__ __forceinline__ void product_any(const float* A, const float* Bs, int pitch, int n, int na, F&& store) {
    switch ((n + 31) >> 5) {  // the launch takes sides above 64; smaller ones come with them in one call
        case 1: product<1, TRANS>(A, Bs, pitch, n, na, store); break;
        case 2: product<2, TRANS>(A, Bs, pitch, n, na, store); break;
        case 3: product<3, TRANS>(A, Bs, pitch, n, na, store); break;
        case 4: product<4, TRANS>(A, Bs, pitch, n, na, store); break;
        default: product<kMaxNB, TRANS>(A, Bs, pitch, n, na, store); break;
    }
}

// Both kernels are bound by shared-memory reads and FP32 FMA.  With four rows and one column
// a thread, five reads served four fma (2.2 ms for 30 boxes of 90^3); with 8 rows and 3 columns
// 14 reads serve 48 (0.8 ms).
__global__ void __launch_bounds__(kThreads, 2) conv_xy_kernel(ConvTCArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int loaded = 0;
    for (TileWalk w(a.toff, a.G, blockIdx.x, gridDim.x); w.valid(); w.next()) {
        const int g = w.g, z = w.local;
        const int n = load_box(a.box + 6 * g).nx(), cp = pitch_of(n);
        float* C = reinterpret_cast<float*>(smem_raw);
        float* Q = C + n * cp;
        float* P = Q + n * cp;
        if (n != loaded) {
            const float* Cg = a.circ + a.circ_off[n];
            for (int q = threadIdx.x; q < n * n; q += kThreads) cp_async_elem(C + (q / n) * cp + q % n, Cg + q);
            loaded = n;
        }
        const float* src = a.in + a.in_off[g] + (long long)z * n * n;
        const int hr = plane_rows(n);
        for (int y0 = 0; y0 < n; y0 += hr) {
            const int ny = min(hr, n - y0);
            for (int q = threadIdx.x; q < ny * n; q += kThreads)
                cp_async_elem(P + (q / n) * cp + q % n, src + y0 * n + q);
            cp_async_wait_all();
            __syncthreads();
            // x: Q[y][x'] = sum_x P[y][x] C[x'][x]
            product_any<true>(P, C, cp, n, ny, [&](int y, int x, float v) { Q[(y0 + y) * cp + x] = v; });
            __syncthreads();
        }
        // y: out[y'][x] = sum_y C[y'][y] Q[y][x]
        float* dst = a.out + a.out_off[g] + (long long)z * n * n;
        product_any<false>(C, Q, cp, n, n, [&](int y, int x, float v) { dst[y * n + x] = v; });
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kThreads, 2) conv_z_kernel(ConvTCArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int loaded = 0;
    for (TileWalk w(a.toff, a.G, blockIdx.x, gridDim.x); w.valid(); w.next()) {
        const int g = w.g, y = w.local;
        const int n = load_box(a.box + 6 * g).nx(), cp = pitch_of(n);
        float* C = reinterpret_cast<float*>(smem_raw);
        float* S = C + n * cp;
        if (n != loaded) {
            const float* Cg = a.circ + a.circ_off[n];
            for (int q = threadIdx.x; q < n * n; q += kThreads) cp_async_elem(C + (q / n) * cp + q % n, Cg + q);
            loaded = n;
        }
        float* io = a.out + a.out_off[g] + (long long)y * n;
        for (int q = threadIdx.x; q < n * n; q += kThreads) {
            const int zz = q / n, x = q % n;
            cp_async_elem(S + zz * cp + x, io + (long long)zz * n * n + x);
        }
        cp_async_wait_all();
        __syncthreads();
        // z: out[z'][x] = sum_z C[z'][z] S[z][x]
        product_any<false>(C, S, cp, n, n, [&](int z, int x, float v) { io[(long long)z * n * n + x] = v; });
        __syncthreads();
    }
}

}  // namespace

void launch_conv_tc(const ConvTCArgs& a, int num_sms, int side_max, cudaStream_t s) {
    static PerDevice configured;
    configured.once([] {
        allow_max_dynamic_smem(conv_xy_kernel);
        allow_max_dynamic_smem(conv_z_kernel);
    });
    size_t xy = 0;  // a side whose plane is staged by halves may need less than a smaller one
    for (int n = 1; n <= side_max; n++)
        xy = std::max(xy, (size_t)(2 * n + plane_rows(n)) * pitch_of(n) * sizeof(float));
    conv_xy_kernel<<<num_sms * 8, kThreads, xy, s>>>(a);
    conv_z_kernel<<<num_sms * 8, kThreads, 2 * sizeof(float) * side_max * pitch_of(side_max), s>>>(a);
}

}  // namespace gg
