// gg_conv_f64.cu -- FP64 Gaussian convolution of every grain box (the plain path).
//
// Stands in for LSbox::executeConvolution / convolutionGeneratorMKL
// (box.cpp:414-427, 685-795): out = IDFT3(DFT3(in) * G) with
// G = exp(-sqrt(2/pi) * S * 4 dt N^2 / n^2 * pi^2) / n^3, S = i2^2 + j2^2 + k2^2.
//
// The reference's MKL transform is replaced by a DFT whose arithmetic is fixed to
// the order of every fused multiply-add (see the oracle's gg_dft.h): each output
// is one fma chain over m = 0..n-1 with twiddle index (k*m) mod n taken from a
// host-built libm table, and G comes from a host-built table per box side.  These
// kernels run exactly those chains, so the FP64 path is bit-identical to the
// oracle.  The transform is split in three batched passes over all boxes:
//   A  per (grain, z-plane): x r2c, then y                    -> spectrum scratch
//   B  per 8 (ky, kx) lines: z forward, multiply by G, z inverse (in place)
//   C  per (grain, z-plane): y inverse, then x c2r            -> output arena
//
// A chain is a row of a product with the twiddle matrix: a complex output's real part is
// sum over m of z.x w.x, then z.y w.y, a dot product of length 2n, and its imaginary part
// the same columns against (z.y, -z.x).  The m8n8k4 FP64 matrix instruction adds its four
// products to the accumulator one fma after the other in k order (a test pins it bit for
// bit against the fma chain), so a chain of length 2n is 2n/4 instructions, each doing 8
// lines x 8 frequencies.  B200's FP64 rate is the same with and without it (37 TFLOP/s
// measured for both); what it removes is everything around the arithmetic.  The scalar
// form of these passes read a 16-byte twiddle and updated an index for every four fma and
// left the lanes past a box's last line idle: 11.5 ms for the 2,000 boxes of a 128^3
// domain (19% of the FP64 rate); this form takes 4.04 ms, its passes 59%, 73% and 52% of the matrix
// pipe's cycles, the rest going to barriers, operand loads and the tails of fragments (at
// n = 35 the frequencies fill 35 of 40 columns).  A step that pads a chain adds
// (-0) x (+0) = -0, which leaves any accumulator as it is.
//
// B operands come from the side's n twiddles in shared memory, at an index each lane
// advances (one add and one conditional subtraction per fragment), not from a stored
// matrix: 2 n^2 doubles would take 65 KB at n = 64 and leave no room for the planes.
#include "gg_common.cuh"
#include "gg_conv.cuh"

#include <algorithm>

namespace gg {

namespace {

constexpr int kThreads = 192;      // passes A and C: a warp per column fragment of sides up to 48
constexpr int kWarps = kThreads / 32;
constexpr int kThreadsB = 256;     // pass B (its warps are independent)
constexpr int kLineChunk = 6;      // line fragments of a complex product held in registers at once
constexpr int kRealChunk = 10;     // of a real one
constexpr int kPlanes = 4;         // most planes a tile of passes A and C takes together
constexpr int kTileBytes = 64 * 1024;  // shared memory of a tile of several planes: three CTAs an SM
constexpr int kColChunk = 8;   // column fragments of a pass B product held in registers at once
constexpr int kLP = 12;        // pitch of pass B's 8 lines

// Pitches in elements.  The 16 lanes of a half warp read 4 lines x (2 rows of m) x (x, y)
// of a complex [m][line] buffer, or 4 lines x 4 m of a [line][m] one: 128 bytes on
// distinct banks when the pitch is 4 modulo 8, or 2 modulo 4 for complex [line][m].
__host__ __device__ constexpr int pitch4(int v) { return (v + 3) / 8 * 8 + 4; }
__host__ __device__ constexpr int pitch2(int v) { return (v + 1) / 4 * 4 + 2; }

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// v, or -0 / +0 in a lane that pads its chain (keep = 0): bit operations rather than a
// branch, so that the 32 lanes reach every matrix instruction together.
__device__ __forceinline__ double keep_or(double v, int keep, int sign) {  // keep = 0 or -1, sign = 0 or 1
    return __hiloint2double((__double2hiint(v) & keep) | (~keep & (sign << 31)), __double2loint(v) & keep);
}

__device__ __forceinline__ double neg_if(double v, int s) {  // s = 0 or 1
    return __hiloint2double(__double2hiint(v) ^ (s << 31), __double2loint(v));
}

// A lane's place in the operands of one instruction: row r of A (a line), or column r of B
// (a frequency), at k = q, that is part p (real, imaginary) of element dm of a pair.
struct Lane {
    int lane, r, q, p, dm;
    __device__ Lane() : lane(threadIdx.x & 31), r(lane >> 2), q(lane & 3), p(q & 1), dm(q >> 1) {}
};

// Complex DFT of MT fragments of 8 lines (the first line at src, element (m, l) at
// src[m * sm + 2 l]) at NT fragments of 8 frequencies from kf: acc[j][c] = lines j,
// frequencies c, columns 2 (lane & 3) + {0, 1}.
template <bool INV, int MT, int NT>
__device__ __forceinline__ void cdft(const double* __restrict__ src, int sm, int n, int kf,
                                     const double* __restrict__ tw, const Lane& L, double (&re)[MT][NT][2],
                                     double (&im)[MT][NT][2]) {
    int t[NT], inc[NT];
#pragma unroll
    for (int c = 0; c < NT; c++) {
        const int k = ((kf + c) * 8 + L.r) % n;
        t[c] = L.dm ? k : 0;
        inc[c] = 2 * k >= n ? 2 * k - n : 2 * k;
#pragma unroll
        for (int j = 0; j < MT; j++) re[j][c][0] = re[j][c][1] = im[j][c][0] = im[j][c][1] = 0.0;
    }
    const double* s = src + L.dm * sm + 2 * L.r;
    const int own = L.p, oth = L.p ^ 1;
    // keep = -1, or 0 in the lanes whose element lies past the chain's end (n odd); those read
    // element n - 1 instead
    auto step = [&](int keep) {
        double b[NT];
#pragma unroll
        for (int c = 0; c < NT; c++) {
            b[c] = keep_or(tw[2 * t[c] + L.p], keep, 0);
            t[c] += inc[c];
            if (t[c] >= n) t[c] -= n;
        }
#pragma unroll
        for (int j = 0; j < MT; j++) {
            // forward: re (x, y), im (y, -x); inverse: re (x, -y), im (y, x)
            const double x = keep_or(neg_if(s[16 * j + own], INV ? L.p : 0), keep, 1);
            const double y = keep_or(neg_if(s[16 * j + oth], INV ? 0 : L.p), keep, 1);
#pragma unroll
            for (int c = 0; c < NT; c++) {
                mma_f64(re[j][c], x, b[c]);
                mma_f64(im[j][c], y, b[c]);
            }
        }
    };
    const int pairs = n >> 1;
#pragma unroll 2
    for (int i = 0; i < pairs; i++) {
        step(-1);
        s += 2 * sm;
    }
    if (n & 1) {
        s -= L.dm * sm;
        step(L.dm - 1);
    }
}

// Calls f(integral constant) for the value v in 1..MAX.
template <int V>
struct Int {
    static constexpr int value = V;
};
template <int MAX, typename F>
__device__ __forceinline__ void dispatch(int v, F&& f) {
    if constexpr (MAX > 1) {
        if (v < MAX) {
            dispatch<MAX - 1>(v, f);
            return;
        }
    }
    f(Int<MAX>{});
}

// Complex DFT along the nl lines of a [m][line] plane in shared memory, one item per (8
// frequencies, chunk of lines); rot carries the round robin over the warps from one step
// to the next so that every scheduler gets the same share.  store(l, k, re, im).
template <bool INV, typename F>
__device__ __forceinline__ void cdft_plane(const double2* src, int sm, int n, int nl, const double2* tw, int& rot,
                                           F&& store) {
    const Lane L;
    const int lf = (nl + 7) / 8, cf = (n + 7) / 8;
    const int chunks = (lf + kLineChunk - 1) / kLineChunk, per = (lf + chunks - 1) / chunks;
    const int items = cf * chunks;
    for (int it = ((threadIdx.x >> 5) + kWarps - rot) % kWarps; it < items; it += kWarps) {
        const int kf = it / chunks, l0 = (it - kf * chunks) * per;
        __syncwarp();
        dispatch<kLineChunk>(min(per, lf - l0), [&](auto mt) {
            constexpr int MT = decltype(mt)::value;
            double re[MT][1][2], im[MT][1][2];
            cdft<INV, MT, 1>(reinterpret_cast<const double*>(src + l0 * 8), 2 * sm, n, kf,
                             reinterpret_cast<const double*>(tw), L, re, im);
#pragma unroll
            for (int j = 0; j < MT; j++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int l = (l0 + j) * 8 + L.r, k = kf * 8 + 2 * L.q + e;
                    if (l < nl && k < n) store(l, k, re[j][0][e], im[j][0][e]);
                }
        });
    }
    rot = (rot + items) % kWarps;
}

// Real-input DFT (x axis, r2c) along the nl lines of a [line][m] plane: frequencies k < nk.
template <typename F>
__device__ __forceinline__ void r2c_plane(const double* src, int sl, int n, int nl, int nk, const double2* tw, int& rot,
                                          F&& store) {
    const Lane L;
    const int lf = (nl + 7) / 8, cf = (nk + 7) / 8;
    const int chunks = lf > kLineChunk ? (lf + kLineChunk - 1) / kLineChunk : (lf > 1 ? 2 : 1);
    const int per = (lf + chunks - 1) / chunks;
    const int items = cf * chunks;
    for (int it = ((threadIdx.x >> 5) + kWarps - rot) % kWarps; it < items; it += kWarps) {
        const int kf = it / chunks, l0 = (it - kf * chunks) * per;
        if (l0 >= lf) continue;
        __syncwarp();
        dispatch<kLineChunk>(min(per, lf - l0), [&](auto mt) {
            constexpr int MT = decltype(mt)::value;
            double re[MT][2], im[MT][2];
#pragma unroll
            for (int j = 0; j < MT; j++) re[j][0] = re[j][1] = im[j][0] = im[j][1] = 0.0;
            const int k = (kf * 8 + L.r) % n;
            int t = (L.q * k) % n;
            const int inc = (4 * k) % n;
            const double* s = src + (l0 * 8 + L.r) * sl + L.q;
            auto step = [&](int keep) {
                const double2 w = tw[t];
                const double c = keep_or(w.x, keep, 0), d = keep_or(-w.y, keep, 0);
                t += inc;
                if (t >= n) t -= n;
#pragma unroll
                for (int j = 0; j < MT; j++) {
                    const double x = keep_or(s[8 * j * sl], keep, 1);
                    mma_f64(re[j], x, c);
                    mma_f64(im[j], x, d);
                }
            };
            const int quads = n >> 2, rest = n & 3;
#pragma unroll 2
            for (int i = 0; i < quads; i++) {
                step(-1);
                s += 4;
            }
            if (rest) {
                s -= max(L.q - (rest - 1), 0);  // lanes past the end read element n - 1
                step(L.q < rest ? -1 : 0);
            }
#pragma unroll
            for (int j = 0; j < MT; j++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int l = (l0 + j) * 8 + L.r, ko = kf * 8 + 2 * L.q + e;
                    if (l < nl && ko < nk) store(l, ko, re[j][e], im[j][e]);
                }
        });
    }
    rot = (rot + items) % kWarps;
}

// Half-spectrum to real (x axis, c2r) of a complex [line][k] plane, k < n/2+1: the chain of
// output m starts at X(0).x and takes 2 X(k).x w.x, then -2 X(k).y w.y, for k = 1, 2, ...; at
// the Nyquist frequency (2k = n) X(k).x w.x alone.
template <typename F>
__device__ __forceinline__ void c2r_plane(const double2* src, int sl, int n, int nl, const double2* tw, int& rot,
                                          F&& store) {
    const Lane L;
    const int h = n / 2 + 1;
    const int lf = (nl + 7) / 8, cf = (n + 7) / 8;
    const int chunks = (lf + kRealChunk - 1) / kRealChunk, per = (lf + chunks - 1) / chunks;
    const int items = cf * chunks;
    for (int it = ((threadIdx.x >> 5) + kWarps - rot) % kWarps; it < items; it += kWarps) {
        const int mf = it / chunks, l0 = (it - mf * chunks) * per;
        __syncwarp();
        dispatch<kRealChunk>(min(per, lf - l0), [&](auto mt) {
            constexpr int MT = decltype(mt)::value;
            double acc[MT][2];
#pragma unroll
            for (int j = 0; j < MT; j++) acc[j][0] = acc[j][1] = 0.0;
            const int m = (mf * 8 + L.r) % n;
            int t = L.dm ? m : 0;
            const int inc = 2 * m >= n ? 2 * m - n : 2 * m;
            const double* twd = reinterpret_cast<const double*>(tw);
            const double* s = reinterpret_cast<const double*>(src + (l0 * 8 + L.r) * sl) + L.q;
            const int pairs = (h + 1) >> 1;
            for (int i = 0; i < pairs; i++) {
                const int k = 2 * i + L.dm;
                const int in = k < h ? -1 : 0;
                const bool edge = k == 0 || 2 * k == n;
                const double f = edge ? 1.0 : (L.p ? -2.0 : 2.0);
                const int keep = edge && L.p ? 0 : in;
                const double b = keep_or(twd[2 * t + L.p], in, 0);
                t += inc;
                if (t >= n) t -= n;
                const double* e = s + (in ? 0 : -2);  // past the end: element h - 1
#pragma unroll
                for (int j = 0; j < MT; j++) mma_f64(acc[j], keep_or(f * e[16 * j * sl], keep, 1), b);
                s += 4;
            }
#pragma unroll
            for (int j = 0; j < MT; j++) {
                const int l = (l0 + j) * 8 + L.r, mo = mf * 8 + 2 * L.q;
                if (l < nl && mo < n) store(l, mo, acc[j][0]);
                if (l < nl && mo + 1 < n) store(l, mo + 1, acc[j][1]);
            }
        });
    }
    rot = (rot + items) % kWarps;
}

// Which plane of a tile a flat line belongs to, n lines a plane.
__device__ __forceinline__ int plane_of(int l, int n) {
    int u = 0;
#pragma unroll
    for (int i = 1; i < kPlanes; i++) u += l >= i * n;
    return u;
}

__device__ __forceinline__ void load_twiddles(double2* tw_s, const double2* __restrict__ tw, int n, int id, int step) {
    for (int j = id; j < n; j += step) tw_s[j] = tw[j];
}

// Elements of u planes' buffers (the last fragment of lines may read up to 7 lines past the
// end): [line][m] real, [m][line] complex, [line][k] complex.
__host__ __device__ constexpr int real_planes(int n, int u) { return (u * n + 7) / 8 * 8 * pitch4(n) + 8; }
__host__ __device__ constexpr int spec_planes_ml(int n, int u) { return n * pitch4(u * (n / 2 + 1)) + 8; }
__host__ __device__ constexpr int spec_planes_lm(int n, int u) { return (u * n + 7) / 8 * 8 * pitch2(n / 2 + 1) + 4; }
__host__ __device__ constexpr int pass_a_bytes(int n, int u) {
    return 16 * (n + spec_planes_ml(n, u)) + 8 * real_planes(n, u);
}
__host__ __device__ constexpr int pass_c_bytes(int n, int u) {
    const int pk = 16 * spec_planes_ml(n, u), xo = 8 * u * n * pitch4(n);
    return 16 * (n + spec_planes_lm(n, u)) + (pk > xo ? pk : xo);
}
// Planes a tile takes together: as many as keep three CTAs on an SM.  The h = n/2 + 1 lines of
// one plane fill their fragments badly (18 of 24 at n = 35); those of two or more planes run
// on (36 of 40), and each block barrier covers more work.
__host__ __device__ constexpr int tile_planes(int n) {
    int u = 1;
    while (u < kPlanes && pass_a_bytes(n, u + 1) <= kTileBytes && pass_c_bytes(n, u + 1) <= kTileBytes) u++;
    return u;
}

// Pass A: x r2c then y forward, up to tile_planes(n) consecutive z-planes of a grain at a time.
__global__ void __launch_bounds__(kThreads, 3) conv_pass_a(ConvArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int rot = 0;
    for (TileWalk w(a.toff, a.G, blockIdx.x, gridDim.x); w.valid();) {
        const int g = w.g, z = w.local;
        const Box b = load_box(a.in_box + 6 * g);
        const int n = b.nx(), h = n / 2 + 1;
        const int U = min(min(tile_planes(n), w.count - z), w.end - w.t);
        const int P = pitch4(n), Hp = pitch4(U * h);
        double2* tw_s = reinterpret_cast<double2*>(smem_raw);
        double2* A = tw_s + n;  // [y][plane, kx]
        double* xp = reinterpret_cast<double*>(A + spec_planes_ml(n, U));  // [plane, y][x]
        load_twiddles(tw_s, a.tw + a.tw_off[n], n, threadIdx.x, kThreads);
        const double* src = a.in + a.in_off[g] + (long long)z * n * n;
        for (int q = threadIdx.x; q < U * n * n; q += kThreads) {
            const int y = q / n, x = q - y * n;
            cp_async_elem(xp + y * P + x, src + q);
        }
        cp_async_wait_all();
        __syncthreads();
        r2c_plane(xp, P, n, U * n, h, tw_s, rot, [&](int l, int k, double re, double im) {
            const int u = plane_of(l, n);
            A[(l - u * n) * Hp + u * h + k] = make_double2(re, im);
        });
        __syncthreads();
        double2* dst = a.spec + a.spec_off[g] + (long long)z * n * h;
        cdft_plane<false>(A, Hp, n, U * h, tw_s, rot, [&](int l, int ky, double re, double im) {
            const int u = plane_of(l, h);
            dst[(u * n + ky) * h + (l - u * h)] = make_double2(re, im);
        });
        __syncthreads();
        for (int u = 0; u < U; u++) w.next();
    }
}

// Pass B: z forward, Gaussian multiply, z inverse, 8 consecutive (ky, kx) lines per warp at a
// time: a warp's lines, twiddles and products are its own, so nothing waits on a block
// barrier.  A grain's n tiles share its n h lines in fragments of 8 without padding.
__global__ void __launch_bounds__(kThreadsB, 2) conv_pass_b(ConvArgs a, int warp_bytes) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Lane L;
    const int warp = threadIdx.x >> 5;
    double2* tw_s = reinterpret_cast<double2*>(smem_raw + (size_t)warp * warp_bytes);
    const double* twd = reinterpret_cast<const double*>(tw_s);
    int n_tw = 0;
    const int warps = blockDim.x >> 5;
    for (TileWalk w(a.toff, a.G, blockIdx.x * warps + warp, gridDim.x * warps); w.valid(); w.next()) {
        const int g = w.g;
        const Box b = load_box(a.in_box + 6 * g);
        const int n = b.nx(), h = n / 2 + 1;
        const int lines = n * h, frags = (lines + 7) / 8, cf = (n + 7) / 8;
        if (n != n_tw) load_twiddles(tw_s, a.tw + a.tw_off[n], n, L.lane, 32);
        n_tw = n;
        double2* S = tw_s + n;
        double2* T = cf > kColChunk ? S + n * kLP : S;  // one chunk: the products replace the lines in place
        double2* spec = a.spec + a.spec_off[g];
        const double* G = a.gtab + a.g_off[n];
        const int f1 = (int)((long long)(w.local + 1) * frags / n);
        for (int f = (int)((long long)w.local * frags / n); f < f1; f++) {
            const int l0 = f * 8;
            {
                const int l = L.lane & 7;
                if (l0 + l < lines)
                    for (int z = L.lane >> 3; z < n; z += 4)
                        cp_async16(S + z * kLP + l, spec + (long long)z * lines + l0 + l);
            }
            cp_async_wait_all();
            __syncwarp();
            // this lane's products belong to line l0 + r
            const int line = min(l0 + L.r, lines - 1), ky = line / h, kx = line - ky * h;
            const int i2 = min(ky, n - ky), j2 = min(kx, n - kx), ij = i2 * i2 + j2 * j2;
            for (int c0 = 0; c0 < cf; c0 += kColChunk)
                dispatch<kColChunk>(min(kColChunk, cf - c0), [&](auto nt) {
                    constexpr int NT = decltype(nt)::value;
                    double re[1][NT][2], im[1][NT][2];
                    cdft<false, 1, NT>(reinterpret_cast<const double*>(S), 2 * kLP, n, c0, twd, L, re, im);
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < NT; c++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int kz = (c0 + c) * 8 + 2 * L.q + e;
                            if (kz < n) {
                                const int k2 = min(kz, n - kz);
                                const double gv = __ldg(G + (ij + k2 * k2));
                                T[kz * kLP + L.r] = make_double2(re[0][c][e] * gv, im[0][c][e] * gv);
                            }
                        }
                });
            __syncwarp();
            for (int c0 = 0; c0 < cf; c0 += kColChunk)
                dispatch<kColChunk>(min(kColChunk, cf - c0), [&](auto nt) {
                    constexpr int NT = decltype(nt)::value;
                    double re[1][NT][2], im[1][NT][2];
                    cdft<true, 1, NT>(reinterpret_cast<const double*>(T), 2 * kLP, n, c0, twd, L, re, im);
                    if (l0 + L.r < lines) {
#pragma unroll
                        for (int c = 0; c < NT; c++)
#pragma unroll
                            for (int e = 0; e < 2; e++) {
                                const int z = (c0 + c) * 8 + 2 * L.q + e;
                                if (z < n)
                                    spec[(long long)z * lines + l0 + L.r] = make_double2(re[0][c][e], im[0][c][e]);
                            }
                    }
                });
            __syncwarp();
        }
    }
}

// Pass C: y inverse then x c2r, the planes of a tile as in pass A, written to the output arena.
__global__ void __launch_bounds__(kThreads, 3) conv_pass_c(ConvArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int rot = 0;
    for (TileWalk w(a.toff, a.G, blockIdx.x, gridDim.x); w.valid();) {
        const int g = w.g, z = w.local;
        const Box b = load_box(a.in_box + 6 * g);
        const int n = b.nx(), h = n / 2 + 1;
        const int U = min(min(tile_planes(n), w.count - z), w.end - w.t);
        const int P = pitch4(n), Hp = pitch4(U * h), Hl = pitch2(h);
        double2* tw_s = reinterpret_cast<double2*>(smem_raw);
        double2* Ay = tw_s + n;                      // [plane, y][kx], pitch Hl
        double2* Pk = Ay + spec_planes_lm(n, U);     // [ky][plane, kx], pitch Hp
        double* xo = reinterpret_cast<double*>(Pk);  // [plane, y][x], pitch P, once the spectrum is read
        load_twiddles(tw_s, a.tw + a.tw_off[n], n, threadIdx.x, kThreads);
        const double2* spec = a.spec + a.spec_off[g] + (long long)z * n * h;
        for (int q = threadIdx.x; q < U * n * h; q += kThreads) {
            const int row = q / h, kx = q - row * h, u = plane_of(row, n);
            cp_async16(Pk + (row - u * n) * Hp + u * h + kx, spec + q);
        }
        cp_async_wait_all();
        __syncthreads();
        cdft_plane<true>(Pk, Hp, n, U * h, tw_s, rot, [&](int l, int y, double re, double im) {
            const int u = plane_of(l, h);
            Ay[(u * n + y) * Hl + (l - u * h)] = make_double2(re, im);
        });
        __syncthreads();
        c2r_plane(Ay, Hl, n, U * n, tw_s, rot, [&](int l, int x, double v) { xo[l * P + x] = v; });
        __syncthreads();
        double* dst = a.out + a.out_off[g] + (long long)z * n * n;
        for (int q = threadIdx.x; q < U * n * n; q += kThreads) {
            const int y = q / n, x = q - y * n;
            dst[q] = xo[y * P + x];
        }
        __syncthreads();
        for (int u = 0; u < U; u++) w.next();
    }
}

constexpr size_t kMaxSmem = 227 * 1024;
size_t pass_b_warp_bytes(int n) {
    return 16 * (size_t)n * (1 + kLP * ((n + 7) / 8 > kColChunk ? 2 : 1)) + 16 * 8;
}

// CTAs of kernel k: a whole number of waves of those that fit the device at once, near
// `grid` (a wave that is two thirds empty at the end cost 11% of a pass).
template <typename K>
int whole_waves(K kernel, int threads, size_t smem, int grid) {
    int dev = 0, sms = 148, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    const int wave = sms * (per_sm > 0 ? per_sm : 1);
    return wave * (grid > wave ? (grid + wave / 2) / wave : 1);
}

}  // namespace

void launch_conv_f64(const ConvArgs& a, int grid, int nmax, cudaStream_t s) {
    static PerDevice configured;
    configured.once([] {
        allow_max_dynamic_smem(conv_pass_a);
        allow_max_dynamic_smem(conv_pass_b);
        allow_max_dynamic_smem(conv_pass_c);
    });
    // a tile of several planes of a smaller side may need more than one plane of the largest
    size_t sa = 0, sc = 0;
    for (int n = 1; n <= nmax; n++) {
        sa = std::max(sa, (size_t)pass_a_bytes(n, tile_planes(n)));
        sc = std::max(sc, (size_t)pass_c_bytes(n, tile_planes(n)));
    }
    const int warp_bytes = (int)pass_b_warp_bytes(nmax);
    // sides above 64 keep two line buffers a warp, and as many warps as then fit
    const int warps = std::min((int)(kMaxSmem / warp_bytes), kThreadsB / 32);
    const size_t sb = (size_t)warps * warp_bytes;
    conv_pass_a<<<whole_waves(conv_pass_a, kThreads, sa, grid), kThreads, sa, s>>>(a);
    conv_pass_b<<<whole_waves(conv_pass_b, 32 * warps, sb, grid), 32 * warps, sb, s>>>(a, warp_bytes);
    conv_pass_c<<<whole_waves(conv_pass_c, kThreads, sc, grid), kThreads, sc, s>>>(a);
}

}  // namespace gg
