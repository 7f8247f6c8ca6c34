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
// oracle.  The transform runs in five batched passes over all boxes' lines:
//   x forward (real to half spectrum) -> spectrum scratch; y forward, in place; z forward,
//   multiply by G, z inverse, in place; y inverse, in place; x inverse -> output arena.
// A warp takes 8 lines (16 rows in x) at a time: its lines, twiddles and products are its own,
// so nothing waits on a block barrier, and lines are numbered through a whole box, so that
// only a box's last fragment is part-full.
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
// domain (19% of the FP64 rate).  With x and y of a plane in one block (three passes, less
// traffic) the matrix pipe was 52-59% busy, waiting at barriers, and the passes took 4.0 ms;
// these take 3.5 ms, the pipe 70-73% busy in y and z and 51% in x.  The frequencies still pad
// (35 of 40 columns at n = 35).  A step that pads a chain adds (-0) x (+0) = -0, which leaves
// any accumulator as it is.
//
// B operands come from the side's n twiddles in shared memory, at an index each lane
// advances (one add and one conditional subtraction per fragment), not from a stored
// matrix: 2 n^2 doubles would take 65 KB at n = 64 and leave no room for the lines.
#include "gg_common.cuh"
#include "gg_conv.cuh"

#include <algorithm>

namespace gg {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kColChunk = 8;   // column fragments of a product held in registers at once (8 lines)
constexpr int kRowFrags = 2;   // fragments of 8 rows an x pass takes
constexpr int kRowChunk = 4;   // column fragments of x forward held in registers at once (16 rows)
constexpr int kLP = 12;        // pitch of 8 complex lines

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

__device__ __forceinline__ void load_twiddles(double2* tw_s, const double2* __restrict__ tw, int n, int lane) {
    for (int j = lane; j < n; j += 32) tw_s[j] = tw[j];
}

// One warp's walk over the fragments of `per` lines of all boxes: calls f(g, n, twiddles,
// buffer, first line, lines of the box).  A grain's n tiles share its fragments, two or three
// each; with few tiles for the warps, four warps share a tile's.
template <typename F>
__device__ __forceinline__ void warp_fragments(const ConvArgs& a, int warp_bytes, int per, bool rows, F&& f) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    double2* tw_s = reinterpret_cast<double2*>(smem_raw + (size_t)warp * warp_bytes);
    const int parts = gridDim.x * warps, part = blockIdx.x * warps + warp;
    const int share = a.toff[a.G + 1] < 2 * parts ? 4 : 1, mine = part % share;
    if (part / share >= parts / share) return;
    int n_tw = 0;
    for (TileWalk w(a.toff, a.G, part / share, parts / share); w.valid(); w.next()) {
        const int n = load_box(a.in_box + 6 * w.g).nx();
        const int lines = rows ? n * n : n * (n / 2 + 1), frags = (lines + per - 1) / per;
        if (n != n_tw) load_twiddles(tw_s, a.tw + a.tw_off[n], n, lane);
        n_tw = n;
        const long long t = (long long)w.local * share + mine, tiles = (long long)n * share;
        const int f1 = (int)((t + 1) * frags / tiles);
        for (int i = (int)(t * frags / tiles); i < f1; i++) f(w.g, n, tw_s, tw_s + n, i * per, lines);
    }
}

// x forward: kRowFrags x 8 consecutive rows (z, y), each a chain per frequency k < n/2 + 1:
// re = sum of x w.x, im = sum of x (-w.y).
__global__ void __launch_bounds__(kThreads, 2) conv_x_forward(ConvArgs a, int warp_bytes) {
    const Lane L;
    warp_fragments(a, warp_bytes, 8 * kRowFrags, true, [&](int g, int n, const double2* tw, double2* buf, int r0, int rows) {
        const int h = n / 2 + 1, P = pitch4(n), cf = (h + 7) / 8;
        double* X = reinterpret_cast<double*>(buf);  // [row][x]
        const double* src = a.in + a.in_off[g] + (long long)r0 * n;
        const int count = min(8 * kRowFrags, rows - r0) * n;
        for (int q = L.lane; q < count; q += 32) {
            const int r = q / n;
            cp_async_elem(X + r * P + (q - r * n), src + q);
        }
        cp_async_wait_all();
        __syncwarp();
        double2* dst = a.spec + a.spec_off[g] + (long long)r0 * h;
        for (int c0 = 0; c0 < cf; c0 += kRowChunk) {
            __syncwarp();
            dispatch<kRowChunk>(min(kRowChunk, cf - c0), [&](auto nt) {
                constexpr int NT = decltype(nt)::value;
                double re[kRowFrags][NT][2], im[kRowFrags][NT][2];
                int t[NT], inc[NT];
#pragma unroll
                for (int c = 0; c < NT; c++) {
                    const int k = ((c0 + c) * 8 + L.r) % n;
                    t[c] = (L.q * k) % n;
                    inc[c] = (4 * k) % n;
#pragma unroll
                    for (int j = 0; j < kRowFrags; j++) re[j][c][0] = re[j][c][1] = im[j][c][0] = im[j][c][1] = 0.0;
                }
                const double* s = X + L.r * P + L.q;
                auto step = [&](int keep) {
                    double x[kRowFrags];
#pragma unroll
                    for (int j = 0; j < kRowFrags; j++) x[j] = keep_or(s[8 * j * P], keep, 1);
#pragma unroll
                    for (int c = 0; c < NT; c++) {
                        const double2 w = tw[t[c]];
                        const double wx = keep_or(w.x, keep, 0), wy = keep_or(-w.y, keep, 0);
                        t[c] += inc[c];
                        if (t[c] >= n) t[c] -= n;
#pragma unroll
                        for (int j = 0; j < kRowFrags; j++) {
                            mma_f64(re[j][c], x[j], wx);
                            mma_f64(im[j][c], x[j], wy);
                        }
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
                for (int j = 0; j < kRowFrags; j++)
#pragma unroll
                    for (int c = 0; c < NT; c++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int r = 8 * j + L.r, k = (c0 + c) * 8 + 2 * L.q + e;
                            if (r0 + r < rows && k < h) dst[r * h + k] = make_double2(re[j][c][e], im[j][c][e]);
                        }
            });
        }
        __syncwarp();
    });
}

// Stages 8 lines (the one of lane l & 7 at src, elements `stride` apart) as [m][line].
__device__ __forceinline__ void stage_lines(double2* S, const double2* src, bool have, int n, int stride, int lane) {
    if (have)
        for (int m = lane >> 3; m < n; m += 4) cp_async16(S + m * kLP + (lane & 7), src + (long long)m * stride);
    cp_async_wait_all();
    __syncwarp();
}

// y, forward or inverse, in place: 8 consecutive lines (z, kx).
template <bool INV>
__global__ void __launch_bounds__(kThreads, 2) conv_y(ConvArgs a, int warp_bytes) {
    const Lane L;
    warp_fragments(a, warp_bytes, 8, false, [&](int g, int n, const double2* tw, double2* S, int l0, int lines) {
        const int h = n / 2 + 1, cf = (n + 7) / 8;
        double2* spec = a.spec + a.spec_off[g];
        auto line_at = [&](int l) {  // line (z, kx) starts at z n h + kx
            const int z = l / h;
            return spec + (z * n * h + (l - z * h));
        };
        stage_lines(S, line_at(min(l0 + (L.lane & 7), lines - 1)), l0 + (L.lane & 7) < lines, n, h, L.lane);
        double2* dst = line_at(min(l0 + L.r, lines - 1));
        for (int c0 = 0; c0 < cf; c0 += kColChunk) {
            __syncwarp();
            dispatch<kColChunk>(min(kColChunk, cf - c0), [&](auto nt) {
                constexpr int NT = decltype(nt)::value;
                double re[1][NT][2], im[1][NT][2];
                cdft<INV, 1, NT>(reinterpret_cast<const double*>(S), 2 * kLP, n, c0, reinterpret_cast<const double*>(tw), L,
                                 re, im);
                if (l0 + L.r < lines) {
#pragma unroll
                    for (int c = 0; c < NT; c++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int k = (c0 + c) * 8 + 2 * L.q + e;
                            if (k < n) dst[k * h] = make_double2(re[0][c][e], im[0][c][e]);
                        }
                }
            });
        }
        __syncwarp();
    });
}

// z forward, Gaussian multiply, z inverse, in place: 8 consecutive lines (ky, kx).
__global__ void __launch_bounds__(kThreads, 2) conv_z(ConvArgs a, int warp_bytes) {
    const Lane L;
    warp_fragments(a, warp_bytes, 8, false, [&](int g, int n, const double2* tw, double2* S, int l0, int lines) {
        const int h = n / 2 + 1, cf = (n + 7) / 8;
        const double* twd = reinterpret_cast<const double*>(tw);
        double2* T = cf > kColChunk ? S + n * kLP : S;  // one chunk: the products replace the lines in place
        double2* spec = a.spec + a.spec_off[g];
        const double* G = a.gtab + a.g_off[n];
        stage_lines(S, spec + min(l0 + (L.lane & 7), lines - 1), l0 + (L.lane & 7) < lines, n, lines, L.lane);
        // this lane's products belong to line l0 + r
        const int line = min(l0 + L.r, lines - 1), ky = line / h, kx = line - ky * h;
        const int i2 = min(ky, n - ky), j2 = min(kx, n - kx), ij = i2 * i2 + j2 * j2;
        for (int c0 = 0; c0 < cf; c0 += kColChunk) {
            __syncwarp();
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
        }
        __syncwarp();
        for (int c0 = 0; c0 < cf; c0 += kColChunk) {
            __syncwarp();
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
                            if (z < n) spec[(long long)z * lines + l0 + L.r] = make_double2(re[0][c][e], im[0][c][e]);
                        }
                }
            });
        }
        __syncwarp();
    });
}

// x inverse (half spectrum to real): the chain of output m starts at X(0).x and takes 2 X(k).x
// w.x, then -2 X(k).y w.y, for k = 1, 2, ...; at the Nyquist frequency (2k = n) X(k).x w.x alone.
__global__ void __launch_bounds__(kThreads, 2) conv_x_inverse(ConvArgs a, int warp_bytes) {
    const Lane L;
    warp_fragments(a, warp_bytes, 8 * kRowFrags, true, [&](int g, int n, const double2* tw, double2* X, int r0, int rows) {
        const int h = n / 2 + 1, P = pitch2(h), cf = (n + 7) / 8;
        const double* twd = reinterpret_cast<const double*>(tw);
        const double2* src = a.spec + a.spec_off[g] + (long long)r0 * h;  // X: [row][k]
        const int count = min(8 * kRowFrags, rows - r0) * h;
        for (int q = L.lane; q < count; q += 32) {
            const int r = q / h;
            cp_async16(X + r * P + (q - r * h), src + q);
        }
        cp_async_wait_all();
        __syncwarp();
        double* dst = a.out + a.out_off[g] + (long long)r0 * n;
        for (int c0 = 0; c0 < cf; c0 += kColChunk) {
            __syncwarp();
            dispatch<kColChunk>(min(kColChunk, cf - c0), [&](auto nt) {
                constexpr int NT = decltype(nt)::value;
                double acc[kRowFrags][NT][2];
                int t[NT], inc[NT];
#pragma unroll
                for (int c = 0; c < NT; c++) {
                    const int m = ((c0 + c) * 8 + L.r) % n;
                    t[c] = L.dm ? m : 0;
                    inc[c] = 2 * m >= n ? 2 * m - n : 2 * m;
#pragma unroll
                    for (int j = 0; j < kRowFrags; j++) acc[j][c][0] = acc[j][c][1] = 0.0;
                }
                const double* s = reinterpret_cast<const double*>(X + L.r * P) + L.q;
                const int pairs = (h + 1) >> 1;
#pragma unroll 2
                for (int i = 0; i < pairs; i++) {
                    const int k = 2 * i + L.dm;
                    const int in = k < h ? -1 : 0;
                    const bool edge = k == 0 || 2 * k == n;
                    const double f = edge ? 1.0 : (L.p ? -2.0 : 2.0);
                    const int keep = edge && L.p ? 0 : in;
                    const double* e = s + (in ? 0 : -2);  // past the end: element h - 1
                    double x[kRowFrags];
#pragma unroll
                    for (int j = 0; j < kRowFrags; j++) x[j] = keep_or(f * e[16 * j * P], keep, 1);
#pragma unroll
                    for (int c = 0; c < NT; c++) {
                        const double b = keep_or(twd[2 * t[c] + L.p], in, 0);
                        t[c] += inc[c];
                        if (t[c] >= n) t[c] -= n;
#pragma unroll
                        for (int j = 0; j < kRowFrags; j++) mma_f64(acc[j][c], x[j], b);
                    }
                    s += 4;
                }
#pragma unroll
                for (int j = 0; j < kRowFrags; j++)
#pragma unroll
                    for (int c = 0; c < NT; c++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int r = 8 * j + L.r, m = (c0 + c) * 8 + 2 * L.q + e;
                            if (r0 + r < rows && m < n) dst[r * n + m] = acc[j][c][e];
                        }
            });
        }
        __syncwarp();
    });
}

// Shared memory of a warp of each pass, in bytes, at side n: its twiddles and its lines (and
// z's products, above kColChunk fragments).
constexpr int kSlack = 16 * 8;
constexpr int kMaxSmem = 227 * 1024;
constexpr int x_forward_bytes(int n) { return 16 * n + 8 * 8 * kRowFrags * pitch4(n) + kSlack; }
constexpr int y_bytes(int n) { return 16 * n * (1 + kLP) + kSlack; }
constexpr int z_bytes(int n) { return 16 * n * (1 + kLP * ((n + 7) / 8 > kColChunk ? 2 : 1)) + kSlack; }
constexpr int x_inverse_bytes(int n) { return 16 * n + 16 * 8 * kRowFrags * pitch2(n / 2 + 1) + kSlack; }

static_assert(x_forward_bytes(kConvF64MaxSide) <= kMaxSmem && y_bytes(kConvF64MaxSide) <= kMaxSmem &&
                  z_bytes(kConvF64MaxSide) <= kMaxSmem && x_inverse_bytes(kConvF64MaxSide) <= kMaxSmem,
              "a warp's buffers fit a CTA at the largest side");

// CTAs of as many warps as fit (8 at most), whole waves of the CTAs that fit the device at once:
// one wave for a few boxes, where every wave pays its start (0.100 -> 0.082 ms for 20 grains of
// 32^3 against four), up to eight, which even out the boxes' sides, for many (3.95 -> 3.52 ms
// for 2,000 of 128^3 against one).
template <typename K>
void launch_pass(K kernel, const ConvArgs& a, int warp_bytes, int nmax, cudaStream_t s) {
    const int warps = std::min(kMaxSmem / warp_bytes, kWarps);
    const size_t smem = (size_t)warps * warp_bytes;
    int dev = 0, sms = 148, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * warps, smem);
    const int wave = sms * (per_sm > 0 ? per_sm : 1);
    const long long tiles = (long long)a.G * nmax;  // at most
    const int waves = (int)std::min(8LL, std::max(1LL, tiles / (4LL * wave * warps)));
    kernel<<<wave * waves, 32 * warps, smem, s>>>(a, warp_bytes);
}

}  // namespace

void launch_conv_f64(const ConvArgs& a, int nmax, cudaStream_t s) {
    static PerDevice configured;
    configured.once([] {
        allow_max_dynamic_smem(conv_x_forward);
        allow_max_dynamic_smem(conv_y<false>);
        allow_max_dynamic_smem(conv_z);
        allow_max_dynamic_smem(conv_y<true>);
        allow_max_dynamic_smem(conv_x_inverse);
    });
    launch_pass(conv_x_forward, a, x_forward_bytes(nmax), nmax, s);
    launch_pass(conv_y<false>, a, y_bytes(nmax), nmax, s);
    launch_pass(conv_z, a, z_bytes(nmax), nmax, s);
    launch_pass(conv_y<true>, a, y_bytes(nmax), nmax, s);
    launch_pass(conv_x_inverse, a, x_inverse_bytes(nmax), nmax, s);
}

}  // namespace gg
