// gg_conv_tc.cuh -- mixed-precision (FP32-storage) Gaussian convolution.
//
// The reference's multiplier G (box.cpp:760-761) is exp(-c (i2^2 + j2^2 + k2^2)) / n^3,
// a product of one factor per axis, so IDFT3(DFT3(in) G) equals three applications
// of one real symmetric circulant matrix C_n = F^-1 diag(g) F / n along x, y and z.
// The mixed path runs those three contractions as dense per-axis GEMMs.
#pragma once

#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <new>
#include <thread>
#include <vector>

namespace gg {

// f(n) for every n in [lo, hi], the largest first, on up to 16 host threads.  The tables of one
// side do not depend on another's, so who computes them does not matter; where no thread can be
// started the caller does them all.  Throws when f has thrown.
template <typename F>
void for_sides(int lo, int hi, F&& f) {
    std::atomic<int> next{hi};
    std::atomic<bool> failed{false};
    auto work = [&] {
        try {
            for (int n = next.fetch_sub(1); n >= lo; n = next.fetch_sub(1)) f(n);
        } catch (...) {
            failed = true;
        }
    };
    std::vector<std::thread> threads;
    const int count = std::min({(int)std::thread::hardware_concurrency(), 16, hi - lo + 1});
    // below side 24 or so a thread costs more than all of the tables
    if (hi >= 24) try {
        for (int i = 1; i < count; i++) threads.emplace_back(work);
    } catch (...) {
    }
    work();
    for (auto& t : threads) t.join();
    if (failed) throw std::bad_alloc();  // the only thing the tables can fail by
}

struct ConvTCArgs {
    int G;
    const int* toff;          // one tile per convolved grain
    const float* in;
    const int* box;
    const long long* in_off;
    float* out;
    const long long* out_off;
    const float* circ;        // C_n row-major (n x n) for every side n at circ_off[n]
    const long long* circ_off;
    int* err;
};

// Write C_n (row-major, FP32, n x n) for box side n, domain size N and TimeStepSize.
void circulant_matrix(int n, int N, double time_step, float* out);
// C_n of the sides lo..hi (those with need[n], when need is given) one after the other in
// `out`, side n at off[n] (off sized hi + 2 or more by the caller).
void circulant_tables(int N, double time_step, int lo, int hi, const std::vector<char>* need, std::vector<float>& out,
                      std::vector<long long>& off);

// toff holds n tiles per grain (z-planes, then y-rows).
void launch_conv_tc(const ConvTCArgs& a, int num_sms, int side_max, cudaStream_t s);

// ---- tcgen05 tensor-core path (gg_conv_umma.cu) ----
constexpr int kUmmaMaxSide = 64;  // largest box side of the tensor-core kernel (TMEM, shared memory)
constexpr int kUmmaRows = 128;    // box rows per MMA tile

// One rotating pass: dst[c'][a][b] = sum_c C_n[c'][c] src[a][b][c] for every box.
struct UmmaPassArgs {
    int G;
    const int* toff;          // ceil(n^2 / 128) row tiles per grain
    const int* box;           // 6 ints per grain, cubic
    const float* src;
    const long long* src_off;
    float* dst;
    const long long* dst_off;
    const uint16_t* bmat;     // 2^8 C_n split into FP16 hi and lo, MMA operand layout, per side
    const long long* boff;
    int side_max;             // largest side in the launch (sizes the shared memory)
    int* err;
};

// The three passes: in -> out -> scratch -> out (scratch shares out's offsets).
struct UmmaConvArgs {
    int G;
    const int* toff;
    const int* box;
    const float* in;
    const long long* in_off;
    float* out;
    const long long* out_off;
    float* scratch;
    const uint16_t* bmat;
    const long long* boff;
    int* err;
};

int umma_side_limit();
// True when the tensor-core kernel takes boxes up to side_max (else the SIMT kernels).
bool umma_supported(int side_max);
// C_n of every side 1..nmax (those with need[n], when need is given) as the MMA's B operand (hi
// block, then lo block).
void umma_tables(int N, double time_step, int nmax, const std::vector<char>* need, std::vector<uint16_t>& bmat,
                 std::vector<long long>& boff);
void launch_conv_umma(const UmmaConvArgs& a, int num_sms, int side_max, cudaStream_t s);

}  // namespace gg
