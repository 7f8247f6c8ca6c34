// gg_compare.cu -- comparison, boundary condition and set-comparison of every grain.
//
// Stands in for LSbox::executeComparison (box.cpp:891-966), boundaryCondition
// (box.cpp:997-1088) and executeSetComparison (box.cpp:814-878).
//
// The reference, per grain A and voxel v of A's box, walks A's comparison list in
// order and keeps the first neighbour whose value at v is strictly greater than
// everything before it (starting from -1).  That is: the largest value among the
// listed neighbours whose box contains v, ties going to the earliest list
// position.  Each box voxel is read about thirty times that way.  Here the work is
// turned around and done per domain tile instead of per grain:
//
//   1. bin: every tile of kTX x kTY x kTZ domain voxels gets the IDs of the
//      grains whose boxes reach it (count, scan, fill);
//   2. compare: one CTA per tile loads every covering box's values over the tile
//      into shared memory once and looks up, in each covering grain's position
//      table (built once per step from its comparison list), the position of every
//      voxel's two largest in its list.  Per voxel it keeps the kTop
//      largest values; every (grain, voxel) pair then picks the first candidate
//      that is in that grain's list, resolving equal values by list position --
//      falling back to a full scan of the tile's boxes whenever the kTop
//      candidates cannot decide.  The boundary condition, the set comparison, the
//      outputs and the new bounding box follow in the same pass.
//   3. copy_lists: m_secondOrderNeighbours = m_comparisonList for the next step.
//
// Every value is read once and written once (12 B per voxel on the FP32 path),
// and the result is bit-identical to the sequential walk.  Voxels no listed
// neighbour covers keep their IDLocal from the previous layout by the reference's
// flat-prefix resize (dimensionalBuffer.h:120-131).
#include "gg_kernels.cuh"

#include <math_constants.h>

#include <climits>

namespace gg {

namespace {

constexpr int kThreads = 256;
constexpr int kTV = kTX * kTY * kTZ;   // voxels per tile (64)
constexpr int kTop = 3;                // candidates kept per voxel
constexpr int kParts = kThreads / kTV; // threads scanning the boxes of one voxel
// row stride of the staged values: the kParts lanes of a voxel read kVS apart, which
// puts the 32 lanes of a warp on 32 different banks
constexpr int kVS = kTV + 8;
static_assert(kTV % 32 == 0 && kThreads % kTV == 0, "a warp's lanes share one tile entry per pair sweep");
static_assert(kThreads == kTV * kParts && (kParts & (kParts - 1)) == 0, "merge layout");
static_assert(kTX == 8 && kTY == 4 && kTZ == 2, "an entry's coverage of a tile is two 32-bit masks, a byte per row");
constexpr unsigned kNone = 0xFFFFFFFFu;
constexpr unsigned short kNotListed = 0xFFFF;
constexpr int kUCap = 32;              // candidate columns of the position matrix

// One branch of the reference's boundary distance (box.cpp:1017-1082).  Returns
// false where no branch assigns `dist`, in which case the reference keeps the value
// of the previous voxel in its loop order.
__device__ bool bc_assign(int i, int j, int k, int m, int gb, double& dist) {
    const double distXMax = (j - (m - 1 - gb));
    const double distYMax = (i - (m - 1 - gb));
    const double distZMax = (k - (m - 1 - gb));
    const double distXMin = -(j - gb + 1);
    const double distYMin = -(i - gb + 1);
    const double distZMin = -(k - gb + 1);
    const double distX = fabs(distXMin) < fabs(distXMax) ? distXMin : distXMax;
    const double distY = fabs(distYMin) < fabs(distYMax) ? distYMin : distYMax;
    const double distZ = fabs(distZMin) < fabs(distZMax) ? distZMin : distZMax;
    if (distX > 0 && distY > 0 && distZ > 0) {
        dist = sqrt((double)distX * distX + distY * distY + distZ * distZ);
        return true;
    }
    if (distX < 0 && distY < 0 && distZ < 0) {
        double d = distX < distY ? distY : distX;
        dist = d < distZ ? distZ : d;
        return true;
    }
    if (distX >= 0) {
        if (distY < 0 && distZ < 0) { dist = distX; return true; }
        if (distY < 0 && distZ >= 0) { dist = sqrt((double)distX * distX + distZ * distZ); return true; }
        if (distY >= 0 && distZ < 0) { dist = sqrt((double)distX * distX + distY * distY); return true; }
        return false;
    }
    if (distY >= 0) {
        if (distZ < 0 && distX < 0) { dist = distY; return true; }
        if (distX < 0 && distZ >= 0) { dist = sqrt((double)distY * distY + distZ * distZ); return true; }
        return false;
    }
    if (distZ >= 0) {
        if (distY < 0 && distX < 0) { dist = distZ; return true; }
        return false;
    }
    return false;
}

// The value `dist` holds at voxel (i, j, k) of the boundary loop over box b.
__device__ double bc_dist(const Box& b, int i, int j, int k, int m, int gb) {
    double d;
    if (bc_assign(i, j, k, m, gb, d)) return d;
    int ii = i, jj = j, kk = k;
    for (;;) {
        if (--jj < b.x0) {
            jj = b.x1 - 1;
            if (--ii < b.y0) {
                ii = b.y1 - 1;
                if (--kk < b.z0) return 0.0;  // initial value, box.cpp:1001
            }
        }
        if (bc_assign(ii, jj, kk, m, gb, d)) return d;
    }
}

// ---------------------------------------------------------------------------------
// 1. m_secondOrderNeighbours = m_comparisonList (box.cpp:895), for the next list update
// ---------------------------------------------------------------------------------
__global__ void copy_lists_kernel(ListCopyArgs a) {
    const int total = a.toff[a.G + 1];
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        const int g = tile_grain(a.toff, a.G, t);
        const int K = a.n_cmp[g];
        const uint32_t* list = a.cmp + (long long)g * a.list_cap;
        uint32_t* son = a.son + (long long)g * a.list_cap;
        for (int i = threadIdx.x; i < K; i += blockDim.x) son[i] = list[i];
        if (threadIdx.x == 0) a.n_son[g] = K;
    }
}

// ---------------------------------------------------------------------------------
// 2. binning of grain boxes to domain tiles: `parts` warps per grain, lanes over its tiles
// ---------------------------------------------------------------------------------
template <bool FILL>
__global__ void bin_kernel(TileBins tb, int G, int parts, const int* exists, const int* box, int* err) {
    const int lane = threadIdx.x & 31;
    const int wi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int g = 1 + wi / parts, part = wi % parts;
    if (g <= G) {
        if (!exists[g]) return;
        const Box b = load_box(box + 6 * g);
        if (b.nx() <= 0) return;
        const int tx0 = b.x0 / kTX, nbx = (b.x1 - 1) / kTX - tx0 + 1;
        const int ty0 = b.y0 / kTY, nby = (b.y1 - 1) / kTY - ty0 + 1;
        const int tz0 = b.z0 / kTZ, nbz = (b.z1 - 1) / kTZ - tz0 + 1;
        const int n = nbx * nby * nbz;
        for (int i = part * 32 + lane; i < n; i += 32 * parts) {
            const int tx = tx0 + i % nbx, ty = ty0 + (i / nbx) % nby, tz = tz0 + i / (nbx * nby);
            const int t = (tz * tb.nty + ty) * tb.ntx + tx;
            if (!FILL) {
                atomicAdd(tb.count + t, 1);
            } else {
                const long long slot = (long long)tb.off[t] + atomicAdd(tb.cursor + t, 1);
                if (slot >= 0 && slot < tb.capacity) tb.entries[slot] = (uint32_t)g;
                else atomicOr(err, ERR_POOL);
            }
        }
    }
}

// After the device-wide exclusive scan of the tile counts: the largest count and the
// capacity check (off[n_tiles] is the total, count[n_tiles] being 0).
__global__ void bin_check_kernel(TileBins tb, int n_tiles, int* err) {
    int m = 0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n_tiles; t += gridDim.x * blockDim.x) m = max(m, tb.count[t]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(tb.max_count, m);
    if (blockIdx.x == 0 && threadIdx.x == 0 && ((long long)tb.off[n_tiles] > tb.capacity || tb.off[n_tiles] < 0))
        atomicOr(err, ERR_POOL);
}

// Exclusive scan of the tile counts (one CTA), largest count, capacity check.
__global__ void __launch_bounds__(1024) bin_scan_kernel(TileBins tb, int n_tiles, int* err) {
    __shared__ long long sums[33];
    __shared__ int mx[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (n_tiles + blockDim.x - 1) / blockDim.x;
    const int t0 = threadIdx.x * per, t1 = min(n_tiles, t0 + per);
    long long mine = 0;
    int m = 0;
    for (int t = t0; t < t1; t++) {
        mine += tb.count[t];
        m = max(m, tb.count[t]);
    }
    long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 31) sums[warp] = incl;
    if (lane == 0) mx[warp] = m;
    __syncthreads();
    if (warp == 0) {
        const long long w = sums[lane];
        long long wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += u;
        }
        sums[lane] = wi - w;
        if (lane == 31) sums[32] = wi;
        int mm = mx[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mm = max(mm, __shfl_xor_sync(0xffffffffu, mm, o));
        if (lane == 0) mx[0] = mm;
    }
    __syncthreads();
    long long run = sums[warp] + incl - mine;
    for (int t = t0; t < t1; t++) {
        tb.off[t] = (int)run;
        run += tb.count[t];
    }
    if (threadIdx.x == 0) {
        tb.off[n_tiles] = (int)sums[32];
        *tb.max_count = mx[0];
        if (sums[32] > tb.capacity) atomicOr(err, ERR_POOL);
    }
}

// ---------------------------------------------------------------------------------
// 3. the per-tile comparison
// ---------------------------------------------------------------------------------
// One grain box reaching the tile.  Element offsets are of the tile's first voxel (they may
// point before the box; only covered voxels are touched): voxel (dx, dy, dz) of the tile
// lies dz * nxy + dy * nx + dx further.
struct alignas(16) Entry {
    long long in, out, idn;     // field, output and IDLocal
    int nx, nxy;                // strides of its box
    unsigned cover[2];          // covered voxels of the tile, one bit each, per z
    uint32_t id;
    unsigned flags;             // kBoundary, kActive
};
constexpr unsigned kBoundary = 1;  // the box reaches the boundary grain's zone
constexpr unsigned kActive = 2;    // the grain is compared (recalculateIDLocal leaves non-existing ones alone)
static_assert(sizeof(Entry) == 48, "three 16-byte loads");

template <typename T>
struct TileSmem {
    Entry* ent;
    T* val;             // [entry][voxel]
    T* topv;            // [kTop][voxel]
    T* bthr;            // per voxel: the boundary distance's value wins over any neighbour value below this,
    T* bset;            //   and is this
    unsigned (*pmask)[2];  // per entry: voxels whose result is >= 0
    int* tsize;         // per entry: size of its position table
    unsigned* umask;    // 8 words: entries among some voxel's two largest
    int* nu;            // their count
    unsigned short* pos;// [entry a][column of b]: position of b in a's list, or kNotListed
    unsigned char* ulist;  // column -> entry
    unsigned char* ucol;   // entry -> column of pos (the first kUCap of ulist), 0xFF: none
    unsigned char* topi;   // [kTop][voxel]
    unsigned char* bunk;   // per voxel: no branch of the reference assigns its boundary distance
};

template <typename T>
__host__ __device__ constexpr size_t tile_smem_bytes(int mcap) {
    return (sizeof(Entry) + sizeof(T) * kVS + 8 + 4 + 2 * kUCap) * (size_t)mcap + sizeof(T) * kTV * (kTop + 2) + 48 + 512 +
           kTV * (kTop + 1) + 64;
}

template <typename T>
__device__ TileSmem<T> carve(unsigned char* base, int mcap) {
    TileSmem<T> s;
    unsigned char* p = base;
    s.ent = reinterpret_cast<Entry*>(p); p += sizeof(Entry) * mcap;
    s.val = reinterpret_cast<T*>(p); p += sizeof(T) * (size_t)mcap * kVS;
    s.topv = reinterpret_cast<T*>(p); p += sizeof(T) * kTV * kTop;
    s.bthr = reinterpret_cast<T*>(p); p += sizeof(T) * kTV;
    s.bset = reinterpret_cast<T*>(p); p += sizeof(T) * kTV;
    s.pmask = reinterpret_cast<unsigned (*)[2]>(p); p += 8 * mcap;
    s.tsize = reinterpret_cast<int*>(p); p += 4 * mcap;
    s.umask = reinterpret_cast<unsigned*>(p); p += 4 * 8;
    s.nu = reinterpret_cast<int*>(p); p += 16;
    s.pos = reinterpret_cast<unsigned short*>(p); p += 2 * (size_t)mcap * kUCap;
    s.ulist = p; p += 256;
    s.ucol = p; p += 256;
    s.topi = p; p += kTV * kTop;
    s.bunk = p;
    return s;
}

// Bits lo .. hi - 1 of an n-bit row.
__device__ __forceinline__ unsigned span_bits(int lo, int hi, int n) {
    lo = max(lo, 0);
    hi = min(hi, n);
    return hi > lo ? ((1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
}

// The least T that is not below d: v < d, d in FP64, exactly when v is below it.
template <typename T>
__device__ __forceinline__ T not_below(double d);
template <>
__device__ __forceinline__ double not_below<double>(double d) { return d; }
template <>
__device__ __forceinline__ float not_below<float>(double d) { return __double2float_ru(d); }

template <typename T>
__device__ __forceinline__ T neg_inf();
template <>
__device__ __forceinline__ double neg_inf<double>() { return -CUDART_INF; }
template <>
__device__ __forceinline__ float neg_inf<float>() { return -CUDART_INF_F; }

// Keep the kTop largest values seen so far in descending order, without branches.
template <typename T>
__device__ __forceinline__ void top_insert(T (&tv)[kTop], int (&ti)[kTop], T w, int e) {
    bool above[kTop];
#pragma unroll
    for (int k = 0; k < kTop; k++) above[k] = w > tv[k];
#pragma unroll
    for (int k = kTop - 1; k > 0; k--) {
        tv[k] = above[k - 1] ? tv[k - 1] : (above[k] ? w : tv[k]);
        ti[k] = above[k - 1] ? ti[k - 1] : (above[k] ? e : ti[k]);
    }
    tv[0] = above[0] ? w : tv[0];
    ti[0] = above[0] ? e : ti[0];
}

__device__ __forceinline__ unsigned pos_home(uint32_t id, int size) { return (id * 2654435761u) & (unsigned)(size - 1); }

// Position of grain b in grain a's comparison list (a's position table of tsize slots),
// or kNotListed.
template <typename T>
__device__ unsigned short list_position(const CompareArgs<T>& a, uint32_t ga, int tsize, uint32_t gb) {
    const unsigned long long* tab = a.pos_table + (long long)ga * a.pos_cap;
    unsigned h = pos_home(gb, tsize);
    for (int probe = 0; probe < tsize; probe++) {
        const unsigned long long e = __ldg(tab + h);
        const uint32_t k = (uint32_t)(e >> 32);
        if (k == gb) return (unsigned short)(e & 0xFFFFu);
        if (k == kNone) return kNotListed;
        h = (h + 1) & (unsigned)(tsize - 1);
    }
    return kNotListed;
}

template <typename T>
__device__ __forceinline__ unsigned short pair_position(const TileSmem<T>& s, const CompareArgs<T>& a, int ea, int eb) {
    const int col = s.ucol[eb];
    return col != 0xFF ? s.pos[ea * kUCap + col] : list_position(a, s.ent[ea].id, s.tsize[ea], s.ent[eb].id);
}

// The neighbour entry that grain entry ea takes at voxel v, or -1: the largest listed value,
// ties to the earliest position.  The general case: ties, unlisted candidates, no candidate.
template <typename T>
__device__ int decide_pair(const TileSmem<T>& s, const CompareArgs<T>& a, int ea, int v, int m) {
    int best = -1;
    unsigned short bpos = kNotListed;
    T level = neg_inf<T>();
    for (int k = 0; k < kTop; k++) {
        const int eb = s.topi[k * kTV + v];
        if (eb == 0xFF) return best;  // every covering candidate was among those examined
        const T w = s.topv[k * kTV + v];
        if (best >= 0 && !(w == level)) return best;
        if (eb == ea) continue;
        const unsigned short p = pair_position(s, a, ea, eb);
        if (p == kNotListed) continue;
        if (best < 0 || p < bpos) { best = eb; bpos = p; level = w; }
    }
    best = -1;  // full scan of the tile's boxes at this voxel
    bpos = kNotListed;
    for (int eb = 0; eb < m; eb++) {
        if (eb == ea) continue;
        const T w = s.val[eb * kVS + v];
        if (!(w > T(-1))) continue;
        if (best >= 0 && w < level) continue;
        const unsigned short p = pair_position(s, a, ea, eb);
        if (p == kNotListed) continue;
        if (best < 0 || w > level || (w == level && p < bpos)) { best = eb; bpos = p; level = w; }
    }
    return best;
}

// The neighbour value and ID of a pair that its voxel's two largest values do not decide.  Not
// inlined, and given the shared memory's base instead of the pointers into it: it is rare,
// and the row loop keeps its registers.
template <typename T>
struct Neighbour {
    T value;
    uint32_t id;
};
template <typename T>
__device__ __noinline__ Neighbour<T> slow_pair(unsigned char* smem, const CompareArgs<T>& a, int ea, int v, int m,
                                               int y, int x, int z) {
    const TileSmem<T> s = carve<T>(smem, a.mcap);
    const int best = decide_pair(s, a, ea, v, m);
    if (best >= 0) return Neighbour<T>{s.val[best * kVS + v], s.ent[best].id};
    // no listed neighbour covers the voxel: value -1, IDLocal kept
    const uint32_t g = s.ent[ea].id;
    const Box A = load_box(a.in.box + 6 * g), Bold = load_box(a.idbox_old + 6 * g);
    const long long f = A.at(y, x, z);
    return Neighbour<T>{T(-1), f < Bold.count() ? a.id_old[a.idoff_old[g] + f] : 0u};
}
// The boundary distance where no branch assigns it at the voxel itself.
template <typename T>
__device__ __noinline__ double carried_dist(const CompareArgs<T>& a, uint32_t g, int y, int x, int z) {
    return bc_dist(load_box(a.in.box + 6 * g), y, x, z, a.geo.M, a.geo.gb);
}

// One CTA per tile.  Bound by instruction issue: a tile of 64 voxels has ~50 boxes, so ~100
// (box, 32 voxels) rows are staged, searched and written.  What a row needs is therefore
// prepared once per box (one record with the three offsets, the strides and the covered
// voxels as bit masks) or once per voxel and held in its thread's registers, whose voxel
// stays the same over the boxes (candidates, their IDs, the boundary distance, which does
// not depend on the box); the positive voxels of a row are one ballot, turned into the box's
// extents at the end.  Per (box, voxel) pair this had been a walk over four candidates with
// the boundary distance in FP64: 14.4 -> 8.3 ms for 820 M pairs (256^3 / 20,000 grains, FP32
// storage), 2.75 -> 1.57 ms for 90 M (128^3 / 2,000, FP64); issue slots 61% busy, the ALU
// pipe 59%.  Two voxels a lane (one row of both z) spill registers and took 9.1 ms.
template <typename T>
__global__ void __launch_bounds__(kThreads, 4) compare_kernel(const __grid_constant__ CompareArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileSmem<T> s = carve<T>(smem_raw, a.mcap);
    const TileBins& tb = a.bins;
    const int n_tiles = tb.ntx * tb.nty * tb.ntz;
    const T NEG = neg_inf<T>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // this thread's voxel of the tile in the row loops (staging: half 0)
    const int dx = lane & 7, dy = lane >> 3;
    const T lim = not_below<T>(0.7 * a.geo.delta);
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        const int e0 = tb.off[t], m = tb.off[t + 1] - e0;
        if (m == 0) continue;
        if (m > a.mcap) {
            if (threadIdx.x == 0) atomicOr(a.err, ERR_BOX);
            continue;
        }
        const int tx = t % tb.ntx, ty = (t / tb.ntx) % tb.nty, tz = t / (tb.ntx * tb.nty);
        const int X0 = tx * kTX, Y0 = ty * kTY, Z0 = tz * kTZ;
        for (int e = threadIdx.x; e < m; e += kThreads) {
            const uint32_t g = tb.entries[e0 + e];
            const Box B = load_box(a.in.box + 6 * g);
            Entry r;
            r.nx = B.nx();
            r.nxy = B.nx() * B.ny();
            const long long at = (long long)(Z0 - B.z0) * r.nxy + (long long)(Y0 - B.y0) * r.nx + (X0 - B.x0);
            r.in = a.in.off[g] + at;
            r.out = a.out.off[g] + at;
            r.idn = a.idoff_new[g] + at;
            const unsigned ym = span_bits(B.y0 - Y0, B.y1 - Y0, kTY);
            const unsigned rows = span_bits(B.x0 - X0, B.x1 - X0, kTX) *
                                  ((ym & 1) | ((ym & 2) << 7) | ((ym & 4) << 14) | ((ym & 8) << 21));
            r.cover[0] = B.z0 <= Z0 && Z0 < B.z1 ? rows : 0u;
            r.cover[1] = B.z0 <= Z0 + 1 && Z0 + 1 < B.z1 ? rows : 0u;
            r.id = g;
            const bool inner = B.x0 > a.geo.gb && B.x1 < a.geo.M - a.geo.gb && B.y0 > a.geo.gb &&
                               B.y1 < a.geo.M - a.geo.gb && B.z0 > a.geo.gb && B.z1 < a.geo.M - a.geo.gb;
            r.flags = (inner ? 0u : kBoundary) | (a.set_comparison || a.exists[g] ? kActive : 0u);
            s.ent[e] = r;
            s.tsize[e] = pos_table_size(a.n_cmp[g], a.pos_cap);
            s.pmask[e][0] = s.pmask[e][1] = 0u;
            s.ucol[e] = 0xFF;
        }
        if (threadIdx.x < 8) s.umask[threadIdx.x] = 0u;
        if (threadIdx.x == 8) s.nu[0] = 0;
        __syncthreads();
        // values of every covering box over the tile (-inf outside the box), copied with
        // cp.async so that no thread waits on one load before issuing the next
        for (int e = warp; e < m; e += kThreads / 32) {
            const Entry& r = s.ent[e];
            const T* src = a.in.data + r.in + (dy * r.nx + dx);
            T* dst = s.val + e * kVS + lane;
            if ((r.cover[0] >> lane) & 1u) cp_async_elem(dst, src);
            else dst[0] = NEG;
            if ((r.cover[1] >> lane) & 1u) cp_async_elem(dst + 32, src + r.nxy);
            else dst[32] = NEG;
        }
        // the boundary distance of this voxel (box.cpp:997-1088): a voxel at least gb from
        // every face of the boundary grain's zone gets an all-negative distance <= -gb,
        // which changes nothing
        if (threadIdx.x < kTV) {
            const int v = threadIdx.x, x = X0 + v % kTX, y = Y0 + (v / kTX) % kTY, z = Z0 + v / (kTX * kTY);
            const int lo_in = 2 * a.geo.gb - 1, hi_in = a.geo.M - 1 - 2 * a.geo.gb;
            T thr = NEG, set = T(0);
            bool unk = false;
            if (!(x >= lo_in && x <= hi_in && y >= lo_in && y <= hi_in && z >= lo_in && z <= hi_in)) {
                double d = 0.0;
                unk = !bc_assign(y, x, z, a.geo.M, a.geo.gb, d);
                if (!unk && d > -a.geo.gb) {
                    thr = not_below<T>(d * a.geo.h);
                    set = (T)(d * a.geo.h);
                }
            }
            s.bthr[v] = thr;
            s.bset[v] = set;
            s.bunk[v] = unk;
        }
        cp_async_wait_all();
        __syncthreads();
        // per voxel: the kTop largest values > -1.  The kParts lanes of a voxel are
        // neighbours in one warp; each keeps the top of every kParts-th box, then two
        // shuffle rounds merge their lists into the first lane's.
        {
            const int part = lane & (kParts - 1), v = warp * (32 / kParts) + (lane / kParts);
            T tv[kTop];
            int ti[kTop];
#pragma unroll
            for (int k = 0; k < kTop; k++) { tv[k] = T(-1); ti[k] = 0xFF; }
            for (int e = part; e < m; e += kParts) top_insert(tv, ti, s.val[e * kVS + v], e);
#pragma unroll
            for (int o = 1; o < kParts; o <<= 1) {
                T pv[kTop];
                int pi[kTop];
#pragma unroll
                for (int k = 0; k < kTop; k++) {
                    pv[k] = __shfl_down_sync(0xffffffffu, tv[k], o);
                    pi[k] = __shfl_down_sync(0xffffffffu, ti[k], o);
                }
#pragma unroll
                for (int k = 0; k < kTop; k++) top_insert(tv, ti, pv[k], pi[k]);
            }
            if (part == 0) {
#pragma unroll
                for (int k = 0; k < kTop; k++) {
                    s.topv[k * kTV + v] = ti[k] != 0xFF ? tv[k] : NEG;
                    s.topi[k * kTV + v] = (unsigned char)ti[k];
                }
                // a column of pos for every entry among some voxel's two largest
#pragma unroll
                for (int k = 0; k < 2; k++)
                    if (ti[k] != 0xFF && !((s.umask[ti[k] >> 5] >> (ti[k] & 31)) & 1u)) {
                        const unsigned bit = 1u << (ti[k] & 31);
                        if (!(atomicOr(s.umask + (ti[k] >> 5), bit) & bit)) {
                            const int col = atomicAdd(s.nu, 1);
                            if (col < kUCap) {
                                s.ulist[col] = (unsigned char)ti[k];
                                s.ucol[ti[k]] = (unsigned char)col;
                            }
                        }
                    }
            }
        }
        __syncthreads();
        // pos[a][column of b] = position of b in a's list, from a's position table; kBatch
        // lookups advance together, each round issuing all their next probes.  Columns beyond
        // kUCap are looked up when needed.
        {
            constexpr int kBatch = 2;
            const int nu = min(s.nu[0], kUCap);
            const int mm = m * nu;
            for (int q0 = 0; q0 < mm; q0 += kBatch * kThreads) {
                unsigned long long e[kBatch];
                const unsigned long long* tab[kBatch];
                unsigned h[kBatch], mask[kBatch];
                uint32_t id[kBatch];
                bool live[kBatch];
                int dst[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; u++) {
                    const int q = q0 + u * kThreads + threadIdx.x;
                    const int ea = q / nu, col = q - ea * nu, eb = q < mm ? s.ulist[col] : 0;
                    live[u] = q < mm && ea != eb;
                    dst[u] = ea * kUCap + col;
                    tab[u] = nullptr;
                    h[u] = mask[u] = id[u] = 0;
                    e[u] = 0;
                    if (live[u]) {
                        tab[u] = a.pos_table + (long long)s.ent[ea].id * a.pos_cap;
                        mask[u] = (unsigned)s.tsize[ea] - 1;
                        id[u] = s.ent[eb].id;
                        h[u] = pos_home(id[u], s.tsize[ea]);
                        e[u] = __ldg(tab[u] + h[u]);
                    }
                }
                for (int round = 0; round < a.pos_cap; round++) {
                    bool more = false;
#pragma unroll
                    for (int u = 0; u < kBatch; u++) {
                        if (!live[u]) continue;
                        const uint32_t k = (uint32_t)(e[u] >> 32);
                        if (k == id[u] || k == kNone) {
                            s.pos[dst[u]] = k == id[u] ? (unsigned short)(e[u] & 0xFFFFu) : kNotListed;
                            live[u] = false;
                        } else {
                            h[u] = (h[u] + 1) & mask[u];
                            more = true;
                        }
                    }
                    if (!more) break;
#pragma unroll
                    for (int u = 0; u < kBatch; u++)
                        if (live[u]) e[u] = __ldg(tab[u] + h[u]);
                }
            }
        }
        __syncthreads();
        // every (grain, voxel) pair of the tile: a thread keeps its voxel, a warp shares the
        // entry (kTV and kThreads are multiples of 64)
        {
            const int v = threadIdx.x % kTV, dz = v / 32;
            const T w0 = s.topv[v], w1 = s.topv[kTV + v], w2 = s.topv[2 * kTV + v];
            const int i0 = s.topi[v], i1 = s.topi[kTV + v];
            const int c0 = i0 != 0xFF ? s.ucol[i0] : 0xFF, c1 = i1 != 0xFF ? s.ucol[i1] : 0xFF;
            const uint32_t g0 = i0 != 0xFF ? s.ent[i0].id : 0u, g1 = i1 != 0xFF ? s.ent[i1].id : 0u;
            const T bthr = s.bthr[v], bset = s.bset[v];
            const bool bunk = s.bunk[v];
            for (int ea = threadIdx.x / kTV; ea < m; ea += kThreads / kTV) {
                const Entry& r = s.ent[ea];
                const unsigned flags = r.flags;
                bool positive = false;
                // else the voxel is outside this grain's box, or (recalculateIDLocal) the
                // grain does not exist and executeComparison leaves it alone
                if (((r.cover[dz] >> lane) & 1u) && (flags & kActive)) {
                    const T in = s.val[ea * kVS + v];
                    const int f = dz * r.nxy + dy * r.nx + dx;
                    // the largest other value, decided when it is listed and the next differs
                    const bool self = i0 == ea;
                    const int col = self ? c1 : c0;
                    T cmpv = self ? w1 : w0;
                    uint32_t idv = self ? g1 : g0;
                    const T next = self ? w2 : w1;
                    if (col == 0xFF || next == cmpv || s.pos[ea * kUCap + col] == kNotListed) {
                        const Neighbour<T> n = slow_pair(smem_raw, a, ea, v, m, Y0 + dy, X0 + dx, Z0 + dz);
                        cmpv = n.value;
                        idv = n.id;
                    }
                    if (flags & kBoundary) {  // the boundary condition near the zone's faces
                        if (bunk) {  // the value of an earlier voxel of this box's loop
                            const double d = carried_dist(a, r.id, Y0 + dy, X0 + dx, Z0 + dz);
                            if (d > -a.geo.gb)
                                if (d * a.geo.h > (double)cmpv) {
                                    cmpv = (T)(d * a.geo.h);
                                    idv = 0;
                                }
                        } else if (cmpv < bthr) {
                            cmpv = bset;
                            idv = 0;
                        }
                    }
                    T res;
                    if (!a.set_comparison) res = cmpv;
                    else if (fabs(in) < lim) res = T(0.5) * (in - cmpv);
                    else res = in;
                    a.out.data[r.out + f] = res;
                    a.id_new[r.idn + f] = idv;
                    positive = a.set_comparison && res >= 0;
                }
                // the voxels of the new bounding box (executeSetComparison, box.cpp:858-877)
                const unsigned bal = __ballot_sync(0xffffffffu, positive);
                if (bal && lane == 0) s.pmask[ea][dz] = bal;
            }
        }
        __syncthreads();
        for (int e = threadIdx.x; e < m; e += kThreads) {
            const unsigned p0 = s.pmask[e][0], p1 = s.pmask[e][1], p = p0 | p1;
            if (!p) continue;
            unsigned row = p | (p >> 16);
            row = (row | (row >> 8)) & 0xFFu;  // the x of any row; a byte per y
            int* nb = a.newbox + 6 * s.ent[e].id;
            atomicMin(nb + 0, X0 + __ffs(row) - 1); atomicMax(nb + 1, X0 + 31 - __clz(row));
            atomicMin(nb + 2, Y0 + ((__ffs(p) - 1) >> 3)); atomicMax(nb + 3, Y0 + ((31 - __clz(p)) >> 3));
            atomicMin(nb + 4, Z0 + (p0 ? 0 : 1)); atomicMax(nb + 5, Z0 + (p1 ? 1 : 0));
        }
        __syncthreads();
    }
}

__global__ void newbox_init_kernel(int G, const int* present, const int* exists, const int* box, int* newbox) {
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g <= G; g += gridDim.x * blockDim.x) {
        if (g == 0 || !present[g] || !exists[g]) continue;
        const Box b = load_box(box + 6 * g);
        // executeSetComparison starts from the inverted out box, box.cpp:815-820
        int* nb = newbox + 6 * g;
        nb[0] = b.x1; nb[1] = b.x0; nb[2] = b.y1; nb[3] = b.y0; nb[4] = b.z1; nb[5] = b.z0;
    }
}

}  // namespace

size_t compare_smem_bytes(int mcap, bool fp64) {
    return fp64 ? tile_smem_bytes<double>(mcap) : tile_smem_bytes<float>(mcap);
}

long long bin_capacity(int G, int side) {
    const long long tx = side / kTX + 2, ty = side / kTY + 2, tz = side / kTZ + 2;
    return (long long)G * tx * ty * tz;
}

void launch_copy_lists(const ListCopyArgs& a, int grid, cudaStream_t s) {
    copy_lists_kernel<<<grid, 256, 0, s>>>(a);
}

void launch_bin(const TileBins& tb, int G, const int* exists, const int* box, int* err, cudaStream_t s) {
    const int n_tiles = tb.ntx * tb.nty * tb.ntz;
    cudaMemsetAsync(tb.count, 0, sizeof(int) * (n_tiles + 1), s);
    cudaMemsetAsync(tb.cursor, 0, sizeof(int) * (n_tiles + 1), s);
    // a warp per grain leaves few grains' thousands of tiles to few warps (0.52 ms for 30 grains
    // of 90^3, of a comparison of 1.0 ms): enough warps for 32 an SM
    const int parts = G >= 4736 ? 1 : (4736 + G - 1) / G;
    const int grid = (G * parts + 3) / 4;  // 4 warps per block
    bin_kernel<false><<<grid, 128, 0, s>>>(tb, G, parts, exists, box, err);
    if (tb.temp) {  // device-wide: the one-CTA scan below walks the tiles serially
        launch_exclusive_scan(tb.temp, tb.temp_bytes, tb.count, tb.off, n_tiles + 1, s);
        cudaMemsetAsync(tb.max_count, 0, sizeof(int), s);
        bin_check_kernel<<<(n_tiles + 255) / 256 < 1184 ? (n_tiles + 255) / 256 : 1184, 256, 0, s>>>(tb, n_tiles, err);
    } else {
        bin_scan_kernel<<<1, 1024, 0, s>>>(tb, n_tiles, err);
    }
    bin_kernel<true><<<grid, 128, 0, s>>>(tb, G, parts, exists, box, err);
}

// A tile's work follows its number of boxes, so equal shares of the tiles are unequal shares of
// the work and the grid's last CTAs decide when it ends.  Shares kGridShares times smaller let
// the hardware deal them out as CTAs retire; a CTA's start costs little beside one tile, so only
// a grid beyond the tiles themselves is a loss (measured with 4096 CTAs per SM: 0.97 -> 1.24 ms
// for 128^3, 2000 grains, float).  Measured with 4 -> 64 CTAs per SM: 256^3, 20,000 grains, float
// 8.83 -> 7.95 ms; 208^3, 16,800 grains, float 4.99 -> 4.66; 128^3, 2000 grains, float
// 1.09 -> 0.97, double 1.68 -> 1.25; 64^3, 200 grains, float 0.213 -> 0.211.
constexpr int kGridShares = 16;

template <typename T>
void launch_compare(const CompareArgs<T>& a, int grid, cudaStream_t s) {
    static PerDevice configured;
    configured.once([] {
        allow_max_dynamic_smem(compare_kernel<T>);
    });
    const int tiles = a.bins.ntx * a.bins.nty * a.bins.ntz;
    const int ctas = min(max(tiles, grid), kGridShares * grid);
    compare_kernel<T><<<ctas, kThreads, compare_smem_bytes(a.mcap, sizeof(T) == 8), s>>>(a);
}

void launch_newbox_init(int G, const int* present, const int* exists, const int* box, int* newbox, cudaStream_t s) {
    newbox_init_kernel<<<(G + 256) / 256, 256, 0, s>>>(G, present, exists, box, newbox);
}

template void launch_compare<double>(const CompareArgs<double>&, int, cudaStream_t);
template void launch_compare<float>(const CompareArgs<float>&, int, cudaStream_t);

}  // namespace gg
