// Root cubes, Morton keys, LSD radix sort and the permutation gather.
//
// All of these are HBM/L2-bound integer and byte moves: coalesced loads,
// grid sizes in multiples of the SM count, no tensor-core reshaping.
#include <cfloat>

#include "sph3_internal.cuh"

namespace sph3 {

// ------------------------------------------------------------ root cubes
// Two kernels (the allocation-free sort), or one (the context, k_move_box).
// k_box_partial: one block per work item (a run of at most
// kBoxChunk particles of one cloud; the item table is fixed per particle
// layout) writes the FP64 min/max of its run.  k_cloud_boxes: one block per
// cloud reduces its items and sets a power-of-two cube [origin, origin + size)
// that contains the cloud, origin on the size/2 grid.  Periodic runs use the
// fixed cube [0, 2^ceil(log2 L)).
// The block's minimum and maximum of each coordinate over its 256 threads, to
// thread 0..2 (one coordinate each) of the block; bad: non-finite input seen.
__device__ __forceinline__ void block_box(double (&mn)[3], double (&mx)[3], int bad, double *part6, unsigned *status) {
    __shared__ double smin[3][8], smax[3][8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double a = warp_min(mn[d]), b = warp_max(mx[d]);
        if (lane == 0) {
            smin[d][wid] = a;
            smax[d][wid] = b;
        }
    }
    if (__any_sync(kFull, bad) && lane == 0) atomicOr(status, SPH3_STATUS_NAN_INPUT);
    __syncthreads();
    if (threadIdx.x < 3) {
        const int d = threadIdx.x;
        double lo = DBL_MAX, hi = -DBL_MAX;
        for (int w = 0; w < 8; ++w) {
            lo = fmin(lo, smin[d][w]);
            hi = fmax(hi, smax[d][w]);
        }
        part6[d] = lo;
        part6[3 + d] = hi;
    }
    __syncthreads();
}

__device__ __forceinline__ void box_add(double x, double &mn, double &mx, int &bad) {
    if (!isfinite(x)) {
        bad = 1;
        return;
    }
    mn = fmin(mn, x);
    mx = fmax(mx, x);
}

// The root cube of one cloud from its extent (one thread)
__device__ void set_root_cube(Cloud &cl, const double (&lo)[3], const double (&hi)[3], int max_level, int periodic,
                              double Lx, double Ly, double Lz) {
    double size;
    double org[3];
    if (periodic) {
        double L = fmax(Lx, fmax(Ly, Lz));
        int e;
        frexp(L, &e);  // L = f * 2^e, f in [0.5, 1)
        size = ldexp(1.0, e);
        if (size * 0.5 >= L) size *= 0.5;
        org[0] = org[1] = org[2] = 0.0;
    } else {
        double ext = fmax(hi[0] - lo[0], fmax(hi[1] - lo[1], hi[2] - lo[2]));
        if (!(ext > 0.0) || !isfinite(ext)) ext = 1.0;
        int e;
        frexp(ext, &e);
        size = ldexp(1.0, e);  // >= ext
        for (int attempt = 0; attempt < 64; ++attempt) {
            double half = 0.5 * size;
            bool ok = true;
            for (int d = 0; d < 3; ++d) {
                org[d] = floor(lo[d] / half) * half;
                if (!(org[d] + size > hi[d])) ok = false;
            }
            if (ok) break;
            size *= 2.0;
        }
    }
    for (int d = 0; d < 3; ++d) cl.origin[d] = org[d];
    cl.size = size;
    cl.inv_cell = ldexp(1.0, max_level) / size;
    cl.s10 = (float)(size / 1024.0);
}

__global__ void __launch_bounds__(256) k_box_partial(const int4 *items, const double *pos, int64_t n,
                                                     double *part, unsigned *status) {
    const int4 it = items[blockIdx.x];  // {cloud, begin, end, 0}
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    int bad = 0;
    for (int64_t k = it.y + threadIdx.x; k < it.z; k += blockDim.x)
#pragma unroll
        for (int d = 0; d < 3; ++d) box_add(pos[d * n + k], mn[d], mx[d], bad);
    block_box(mn, mx, bad, part + (size_t)blockIdx.x * 6, status);
}

__global__ void k_cloud_boxes(Cloud *clouds, const int *item_begin, const double *part, int max_level,
                              int periodic, double Lx, double Ly, double Lz) {
    // one warp: lanes stride over the cloud's items, then a warp reduction
    double lo[3], hi[3];
    for (int d = 0; d < 3; ++d) {
        lo[d] = DBL_MAX;
        hi[d] = -DBL_MAX;
        for (int it = item_begin[blockIdx.x] + (int)threadIdx.x; it < item_begin[blockIdx.x + 1]; it += 32) {
            lo[d] = fmin(lo[d], part[it * 6 + d]);
            hi[d] = fmax(hi[d], part[it * 6 + 3 + d]);
        }
        lo[d] = warp_min(lo[d]);
        hi[d] = warp_max(hi[d]);
        if (lo[d] > hi[d]) lo[d] = hi[d] = 0.0;  // empty cloud
    }
    if (threadIdx.x == 0) set_root_cube(clouds[blockIdx.x], lo, hi, max_level, periodic, Lx, Ly, Lz);
}

// The context's form: the opening kick and drift (MOVE), the extents and the
// root cubes in one launch.  A block moves and reduces one item; the block that
// completes a cloud's items (counted in `arrive`) reduces them and sets the
// cube.  Three launches took 18 us at 2,000 particles and 37 at 1,048,576; 7
// and 32 now (HBM: 120 B a particle, and the last block's tail).
struct MoveArgs {
    double dt;
    double *pos, *vel;
    const double *acc;
};

template <bool MOVE>
__global__ void __launch_bounds__(256) k_move_box(const int4 *items, int64_t n, MoveArgs m, double *part, int *arrive,
                                                  Cloud *clouds, const int *item_begin, int ncloud, int max_level,
                                                  int periodic, double Lx, double Ly, double Lz, unsigned *status) {
    __shared__ int s_last;
    __shared__ double s_box[6];
    const int4 it = items[blockIdx.x];  // {cloud, begin, end, 0}
    const double L[3] = {Lx, Ly, Lz};
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    int bad = 0;
    for (int64_t k = it.y + threadIdx.x; k < it.z; k += 256) {
        double x[3], v[3], a[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {  // all loads of a particle in flight together
            x[d] = m.pos[d * n + k];
            v[d] = MOVE ? m.vel[d * n + k] : 0.0;
            a[d] = MOVE ? m.acc[d * n + k] : 0.0;
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (MOVE) {
                // v + acc * dt / 2.0 and r + v * dt, rounded as NumPy does (no FMA)
                v[d] = __dadd_rn(v[d], __dmul_rn(__dmul_rn(a[d], m.dt), 0.5));
                x[d] = __dadd_rn(x[d], __dmul_rn(v[d], m.dt));
                if (L[d] > 0.0) {
                    if (x[d] < 0.0) x[d] += L[d];
                    if (x[d] >= L[d]) x[d] -= L[d];
                }
                m.vel[d * n + k] = v[d];
                m.pos[d * n + k] = x[d];
            }
            box_add(x[d], mn[d], mx[d], bad);
        }
    }
    block_box(mn, mx, bad, part + (size_t)blockIdx.x * 6, status);
    const int i0 = item_begin[it.x], i1 = item_begin[it.x + 1];
    if (threadIdx.x < 3) __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(arrive + it.x, 1) == i1 - i0 - 1;
        __threadfence();
    }
    __syncthreads();
    if (s_last) {
        double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
        for (int q = i0 + (int)threadIdx.x; q < i1; q += 256)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                lo[d] = fmin(lo[d], __ldcg(part + (size_t)q * 6 + d));
                hi[d] = fmax(hi[d], __ldcg(part + (size_t)q * 6 + 3 + d));
            }
        block_box(lo, hi, 0, s_box, status);
        if (threadIdx.x == 0) {
            for (int d = 0; d < 3; ++d) {
                lo[d] = s_box[d];
                hi[d] = s_box[3 + d];
                if (lo[d] > hi[d]) lo[d] = hi[d] = 0.0;  // no finite coordinate
            }
            set_root_cube(clouds[it.x], lo, hi, max_level, periodic, Lx, Ly, Lz);
            arrive[it.x] = 0;
        }
    }
    if (blockIdx.x == 0) {  // clouds without particles
        const double zero[3] = {0.0, 0.0, 0.0};
        for (int c = threadIdx.x; c < ncloud; c += 256)
            if (item_begin[c] == item_begin[c + 1])
                set_root_cube(clouds[c], zero, zero, max_level, periodic, Lx, Ly, Lz);
    }
}

// Particles per item: one per thread in small sets, so that a block's chain is
// short; two and four in larger ones, so that the block that completes a cloud
// has at most a few thousand items to reduce.
int box_chunk(int64_t n) { return n <= 65536 ? 256 : (n <= (1 << 21) ? 512 : 1024); }

void launch_move_box(State &S, const Params &P, const double *dt, cudaStream_t st) {
    if (S.n == 0) return;
    const MoveArgs m = {dt ? *dt : 0.0, S.pos, S.vel, S.acc};
    auto *kern = dt ? k_move_box<true> : k_move_box<false>;
    kern<<<S.nbox_items, 256, 0, st>>>(S.box_items, S.n, m, S.box_part, S.box_arrive, S.clouds, S.box_item_begin,
                                      S.ncloud, S.max_level, P.periodic, P.box[0], P.box[1], P.box[2], S.status);
}

// ------------------------------------------------------------ keys
__device__ __forceinline__ int cloud_of_sorted(const Cloud *clouds, int ncloud, int64_t k) {
    int lo = 0, hi = ncloud - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (clouds[mid].begin <= k) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void k_keys(const Cloud *clouds, int ncloud, const double *pos, int64_t n,
                       int max_level, uint64_t *key, uint32_t *perm) {
    const uint32_t maxq = (1u << max_level) - 1u;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        const int c = cloud_of_sorted(clouds, ncloud, k);
        const Cloud &cl = clouds[c];
        uint32_t ix = quantise(pos[k], cl.origin[0], cl.inv_cell, maxq);
        uint32_t iy = quantise(pos[n + k], cl.origin[1], cl.inv_cell, maxq);
        uint32_t iz = quantise(pos[2 * n + k], cl.origin[2], cl.inv_cell, maxq);
        uint64_t mort = spread3(ix) | (spread3(iy) << 1) | (spread3(iz) << 2);
        key[k] = ((uint64_t)c << (3 * max_level)) | mort;
        perm[k] = (uint32_t)k;
    }
}

static bool keys_start_in_alt(const State &S);

// unsorted keys and the identity permutation, where launch_radix_sort takes them from
void launch_keys(State &S, const Params &P, cudaStream_t st) {
    if (S.n == 0) return;
    int blocks = (int)std::min<int64_t>((S.n + 255) / 256, (int64_t)S.num_sms * 8);
    const bool alt = keys_start_in_alt(S);
    k_keys<<<blocks, 256, 0, st>>>(S.clouds, S.ncloud, S.pos, S.n, S.max_level, alt ? S.key_alt : S.key,
                                   alt ? S.perm_alt : S.perm);
}

// ------------------------------------------------------------ radix sort
// LSD, 8-bit digits, stable.  Per pass of the fixed-scratch form: a tile
// histogram, one scan of the digit-major histogram table, and a stable scatter
// that ranks each key within its tile (order = memory order inside a warp's
// segment, then warp order).
constexpr int kRsThreads = 256;
constexpr int kRsItems = kRsTileKeys / kRsThreads;
constexpr int kRsTile = kRsThreads * kRsItems;
constexpr int kRsWarps = kRsThreads / 32;

__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const uint64_t *key, int64_t n, int shift,
                                                        uint32_t *hist, int nblocks) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kRsTile;
#pragma unroll
    for (int t = 0; t < kRsItems; ++t) {
        int64_t k = base + t * kRsThreads + threadIdx.x;
        if (k < n) atomicAdd(&h[(key[k] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[blockIdx.x * 256 + threadIdx.x] = h[threadIdx.x];  // block-major table
}

// Exclusive prefix of the block-major digit histogram, in place: hist[b][d]
// becomes the number of keys with digit d in blocks before b, and
// hist[nblocks][d] the number of keys with a smaller digit.  One block of
// kRsOffsetThreads threads: 256 digits x kOffQ block ranges; each range is
// summed with kOffU independent loads in flight, the ranges and digits are
// combined in shared memory, and a second pass over the (L2-resident) table
// writes the prefixes.
constexpr int kOffQ = kRsOffsetThreads / 256;
constexpr int kOffU = 16;

__global__ void __launch_bounds__(kRsOffsetThreads) k_rs_offsets(uint32_t *hist, int nblocks) {
    __shared__ uint32_t part[kOffQ][256];
    __shared__ uint32_t tot[256];
    const int d = threadIdx.x & 255, q = threadIdx.x >> 8;
    const int per = (nblocks + kOffQ - 1) / kOffQ;
    const int b0 = min(nblocks, q * per), b1 = min(nblocks, b0 + per);
    uint32_t s = 0;
    int b = b0;
    for (; b + kOffU <= b1; b += kOffU) {
        uint32_t v[kOffU];
#pragma unroll
        for (int k = 0; k < kOffU; ++k) v[k] = hist[(size_t)(b + k) * 256 + d];
#pragma unroll
        for (int k = 0; k < kOffU; ++k) s += v[k];
    }
    for (; b < b1; ++b) s += hist[(size_t)b * 256 + d];
    part[q][d] = s;
    __syncthreads();
    if (q == 0) {
        uint32_t run = 0;
#pragma unroll
        for (int k = 0; k < kOffQ; ++k) {
            const uint32_t t = part[k][d];
            part[k][d] = run;
            run += t;
        }
        tot[d] = run;
    }
    __syncthreads();
    const uint32_t own = tot[d];
    for (int o = 1; o < 256; o <<= 1) {
        const uint32_t v = (q == 0 && d >= o) ? tot[d - o] : 0u;
        __syncthreads();
        if (q == 0) tot[d] += v;
        __syncthreads();
    }
    uint32_t run = part[q][d];
    b = b0;
    for (; b + kOffU <= b1; b += kOffU) {
        uint32_t v[kOffU];
#pragma unroll
        for (int k = 0; k < kOffU; ++k) v[k] = hist[(size_t)(b + k) * 256 + d];
#pragma unroll
        for (int k = 0; k < kOffU; ++k) {
            hist[(size_t)(b + k) * 256 + d] = run;
            run += v[k];
        }
    }
    for (; b < b1; ++b) {
        const uint32_t v = hist[(size_t)b * 256 + d];
        hist[(size_t)b * 256 + d] = run;
        run += v;
    }
    if (q == 0) hist[(size_t)nblocks * 256 + d] = tot[d] - own;  // exclusive digit base
}

// Lanes of the warp holding the same 8-bit digit: one ballot per digit bit
// (independent of the data, where a warp match takes a round per distinct
// digit).  Lanes with ok = false form a class of their own.
__device__ __forceinline__ unsigned digit_peers(int d, bool ok) {
    unsigned peers = __ballot_sync(kFull, ok);
    if (!ok) peers = ~peers;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1;
        const unsigned bal = __ballot_sync(kFull, bit);
        peers &= bit ? bal : ~bal;
    }
    return peers;
}

// Stable scatter of one tile of 256 ITEMS keys.  Each key's rank inside the
// tile (digit start in the tile + earlier warps' count of the digit + rank
// inside its warp, in memory order) comes from digit ballots; the tile is then
// staged in shared memory in digit order, so that every digit's run leaves
// as consecutive addresses (coalesced stores instead of one scattered 8-byte
// store per key).  The output is the same as scattering each key directly.
// offsets(d, count of digit d in this tile) gives the output start of the
// tile's keys of digit d (called by thread d once the counts are known).
template <int ITEMS, class Offsets>
__device__ __forceinline__ void rs_scatter_tile(const uint64_t *key_in, const uint32_t *val_in, uint64_t *key_out,
                                                uint32_t *val_out, int64_t n, int shift, int tile_index,
                                                Offsets &offsets) {
    constexpr int TILE = kRsThreads * ITEMS;
    __shared__ uint32_t wcnt[kRsWarps][256];
    __shared__ uint32_t goff[256];  // output start of the tile's keys of digit d, less the digit's start in the tile
    __shared__ uint32_t toff[256];  // start of digit d inside the tile
    __shared__ uint32_t wsum[kRsWarps];
    // keys and values in tile order; the largest tile stages its values in the
    // keys' place after the keys have left (48 KB of static shared memory)
    constexpr bool kTwoPhase = ITEMS > 8;
    __shared__ uint64_t skey[TILE];
    __shared__ uint32_t sval_own[kTwoPhase ? 1 : TILE];
    uint32_t *sval = kTwoPhase ? reinterpret_cast<uint32_t *>(skey) : sval_own;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t tile = (int64_t)tile_index * TILE;
    const int64_t base = tile + (int64_t)w * (ITEMS * 32);
    uint64_t kk[ITEMS];
    uint32_t vv[ITEMS];
#pragma unroll
    for (int t = 0; t < ITEMS; ++t) {
        const int64_t k = base + t * 32 + lane;
        kk[t] = k < n ? key_in[k] : 0ull;
        vv[t] = k < n ? val_in[k] : 0u;
    }
    for (int i = lane; i < 256; i += 32) wcnt[w][i] = 0;
    __syncwarp();
    uint32_t rank[ITEMS];
    const unsigned lt = lanemask_lt();
#pragma unroll
    for (int t = 0; t < ITEMS; ++t) {
        const bool ok = base + t * 32 + lane < n;
        const int d = (int)((kk[t] >> shift) & 255u);
        const unsigned peers = digit_peers(d, ok);
        const uint32_t b = wcnt[w][d];
        __syncwarp();
        if (ok && (peers & lt) == 0) wcnt[w][d] = b + __popc(peers);
        __syncwarp();
        rank[t] = b + __popc(peers & lt);
    }
    __syncthreads();
    // prefix over warps for each digit, and the tile's count of the digit
    uint32_t cnt_d;
    {
        const int d = threadIdx.x;
        uint32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < kRsWarps; ++ww) {
            uint32_t c = wcnt[ww][d];
            wcnt[ww][d] = run;
            run += c;
        }
        cnt_d = run;
    }
    // exclusive scan of the digit counts over the tile (256 threads = 256 digits)
    const uint32_t incl = (uint32_t)warp_incl_scan((int)cnt_d);
    if (lane == 31) wsum[w] = incl;
    const uint32_t gstart = offsets(threadIdx.x, cnt_d);  // output start of the tile's keys of the digit
    __syncthreads();
    {
        uint32_t pre = 0;
#pragma unroll
        for (int ww = 0; ww < kRsWarps; ++ww) pre += ww < w ? wsum[ww] : 0u;
        const uint32_t start = pre + incl - cnt_d;
        toff[threadIdx.x] = start;
        goff[threadIdx.x] = gstart - start;
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < ITEMS; ++t) {
        if (base + t * 32 + lane < n) {
            const int d = (int)((kk[t] >> shift) & 255u);
            rank[t] += toff[d] + wcnt[w][d];  // place in the tile
            skey[rank[t]] = kk[t];
            if (!kTwoPhase) sval[rank[t]] = vv[t];
        }
    }
    __syncthreads();
    const int cnt = (int)min((int64_t)TILE, n - tile);
    uint32_t at[ITEMS];
#pragma unroll
    for (int t = 0; t < ITEMS; ++t) {
        const int j = t * kRsThreads + threadIdx.x;
        at[t] = 0;
        if (j < cnt) {
            const uint64_t kv = skey[j];
            at[t] = goff[(int)((kv >> shift) & 255u)] + (uint32_t)j;
            key_out[at[t]] = kv;
            if (!kTwoPhase) val_out[at[t]] = sval[j];
        }
    }
    if (!kTwoPhase) return;
    __syncthreads();
#pragma unroll
    for (int t = 0; t < ITEMS; ++t)
        if (base + t * 32 + lane < n) sval[rank[t]] = vv[t];
    __syncthreads();
#pragma unroll
    for (int t = 0; t < ITEMS; ++t) {
        const int j = t * kRsThreads + threadIdx.x;
        if (j < cnt) val_out[at[t]] = sval[j];
    }
}

// The tile scatter with offsets from the digit-major table of k_rs_offsets
// (one tile per block, in block order).
__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const uint64_t *key_in,
                                                           const uint32_t *val_in, uint64_t *key_out,
                                                           uint32_t *val_out, int64_t n, int shift,
                                                           const uint32_t *hist, int nblocks) {
    auto offsets = [&](int d, uint32_t) { return hist[nblocks * 256 + d] + hist[blockIdx.x * 256 + d]; };
    rs_scatter_tile<kRsItems>(key_in, val_in, key_out, val_out, n, shift, blockIdx.x, offsets);
}

// ---- one sweep per digit pass (the context's sort above kRankMax keys)
// All passes' digit histograms in one read of the keys (a private table in
// shared memory, then one atomic per bin and block); the scatter of each pass
// then takes its tiles in order from an atomic counter and finds each digit's
// offset over the earlier tiles by decoupled look-back: a tile publishes its
// count of each digit (AGG), adds up its predecessors' counts back to one
// that knows its inclusive prefix (INCL) and publishes its own.  The look-back
// reads kOsBatch predecessors at a time (independent loads): with every tile
// resident, a tile starts when none of its predecessors has its prefix yet,
// and one dependent L2 round trip per predecessor was most of a pass.
// One launch per pass instead of histogram + table scan + scatter.  Every
// predecessor tile was taken by a running block, so each wait ends; waits are
// bounded all the same and raise SPH3_STATUS_SORT if one ever ran out.
constexpr int kHaThreads = 256;
constexpr int kMaxPasses = 8;
constexpr uint32_t kOsAgg = 1u << 30, kOsIncl = 2u << 30, kOsMask = (1u << 30) - 1u;
constexpr int kOsMaxSpin = 1 << 22;
constexpr int kOsBatch = 8;

__global__ void __launch_bounds__(kHaThreads) k_rs_hist_all(const uint64_t *key, int64_t n, int passes,
                                                            uint32_t *hist_all) {
    __shared__ uint32_t h[kMaxPasses][256];
    for (int i = threadIdx.x; i < passes * 256; i += kHaThreads) (&h[0][0])[i] = 0;
    __syncthreads();
    for (int64_t k = (int64_t)blockIdx.x * kHaThreads + threadIdx.x; k < n; k += (int64_t)gridDim.x * kHaThreads) {
        const uint64_t kv = key[k];
        for (int p = 0; p < passes; ++p) {
            // neighbouring keys share their upper digits: one shared atomic per run of equal digits
            const unsigned act = __activemask();
            const uint32_t d = (uint32_t)(kv >> (8 * p)) & 255u;
            int same;
            __match_all_sync(act, d, &same);
            if (same) {
                if ((int)(threadIdx.x & 31) == __ffs(act) - 1) atomicAdd(&h[p][d], (uint32_t)__popc(act));
            } else {
                atomicAdd(&h[p][d], 1u);
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += kHaThreads) {
        const uint32_t t = (&h[0][0])[i];
        if (t) atomicAdd(hist_all + i, t);
    }
}

// look-back words hold their flag and value in one 32-bit word, so relaxed
// device-scope accesses are enough
__device__ __forceinline__ uint32_t ld_word(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(uint32_t *p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

template <int ITEMS>
__global__ void __launch_bounds__(kRsThreads) k_rs_onesweep(const uint64_t *key_in, const uint32_t *val_in,
                                                            uint64_t *key_out, uint32_t *val_out, int64_t n,
                                                            int pass, const uint32_t *hist_all, uint32_t *state,
                                                            int *tile_ctr, unsigned *status) {
    __shared__ int s_tile;
    __shared__ uint32_t wtot[kRsWarps];
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_ctr + pass, 1);
    // exclusive scan over digits of this pass's global histogram: digit bases
    const int d0 = threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t hd = hist_all[pass * 256 + d0];
    const uint32_t incl = (uint32_t)warp_incl_scan((int)hd);
    if (lane == 31) wtot[w] = incl;
    __syncthreads();
    uint32_t dbase = incl - hd;
#pragma unroll
    for (int q = 0; q < kRsWarps; ++q) dbase += q < w ? wtot[q] : 0u;
    const int tile = s_tile;
    auto offsets = [&](int d, uint32_t cnt) -> uint32_t {
        uint32_t *st = state + (size_t)tile * 256 + d;
        if (tile == 0) {
            st_word(st, kOsIncl | cnt);
            return dbase;
        }
        st_word(st, kOsAgg | cnt);
        uint32_t excl = 0;
        int j = tile - 1, spins = 0;
        while (j >= 0) {
            uint32_t v[kOsBatch];
#pragma unroll
            for (int q = 0; q < kOsBatch; ++q)
                v[q] = j - q >= 0 ? ld_word(state + (size_t)(j - q) * 256 + d) : kOsIncl;
            // take the published words nearest first, up to an inclusive one
            int used = 0;
            bool done = false, open = true;
#pragma unroll
            for (int q = 0; q < kOsBatch; ++q) {
                open = open && !done && (v[q] & ~kOsMask) != 0u;
                if (open) {
                    excl += v[q] & kOsMask;
                    done = (v[q] & ~kOsMask) == kOsIncl;
                    ++used;
                }
            }
            if (done) break;
            j -= used;
            if (used == 0) {
                if (++spins > kOsMaxSpin) {
                    atomicOr(status, SPH3_STATUS_SORT);
                    break;
                }
                __nanosleep(20);
            }
        }
        st_word(st, kOsIncl | (excl + cnt));
        return dbase + excl;
    };
    rs_scatter_tile<ITEMS>(key_in, val_in, key_out, val_out, n, 8 * pass, tile, offsets);
}

// ---- rank sort (up to kRankMax keys)
// rank(i) = #{j : key_j < key_i, or key_j = key_i and j < i}, by comparing
// every pair: n^2 compares spread over the whole chip are cheaper than six
// dependent digit passes of a few tiles each.  A block ranks 32 keys; its
// warps take chunks of 256 sources, eight per lane in registers, and run them
// against the 32 targets, whose thresholds are broadcast from shared memory
// and whose counts stay in registers (a target per lane and the sources
// broadcast took 55 us against 45 at 16,000 keys).  The tie rule needs j < i
// only in the chunk that holds the block's own keys; elsewhere the threshold
// is key_i + 1 (earlier keys) or key_i (later ones).
// Bound: the compares.  Keys of at most 62 bits are, as bit patterns, finite
// non-negative doubles and order as the integers do: one FP64 compare a pair
// where a 64-bit integer compare takes two instructions (61 us at 16,000).
// The padding is a NaN, below nothing.
// 2,000 keys: 6 us, against 7 launches and 45 us in one-sweep passes; 10,000:
// 25 against 50; 16,000: 45 against 52; 24,000: 91 against 53.
constexpr int kRankThreads = 256;
constexpr int kRankPer = 8;  // sources per lane and chunk

__device__ __forceinline__ double as_f64(uint64_t k) { return __longlong_as_double((long long)k); }

__global__ void __launch_bounds__(kRankThreads) k_rank_sort(const uint64_t *__restrict__ key_in, int n,
                                                            uint64_t *__restrict__ key_out,
                                                            uint32_t *__restrict__ perm_out) {
    __shared__ double thr[2][32];  // key_i, key_i + 1
    __shared__ int part[kRankThreads / 32][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int b0 = blockIdx.x * 32;
    if (w == 0) {
        const uint64_t ki = b0 + lane < n ? key_in[b0 + lane] : 0ull;
        thr[0][lane] = as_f64(ki);
        thr[1][lane] = as_f64(ki + 1ull);
    }
    __syncthreads();
    int cnt[32];
#pragma unroll
    for (int t = 0; t < 32; ++t) cnt[t] = 0;
    for (int j0 = w * 32 * kRankPer; j0 < n; j0 += kRankThreads * kRankPer) {
        double v[kRankPer];
#pragma unroll
        for (int q = 0; q < kRankPer; ++q) {
            const int j = j0 + 32 * q + lane;
            v[q] = as_f64(j < n ? key_in[j] : ~0ull);
        }
        if (j0 <= b0 && b0 < j0 + 32 * kRankPer) {  // the chunk with the block's own keys
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                const double lo = thr[0][t], hi = thr[1][t];
#pragma unroll
                for (int q = 0; q < kRankPer; ++q) cnt[t] += v[q] < (j0 + 32 * q + lane < b0 + t ? hi : lo);
            }
        } else {
            const double *th = thr[j0 < b0 ? 1 : 0];
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                const double x = th[t];
#pragma unroll
                for (int q = 0; q < kRankPer; ++q) cnt[t] += v[q] < x;
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 32; ++t) {
        const int s = __reduce_add_sync(kFull, cnt[t]);
        if (lane == 0) part[w][t] = s;
    }
    __syncthreads();
    if (w == 0 && b0 + lane < n) {
        int r = 0;
#pragma unroll
        for (int q = 0; q < kRankThreads / 32; ++q) r += part[q][lane];
        key_out[r] = key_in[b0 + lane];
        perm_out[r] = (uint32_t)(b0 + lane);
    }
}

// Which way a set of n keys is sorted, and whether its unsorted keys start in
// the alternate buffers, so that the sorted ones always end in key/perm.
static bool sort_by_rank(const State &S) { return S.n <= kRankMax && S.key_bits <= 62; }
// Keys per thread of the radix tiles: few enough that a pass has tiles for
// most SMs, since one tile's chain of loads, ballots and scatter is what a pass
// of a small set waits for (17 us with one 4096-key tile, 8 with 1024; at
// 1,048,576 keys 30 us with 4096-key tiles, 23 with 2048).
static int sort_items(int64_t n) { return n <= kSortItems4 ? 4 : (n <= kSortItems8 ? 8 : 16); }
static bool keys_start_in_alt(const State &S) {
    return S.n > 1 && (sort_by_rank(S) || ((S.key_bits + 7) / 8) % 2 != 0);
}

void launch_radix_sort(State &S, cudaStream_t st) {
    if (S.n <= 1) return;
    if (sort_by_rank(S)) {
        k_rank_sort<<<(int)((S.n + 31) / 32), kRankThreads, 0, st>>>(S.key_alt, (int)S.n, S.key, S.perm);
        return;
    }
    const int items = sort_items(S.n);
    const int nb = (int)((S.n + kRsThreads * items - 1) / (kRsThreads * items));
    const int passes = (S.key_bits + 7) / 8;
    uint64_t *kin = S.key, *kout = S.key_alt;
    uint32_t *vin = S.perm, *vout = S.perm_alt;
    if (keys_start_in_alt(S)) {
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    // scratch: all passes' histograms, the tile counters, the look-back words
    uint32_t *hist_all = S.sort_hist;
    int *tile_ctr = reinterpret_cast<int *>(S.sort_hist + kMaxPasses * 256);
    uint32_t *state = S.sort_hist + kMaxPasses * 256 + 64;
    cudaMemsetAsync(S.sort_hist, 0, sizeof(uint32_t) * ((size_t)kMaxPasses * 256 + 64 + (size_t)passes * nb * 256), st);
    const int hblocks = (int)std::min<int64_t>((S.n + 1023) / 1024, (int64_t)S.num_sms * 4);
    k_rs_hist_all<<<hblocks, kHaThreads, 0, st>>>(kin, S.n, passes, hist_all);
    auto *sweep = items == 4 ? k_rs_onesweep<4> : (items == 8 ? k_rs_onesweep<8> : k_rs_onesweep<16>);
    for (int p = 0; p < passes; ++p) {
        sweep<<<nb, kRsThreads, 0, st>>>(kin, vin, kout, vout, S.n, p, hist_all, state + (size_t)p * nb * 256,
                                         tile_ctr, S.status);
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
}

size_t sort_scratch_words(int64_t n) {
    // the smallest tile of the size's range bounds the number of tiles
    const int64_t tile = (int64_t)kRsThreads * sort_items(n);
    return (size_t)kMaxPasses * 256 + 64 + (size_t)kMaxPasses * 256 * (size_t)((n + tile - 1) / tile + 1);
}

// ------------------------------------------------------------ gather
constexpr int kMaxGather = 40;
struct GatherArgs {
    const double *src[kMaxGather];
    double *dst[kMaxGather];
    int nf;
};

__global__ void k_gather(const uint32_t *perm, GatherArgs a, int64_t n) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t j = perm[k];
        for (int f = 0; f < a.nf; ++f) a.dst[f][k] = a.src[f][j];
    }
}

void launch_gather(State &S, const double *const *src, double *const *dst, int nfields,
                   const int *ncomp, cudaStream_t st) {
    if (S.n == 0) return;
    GatherArgs a;
    a.nf = 0;
    for (int f = 0; f < nfields; ++f) {
        for (int c = 0; c < ncomp[f]; ++c) {
            if (a.nf == kMaxGather) {
                int blocks = (int)std::min<int64_t>((S.n + 255) / 256, (int64_t)S.num_sms * 8);
                k_gather<<<blocks, 256, 0, st>>>(S.perm, a, S.n);
                a.nf = 0;
            }
            a.src[a.nf] = src[f] + (int64_t)c * S.n;
            a.dst[a.nf] = dst[f] + (int64_t)c * S.n;
            ++a.nf;
        }
    }
    if (a.nf) {
        int blocks = (int)std::min<int64_t>((S.n + 255) / 256, (int64_t)S.num_sms * 8);
        k_gather<<<blocks, 256, 0, st>>>(S.perm, a, S.n);
    }
}

// ------------------------------------------------------------ packs
// The step's gather: the carried fields and the caller's indices in the new
// order, and the packs of positions, {h, m, eps} and velocities from the values
// in hand.  Three launches took 17 us at 2,000 particles and 71 at 1,048,576,
// 4 and 42 now (HBM: 256 B a particle).
constexpr int kCarriedFields = 12;  // pos(3) vel(3) u u_prev dudt_prev m h eps

__global__ void __launch_bounds__(256) k_gather_carried(const uint32_t *perm, const double *src, double *dst,
                                                        const int64_t *orig_in, int64_t *orig_out, int64_t n,
                                                        const Cloud *clouds, const uint64_t *key, int max_level,
                                                        float4 *pk_pos, float4 *pk_hme, float4 *pk_vel) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = perm[k];
        double v[kCarriedFields];
#pragma unroll
        for (int f = 0; f < kCarriedFields; ++f) v[f] = src[f * n + j];
        const int64_t o = orig_in[j];
        const Cloud &cl = clouds[(int)(key[k] >> (3 * max_level))];
#pragma unroll
        for (int f = 0; f < kCarriedFields; ++f) dst[f * n + k] = v[f];
        orig_out[k] = o;
        const CellRel r = make_cellrel(v[0], v[1], v[2], cl);
        pk_pos[k] = make_float4(r.ox, r.oy, r.oz, __int_as_float(r.cell));
        pk_vel[k] = make_float4((float)v[3], (float)v[4], (float)v[5], 0.f);
        pk_hme[k] = make_float4((float)v[10], (float)v[9], (float)v[11], 0.f);
    }
}

void launch_gather_carried(State &S, const double *src, double *dst, const int64_t *orig_in, int64_t *orig_out,
                           cudaStream_t st) {
    if (S.n == 0) return;
    const int blocks = (int)std::min<int64_t>((S.n + 255) / 256, (int64_t)S.num_sms * 8);
    k_gather_carried<<<blocks, 256, 0, st>>>(S.perm, src, dst, orig_in, orig_out, S.n, S.clouds, S.key, S.max_level,
                                             S.pk_pos, S.pk_hme, S.pk_vel);
}

__global__ void k_pack(int64_t n, const double *vel, const double *h, const double *m, const double *eps,
                       const double *rho, const double *P, const double *c, const double *bal, float4 *pk_hme,
                       float4 *pk_vel, float4 *pk_thm, unsigned which) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        if (which & kPackHme) pk_hme[k] = make_float4((float)h[k], (float)m[k], (float)eps[k], 0.f);
        if (which & kPackVel)
            pk_vel[k] = make_float4((float)vel[k], (float)vel[n + k], (float)vel[2 * n + k], 0.f);
        if (which & kPackThm) {
            double r = rho[k];
            double pr = r > 0.0 ? P[k] / (r * r) : 0.0;
            pk_thm[k] = make_float4((float)r, (float)pr, (float)c[k], (float)bal[k]);
        }
    }
}

void launch_pack(State &S, const Params &P, unsigned which, cudaStream_t st) {
    if (S.n == 0 || which == 0) return;
    (void)P;
    int blocks = (int)std::min<int64_t>((S.n + 255) / 256, (int64_t)S.num_sms * 8);
    k_pack<<<blocks, 256, 0, st>>>(S.n, S.vel, S.h, S.m, S.eps, S.rho, S.P, S.c, S.bal, S.pk_hme, S.pk_vel, S.pk_thm,
                                   which);
}

}  // namespace sph3
