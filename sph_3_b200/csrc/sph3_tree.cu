// Linear octree from Morton-sorted keys, built in two launches, then moments
// bottom-up.
//
// A node is a contiguous run [first, first + count) of sorted particles whose
// keys share a common prefix; its level is the deepest level whose cell holds
// the whole run.  A node with more than leaf_size particles (and level below
// max_level) is split on the next 3-bit digit into its 2..8 non-empty
// sub-runs.  Single-child chains never appear, so nodes < 2 * particles.
//
// Every node but a root starts at a particle s and is a child of a split node
// of some level p ("plane" p holds the children of the level-p nodes).  Which
// planes have a node starting at s follows from the keys around s alone, so
// the first launch (k_tree_topo) finds all nodes of all depths at once: one
// bit per particle and plane, and the number of earlier bits of every plane
// per 32 particles.  A node's index is its plane's start plus its rank in the
// plane, so the children of a node are contiguous, planes follow one another
// (a node's children lie in a later plane than the node), and the layout, and
// every sum over it, is deterministic; the second launch (k_tree_emit) writes
// the nodes.
// Compared with the reference's pointer octree (bh_tree_iteration_v2.h:149-450:
// one block, atomicCAS locks, a DFS sort that spins on its parent) there are
// no locks and no waits.
#include <algorithm>
#include <cfloat>

#include "sph3_internal.cuh"

namespace sph3 {

__device__ __forceinline__ int common_level(uint64_t a, uint64_t b, int max_level) {
    uint64_t x = a ^ b;
    if (x == 0) return max_level;
    int hb = 63 - __clzll((long long)x);
    return max_level - 1 - hb / 3;
}

// ------------------------------------------------------------ topology
constexpr int kTopoThreads = 512;              // particles per tile of the topology pass
constexpr int kTopoWords = kTopoThreads / 32;
constexpr int kTopoHalo = 64;                  // keys staged on either side of a tile (leaf_size <= 64)
// nodes that can start inside one tile: at most one leaf and one internal node
// per particle, one more internal node per level whose run crosses the tile's
// end, and the roots
constexpr int kTopoNodes = 2 * kTopoThreads + 64;
constexpr int kTopoScan = 8;

struct TopoArgs {
    const uint64_t *key;
    int n;
    const Cloud *clouds;
    int ncloud;
    int leaf_size, max_level;
    int nwords;  // 32-particle words, n / 32 + 1
    int ntiles;
    unsigned *status;
    unsigned long long *counters;
};

// The topology pass.  Particle s starts nodes if it is a cloud's first
// particle (then also the root), or if the smallest cell holding s - 1 and s
// (level p) has more than leaf_size particles.  The first node at s is then the
// child of that cell; it is followed by its own first child, and so on down to a
// leaf.  A first node that is a leaf (nearly all) is settled from the staged
// keys; otherwise the warp searches the ends of the runs of all deeper levels
// together, a lane per level, doubling the distance and then bisecting.
// The ranks of a plane are counted inside the tile here; the last tile to
// finish turns the tiles' counts into prefixes (no tile waits for another).
// Bound: latency of the searches.  This launch and k_tree_emit replaced one
// launch per level, each waiting on the last (17 launches, 75 us at 2,000
// particles, 228 us at 1,048,576; now 16 and 66 us for
// the two).
__global__ void __launch_bounds__(kTopoThreads) k_tree_topo(Tree T, TopoArgs A) {
    __shared__ uint64_t sk[kTopoThreads + 2 * kTopoHalo + 1];
    __shared__ uint32_t sbits[kTopoWords][kTreePlanes];
    __shared__ int s_end[kTopoNodes];
    __shared__ uint32_t s_node[kTopoNodes];  // start in the tile | plane + 1 << 16 | level << 24
    __shared__ uint32_t s_mask[kTopoThreads];   // planes with a node starting at the particle
    __shared__ uint32_t s_heavy[kTopoThreads];  // particle in the tile | level of the split cell << 16
    __shared__ int s_cnt, s_base, s_last, s_nheavy;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int L = A.max_level, leaf = A.leaf_size, n = A.n;
    const uint64_t *key = A.key;
    if (threadIdx.x == 0) s_cnt = s_nheavy = 0;
    const int tile = blockIdx.x;
    const int s0 = tile * kTopoThreads;
    // keys outside the set read as ~0, in no cell of any (63-bit) key
    for (int i = threadIdx.x; i < kTopoThreads + 2 * kTopoHalo + 1; i += kTopoThreads) {
        const int j = s0 - kTopoHalo + i;
        sk[i] = j >= 0 && j < n ? key[j] : ~0ull;
    }
    __syncthreads();
    const int s = s0 + (int)threadIdx.x, at = kTopoHalo + (int)threadIdx.x;
    const uint64_t k = sk[at], prev = sk[at - 1];
    auto push = [&](int x, int plane, int end, int lvl) {
        const int q = atomicAdd(&s_cnt, 1);
        if (q < kTopoNodes) {
            s_end[q] = end;
            s_node[q] = (uint32_t)x | ((uint32_t)(plane + 1) << 16) | ((uint32_t)lvl << 24);
        }
    };
    unsigned mask = 0;
    int p = 0;
    bool go = false;
    if (s < n) {
        if ((k >> (3 * L)) != (prev >> (3 * L))) {  // a cloud's first particle: its root
            const int e = (int)A.clouds[(int)(k >> (3 * L))].end;
            p = common_level(k, key[e - 1], L);
            push(threadIdx.x, -1, e, p);
            go = e - s > leaf && p < L;
        } else {
            p = common_level(prev, k, L);
            if (p < L) {
                const int sh = 3 * (L - p);
                const uint64_t c = k >> sh;
                go = (sk[at - leaf] >> sh) == c || (sk[at + leaf] >> sh) == c;
                if (!go) {  // count the cell's particles on either side
                    int lo = at - leaf, hi = at - 1;  // sk[lo] outside, sk[hi] inside
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if ((sk[mid] >> sh) == c) hi = mid;
                        else lo = mid;
                    }
                    int in = at, out = at + leaf;
                    while (out - in > 1) {
                        const int mid = (in + out) >> 1;
                        if ((sk[mid] >> sh) == c) in = mid;
                        else out = mid;
                    }
                    go = out - hi > leaf;
                }
            }
        }
    }
    if (go) {
        const int sh = 3 * (L - p - 1);
        const uint64_t c = k >> sh;
        if ((sk[at + leaf] >> sh) == c) {
            s_heavy[atomicAdd(&s_nheavy, 1)] = threadIdx.x | ((uint32_t)p << 16);
        } else {  // a leaf of the split cell
            int in = at, out = at + leaf;
            while (out - in > 1) {
                const int mid = (in + out) >> 1;
                if ((sk[mid] >> sh) == c) in = mid;
                else out = mid;
            }
            mask = 1u << p;
            push(threadIdx.x, p, s0 - kTopoHalo + out, common_level(k, sk[in], L));
        }
    }
    s_mask[threadIdx.x] = mask;
    __syncthreads();
    // particles whose first node is split further, dealt out to the warps
    for (int t = w; t < s_nheavy; t += kTopoThreads / 32) {
        const int x0 = (int)(s_heavy[t] & 0xffffu), ps = (int)(s_heavy[t] >> 16);
        const int ss = s0 + x0;
        const uint64_t kq = sk[kTopoHalo + x0];
        const int lv = ps + 1 + lane;  // this lane's level
        const int sh = lv <= L ? 3 * (L - lv) : 0;
        const uint64_t c = kq >> sh;
        int e = ss + 1, lvl = L;
        if (lv <= L) {
            int in = ss, d = leaf;  // key[in] inside the run
            while (ss + d < n && (key[ss + d] >> sh) == c) {
                in = ss + d;
                d *= 2;
            }
            int out = min(ss + d, n);
            while (out - in > 1) {
                const int mid = (in + out) >> 1;
                if ((key[mid] >> sh) == c) in = mid;
                else out = mid;
            }
            e = out;
            lvl = common_level(kq, key[in], L);
        }
        unsigned chain = 0;
        for (int q = ps;;) {
            const int x = q - ps;  // the lane of level q + 1
            const int eq = __shfl_sync(kFull, e, x), lq = __shfl_sync(kFull, lvl, x);
            chain |= 1u << q;
            if (lane == x) push(x0, q, e, lvl);
            if (eq - ss > leaf && lq < L) q = lq;
            else break;
        }
        if (lane == 0) s_mask[x0] = chain;
    }
    __syncthreads();
    mask = s_mask[threadIdx.x];
    for (int q = 0; q < L; ++q) {
        const unsigned b = __ballot_sync(kFull, (mask >> q) & 1u);
        if (lane == 0) sbits[w][q] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_cnt > kTopoNodes) {  // cannot happen, see kTopoNodes
            atomicOr(A.status, SPH3_STATUS_TREE_CAPACITY);
            s_cnt = kTopoNodes;
        }
        s_base = atomicAdd(T.lvl + 1, s_cnt);
    }
    __syncthreads();
    // the tile's nodes, in any order, for k_tree_emit
    int4 *tmp = reinterpret_cast<int4 *>(T.box_c);
    for (int q = threadIdx.x; q < s_cnt; q += kTopoThreads) {
        const uint32_t v = s_node[q];
        const int first = s0 + (int)(v & 0xffffu);
        if (s_base + q < T.cap) tmp[s_base + q] = make_int4(first, s_end[q], (int)((v >> 16) & 255u) - 1, (int)(v >> 24));
    }
    // ranks inside the tile and the tile's counts: a warp per plane
    for (int q = w; q < L; q += kTopoThreads / 32) {
        const unsigned b = lane < kTopoWords ? sbits[lane][q] : 0u;
        const int incl = warp_incl_scan(__popc(b));
        const int word = tile * kTopoWords + lane;
        if (lane < kTopoWords && word < A.nwords) {
            T.plane_bits[(size_t)q * A.nwords + word] = b;
            T.plane_rank[(size_t)q * A.nwords + word] = incl - __popc(b);
        }
        if (lane == 31) T.tile_rank[(size_t)q * (A.ntiles + 1) + tile] = incl;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(T.lvl, 1) == A.ntiles - 1;
    __syncthreads();
    if (!s_last) return;
    // the last tile: exclusive prefixes of the tiles' counts, a warp per plane,
    // kTopoScan chunks of 32 tiles in flight
    __threadfence();
    for (int q = w; q < L; q += kTopoThreads / 32) {
        int *cnt = T.tile_rank + (size_t)q * (A.ntiles + 1);
        int run = 0;
        for (int t0 = 0; t0 < A.ntiles; t0 += 32 * kTopoScan) {
            int v[kTopoScan];
#pragma unroll
            for (int x = 0; x < kTopoScan; ++x) {
                const int t = t0 + 32 * x + lane;
                v[x] = t < A.ntiles ? __ldcg(cnt + t) : 0;
            }
#pragma unroll
            for (int x = 0; x < kTopoScan; ++x) {
                const int t = t0 + 32 * x + lane;
                const int incl = warp_incl_scan(v[x]);
                if (t < A.ntiles) cnt[t] = run + incl - v[x];
                run += __shfl_sync(kFull, incl, 31);
            }
        }
        if (lane == 0) {
            cnt[A.ntiles] = run;
            if (A.ntiles * kTopoWords < A.nwords) {  // n a multiple of the tile: the word past the end
                T.plane_bits[(size_t)q * A.nwords + A.nwords - 1] = 0u;
                T.plane_rank[(size_t)q * A.nwords + A.nwords - 1] = 0;
            }
        }
    }
}

// Writes the nodes: a thread per node of the list, its index and its
// children's from the plane ranks.  Also the plane starts (depth_begin: the
// roots, then one plane after another) and the node and leaf counters.
__global__ void __launch_bounds__(256) k_tree_emit(Tree T, TopoArgs A) {
    __shared__ int s_plane[kTreePlanes + 1];
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        const int t = lane < A.max_level ? T.tile_rank[(size_t)lane * (A.ntiles + 1) + A.ntiles] : 0;
        const int incl = warp_incl_scan(t);
        if (lane <= A.max_level) s_plane[lane] = A.ncloud + incl - t;  // s_plane[max_level]: the node count
    }
    __syncthreads();
    const int L = A.max_level;
    const int nlist = T.lvl[1];
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            T.depth_begin[0] = 0;
            T.depth_begin[L + 2] = s_plane[L];
            A.counters[6] = (unsigned long long)s_plane[L];
        }
        if (threadIdx.x <= L) T.depth_begin[1 + threadIdx.x] = s_plane[threadIdx.x];
    }
    auto rank = [&](int plane, int x) {
        const size_t q = (size_t)plane * A.nwords + (x >> 5);
        return T.tile_rank[(size_t)plane * (A.ntiles + 1) + x / kTopoThreads] + T.plane_rank[q] +
               __popc(T.plane_bits[q] & ((1u << (x & 31)) - 1u));
    };
    unsigned long long leaves = 0;
    const int4 *tmp = reinterpret_cast<const int4 *>(T.box_c);
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, dt = gridDim.x * blockDim.x;
    for (int t = t0; t < nlist; t += dt) {
        const int4 v = tmp[t];  // {first, end, plane, level}
        const int id = v.z < 0 ? (int)(A.key[v.x] >> (3 * L)) : s_plane[v.z] + rank(v.z, v.x);
        int cf = -1, nch = 0;
        if (v.y - v.x > A.leaf_size && v.w < L) {
            const int r0 = rank(v.w, v.x);
            cf = s_plane[v.w] + r0;
            nch = rank(v.w, v.y) - r0;
        }
        T.range[id] = make_int2(v.x, v.y - v.x);
        T.child[id] = make_int2(cf, nch | (v.w << 8));
        for (int c = 0; c < nch; ++c) T.parent[cf + c] = id;
        if (v.z < 0) T.parent[id] = -1;
        leaves += nch == 0;
    }
    for (int c = t0; c < A.ncloud; c += dt) {
        const Cloud &cl = A.clouds[c];
        if (cl.end > cl.begin) continue;
        T.range[c] = make_int2((int)cl.begin, 0);  // an empty cloud's root
        T.child[c] = make_int2(-1, L << 8);
        T.parent[c] = -1;
        ++leaves;
    }
    leaves = warp_sum(leaves);
    if (lane == 0 && leaves) atomicAdd(&A.counters[7], leaves);
}

// ------------------------------------------------------------ moments
struct MomArgs {
    const double *pos, *m, *h, *eps;
    int64_t n;
    const Cloud *clouds;
    const uint64_t *key;
    int max_level;
    double inv_theta;  // 1/theta (inf for theta = 0)
    int mac_offset;    // add the com offset to the opening radius
};

// Four threads per node: a leaf's particles and an internal node's children
// are shared out round-robin and the partial sums (FP64), minima and maxima
// are combined with two shuffles, so a warp reads eight nodes' particle runs
// four consecutive entries at a time.  The combination order is fixed, so the
// moments are deterministic.
__device__ __forceinline__ void node_moments(const Tree &T, const MomArgs &a, int i, int2 r, int2 ch, int quad) {
    const int cap = T.cap;
    const int64_t n = a.n;
    const int qt = threadIdx.x & 3;
    const unsigned qmask = 0xFu << (threadIdx.x & 28);
    auto qsum = [&](double v) {
        v += __shfl_xor_sync(qmask, v, 1);
        return v + __shfl_xor_sync(qmask, v, 2);
    };
    auto qmin = [&](double v) {
        v = fmin(v, __shfl_xor_sync(qmask, v, 1));
        return fmin(v, __shfl_xor_sync(qmask, v, 2));
    };
    auto qmax = [&](double v) {
        v = fmax(v, __shfl_xor_sync(qmask, v, 1));
        return fmax(v, __shfl_xor_sync(qmask, v, 2));
    };
    const int nch = ch.y & 255;
    double M = 0, sx = 0, sy = 0, sz = 0;
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    double hm = 0, em = 0;
    double cm[2], cc[2][3], cq[2][6];  // the (at most two) children of this thread
    if (nch == 0) {
#pragma unroll 4
        for (int k = r.x + qt; k < r.x + r.y; k += 4) {
            const double mk = a.m[k];
            const double x = a.pos[k], y = a.pos[n + k], z = a.pos[2 * n + k];
            M += mk;
            sx += mk * x;
            sy += mk * y;
            sz += mk * z;
            lo[0] = fmin(lo[0], x); hi[0] = fmax(hi[0], x);
            lo[1] = fmin(lo[1], y); hi[1] = fmax(hi[1], y);
            lo[2] = fmin(lo[2], z); hi[2] = fmax(hi[2], z);
            hm = fmax(hm, a.h[k]);
            em = fmax(em, a.eps[k]);
        }
    } else {
        // fixed trip count with a guard: the loads of all children are
        // issued together (a node has at most 8), same summation order
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (qt + 4 * q >= nch) continue;
            const int c = ch.x + qt + 4 * q;
            cm[q] = __ldcg(T.mass + c);
            cc[q][0] = __ldcg(T.com + c);
            cc[q][1] = __ldcg(T.com + cap + c);
            cc[q][2] = __ldcg(T.com + 2 * cap + c);
            if (quad)
                for (int k = 0; k < 6; ++k) cq[q][k] = __ldcg(T.quad + (size_t)k * cap + c);
            for (int k = 0; k < 3; ++k) {
                lo[k] = fmin(lo[k], __ldcg(T.bmin + k * cap + c));
                hi[k] = fmax(hi[k], __ldcg(T.bmax + k * cap + c));
            }
            hm = fmax(hm, __ldcg(T.hmax + c));
            em = fmax(em, __ldcg(T.epsmax + c));
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (qt + 4 * q >= nch) continue;
            M += cm[q];
            sx += cm[q] * cc[q][0];
            sy += cm[q] * cc[q][1];
            sz += cm[q] * cc[q][2];
        }
    }
    M = qsum(M);
    sx = qsum(sx);
    sy = qsum(sy);
    sz = qsum(sz);
    for (int q = 0; q < 3; ++q) {
        lo[q] = qmin(lo[q]);
        hi[q] = qmax(hi[q]);
    }
    hm = qmax(hm);
    em = qmax(em);
    if (r.y == 0) {
        lo[0] = lo[1] = lo[2] = 0.0;
        hi[0] = hi[1] = hi[2] = 0.0;
    }
    double cx, cy, cz;
    if (M > 0) {
        cx = sx / M; cy = sy / M; cz = sz / M;
    } else {
        cx = 0.5 * (lo[0] + hi[0]); cy = 0.5 * (lo[1] + hi[1]); cz = 0.5 * (lo[2] + hi[2]);
    }
    if (qt == 0) {
        T.mass[i] = M;
        T.com[i] = cx; T.com[cap + i] = cy; T.com[2 * cap + i] = cz;
        for (int q = 0; q < 3; ++q) {
            T.bmin[q * cap + i] = lo[q];
            T.bmax[q * cap + i] = hi[q];
        }
        T.hmax[i] = hm;
        T.epsmax[i] = em;
    }
    double Q[6] = {0, 0, 0, 0, 0, 0};
    if (quad) {
        if (nch == 0) {
#pragma unroll 4
            for (int k = r.x + qt; k < r.x + r.y; k += 4) {
                const double mk = a.m[k];
                const double dx = a.pos[k] - cx, dy = a.pos[n + k] - cy, dz = a.pos[2 * n + k] - cz;
                const double d2 = dx * dx + dy * dy + dz * dz;
                Q[0] += mk * (3 * dx * dx - d2);
                Q[1] += mk * (3 * dx * dy);
                Q[2] += mk * (3 * dx * dz);
                Q[3] += mk * (3 * dy * dy - d2);
                Q[4] += mk * (3 * dy * dz);
                Q[5] += mk * (3 * dz * dz - d2);
            }
        } else {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (qt + 4 * q >= nch) continue;
                const double mc = cm[q];
                const double dx = cc[q][0] - cx, dy = cc[q][1] - cy, dz = cc[q][2] - cz;
                const double d2 = dx * dx + dy * dy + dz * dz;
                Q[0] += cq[q][0] + mc * (3 * dx * dx - d2);
                Q[1] += cq[q][1] + mc * (3 * dx * dy);
                Q[2] += cq[q][2] + mc * (3 * dx * dz);
                Q[3] += cq[q][3] + mc * (3 * dy * dy - d2);
                Q[4] += cq[q][4] + mc * (3 * dy * dz);
                Q[5] += cq[q][5] + mc * (3 * dz * dz - d2);
            }
        }
    }
    for (int q = 0; q < 6; ++q) Q[q] = qsum(Q[q]);
    if (qt == 0)  // one thread of the four writes the node
        for (int q = 0; q < 6; ++q) T.quad[q * cap + i] = Q[q];
}

// Last-arrival climb: after finishing node c, a thread counts itself in at
// c's parent p (with nch children); the thread that completes the count (all
// the children's results are written and fenced) goes on with the parent.  No
// thread ever waits, and each internal node is done exactly once.  The counter
// is put back to zero for the next pass.  The parent's record is read by the
// caller before c's own work, so that a climb step waits on one atomic only.
__device__ __forceinline__ bool arrive_last(const Tree &T, int p, int nch) {
    __threadfence();
    if (atomicAdd(T.arrive + p, 1) != nch - 1) return false;
    __threadfence();
    T.arrive[p] = 0;
    return true;
}

// climbs from node i (its four threads) while its parents' counts complete
__device__ __forceinline__ void moments_up(const Tree &T, const MomArgs &a, int i, int max_depth, int quad) {
    const unsigned qmask = 0xFu << (threadIdx.x & 28);
    int2 r = T.range[i], ch = T.child[i];
    for (int up = 0; up < max_depth; ++up) {
        const int p = T.parent[i];
        const int2 rp = p >= 0 ? T.range[p] : make_int2(0, 0), cp = p >= 0 ? T.child[p] : make_int2(0, 0);
        node_moments(T, a, i, r, ch, quad);
        int last = 0;
        if (p >= 0 && (threadIdx.x & 3) == 0) last = arrive_last(T, p, cp.y & 255);
        if (!__shfl_sync(qmask, last, 0, 4)) break;
        __syncwarp(qmask);
        i = p;
        r = rp;
        ch = cp;
    }
}

// Moments in one launch (up to kClimbMax particles): four threads per leaf,
// then up the last-arrival chain.  Children are read through L2, where other
// threads of the launch wrote them.
// Larger sets take two launches: here the leaves only, the thread that
// completes a parent made of leaves noting it in `ready`; then
// k_tree_moments_ready climbs from those.  (Climbing from the leaves of a
// large set keeps whole warps waiting on their longest chain: 300 us at
// 1,048,576 particles.)
__global__ void __launch_bounds__(128) k_tree_moments_leaves(Tree T, MomArgs a, int max_depth, int quad, int *ready) {
    const int nn = T.depth_begin[max_depth];
    for (int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 2); i < nn;
         i += (int)((gridDim.x * blockDim.x) >> 2)) {
        const int2 ch = T.child[i];
        if ((ch.y & 255) != 0) continue;
        if (!ready) {
            moments_up(T, a, i, max_depth, quad);
            continue;
        }
        const int p = T.parent[i];
        const int np = p >= 0 ? T.child[p].y & 255 : 0;
        node_moments(T, a, i, T.range[i], ch, quad);
        if (p >= 0 && (threadIdx.x & 3) == 0 && arrive_last(T, p, np)) ready[atomicAdd(T.lvl + 2, 1)] = p;
    }
}

// the internal nodes, from the noted parents of leaves up
__global__ void __launch_bounds__(128) k_tree_moments_ready(Tree T, MomArgs a, int max_depth, int quad,
                                                            const int *ready) {
    const int nr = T.lvl[2];
    for (int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 2); i < nr;
         i += (int)((gridDim.x * blockDim.x) >> 2))
        moments_up(T, a, ready[i], max_depth, quad);
}

// Node hmax from the current h (after an h search): a leaf from its
// particles, an internal node from its children (read through L2: they were
// written by other threads of the same launch).  With eps = h (eps_from_h)
// the softening maximum and the softening reach r_soft = bmax + eps_max
// follow as well.
__device__ __forceinline__ void node_refit_h(const Tree &T, const double *h, int i, int2 r, int2 ch, int refit_eps,
                                             const uint64_t *key, const Cloud *clouds, int max_level) {
    const int cap = T.cap;
    const int nch = ch.y & 255;
    double hm = 0;
    if (nch == 0) {
#pragma unroll 4
        for (int k = r.x; k < r.x + r.y; ++k) hm = fmax(hm, h[k]);
    } else {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (q < nch) hm = fmax(hm, __ldcg(T.hmax + ch.x + q));
    }
    T.hmax[i] = hm;
    T.box_h[i].w = (float)(hm * (1.0 + 1e-6));
    T.sw[3 * i + 1].w = (float)(hm * (1.0 + 1e-6));
    if (refit_eps && r.y > 0) {
        T.epsmax[i] = hm;
        const Cloud &cl = clouds[(int)(key[r.x] >> (3 * max_level))];
        const double cx = T.com[i], cy = T.com[cap + i], cz = T.com[2 * cap + i];
        const double ex = fmax(fabs(T.bmax[i] - cx), fabs(cx - T.bmin[i]));
        const double ey = fmax(fabs(T.bmax[cap + i] - cy), fabs(cy - T.bmin[cap + i]));
        const double ez = fmax(fabs(T.bmax[2 * cap + i] - cz), fabs(cz - T.bmin[2 * cap + i]));
        const double bmax = sqrt(ex * ex + ey * ey + ez * ez);
        const float r_soft = (float)fmin((bmax + hm) * (1.0 + 1e-5) + 1e-6 * cl.size, (double)FLT_MAX);
        T.gw[2 * i + 1].y = r_soft;
    }
}

// one launch: a thread per leaf, then up the last-arrival chain (hmax is a
// maximum, so the order in which children finish does not matter)
__global__ void k_tree_refit_h(Tree T, const double *h, int max_depth, int refit_eps, const uint64_t *key,
                               const Cloud *clouds, int max_level) {
    const int nn = T.depth_begin[max_depth];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        int2 ch = T.child[i];
        if ((ch.y & 255) != 0) continue;
        int2 r = T.range[i];
        int c = i;
        for (int up = 0; up < max_depth; ++up) {
            const int p = T.parent[c];
            const int2 rp = p >= 0 ? T.range[p] : make_int2(0, 0), cp = p >= 0 ? T.child[p] : make_int2(0, 0);
            node_refit_h(T, h, c, r, ch, refit_eps, key, clouds, max_level);
            if (p < 0 || !arrive_last(T, p, cp.y & 255)) break;
            c = p;
            r = rp;
            ch = cp;
        }
    }
}

void launch_tree_refit_h(State &S, const Params &P, cudaStream_t st) {
    if (S.ncloud == 0) return;
    k_tree_refit_h<<<S.num_sms * 8, 128, 0, st>>>(S.tree, S.h, S.max_level + 2, P.eps_from_h, S.key, S.clouds,
                                                   S.max_level);
}

// ------------------------------------------------------------ h start guess
// A starting h for the Newton search when none is given: every particle of a
// leaf gets the h at which a sphere of radius 2h would hold n_ngb particles
// at the leaf's number density (its count over its octree cell's volume).
// The search then converges in a few passes; the exact bootstrap of the
// reference (k-th nearest neighbour, k_boot_h) stays for the reference rule.
__global__ void k_h_guess(Tree T, const Cloud *clouds, const uint64_t *key, int max_level, int n_ngb, double *h,
                          float4 *pk_hme) {
    const int nn = T.depth_begin[max_level + 2];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        const int2 r = T.range[i];
        const int2 ch = T.child[i];
        if ((ch.y & 255) != 0 || r.y == 0) continue;  // leaves only
        const Cloud &cl = clouds[(int)(key[r.x] >> (3 * max_level))];
        const int lvl = ch.y >> 8;
        const double side = ldexp(cl.size, -lvl);
        const double dens = (double)r.y / (side * side * side);
        const double hg = 0.5 * cbrt(3.0 * (double)n_ngb / (4.0 * M_PI * dens));
        for (int k = r.x; k < r.x + r.y; ++k) {
            h[k] = hg;
            pk_hme[k].x = (float)hg;
        }
    }
}

void launch_h_guess(State &S, const Params &P, cudaStream_t st) {
    if (S.ncloud == 0 || S.n == 0) return;
    S.list_valid = false;
    k_h_guess<<<S.num_sms * 4, 256, 0, st>>>(S.tree, S.clouds, S.key, S.max_level, P.n_ngb, S.h, S.pk_hme);
}

// ------------------------------------------------------------ walk groups
// Target groups for the walks: runs of at most kGroup consecutive particles
// whose bounding box is small on the scale of their smoothing lengths (a
// walk's work grows with (group extent + 2h)^3, so one sprawling group can
// stall a whole persistent kernel).
//
// A node is *compact* if it holds <= kGroup particles and its bbox extent is
// at most kGroupSpan * hmax (or it holds one particle, or no h is known yet).
// Every non-compact internal node acts as a parent: it packs its consecutive
// compact children greedily into groups while the merged bbox stays within
// kGroupSpan * (largest hmax) and the count within kGroup; a non-compact leaf
// child is split into kGroup-sized chunks if it is only too populous, or into
// one group per particle if it is sprawling.  A compact root is one group.
// Every particle lands in exactly one group: the first compact node on its
// root-to-leaf chain is packed by its (non-compact) parent, and a chain
// without one ends in a non-compact leaf that its parent splits.  The order
// of the group table does not affect any result.
constexpr double kGroupSpan = 4.0;

__device__ __forceinline__ double node_extent(const Tree &T, int i) {
    const int cap = T.cap;
    return fmax(T.bmax[i] - T.bmin[i],
                fmax(T.bmax[cap + i] - T.bmin[cap + i], T.bmax[2 * cap + i] - T.bmin[2 * cap + i]));
}

// length scale of a node: its largest h, or "any size" before h is known
__device__ __forceinline__ double node_scale(const Tree &T, int i) {
    const double h = T.hmax[i];
    return h > 0.0 ? kGroupSpan * h : DBL_MAX;
}

__device__ __forceinline__ bool compact_node(const Tree &T, int i) {
    const int cnt = T.range[i].y;
    return cnt <= kGroup && (cnt == 1 || node_extent(T, i) <= node_scale(T, i));
}

// groups of a leaf that is not compact: kGroup-sized chunks if it is only too
// populous, one group per particle if it sprawls
__device__ __forceinline__ int split_step(double extent, double scale) { return extent <= scale ? kGroup : 1; }

// FP32 packs of node i for the walks, from its FP64 moments
__device__ __forceinline__ void node_packs(const Tree &T, const MomArgs &a, int i, int2 r, int2 ch) {
    const int cap = T.cap;
    const double M = T.mass[i], cx = T.com[i], cy = T.com[cap + i], cz = T.com[2 * cap + i];
    double lo[3], hi[3], Q[5];
    for (int q = 0; q < 3; ++q) {
        lo[q] = T.bmin[q * cap + i];
        hi[q] = T.bmax[q * cap + i];
    }
    for (int q = 0; q < 5; ++q) Q[q] = T.quad[q * cap + i];
    const double hm = T.hmax[i], em = T.epsmax[i];
    const Cloud &cl = a.clouds[r.y > 0 ? (int)(a.key[r.x] >> (3 * a.max_level)) : 0];
    const double bcx = 0.5 * (lo[0] + hi[0]), bcy = 0.5 * (lo[1] + hi[1]), bcz = 0.5 * (lo[2] + hi[2]);
    const double hx = 0.5 * (hi[0] - lo[0]), hy = 0.5 * (hi[1] - lo[1]), hz = 0.5 * (hi[2] - lo[2]);
    const double pad = 1e-6 * cl.size;
    CellRel b = make_cellrel(bcx, bcy, bcz, cl);
    T.box_c[i] = make_float4(b.ox, b.oy, b.oz, __int_as_float(b.cell));
    T.box_h[i] = make_float4((float)(hx + pad), (float)(hy + pad), (float)(hz + pad),
                             (float)(hm * (1.0 + 1e-6)));
    CellRel cm = make_cellrel(cx, cy, cz, cl);
    const float4 com_c = make_float4(cm.ox, cm.oy, cm.oz, __int_as_float(cm.cell));
    const double ex = fmax(fabs(hi[0] - cx), fabs(cx - lo[0]));
    const double ey = fmax(fabs(hi[1] - cy), fabs(cy - lo[1]));
    const double ez = fmax(fabs(hi[2] - cz), fabs(cz - lo[2]));
    const double bmax = sqrt(ex * ex + ey * ey + ez * ez);
    const double side = 2.0 * fmax(hx, fmax(hy, hz));
    const double delta = sqrt((cx - bcx) * (cx - bcx) + (cy - bcy) * (cy - bcy) + (cz - bcz) * (cz - bcz));
    // s/d < theta (d > s/theta), optionally plus the offset of the centre of
    // mass from the box centre (d > s/theta + delta); theta = 0 never
    // accepts a node (exact sum).  The walks also require d > r_soft
    // (bmax + eps), so an accepted node's particles always lie outside the
    // group's box, whatever theta.
    double r_open = isinf(a.inv_theta) ? (double)FLT_MAX : side * a.inv_theta + (a.mac_offset ? delta : 0.0);
    r_open = fmin(r_open * (1.0 + 1e-5) + pad, (double)FLT_MAX);
    const double r_soft = fmin((bmax + em) * (1.0 + 1e-5) + pad, (double)FLT_MAX);
    T.gn[3 * (size_t)i] = com_c;
    T.gn[3 * (size_t)i + 1] = make_float4((float)M, (float)Q[0], (float)Q[1], (float)Q[2]);
    T.gn[3 * (size_t)i + 2] = make_float4((float)Q[3], (float)Q[4], 0.f, 0.f);
    // walk records: everything one node test needs in one contiguous
    // record, so a walk step is a single round trip to L2
    const int chy = r.y > 0 ? ch.y : -1;  // -1: empty node, never taken
    T.gw[2 * i] = com_c;
    T.gw[2 * i + 1] = make_float4((float)r_open, (float)r_soft, __int_as_float(ch.x), __int_as_float(chy));
    T.sw[3 * i] = T.box_c[i];
    T.sw[3 * i + 1] = T.box_h[i];
    T.sw[3 * i + 2] = make_float4(__int_as_float(ch.x), __int_as_float(chy), __int_as_float(r.y), 0.f);
}

// Walk packs and groups, by blocks of even and odd number.  Packs: a thread
// per node (the moments' four threads would leave three idle).  Groups: a
// warp per eight nodes; those that pack their children are found with a
// ballot and taken four at a time, eight lanes each: a lane reads one child's
// range, box and scale (all reads in flight together), the greedy packing
// then runs over the eight from registers, every lane alike, and each group's
// first lane emits it.  One thread per node reading its children one after
// another took 14 us at 2,000 particles for the groups alone (9 us
// with the packs now).
__global__ void __launch_bounds__(256) k_tree_finish(Tree T, MomArgs a, int ncloud, int max_depth, int2 *groups,
                                                     int *gcl, int *ng) {
    if (blockIdx.x == 0 && threadIdx.x < kLvlCount) T.lvl[threadIdx.x] = 0;  // the build's counters, for the next build
    const int nn = T.depth_begin[max_depth];
    const int cap = T.cap;
    const int lane = threadIdx.x & 31, sub = lane & 7, oct = lane >> 3;
    const int first_thread = (int)((blockIdx.x >> 1) * blockDim.x + threadIdx.x), threads = (int)((gridDim.x >> 1) * blockDim.x);
    if ((blockIdx.x & 1) == 0) {
        for (int i = first_thread; i < nn; i += threads) node_packs(T, a, i, T.range[i], T.child[i]);
        return;
    }
    for (int i0 = (first_thread >> 5) * 8; i0 < nn; i0 += threads >> 2) {
        int2 r = make_int2(0, 0), ch = make_int2(0, 0);
        bool packs = false, ci = false;
        if (lane < 8 && i0 + lane < nn) {
            const int i = i0 + lane;
            r = T.range[i];
            ch = T.child[i];
            // leaves and compact nodes are packed by their parent, a cloud's root by itself
            if (i < ncloud || (ch.y & 255) != 0) ci = compact_node(T, i);
            packs = r.y > 0 && (i < ncloud || (!ci && (ch.y & 255) != 0));
        }
        for (unsigned todo = __ballot_sync(kFull, packs); todo;) {
            // the oct-th packing node left
            unsigned left = todo;
            for (int q = 0; q < oct; ++q) left &= left - 1;
            const int src = left ? __ffs((int)left) - 1 : 0;
            for (int q = 0; q < 4 && todo; ++q) todo &= todo - 1;
            const int i = i0 + src;
            const int rx = __shfl_sync(kFull, r.x, src), ry = __shfl_sync(kFull, r.y, src);
            const int cx = __shfl_sync(kFull, ch.x, src), nch = __shfl_sync(kFull, ch.y, src) & 255;
            const bool own = __shfl_sync(kFull, (int)ci, src) != 0 || nch == 0;
            const int cloud = left ? (int)(a.key[rx] >> (3 * a.max_level)) : 0;
            // the units this node emits: itself (a cloud's root that is compact or a leaf), or its children
            const int units = !left ? 0 : (own ? 1 : nch);
            const int c = own ? i : cx + sub;
            const bool mine = sub < units;
            int2 cr = make_int2(0, 0);
            double lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0}, scale = 0.0, ext = 0.0;
            bool compact = false, leaf = false;
            if (mine) {
                cr = own ? make_int2(rx, ry) : T.range[c];
                leaf = (T.child[c].y & 255) == 0;
                for (int d = 0; d < 3; ++d) {
                    lo[d] = T.bmin[d * cap + c];
                    hi[d] = T.bmax[d * cap + c];
                }
                scale = node_scale(T, c);
                ext = fmax(hi[0] - lo[0], fmax(hi[1] - lo[1], hi[2] - lo[2]));
                compact = cr.y <= kGroup && (cr.y == 1 || ext <= scale);
            }
            // greedy packing of consecutive compact children, the same in every lane of the eight
            int first = -1, count = 0, my_first = -1, my_count = 0, starter = 0;
            double glo[3] = {0, 0, 0}, ghi[3] = {0, 0, 0}, gs = 0.0;
            for (int q = 0; q < 8; ++q) {
                const int qx = __shfl_sync(kFull, cr.x, q, 8), qc = __shfl_sync(kFull, cr.y, q, 8);
                const bool qk = __shfl_sync(kFull, (int)compact, q, 8) != 0;
                double ql[3], qh[3];
                for (int d = 0; d < 3; ++d) {
                    ql[d] = __shfl_sync(kFull, lo[d], q, 8);
                    qh[d] = __shfl_sync(kFull, hi[d], q, 8);
                }
                const double qs = __shfl_sync(kFull, scale, q, 8);
                if (q >= units) continue;
                bool merged = false;
                if (qk && first >= 0 && count + qc <= kGroup) {
                    double e = 0.0;
                    for (int d = 0; d < 3; ++d) e = fmax(e, fmax(ghi[d], qh[d]) - fmin(glo[d], ql[d]));
                    const double sc = fmax(gs, qs);
                    if (e <= sc) {
                        count += qc;
                        for (int d = 0; d < 3; ++d) {
                            glo[d] = fmin(glo[d], ql[d]);
                            ghi[d] = fmax(ghi[d], qh[d]);
                        }
                        gs = sc;
                        merged = true;
                    }
                }
                if (!merged) {
                    first = qk ? qx : -1;
                    count = qk ? qc : 0;
                    starter = q;
                    for (int d = 0; d < 3; ++d) {
                        glo[d] = ql[d];
                        ghi[d] = qh[d];
                    }
                    gs = qs;
                }
                if (qk && sub == starter) {  // the lane of the group's first child holds the group as it grows
                    my_first = first;
                    my_count = count;
                }
            }
            // this lane's groups: the packed one it starts, or the pieces of its non-compact leaf
            int step = kGroup, total = 0;
            if (my_first >= 0) {
                total = my_count;
            } else if (mine && !compact && leaf && cr.y > 0) {
                my_first = cr.x;
                total = cr.y;
                step = split_step(ext, scale);
            }
            if (total > 0) {
                int g = atomicAdd(ng, (total + step - 1) / step);
                for (int f = 0; f < total; f += step, ++g) {
                    groups[g] = make_int2(my_first + f, min(step, total - f));
                    gcl[g] = cloud;
                }
            }
        }
    }
}

// Moments in one launch up to here: 19 us at 2,000 particles, 40 at 100,000
// (19 launches, one per level, took 94 and 115); in two above: 48 us at
// 300,000, 111 at 1,048,576 (a launch per level 162; one launch 300).
constexpr int64_t kClimbMax = 100000;

// tile counts and 32-particle words per plane of n particles' topology pass
size_t topo_tile_words(int64_t n) { return (size_t)kTreePlanes * (size_t)((n + kTopoThreads - 1) / kTopoThreads + 2); }
size_t topo_plane_words(int64_t n) { return (size_t)kTreePlanes * (size_t)(n / 32 + 1); }

void launch_tree_build(State &S, const Params &P, cudaStream_t st) {
    S.list_valid = false;  // a new order invalidates the neighbour lists
    if (S.ncloud == 0) return;
    Tree &T = S.tree;
    const int maxd = S.max_level + 1;  // the roots and max_level planes
    const int blocks = S.num_sms * 4;
    TopoArgs t;
    t.key = S.key;
    t.n = (int)S.n;
    t.clouds = S.clouds;
    t.ncloud = S.ncloud;
    t.leaf_size = P.leaf_size;
    t.max_level = S.max_level;
    t.nwords = (int)(S.n / 32) + 1;
    t.ntiles = std::max(1, (int)((S.n + kTopoThreads - 1) / kTopoThreads));
    t.status = S.status;
    t.counters = S.counters;
    k_tree_topo<<<t.ntiles, kTopoThreads, 0, st>>>(T, t);
    k_tree_emit<<<(int)std::min<int64_t>(blocks, (S.n + 255) / 256 + 1), 256, 0, st>>>(T, t);
    MomArgs a;
    a.pos = S.pos; a.m = S.m; a.h = S.h; a.eps = S.eps; a.n = S.n;
    a.clouds = S.clouds; a.key = S.key; a.max_level = S.max_level;
    a.inv_theta = P.theta > 0 ? 1.0 / P.theta : __builtin_inf();
    a.mac_offset = P.mac == SPH3_MAC_BH_OFFSET;
    const bool two = S.n > kClimbMax;
    int *ready = two ? reinterpret_cast<int *>(S.key_alt) : nullptr;  // free between sorts; at most n / 2 internal nodes
    k_tree_moments_leaves<<<(int)std::min<int64_t>(blocks * 4, S.n / 64 + 1), 128, 0, st>>>(T, a, maxd + 1,
                                                                                           P.quadrupole, ready);
    if (two)
        k_tree_moments_ready<<<(int)std::min<int64_t>(blocks * 4, S.n / 1024 + 1), 128, 0, st>>>(
            T, a, maxd + 1, P.quadrupole, ready);
    cudaMemsetAsync(S.ngroups_dev, 0, sizeof(int), st);
    k_tree_finish<<<2 * (int)std::min<int64_t>(blocks * 2, S.n / 512 + 1), 256, 0, st>>>(
        T, a, S.ncloud, maxd + 1, S.groups, S.group_cloud, S.ngroups_dev);
}

}  // namespace sph3
