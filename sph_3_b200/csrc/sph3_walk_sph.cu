// SPH walks: bootstrap h, h search, density (+ div/curl v, EOS) and the fused
// hydro acceleration + du/dt pass, plus the neighbour-set export used by the
// parity tests.
//
// Every walk is one persistent kernel: warps (in small sets teams of warps) pull
// compact particle groups (<= 32, built from the octree) from an atomic counter,
// walk the octree once per group (sph3_walk.cuh) and stream the candidate leaves
// through a shared-memory tile.  Two instantiations per pass:
//   float  -- mixed precision: positions in the FP32 frame of the group's
//             reference cell (exact integer cell offsets + FP32 in-cell
//             offsets), FP32 kernel arithmetic, FP64 results;
//   double -- the plain FP64 path: absolute FP64 positions and FP64 arithmetic.
//             FP32 distances settle the predicates that are not close; the rest
//             run the reference's own expressions (no FMA contraction in them),
//             so neighbour sets and the reference h rule are bit-exact.
// The kernel formulas follow sph_code/libsx.py (M4 kernel, sigma = 1/pi,
// hbar_ij = (h_i + h_j) / 2, support q <= 2) and sph_code/shear.py.
#include <cfloat>
#include <vector>

#include "sph3_walk.cuh"

namespace sph3 {

constexpr double kSig = 0.31830988618379067154;  // 1/pi
constexpr float kSigF = 0.31830988618379067154f;

// ------------------------------------------------------------ arguments
struct WalkArgs {
    const int2 *groups;
    const int *ngroups_dev;
    const int *group_cloud;
    const Cloud *clouds;
    int ncloud;
    const int2 *range;
    const int2 *child;
    const float4 *box_c;
    const float4 *box_h;
    const float4 *sw;  // walk records [node][3]
    const float4 *pk_pos;
    const double *pos;
    int64_t n;
    int stack_cap;
    int max_depth;
    int node_cap;
    int periodic;
    double box[3];
    int *work;
    unsigned *status;
    unsigned long long *counters;
    int visit_slot;  // counter that accumulates this pass's node visits
};

// division in the pass precision: the FP32 path uses the approximate
// hardware reciprocal, the FP64 path IEEE division
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double fdiv(double a, double b) { return a / b; }

// exact FP64 distance as the reference writes it: sqrt(dx*dx + dy*dy + dz*dz)
__device__ __forceinline__ double exact_dist(double dx, double dy, double dz) {
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
}

// The SPH walks take a node with at most kSphLeaf particles whole, as if it
// were a leaf: below that size descending costs more walk steps than the
// extra candidates it saves (the per-candidate reach test still drops them;
// the gravity walk keeps the tree's own leaves).
constexpr int kSphLeaf = 64;

// Walk the tree for one group, calling flush(nleaf) on full leaf queues.
// A node is kept if the gap between its bbox and the group bbox is at most
// reach = Rg + (node_h ? hmax_node : 0) (times a 4e-5 safety margin; the
// exact pair predicate decides); images shift the nodes by `shift`.
// How the walk treats the block's other warps: kAlone, a group of its own;
// kShare, a team's walk split between its warps (team_share); kAll, every warp
// of a team collects all leaves (the flush shares out the candidates).
enum WalkMode { kAlone, kShare, kAll };

template <WalkMode MODE = kAlone, class Flush>
__device__ void collect_leaves(const WalkArgs &a, const WarpMem &wm, int root, const GroupBox &gb,
                               float Rg, bool node_h, float3 shift, Flush &flush) {
    const int lane = lane_id();
    const int team = MODE == kShare ? (int)(blockDim.x >> 5) : 1, tw = MODE != kAlone ? (int)(threadIdx.x >> 5) : 0;
    bool common = MODE == kShare;  // still on the steps all warps of the team take
    int top = 1;
    if (lane == 0) wm.stack[0] = root;
    __syncwarp();
    int nleaf = 0;
    const float margin = 1.0f + 4e-5f;
    // every node is popped at most once per walk; the bound only trips on a
    // corrupted tree, which then raises a status bit instead of spinning
    unsigned long long visits = 0;
    int guard = 0;
    for (; top > 0; ++guard) {
        if (guard > a.node_cap) {
            if (lane == 0) set_status(a.status, SPH3_STATUS_STACK_OVERFLOW);
            break;
        }
        if (MODE == kShare && common && top >= kTeamSplit) {
            top = team_share(wm.stack, top, team, tw);
            common = false;
            if (top == 0) break;
        }
        const int p = pop_width(top, a.stack_cap, a.max_depth);
        if ((MODE != kAll && !common) || tw == 0) visits += p;
        int node = -1;
        if (lane < p) node = wm.stack[top - 1 - lane];
        __syncwarp();
        top -= p;
        bool take = false;
        int nch = 0, cf = 0;
        if (node >= 0) {
            // one record per node: box, half widths + hmax, children (one round trip)
            const float4 bc = a.sw[3 * node], bh = a.sw[3 * node + 1], w2 = a.sw[3 * node + 2];
            const int chy = __float_as_int(w2.y);
            float3 c = rel_to(bc, gb.ref, gb.s10);
            c.x += shift.x;
            c.y += shift.y;
            c.z += shift.z;
            const float reach = (Rg + (node_h ? bh.w : 0.f)) * margin;
            const float g2 = box_gap2(gb, c, make_float3(bh.x, bh.y, bh.z));
            if (chy >= 0 && g2 <= reach * reach) {
                const int k = chy & 255;
                if (k == 0 || __float_as_int(w2.z) <= kSphLeaf) {
                    take = !common || lane % team == tw;
                } else {
                    nch = k;
                    cf = __float_as_int(w2.x);
                }
            }
        }
        const unsigned tb = __ballot_sync(kFull, take);
        if (take) wm.leafq[nleaf + __popc(tb & lanemask_lt())] = node;
        nleaf += __popc(tb);
        top = push_children(wm.stack, top, a.stack_cap, nch, cf, a.status);
        if (nleaf > kLeafQ - 32) {
            __syncwarp();
            flush(nleaf);
            nleaf = 0;
        }
    }
    __syncwarp();
    if (nleaf > 0) flush(nleaf);
    if (lane == 0) {  // walk statistics: node visits per pass, longest walk (and where)
        atomicAdd(&a.counters[a.visit_slot], visits);
        atomicMax(&a.counters[kCntWalkMaxIter], (unsigned long long)guard);
        atomicMax(&a.counters[kCntWalkMaxWhere],
                  ((unsigned long long)guard << 40) | ((unsigned long long)a.visit_slot << 32) |
                      (unsigned long long)(unsigned)gb.first);
    }
}

// ------------------------------------------------------------ group setup
struct GroupInfo {
    int first, count, cloud, i;
    bool active;
    int ref;
    float s10;
    int root;
    float3 prel;  // target in the group frame (FP32)
};

__device__ __forceinline__ GroupInfo group_info(const WalkArgs &a, int g) {
    GroupInfo gi;
    const int2 gr = a.groups[g];
    gi.first = gr.x;
    gi.count = gr.y;
    gi.cloud = a.group_cloud[g];
    const Cloud &cl = a.clouds[gi.cloud];
    gi.s10 = cl.s10;
    gi.root = cl.root;
    gi.ref = __float_as_int(a.pk_pos[gi.first].w);
    const int lane = lane_id();
    gi.active = lane < gi.count;
    gi.i = gi.first + (gi.active ? lane : 0);
    gi.prel = rel_to(a.pk_pos[gi.i], gi.ref, gi.s10);
    return gi;
}

// source position in the group frame: FP32 relative (mixed) or absolute FP64
template <typename R>
__device__ __forceinline__ V4<R> src_pos(const WalkArgs &a, const GroupInfo &gi, int j, float3 s, R w) {
    V4<R> p;
    if (sizeof(R) == 8) {
        p.x = (R)(a.pos[j] + (double)s.x);
        p.y = (R)(a.pos[a.n + j] + (double)s.y);
        p.z = (R)(a.pos[2 * a.n + j] + (double)s.z);
    } else {
        const float3 q = rel_to(a.pk_pos[j], gi.ref, gi.s10);
        p.x = (R)(q.x + s.x);
        p.y = (R)(q.y + s.y);
        p.z = (R)(q.z + s.z);
    }
    p.w = w;
    return p;
}

// group-frame FP32 position of source j shifted by s (for the reach filter)
__device__ __forceinline__ float3 frame_pos(const WalkArgs &a, const GroupInfo &gi, int j, float3 s) {
    const float3 q = rel_to(a.pk_pos[j], gi.ref, gi.s10);
    return make_float3(q.x + s.x, q.y + s.y, q.z + s.z);
}

// can a source at p with smoothing length hj reach any target of the group
// (gap to the group box <= reach + hj, with the walk's 4e-5 safety margin)?
__device__ __forceinline__ bool reaches(const GroupBox &gb, float3 p, float reach) {
    const float r = reach * (1.0f + 4e-5f);
    return point_gap2(gb, p) <= r * r;
}

// FP32 distances decide nearly every FP64 predicate: relative to the sum of
// the two radii they are good to far better than kNearRel, plus the walks'
// absolute pad for the packed positions' rounding; only pairs inside that band
// are decided by the exact FP64 expressions.
constexpr float kNearRel = 4e-5f;
// Squares below FP32's normal range (lengths below 1e-19 units) are only good to
// the spacing there, 1.4e-45 an operation: the band is widened by more than the
// four or five roundings of a comparison.  Larger squares absorb it.
constexpr float kNearSq = 1e-44f;
__device__ __forceinline__ float near_pad(float s10) { return 1e-6f * 1024.f * s10; }

// ================================================================= h search
struct HArgs {
    WalkArgs w;
    double *h;
    float4 *pk_hme;
    int *nngb;
    int n_ngb, tol, max_iter;
};

constexpr int kHK = 16;  // thresholds per pass in the reference-step mode
constexpr double kNewtonDelta = 0.08;

// fields of the candidate tile: x, y, z and, in FP64, the source index
template <typename R>
constexpr int h_fields() {
    return sizeof(R) == 8 ? 4 : 3;
}
// bytes after a team warp's tile for its counts: K thresholds, 32 lanes
template <int MODE>
constexpr size_t h_count_bytes() {
    return sizeof(int) * 32 * (MODE == SPH3_H_REFSTEP ? kHK : 2);
}

template <typename R, int MODE, bool TEAM>
__device__ __forceinline__ void h_search_body(const HArgs &A) {
    extern __shared__ __align__(16) unsigned char smem[];
    const WalkArgs &a = A.w;
    constexpr bool F64 = sizeof(R) == 8;
    constexpr int NF = h_fields<R>();
    constexpr size_t kFieldBytes = sizeof(float) * 64 * NF;
    constexpr size_t kTileBytes = kFieldBytes + (TEAM ? h_count_bytes<MODE>() : 0);
    WarpMem wm = carve_warp_mem(smem, a.stack_cap, kTileBytes);
    const int lane = lane_id();
    const bool lead_warp = !TEAM || threadIdx.x < 32;  // the warp that writes a team's results
    constexpr int K = MODE == SPH3_H_REFSTEP ? kHK : 2;
    const int up = A.n_ngb + A.tol, low = A.n_ngb - A.tol;
    unsigned long long pairs = 0, passes = 0;
    for (int g = next_group_of<TEAM>(a.work, a.status); g < *a.ngroups_dev;
         g = next_group_of<TEAM>(a.work, a.status)) {
        GroupInfo gi = group_info(a, g);
        const Cloud &cl = a.clouds[gi.cloud];
        const int64_t ncl = cl.end - cl.begin;
        GroupBox gb = group_box(gi.prel, gi.active, gi.ref, gi.s10);
        gb.first = gi.first;
        const double tx = F64 ? a.pos[gi.i] : 0.0, ty = F64 ? a.pos[a.n + gi.i] : 0.0,
                     tz = F64 ? a.pos[2 * a.n + gi.i] : 0.0;
        double h = A.h[gi.i];
        if (!(h > 0.0) || !isfinite(h)) h = (double)gi.s10;  // no usable start: one level-10 cell
        bool conv = !gi.active;
        int ncount = 0;
        int steps = 0;  // reference-rule steps taken
        int dir = 0;    // reference rule: -1 down, +1 up, 0 unknown (first pass)
        double lb = 0.0, hb = DBL_MAX;
        int n_hb = 0;  // count at hb
        bool failed = false;
        const double hcap = 4.0 * cl.size;
        for (int pass = 0; pass < A.max_iter + 2; ++pass) {
            if (__all_sync(kFull, conv)) break;
            double thr[K];
            if (MODE == SPH3_H_REFSTEP) {
                if (dir == 0) {
#pragma unroll
                    for (int k = 0; k < K; ++k) thr[k] = __dmul_rn(2.0, h);
                } else {
                    double hk = h;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const double t = __dmul_rn(0.003, hk);
                        hk = dir < 0 ? __dsub_rn(hk, t) : __dadd_rn(hk, t);
                        thr[k] = __dmul_rn(2.0, hk);
                    }
                }
            } else {
                thr[0] = 2.0 * h;
                // the first pass counts at 2h only (a smaller reach: most groups
                // are already in the window with the previous step's h); later
                // passes also count at 2h (1 + delta) for the measured slope
                thr[1] = pass == 0 ? thr[0] : 2.0 * h * (1.0 + kNewtonDelta);
            }
            float reach = 0.f;
            if (!conv) {
#pragma unroll
                for (int k = 0; k < K; ++k) reach = fmaxf(reach, (float)thr[k]);
            }
            reach = warp_max(reach) * (1.0f + 1e-5f);
            float thr2f[K];
#pragma unroll
            for (int k = 0; k < K; ++k) thr2f[k] = (float)(thr[k] * thr[k]);
            int cnt[K];
#pragma unroll
            for (int k = 0; k < K; ++k) cnt[k] = 0;
            // FP64: distances below `in2` are inside every threshold, above `out2`
            // outside all, settled in FP32; the rest are compared exactly
            float in2 = 0.f, out2 = 0.f;
            if (F64) {
                double tmin = thr[0], tmax = thr[0];
#pragma unroll
                for (int k = 1; k < K; ++k) {
                    tmin = fmin(tmin, thr[k]);
                    tmax = fmax(tmax, thr[k]);
                }
                const float pad = near_pad(gi.s10);
                const float lo = fmaxf((float)tmin * (1.f - kNearRel) - pad, 0.f);
                const float hi = (float)tmax * (1.f + kNearRel) + pad;
                in2 = fmaf(lo, lo, -kNearSq);
                out2 = fmaf(hi, hi, kNearSq);
            }
            int inside = 0;
            const Images ims = group_images(gb, reach, a.box, a.periodic);
            for (int im = 0; im < 27; ++im) {
                float3 s;
                if (!image_shift(ims, im, a.box, s)) continue;
                // candidates staged as coordinate arrays (FP64: and the source
                // index) and tested two per packed instruction
                float *xs = reinterpret_cast<float *>(wm.tile), *ys = xs + 64, *zs = ys + 64, *js = zs + 64;
                auto load = [&](int j, bool &keep) {
                    const float3 q = rel_to(a.pk_pos[j], gi.ref, gi.s10);
                    SoaV<NF> f;
                    f.v[0] = q.x + s.x;
                    f.v[1] = q.y + s.y;
                    f.v[2] = q.z + s.z;
                    if constexpr (F64) f.v[3] = __int_as_float(j);
                    keep = reaches(gb, make_float3(f.v[0], f.v[1], f.v[2]), reach);
                    return f;
                };
                auto interact = [&](int ne) {
                    if (conv) return;
                    pairs += ne;
                    const float2 ntx = make_float2(-gi.prel.x, -gi.prel.x);
                    const float2 nty = make_float2(-gi.prel.y, -gi.prel.y);
                    const float2 ntz = make_float2(-gi.prel.z, -gi.prel.z);
                    unsigned band = 0;
                    for (int e = 0; e < ne; e += 2) {
                        const float2 dx = __fadd2_rn(*reinterpret_cast<const float2 *>(xs + e), ntx);
                        const float2 dy = __fadd2_rn(*reinterpret_cast<const float2 *>(ys + e), nty);
                        const float2 dz = __fadd2_rn(*reinterpret_cast<const float2 *>(zs + e), ntz);
                        float2 d2 = __fmul2_rn(dz, dz);
                        d2 = __ffma2_rn(dy, dy, d2);
                        d2 = __ffma2_rn(dx, dx, d2);
                        if constexpr (F64) {
                            const bool ix = d2.x < in2, iy = d2.y < in2;
                            inside += (int)ix + (int)iy;
                            band |= ((unsigned)(!ix && d2.x <= out2) | ((unsigned)(!iy && d2.y <= out2) << 1)) << e;
                        } else {
#pragma unroll
                            for (int k = 0; k < K; ++k) cnt[k] += (d2.x < thr2f[k]) + (d2.y < thr2f[k]);
                        }
                    }
                    if constexpr (F64) {
                        for (; band; band &= band - 1) {
                            const int j = __float_as_int(js[__ffs(band) - 1]);
                            const double d = exact_dist((a.pos[j] + (double)s.x) - tx, (a.pos[a.n + j] + (double)s.y) - ty,
                                                        (a.pos[2 * a.n + j] + (double)s.z) - tz);
#pragma unroll
                            for (int k = 0; k < K; ++k) cnt[k] += d < thr[k];
                        }
                    }
                };
                // an odd batch's pad passes no comparison, whatever the unit of length
                constexpr SoaV<NF> pad = {{__builtin_nanf(""), __builtin_nanf(""), __builtin_nanf("")}};
                auto flush = [&](int nl) {
                    flush_leaves_compact_soa<NF>(a.range, wm.leafq, nl, xs, pad, load, interact);
                };
                collect_leaves<TEAM ? kShare : kAlone>(a, wm, gi.root, gb, reach, false, s, flush);
            }
#pragma unroll
            for (int k = 0; k < K; ++k) cnt[k] += inside;
            if (TEAM) {  // the team's counts, the same sum in every warp
                auto counts_of = [&](int w) {
                    return reinterpret_cast<int *>(smem + (size_t)w * warp_mem_bytes(a.stack_cap, kTileBytes) +
                                                   warp_mem_bytes(a.stack_cap, 0) + kFieldBytes);
                };
                int *mine = counts_of(threadIdx.x >> 5);
#pragma unroll
                for (int k = 0; k < K; ++k) mine[32 * k + lane] = cnt[k];
                __syncwarp();
                __syncthreads();
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    int sum = 0;
                    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) sum += counts_of(w)[32 * k + lane];
                    cnt[k] = sum;
                }
                __syncthreads();
            }
            if (lead_warp) ++passes;
            // ---- update (lanes already converged keep their h)
            if (conv) {
            } else if (MODE == SPH3_H_REFSTEP) {
                if (dir == 0) {
                    ncount = cnt[0];
                    if (ncount <= up && ncount >= low) conv = true;
                    else dir = ncount > up ? -1 : 1;
                } else {
                    double hk = h;
                    for (int k = 0; k < K; ++k) {
                        if (steps >= A.max_iter) {
                            failed = true;
                            conv = true;
                            break;
                        }
                        const double t = __dmul_rn(0.003, hk);
                        hk = dir < 0 ? __dsub_rn(hk, t) : __dadd_rn(hk, t);
                        ++steps;
                        ncount = cnt[k];
                        h = hk;
                        if (ncount <= up && ncount >= low) {
                            conv = true;
                            break;
                        }
                        const int nd = ncount > up ? -1 : 1;
                        if (nd != dir) {  // crossed the window: the rule turns around
                            dir = nd;
                            break;
                        }
                    }
                }
            } else {
                const int n0 = cnt[0], n1 = cnt[1];
                ncount = n0;
                if (n0 <= up && n0 >= low) {
                    conv = true;
                } else if (pass >= A.max_iter || (n0 < low && (int64_t)n0 >= ncl)) {
                    // out of iterations, or the whole system is inside 2h already
                    failed = true;
                    conv = true;
                } else {
                    // Newton step on ln N(ln h) with the slope measured between
                    // h and h (1 + delta), safeguarded by the bracket [lb, hb]
                    if (n0 > up && h < hb) {
                        hb = h;
                        n_hb = n0;
                    } else if (n0 < low) {
                        lb = fmax(lb, h);
                    }
                }
                if (!conv && lb > 0.0 && hb < DBL_MAX && hb - lb <= 1e-6 * hb) {
                    // the count jumps over the whole window at one radius (a
                    // shell of equidistant neighbours, e.g. on a lattice): no h
                    // reaches the window, take the smallest h above the jump
                    h = hb;
                    ncount = n_hb;
                    conv = true;
                } else if (!conv) {
                    double hn;
                    if (n0 == 0) {
                        hn = 2.0 * h;
                    } else {
                        // slope of ln N over ln h: measured, or 3 (uniform density) on the first pass
                        double sl = pass > 0 && n1 > n0 ? log((double)n1 / (double)n0) / log1p(kNewtonDelta) : 3.0;
                        sl = fmin(fmax(sl, 1.0), 6.0);
                        hn = h * exp((log((double)A.n_ngb) - log((double)n0)) / sl);
                    }
                    hn = fmin(fmax(hn, 0.5 * h), 2.0 * h);
                    if (!(hn > lb && hn < hb)) {
                        if (lb > 0.0 && hb < DBL_MAX) hn = sqrt(lb * hb);
                        else if (hb < DBL_MAX) hn = hb * 0.8;
                        else hn = lb * 1.25;
                    }
                    h = fmin(hn, hcap);
                }
            }
        }
        if (!conv) failed = true;
        if (gi.active && lead_warp) {
            A.h[gi.i] = h;
            A.nngb[gi.i] = ncount;
            A.pk_hme[gi.i].x = (float)h;
            // minimum-image counting needs the kernel support inside half the box
            bool big = false;
            for (int d = 0; d < 3; ++d) big |= a.box[d] > 0.0 && 2.0 * h > 0.5 * a.box[d];
            if (big) set_status(a.status, SPH3_STATUS_BOX_TOO_SMALL);
        }
        const unsigned fb = __ballot_sync(kFull, gi.active && failed);
        if (fb && lane == 0) set_status(a.status, SPH3_STATUS_H_NOT_CONVERGED);
    }
    pairs = warp_sum(pairs);
    if (lane == 0) {
        atomicAdd(&a.counters[4], pairs);
        atomicAdd(&a.counters[5], passes);
    }
}

template <typename R, int MODE, bool TEAM>
__global__ void __launch_bounds__(kWalkWarps * 32, kWalkMinBlocks) k_h_search(HArgs A) {
    h_search_body<R, MODE, TEAM>(A);
}

// The mixed Newton search (the per-step path) capped at 96 registers: 20
// resident warps per SM instead of 16 (its walk is latency-bound).
__global__ void __maxnreg__(96) k_h_search_f32_newton(HArgs A) { h_search_body<float, SPH3_H_NEWTON, false>(A); }

// ============================================================ bootstrap h
// h = 0.5 * (k-th smallest distance, self included), the reference's
// smoothing_length_mpi / do_smoothingX (sph_code/libsx.py:752-800), exact:
// a radius that holds k+1 particles, then a 17-way bisection on the bit
// pattern of the FP64 distance.
struct BootArgs {
    WalkArgs w;
    double *h;
    float4 *pk_hme;
    int k;
};

__global__ void __launch_bounds__(kWalkWarps * 32, kWalkMinBlocks) k_boot_h(BootArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    const WalkArgs &a = A.w;
    using E = V4<double>;
    WarpMem wm = carve_warp_mem(smem, a.stack_cap, sizeof(E) * 64);
    E *tile = reinterpret_cast<E *>(wm.tile);
    for (int g = next_group(a.work, a.status); g < *a.ngroups_dev; g = next_group(a.work, a.status)) {
        GroupInfo gi = group_info(a, g);
        const Cloud &cl = a.clouds[gi.cloud];
        const int64_t ncl = cl.end - cl.begin;
        const int need = (int)std::min<int64_t>((int64_t)A.k, ncl - 1) + 1;
        GroupBox gb = group_box(gi.prel, gi.active, gi.ref, gi.s10);
        gb.first = gi.first;
        const double tx = a.pos[gi.i], ty = a.pos[a.n + gi.i], tz = a.pos[2 * a.n + gi.i];
        // phase 1: grow a common radius until every target has `need` particles within it
        double Rg = 2.0 * (double)fmaxf(gb.hw.x, fmaxf(gb.hw.y, gb.hw.z)) + (double)gi.s10;
        for (int it = 0; it < 64; ++it) {
            int cnt = 0;
            const Images ims = group_images(gb, (float)Rg, a.box, a.periodic);
            for (int im = 0; im < 27; ++im) {
                float3 s;
                if (!image_shift(ims, im, a.box, s)) continue;
                auto load = [&](int j) { return src_pos<double>(a, gi, j, s, 0.0); };
                auto interact = [&](const E *t, int ne) {
                    for (int e = 0; e < ne; ++e) {
                        const E q = t[e];
                        cnt += exact_dist(q.x - tx, q.y - ty, q.z - tz) <= Rg;
                    }
                };
                auto flush = [&](int nl) {
                    flush_leaves(a.range, wm.leafq, nl, tile, load, interact);
                };
                collect_leaves(a, wm, gi.root, gb, (float)Rg * 1.0001f, false, s, flush);
            }
            if (__all_sync(kFull, !gi.active || cnt >= need)) break;
            Rg *= 2.0;
        }
        // phase 2: bisection on the distance bits, 16 thresholds per pass
        unsigned long long lo = 0ull, hi = (unsigned long long)__double_as_longlong(Rg);
        for (int it = 0; it < 40; ++it) {
            if (__all_sync(kFull, !gi.active || lo == hi)) break;
            unsigned long long t[16];
            const unsigned long long span = hi - lo;
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                if (span > 16ull) t[m] = lo + (span / 17ull) * (unsigned long long)(m + 1);
                else t[m] = (unsigned long long)m < span ? lo + m : hi;
            }
            double tv[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) tv[m] = __longlong_as_double((long long)t[m]);
            int c[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) c[m] = 0;
            const Images ims = group_images(gb, (float)Rg, a.box, a.periodic);
            for (int im = 0; im < 27; ++im) {
                float3 s;
                if (!image_shift(ims, im, a.box, s)) continue;
                auto load = [&](int j) { return src_pos<double>(a, gi, j, s, 0.0); };
                auto interact = [&](const E *tl, int ne) {
                    if (lo == hi) return;
                    for (int e = 0; e < ne; ++e) {
                        const E q = tl[e];
                        const double d = exact_dist(q.x - tx, q.y - ty, q.z - tz);
#pragma unroll
                        for (int m = 0; m < 16; ++m) c[m] += d <= tv[m];
                    }
                };
                auto flush = [&](int nl) {
                    flush_leaves(a.range, wm.leafq, nl, tile, load, interact);
                };
                collect_leaves(a, wm, gi.root, gb, (float)Rg * 1.0001f, false, s, flush);
            }
            if (lo != hi) {
                int m = 0;
                while (m < 16 && c[m] < need) ++m;
                if (m == 16) {
                    lo = t[15] + 1;
                } else {
                    const unsigned long long nlo = m > 0 ? t[m - 1] + 1 : lo;
                    hi = t[m];
                    lo = nlo;
                }
                if (lo > hi) lo = hi;
            }
        }
        if (gi.active) {
            const double hv = __longlong_as_double((long long)hi) * 0.5;
            A.h[gi.i] = hv;
            A.pk_hme[gi.i].x = (float)hv;
        }
    }
}

// one rounding each, whatever the compiler would contract
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
// a b - c d as every pass computes it
__device__ __forceinline__ float cross_rn(float a, float b, float c, float d) { return fma_rn(a, b, -mul_rn(c, d)); }

// =================================================== density, EOS, div/curl
struct DArgs {
    WalkArgs w;
    const float4 *pk_hme, *pk_vel;
    const double *h, *m, *vel, *u;
    double *rho, *P, *c, *divV, *curlV, *bal;
    float4 *pk_thm;
    double gamma;
    int keep_rho;
    // neighbour lists for the hydro pass (null: none kept)
    int *list, *nlist;
    int list_cap;
    int *ovf;  // particles with more pairs than list_cap
};

// The candidate tile: arrays of 64 floats {x, y, z, h, source index as float
// bits}, and in the mixed path {m} and, with div and curl, {vx, vy, vz}.
template <typename R, bool DC>
constexpr int density_fields() {
    return sizeof(R) == 8 ? 5 : (DC ? 9 : 6);
}
// The mixed pass with div and curl adds a target's pairs one by one, in the
// order it met them (a run's segments added up apart round differently, and the
// h rule turns any difference in the positions into a step of 3 % in h where a
// neighbour count comes out on the other side of its window): the terms of
// kDcBatch tasks wait in shared memory.  Kelvin-Helmholtz at 4,194,304: 5.75 ms
// in segments, 6.25 in order (batches of 32: 7.43, 64: 6.66, 256: 7.46).
template <typename R, bool DC>
constexpr bool density_in_order() {
    return sizeof(R) == 4 && DC;
}
constexpr int kDcBatch = 128;
// task list of a tile: one (target lane, tile entry) pair per in-support
// candidate, at most 32 x 32
constexpr size_t kTaskBytes = sizeof(unsigned short) * 32 * 32;
constexpr int kOvfStop = 512;
// a team warp's in-support counts of two rounds, one per target lane
constexpr size_t kTeamCountBytes = sizeof(int) * 2 * 32;
// bytes of the fields (a team's sums, five values per lane, fit in them), and
// of a warp's whole tile
template <typename R, bool DC>
constexpr size_t density_field_bytes() {
    return sizeof(float) * 64 * density_fields<R, DC>();
}
template <typename R, bool DC>
constexpr size_t density_tile_bytes() {
    return density_field_bytes<R, DC>() + kTaskBytes + kTeamCountBytes +
           (density_in_order<R, DC>() ? sizeof(float4) * 2 * kDcBatch : 0);
}

// The density pass.  Candidates are staged as arrays of fields and tested two
// per packed FP32 instruction against every target.  The in-support (target,
// entry) pairs of a tile become a task list ordered by target; lane k runs
// task k of each chunk of 32 (target values by shuffle), writes the pair into
// the target's neighbour list, and the density (div and curl) terms are summed
// per target with a segmented warp reduction (fixed order: deterministic), so
// no lane idles while the one with the most neighbours finishes.  The mixed pass
// with div and curl adds them in list order instead (kDcBatch).
// FP64: the tests settle all but a narrow band of distances in FP32 (the rest
// by the exact predicate, so the pair sets are exact) and a pair's FP64 values
// are read by the lane that runs it; testing every candidate with an FP64 root
// and quotient was most of the pass (674 us at 131,072 particles, 327 now;
// the h search, by the same means, 386 and 195).
// TEAM: every warp of the block collects the group's leaves (the same queue),
// the candidate chunks go round the warps, and the warps exchange their
// chunks' in-support counts per target before they write the pairs, so the
// lists hold the same pairs in the same order as a warp's alone.
// LISTS: only the neighbour lists are wanted, for FP64 forces from a given
// density.  A group's walk ends once a list of it overflows (its particles are
// walked by the hydro pass), and no group is begun after kOvfStop particles were
// left to that: where the caller's h gives more pairs than a list holds, the
// walks of the lists would be for nothing (100,000 particles, 262 pairs each, lists
// of 128: 3.05 ms, 2.22 now and 2.26 without lists at all; 82 pairs: 0.53, 0.41
// and 1.06).
template <typename R, bool DC, bool TEAM, bool LISTS = false>
__device__ __forceinline__ void density_body(const DArgs &A) {
    extern __shared__ __align__(16) unsigned char smem[];
    const WalkArgs &a = A.w;
    constexpr bool F64 = sizeof(R) == 8;
    constexpr int NF = density_fields<R, DC>();
    constexpr size_t kFieldBytes = density_field_bytes<R, DC>(), kTileBytes = density_tile_bytes<R, DC>();
    WarpMem wm = carve_warp_mem(smem, a.stack_cap, kTileBytes);
    const int team = TEAM ? (int)(blockDim.x >> 5) : 1, tw = TEAM ? (int)(threadIdx.x >> 5) : 0;
    int round = 0;
    // warp w's tile region
    auto region_of = [&](int w) {
        return smem + (size_t)w * warp_mem_bytes(a.stack_cap, kTileBytes) + warp_mem_bytes(a.stack_cap, 0);
    };
    // The team's exchange: c in-support pairs of this lane's target in this
    // warp's chunk -> those of the earlier warps' chunks, and of all of them
    auto team_counts = [&](int c, int &before, int &all) {
        const size_t at = kFieldBytes + kTaskBytes + sizeof(int) * 32 * (round & 1);
        ++round;
        reinterpret_cast<int *>(region_of(tw) + at)[lane_id()] = c;
        __syncwarp();
        __syncthreads();
        before = all = 0;
        for (int w = 0; w < team; ++w) {
            const int v = reinterpret_cast<const int *>(region_of(w) + at)[lane_id()];
            before += w < tw ? v : 0;
            all += v;
        }
    };
    float *sx = reinterpret_cast<float *>(wm.tile), *sy = sx + 64, *sz = sy + 64, *sh = sz + 64, *sj = sh + 64,
          *sm = sj + 64, *sv = sm + 64;
    unsigned short *tasks =
        reinterpret_cast<unsigned short *>(reinterpret_cast<unsigned char *>(wm.tile) + kFieldBytes);
    constexpr bool kInOrder = density_in_order<R, DC>();
    float4 *terms = reinterpret_cast<float4 *>(reinterpret_cast<unsigned char *>(wm.tile) + kFieldBytes + kTaskBytes +
                                               kTeamCountBytes);
    const int lane = lane_id();
    unsigned long long pairs = 0;
    for (int g = next_group_of<TEAM>(a.work, a.status); g < *a.ngroups_dev;
         g = next_group_of<TEAM>(a.work, a.status)) {
        GroupInfo gi = group_info(a, g);
        GroupBox gb = group_box(gi.prel, gi.active, gi.ref, gi.s10);
        gb.first = gi.first;
        // the target in the group frame, and in the path's precision
        const float fth = A.pk_hme[gi.i].x;
        R tx, ty, tz, th, tvx = 0, tvy = 0, tvz = 0;
        if (F64) {
            tx = (R)a.pos[gi.i]; ty = (R)a.pos[a.n + gi.i]; tz = (R)a.pos[2 * a.n + gi.i];
            th = (R)A.h[gi.i];
            if (DC) { tvx = (R)A.vel[gi.i]; tvy = (R)A.vel[a.n + gi.i]; tvz = (R)A.vel[2 * a.n + gi.i]; }
        } else {
            tx = (R)gi.prel.x; ty = (R)gi.prel.y; tz = (R)gi.prel.z;
            th = (R)fth;
            if (DC) { const float4 v = A.pk_vel[gi.i]; tvx = (R)v.x; tvy = (R)v.y; tvz = (R)v.z; }
        }
        const float hmax_g = warp_max(gi.active ? fth : 0.f);
        const float pad32 = near_pad(gi.s10);
        R rho = 0, sdiv = 0, cx = 0, cy = 0, cz = 0;
        int nkept = 0;  // in-support pairs found (kept in the list while < list_cap)
        bool full = false;  // LISTS: a list of this group has overflowed
        if constexpr (LISTS) {  // the same answer in all warps of a team
            const int over = *reinterpret_cast<const volatile int *>(A.ovf) > kOvfStop;
            full = (TEAM ? __syncthreads_or(threadIdx.x == 0 && over) : __shfl_sync(kFull, over, 0)) != 0;
        }
        const Images ims = group_images(gb, hmax_g + a.box_h[gi.root].w, a.box, a.periodic);
        for (int im = 0; im < 27; ++im) {
            float3 s;
            if (!image_shift(ims, im, a.box, s)) continue;
            auto load = [&](int j, bool &keep) {
                const float4 hm = A.pk_hme[j];
                const float3 q = rel_to(a.pk_pos[j], gi.ref, gi.s10);
                SoaV<NF> v;
                v.v[0] = q.x + s.x;
                v.v[1] = q.y + s.y;
                v.v[2] = q.z + s.z;
                v.v[3] = hm.x;
                v.v[4] = __int_as_float(j);
                if constexpr (!F64) v.v[5] = hm.y;
                if constexpr (!F64 && DC) {
                    const float4 w = A.pk_vel[j];
                    v.v[6] = w.x;
                    v.v[7] = w.y;
                    v.v[8] = w.z;
                }
                keep = reaches(gb, make_float3(v.v[0], v.v[1], v.v[2]), hmax_g + hm.x);
                return v;
            };
            // source j's exact pair geometry (FP64 path): d = r_i - r_j and hbar
            auto exact_pair = [&](int j, double qx, double qy, double qz, double qh, double &dx, double &dy, double &dz,
                                  double &hij) {
                dx = __dsub_rn(qx, a.pos[j] + (double)s.x);
                dy = __dsub_rn(qy, a.pos[a.n + j] + (double)s.y);
                dz = __dsub_rn(qz, a.pos[2 * a.n + j] + (double)s.z);
                hij = __dmul_rn(0.5, __dadd_rn(qh, A.h[j]));
                return exact_dist(dx, dy, dz);
            };
            auto interact = [&](int ne) {
                if (LISTS && full) return;
                if (gi.active) pairs += ne;
                unsigned mask = 0;
                if (gi.active) {
                    unsigned band = 0;
                    const float2 ntx = make_float2(-gi.prel.x, -gi.prel.x);
                    const float2 nty = make_float2(-gi.prel.y, -gi.prel.y);
                    const float2 ntz = make_float2(-gi.prel.z, -gi.prel.z);
                    const float2 th2 = make_float2(fth, fth);
                    auto test = [&](int e) {
                        const float2 dx = __fadd2_rn(*reinterpret_cast<const float2 *>(sx + e), ntx);
                        const float2 dy = __fadd2_rn(*reinterpret_cast<const float2 *>(sy + e), nty);
                        const float2 dz = __fadd2_rn(*reinterpret_cast<const float2 *>(sz + e), ntz);
                        const float2 hs = __fadd2_rn(th2, *reinterpret_cast<const float2 *>(sh + e));
                        float2 d2 = __fmul2_rn(dz, dz);
                        d2 = __ffma2_rn(dy, dy, d2);
                        d2 = __ffma2_rn(dx, dx, d2);
                        if constexpr (F64) {
                            float2 lo = __ffma2_rn(hs, make_float2(1.f - kNearRel, 1.f - kNearRel),
                                                   make_float2(-pad32, -pad32));
                            lo = make_float2(fmaxf(lo.x, 0.f), fmaxf(lo.y, 0.f));
                            const float2 hi = __ffma2_rn(hs, make_float2(1.f + kNearRel, 1.f + kNearRel),
                                                         make_float2(pad32, pad32));
                            const float2 lo2 = __ffma2_rn(lo, lo, make_float2(-kNearSq, -kNearSq));
                            const float2 hi2 = __ffma2_rn(hi, hi, make_float2(kNearSq, kNearSq));
                            mask |= ((unsigned)(d2.x < lo2.x) | ((unsigned)(d2.y < lo2.y) << 1)) << e;
                            band |= ((unsigned)(d2.x <= hi2.x) | ((unsigned)(d2.y <= hi2.y) << 1)) << e;
                        } else {
                            const float2 hs2 = __fmul2_rn(hs, hs);
                            mask |= ((unsigned)(d2.x <= hs2.x) | ((unsigned)(d2.y <= hs2.y) << 1)) << e;
                        }
                    };
                    if constexpr (DC || F64) {
#pragma unroll 2
                        for (int e = 0; e < ne; e += 2) test(e);
                    } else {
                        for (int e = 0; e < ne; e += 2) test(e);
                    }
                    if (ne < 32) {  // the pad entry of an odd batch
                        mask &= (1u << ne) - 1u;
                        band &= (1u << ne) - 1u;
                    }
                    if constexpr (F64) {
                        for (band &= ~mask; band; band &= band - 1) {
                            const int e = __ffs(band) - 1;
                            double dx, dy, dz, hij;
                            const double rr = exact_pair(__float_as_int(sj[e]), tx, ty, tz, th, dx, dy, dz, hij);
                            if (__ddiv_rn(rr, hij) <= 2.0) mask |= 1u << e;
                        }
                    }
                }
                const int c = __popc(mask);
                const int incl = warp_incl_scan(c);
                const int total = __shfl_sync(kFull, incl, 31);
                const int off = incl - c;
                int first_slot = nkept, all = c;
                if (TEAM) {
                    team_counts(c, first_slot, all);
                    first_slot += nkept;
                }
                {
                    int o = off;
                    unsigned mm = mask;
                    while (mm) {
                        const int e = __ffs(mm) - 1;
                        mm &= mm - 1;
                        tasks[o++] = (unsigned short)((lane << 5) | e);
                    }
                }
                __syncwarp();
                for (int k0 = 0; k0 < total; k0 += 32) {
                    const int k = k0 + lane;
                    const bool valid = k < total;
                    const int task = valid ? (int)tasks[k] : 0;
                    const int tl = valid ? task >> 5 : 32;  // key: target lane (32 past the end)
                    const int e = task & 31;
                    const R qx = __shfl_sync(kFull, tx, tl & 31);
                    const R qy = __shfl_sync(kFull, ty, tl & 31);
                    const R qz = __shfl_sync(kFull, tz, tl & 31);
                    const R qh = __shfl_sync(kFull, th, tl & 31);
                    const int base = __shfl_sync(kFull, first_slot - off, tl & 31);
                    R qvx = 0, qvy = 0, qvz = 0;
                    if (DC) {
                        qvx = __shfl_sync(kFull, tvx, tl & 31);
                        qvy = __shfl_sync(kFull, tvy, tl & 31);
                        qvz = __shfl_sync(kFull, tvz, tl & 31);
                    }
                    constexpr int NV = DC ? 5 : 1;  // rho; div, curl
                    R v[NV];
#pragma unroll
                    for (int f = 0; f < NV; ++f) v[f] = 0;
                    if (valid) {
                        const int j = __float_as_int(sj[e]);
                        if (A.list) {
                            const int slot = base + k;
                            if (slot < A.list_cap) A.list[(size_t)(gi.first + tl) * A.list_cap + slot] = j;
                        }
                        if constexpr (LISTS) {
                        } else if constexpr (F64) {
                            double dx, dy, dz, hij;
                            const double rr = exact_pair(j, qx, qy, qz, qh, dx, dy, dz, hij);
                            const double q = __ddiv_rn(rr, hij);
                            const double ih = 1.0 / hij;
                            const double ih3 = ih * ih * ih;
                            const double tq = 2.0 - q;
                            const double W = kSig * ih3 * (q <= 1.0 ? 1.0 - 1.5 * q * q + 0.75 * q * q * q : 0.25 * tq * tq * tq);
                            const double mj = A.m[j];
                            v[0] = mj * W;
                            if constexpr (DC) {
                                const double ih5 = ih3 * ih * ih;
                                double nW;
                                if (q <= 1.0) nW = kSig * ih5 * (-3.0 + 2.25 * q);
                                else nW = -0.75 * kSig * ih5 * tq * tq / (q + 1e-20);
                                const double gx = nW * dx, gy = nW * dy, gz = nW * dz;
                                const double vx = qvx - A.vel[j], vy = qvy - A.vel[a.n + j],
                                             vz = qvz - A.vel[2 * a.n + j];
                                v[1] = -mj * (vx * gx + vy * gy + vz * gz);
                                v[2] = mj * (vy * gz - vz * gy);
                                v[3] = mj * (vz * gx - vx * gz);
                                v[4] = mj * (vx * gy - vy * gx);
                            }
                        } else {
                            const float dx = qx - sx[e];
                            const float dy = qy - sy[e];
                            const float dz = qz - sz[e];
                            const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                            const float ih = __fdividef(2.0f, qh + sh[e]);
                            // |r| as d2 * rsqrt(d2) (0 for the self pair)
                            const float q = (d2 > 0.f ? d2 * rsqrtf(d2) : 0.f) * ih;
                            const float ih3 = ih * ih * ih;
                            const float tq = 2.0f - q;
                            const float w_in = fmaf(q * q, fmaf(0.75f, q, -1.5f), 1.0f);
                            const float w_out = 0.25f * tq * tq * tq;
                            const float W = kSigF * ih3 * (q <= 1.0f ? w_in : w_out);
                            if constexpr (kInOrder) {
                                const float ih5 = ih3 * ih * ih;
                                float nW;
                                if (q <= 1.0f) nW = kSigF * ih5 * fmaf(2.25f, q, -3.0f);
                                else nW = -0.75f * kSigF * ih5 * tq * tq * __fdividef(1.0f, q + 1e-20f);
                                const float vx = qvx - sv[e], vy = qvy - sv[64 + e], vz = qvz - sv[128 + e];
                                const int at = 2 * (k & (kDcBatch - 1));
                                terms[at] = make_float4(sm[e], W, sm[e] * nW, fmaf(vx, dx, fmaf(vy, dy, vz * dz)));
                                terms[at + 1] = make_float4(cross_rn(vy, dz, vz, dy), cross_rn(vz, dx, vx, dz),
                                                            cross_rn(vx, dy, vy, dx), 0.f);
                            } else {
                                v[0] = sm[e] * W;
                            }
                        }
                    }
                    if constexpr (LISTS) {
                    } else if constexpr (kInOrder) {
                        // at the end of a batch each target adds its run of it, pair by pair
                        if ((k0 + 32) % kDcBatch != 0 && k0 + 32 < total) continue;
                        __syncwarp();
                        const int b0 = k0 & ~(kDcBatch - 1);
                        const int t1 = min(off + c - b0, kDcBatch);
                        for (int t = max(off - b0, 0); t < t1; ++t) {
                            const float4 p = terms[2 * t], r = terms[2 * t + 1];
                            rho = fma_rn(p.x, p.y, rho);
                            sdiv = fma_rn(-p.z, p.w, sdiv);
                            cx = fma_rn(p.z, r.x, cx);
                            cy = fma_rn(p.z, r.y, cy);
                            cz = fma_rn(p.z, r.z, cz);
                        }
                        __syncwarp();
                    } else {
                        // segmented suffix sums over equal keys (keys are non-decreasing)
#pragma unroll
                        for (int d = 1; d < 32; d <<= 1) {
                            const int ot = __shfl_down_sync(kFull, tl, d);
                            const bool same = lane + d < 32 && ot == tl;
#pragma unroll
                            for (int f = 0; f < NV; ++f) {
                                const R ov = __shfl_down_sync(kFull, v[f], d);
                                if (same) v[f] += ov;
                            }
                        }
                        // each target takes the sum of its run inside this chunk
                        const int first_pos = off > k0 ? off - k0 : 0;
                        const bool mine = c > 0 && off < k0 + 32 && off + c > k0;
#pragma unroll
                        for (int f = 0; f < NV; ++f) {
                            const R got = __shfl_sync(kFull, v[f], first_pos & 31);
                            R &sum = f == 0 ? rho : (f == 1 ? sdiv : (f == 2 ? cx : (f == 3 ? cy : cz)));
                            if (mine) sum += got;
                        }
                    }
                }
                nkept += all;
                if (LISTS) full = __any_sync(kFull, gi.active && nkept > A.list_cap);
                __syncwarp();
            };
            auto flush = [&](int nl) {
                if (LISTS && full) return;
                constexpr SoaV<NF> pad = {{1e18f, 1e18f, 1e18f}};  // other fields 0
                if constexpr (TEAM) {
                    auto put = [&](int at, const SoaV<NF> &v) {
#pragma unroll
                        for (int f = 0; f < NF; ++f) sx[64 * f + at] = v.v[f];
                    };
                    auto run = [&](int ne) {
                        if ((ne & 1) && lane == 0) {  // entries run in pairs: one far away
#pragma unroll
                            for (int f = 0; f < NF; ++f) sx[64 * f + ne] = pad.v[f];
                        }
                        __syncwarp();
                        interact(ne);
                    };
                    flush_leaves_team(a.range, wm.leafq, nl, team, tw, load, put, run);
                } else {
                    flush_leaves_compact_soa<NF>(a.range, wm.leafq, nl, sx, pad, load, interact);
                }
            };
            collect_leaves<TEAM ? kAll : kAlone>(a, wm, gi.root, gb, hmax_g, true, s, flush);
        }
        if (TEAM && !LISTS) {  // the warps' sums, in warp order
            __syncwarp();
            R *mine = reinterpret_cast<R *>(region_of(tw));
            const R v[5] = {rho, sdiv, cx, cy, cz};
#pragma unroll
            for (int k = 0; k < (DC ? 5 : 1); ++k) mine[32 * k + lane] = v[k];
            __syncwarp();
            __syncthreads();
            if (tw == 0) {
                for (int w = 1; w < team; ++w) {
                    const R *o = reinterpret_cast<const R *>(region_of(w));
                    rho += o[lane];
                    if (DC) {
                        sdiv += o[32 + lane];
                        cx += o[64 + lane];
                        cy += o[96 + lane];
                        cz += o[128 + lane];
                    }
                }
            }
        }
        if (gi.active && tw == 0) {
            const int i = gi.i;
            if (A.list) {
                if (LISTS && full) nkept = A.list_cap + 1;
                A.nlist[i] = nkept;
                if (nkept > A.list_cap) atomicAdd(A.ovf, 1);
            }
            if constexpr (LISTS) continue;
            double r, P, c;
            if (A.keep_rho) {  // div/curl only: divide by the caller's rho
                r = A.rho[i];
                P = A.P[i];
                c = A.c[i];
            } else {
                r = (double)rho;
                const double u = A.u[i];
                P = (A.gamma - 1.0) * r * u;
                c = sqrt(A.gamma * (A.gamma - 1.0) * u);
                A.rho[i] = r;
                A.P[i] = P;
                A.c[i] = c;
            }
            double f = 0.0;
            if (DC) {
                const double inv = r > 0.0 ? 1.0 / r : 0.0;
                const double dv = fabs((double)sdiv) * inv;
                const double cv = sqrt((double)cx * (double)cx + (double)cy * (double)cy + (double)cz * (double)cz) * inv;
                A.divV[i] = dv;
                A.curlV[i] = cv;
                f = dv / (dv + cv + 0.0001 * c / A.h[i]);
                A.bal[i] = f;
            }
            const double pr = r > 0.0 ? P / (r * r) : 0.0;
            A.pk_thm[i] = make_float4((float)r, (float)pr, (float)c, (float)f);
            if (!(r > 0.0)) set_status(a.status, SPH3_STATUS_ZERO_DENSITY);
        }
    }
    pairs = warp_sum(pairs);
    if (lane == 0) atomicAdd(&a.counters[2], pairs);
}

template <typename R, bool DC, bool TEAM>
__global__ void __launch_bounds__(kWalkWarps * 32, kWalkMinBlocks) k_density(DArgs A) {
    density_body<R, DC, TEAM>(A);
}

// the lists alone, for FP64 forces from a given density
template <bool TEAM>
__global__ void __launch_bounds__(kWalkWarps * 32, kWalkMinBlocks) k_make_lists(DArgs A) {
    density_body<double, false, TEAM, true>(A);
}

// The mixed density pass of every step capped at 96 registers: 20 resident
// warps per SM instead of 16.
__global__ void __maxnreg__(96) k_density_f32(DArgs A) { density_body<float, false, false>(A); }

// With div and curl: 128 registers (16 warps; with segmented sums 1.45 ms at
// 1,048,576 particles, 1.50 at 112, 1.93 at 96, 1.81 at 152), pair tests unrolled
// twice.
__global__ void __maxnreg__(128) k_density_dc_f32(DArgs A) { density_body<float, true, false>(A); }

// ============================================================ hydro
struct YArgs {
    WalkArgs w;
    const float4 *pk_hme, *pk_vel, *pk_thm;
    const double *h, *m, *vel, *rho, *P, *c, *bal;
    double *acc_sph, *dudt;
    double *vsig;  // max signal velocity over the pairs (written with the acceleration)
    double alpha, beta, eta;
    // only_overflow: walk only for particles whose neighbour list overflowed
    const int *nlist;
    int list_cap;
    int only_overflow;
    const int *ovf;  // number of overflowed lists (only_overflow: nothing to do when 0)
};

// tile entry: p = {x, y, z, h}, v = {vx, vy, vz, m}, t = {rho, P/rho^2, c, f}
template <typename R>
struct YE {
    V4<R> p, v, t;
};

// One hydro pair, after the pair geometry (d = r_i - r_j, |d|, hbar_ij,
// q = |d| / hbar_ij): the reference's acceleration and du/dt terms
// (sph_code/libsx.py:117-165, :364-417; MG83 :236-246; Balsara
// sph_code/shear.py:193-215) and the pair's signal velocity.  sv = {vx, vy,
// vz, m} and st = {rho, P/rho^2, c, f} of the source.  The terms are kept as
// factors and added by hydro_add with one rounding each, so the walk and the
// list passes run the same arithmetic whichever lane computes a pair.
// Products and sums are written with explicit roundings, so that every kernel
// that inlines them gives the same bits.
template <typename R>
struct HydroTerms {
    R pt, gx, gy, gz;  // acceleration -= pt * grad W
    R ud, vg;          // du/dt += ud * vg
    R vsig;            // signal velocity (time-step estimate)
};

template <typename R, int VISC, bool ACC, bool DU>
__device__ __forceinline__ HydroTerms<R> hydro_terms(R dx, R dy, R dz, R rr, R hij, R q, R tvx, R tvy, R tvz, R trho,
                                                     R tpr, R tc, R tf, const V4<R> &sv, const V4<R> &st, R alpha,
                                                     R beta, R eta2) {
    HydroTerms<R> t;
    const R ih = fdiv((R)1, hij);
    const R ih5 = ih * ih * ih * ih * ih;
    R nW;
    if (q <= (R)1) nW = mul_rn((R)kSig * ih5, fma_rn((R)2.25, q, (R)-3));
    else { const R tq = (R)2 - q; nW = fdiv((R)(-0.75 * kSig) * ih5 * tq * tq, q + (R)1e-20); }
    t.gx = mul_rn(nW, dx);
    t.gy = mul_rn(nW, dy);
    t.gz = mul_rn(nW, dz);
    const R vx = tvx - sv.x, vy = tvy - sv.y, vz = tvz - sv.z;
    const R vr = fma_rn(vz, dz, fma_rn(vx, dx, mul_rn(vy, dy)));
    const R rhoij = (R)0.5 * (trho + st.x);
    R PI = 0, bal = 0, bare = 0;
    t.vsig = 0;
    if (VISC == SPH3_VISC_MG83) {
        const R cij = (R)0.5 * (tc + st.z);
        const R mu = fdiv(mul_rn(hij, vr), fma_rn(mul_rn(hij, hij), eta2, mul_rn(rr, rr)));
        if (vr <= (R)0) PI = fdiv(fma_rn(-mul_rn(alpha, cij), mu, mul_rn(mul_rn(beta, mu), mu)), rhoij);
        if (ACC) t.vsig = fma_rn((R)-3, fdiv(vr, rr + (R)1e-5), tc + st.z);
    } else {
        const R w = fdiv(vr, rr + (R)1e-5);
        t.vsig = fma_rn((R)-3, w, tc + st.z);
        if (vr <= (R)0) PI = fdiv(mul_rn(mul_rn((R)-0.5 * alpha, t.vsig), w), rhoij);
        if (VISC == SPH3_VISC_BALSARA) {
            bal = (R)0.5 * (tf + st.w);
            bare = PI;
            PI = mul_rn(bal, PI);
        }
    }
    const R mj = sv.w;
    const R pr = tpr + st.y;
    // the mixed acceleration alone takes the Balsara product unrounded
    constexpr bool kFused = sizeof(R) == 4 && VISC == SPH3_VISC_BALSARA && ACC && !DU;
    t.pt = ACC ? mul_rn(mj, kFused ? fma_rn(bal, bare, pr) : pr + PI) : (R)0;
    t.ud = DU ? mul_rn(mj, fma_rn((R)0.5, PI, tpr)) : (R)0;
    t.vg = DU ? fma_rn(vz, t.gz, fma_rn(vx, t.gx, mul_rn(vy, t.gy))) : (R)0;
    return t;
}

template <typename R, bool ACC, bool DU>
__device__ __forceinline__ void hydro_add(const HydroTerms<R> &t, R &ax, R &ay, R &az, R &du, R &vmax) {
    if (ACC) {
        if (t.vsig > vmax) vmax = t.vsig;
        ax = fma_rn(-t.pt, t.gx, ax);
        ay = fma_rn(-t.pt, t.gy, ay);
        az = fma_rn(-t.pt, t.gz, az);
    }
    if (DU) du = fma_rn(t.ud, t.vg, du);
}

template <typename R, int VISC, bool ACC, bool DU>
__global__ void __launch_bounds__(kWalkWarps * 32, kWalkMinBlocks) k_hydro(YArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    const WalkArgs &a = A.w;
    using E = YE<R>;
    if (A.only_overflow && *A.ovf == 0) return;  // every list fitted
    WarpMem wm = carve_warp_mem(smem, a.stack_cap, sizeof(E) * 64);
    E *tile = reinterpret_cast<E *>(wm.tile);
    const int lane = lane_id();
    unsigned long long pairs = 0;
    const R alpha = (R)A.alpha, beta = (R)A.beta, eta2 = (R)(A.eta * A.eta);
    for (int g = next_group(a.work, a.status); g < *a.ngroups_dev; g = next_group(a.work, a.status)) {
        GroupInfo gi = group_info(a, g);
        const bool mine = !A.only_overflow || (gi.active && A.nlist[gi.i] > A.list_cap);
        if (A.only_overflow && !__any_sync(kFull, mine)) continue;
        GroupBox gb = group_box(gi.prel, gi.active, gi.ref, gi.s10);
        gb.first = gi.first;
        const int i = gi.i;
        R tx, ty, tz, tvx, tvy, tvz, th, trho, tpr, tc, tf;
        if (sizeof(R) == 8) {
            tx = (R)a.pos[i]; ty = (R)a.pos[a.n + i]; tz = (R)a.pos[2 * a.n + i];
            tvx = (R)A.vel[i]; tvy = (R)A.vel[a.n + i]; tvz = (R)A.vel[2 * a.n + i];
            th = (R)A.h[i]; trho = (R)A.rho[i];
            tpr = (R)(A.P[i] / (A.rho[i] * A.rho[i]));
            tc = (R)A.c[i]; tf = (R)A.bal[i];
        } else {
            tx = (R)gi.prel.x; ty = (R)gi.prel.y; tz = (R)gi.prel.z;
            const float4 v = A.pk_vel[i];
            tvx = (R)v.x; tvy = (R)v.y; tvz = (R)v.z;
            th = (R)A.pk_hme[i].x;
            const float4 t = A.pk_thm[i];
            trho = (R)t.x; tpr = (R)t.y; tc = (R)t.z; tf = (R)t.w;
        }
        const float hmax_g = warp_max(gi.active ? (float)th : 0.f);
        R ax = 0, ay = 0, az = 0, du = 0, vmax = 0;
        const Images ims = group_images(gb, hmax_g + a.box_h[gi.root].w, a.box, a.periodic);
        for (int im = 0; im < 27; ++im) {
            float3 s;
            if (!image_shift(ims, im, a.box, s)) continue;
            auto load = [&](int j, bool &keep) {
                E en;
                float3 f;
                if (sizeof(R) == 8) {
                    f = frame_pos(a, gi, j, s);
                    en.p = src_pos<R>(a, gi, j, s, (R)A.h[j]);
                    en.v.x = (R)A.vel[j]; en.v.y = (R)A.vel[a.n + j]; en.v.z = (R)A.vel[2 * a.n + j];
                    en.v.w = (R)A.m[j];
                    const double rj = A.rho[j];
                    en.t.x = (R)rj;
                    en.t.y = (R)(A.P[j] / (rj * rj));
                    en.t.z = (R)A.c[j];
                    en.t.w = (R)A.bal[j];
                } else {
                    const float4 hm = A.pk_hme[j];
                    en.p = src_pos<R>(a, gi, j, s, (R)hm.x);
                    const float4 v = A.pk_vel[j];
                    en.v.x = (R)v.x; en.v.y = (R)v.y; en.v.z = (R)v.z; en.v.w = (R)hm.y;
                    const float4 t = A.pk_thm[j];
                    en.t.x = (R)t.x; en.t.y = (R)t.y; en.t.z = (R)t.z; en.t.w = (R)t.w;
                    f = make_float3((float)en.p.x, (float)en.p.y, (float)en.p.z);
                }
                keep = reaches(gb, f, hmax_g + (float)en.p.w);
                return en;
            };
            auto interact = [&](const E *tl, int ne) {
                if (!gi.active) return;
                pairs += ne;
                // pass 1: which staged sources lie inside this target's support
                unsigned mask = 0;
                for (int e = 0; e < ne; ++e) {
                    const V4<R> p = tl[e].p;
                    bool in;
                    if (sizeof(R) == 8) {
                        const double ddx = __dsub_rn((double)tx, (double)p.x);
                        const double ddy = __dsub_rn((double)ty, (double)p.y);
                        const double ddz = __dsub_rn((double)tz, (double)p.z);
                        const double hs = __dadd_rn((double)th, (double)p.w);
                        // settled in FP32 but for a narrow band, as the density pass does
                        const float fx = (float)ddx, fy = (float)ddy, fz = (float)ddz, fh = (float)hs;
                        const float d2 = fmaf(fx, fx, fmaf(fy, fy, fz * fz));
                        const float lo = fh * (1.f - kNearRel), hi = fh * (1.f + kNearRel);
                        in = d2 < fmaf(lo, lo, -kNearSq);
                        if (!in && !(d2 > fmaf(hi, hi, kNearSq)))
                            in = __ddiv_rn(exact_dist(ddx, ddy, ddz), __dmul_rn(0.5, hs)) <= 2.0;
                    } else {
                        const float fx = (float)tx - (float)p.x;
                        const float fy = (float)ty - (float)p.y;
                        const float fz = (float)tz - (float)p.z;
                        const float hs = (float)th + (float)p.w;
                        in = fmaf(fx, fx, fmaf(fy, fy, fz * fz)) <= hs * hs;
                    }
                    mask |= (unsigned)in << e;
                }
                // pass 2: each lane runs the pair terms only on its own neighbours
                while (mask) {
                    const int e = __ffs(mask) - 1;
                    mask &= mask - 1;
                    const E en = tl[e];
                    R dx, dy, dz, rr, hij, q;
                    bool in;
                    if (sizeof(R) == 8) {
                        const double ddx = __dsub_rn((double)tx, (double)en.p.x);
                        const double ddy = __dsub_rn((double)ty, (double)en.p.y);
                        const double ddz = __dsub_rn((double)tz, (double)en.p.z);
                        const double drr = exact_dist(ddx, ddy, ddz);
                        const double dh = __dmul_rn(0.5, __dadd_rn((double)th, (double)en.p.w));
                        const double dq = __ddiv_rn(drr, dh);
                        in = dq <= 2.0;
                        dx = (R)ddx; dy = (R)ddy; dz = (R)ddz; rr = (R)drr; hij = (R)dh; q = (R)dq;
                    } else {
                        dx = tx - en.p.x;
                        dy = ty - en.p.y;
                        dz = tz - en.p.z;
                        const R d2 = dx * dx + dy * dy + dz * dz;
                        const R hs = th + en.p.w;
                        in = d2 <= hs * hs;
                        rr = d2 > (R)0 ? (R)((float)d2 * rsqrtf((float)d2)) : (R)0;  // as the list pass
                        hij = (R)0.5 * hs;
                        q = (R)((float)rr * __fdividef(1.0f, (float)hij));
                    }
                    (void)in;
                    hydro_add<R, ACC, DU>(hydro_terms<R, VISC, ACC, DU>(dx, dy, dz, rr, hij, q, tvx, tvy, tvz, trho,
                                                                        tpr, tc, tf, en.v, en.t, alpha, beta, eta2),
                                          ax, ay, az, du, vmax);
                }
            };
            auto flush = [&](int nl) {
                flush_leaves_compact(a.range, wm.leafq, nl, tile, load, interact);
            };
            collect_leaves(a, wm, gi.root, gb, hmax_g, true, s, flush);
        }
        if (gi.active && mine) {
            if (ACC) {
                A.acc_sph[i] = (double)ax;
                A.acc_sph[a.n + i] = (double)ay;
                A.acc_sph[2 * a.n + i] = (double)az;
                A.vsig[i] = (double)vmax;
            }
            if (DU) A.dudt[i] = (double)du;
        }
    }
    pairs = warp_sum(pairs);
    if (lane == 0) atomicAdd(&a.counters[3], pairs);
}

// ============================================================ hydro over lists
// Mixed path: the hydro pass over the neighbour lists kept by the density
// walk, one thread or four lanes per particle.  The lists hold exactly the in-support pairs
// (|r| <= h_i + h_j in FP32, the same test as the walks' first pass) in the
// order the density walk met them, so this is the walk's pair loop without
// the walk: no tree traversal, no candidate tests.  Pair terms are the
// reference's (sph_code/libsx.py:117-165 acceleration, :364-417 du/dt; MG83
// :236-246; Balsara sph_code/shear.py:193-215) in FP32 on positions relative
// to the target's level-10 cell.  Periodic boxes use the minimum image (a
// unique image within the support: 2h < L/2 is checked by the h search).
// Particles whose list overflowed are skipped here and walked instead.
struct LArgs {
    const int *list, *nlist;
    int list_cap;
    const float4 *pk_pos, *pk_hme, *pk_vel, *pk_thm;
    float4 *hrec;  // [n][3] source records, packed by k_pack_hrec
    const uint64_t *key;
    int cloud_shift;
    const Cloud *clouds;
    int64_t n;
    int periodic;
    float box[3];
    double *acc_sph, *dudt, *vsig;
    float alpha, beta, eta2;
    unsigned long long *counters;
    // FP64 path: the masters
    const double *pos, *vel, *h, *m, *rho, *P, *c, *bal;
    double boxd[3];
    double alpha_d, beta_d, eta2_d;
};

// One 48-byte record per source, everything a hydro pair reads from it in two
// 32-byte sectors instead of four (pk_pos, pk_hme, pk_vel, pk_thm).  The
// Balsara factor stays in pk_thm: 64-byte records with it made the pass slower
// (Kelvin-Helmholtz at 4,194,304, one pass: 2.51 against 1.78 ms).
__global__ void k_pack_hrec(LArgs A) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < A.n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float4 hm = A.pk_hme[i], v = A.pk_vel[i], t = A.pk_thm[i];
        A.hrec[3 * i] = A.pk_pos[i];
        A.hrec[3 * i + 1] = make_float4(v.x, v.y, v.z, hm.y);
        A.hrec[3 * i + 2] = make_float4(t.x, t.y, t.z, hm.x);
    }
}

__device__ __forceinline__ float min_image(float d, float L) {
    if (L > 0.f) d -= L * rintf(d * (1.0f / L));
    return d;
}

// The pairs are added in list order, whichever way a particle is run: partial
// sums round differently, and the h rule turns any difference in the positions
// into a step of 3 % in h where a neighbour count comes out on the other side of
// its window.
// LPP = 1: a thread per particle.  LPP = 4: four lanes share a particle, each
// computing every fourth pair; they transpose the factors of their four pairs
// and each adds those of one output (ax, ay, az, du/dt).
__device__ __forceinline__ void transpose4(float (&v)[4], unsigned mask, int sub) {
    // v[x] of lane c becomes v[c] of lane x, over the four lanes of `mask`
    const bool b0 = sub & 1, b1 = sub & 2;
#pragma unroll
    for (int x = 0; x < 4; x += 2) {
        const float r = __shfl_xor_sync(mask, b0 ? v[x] : v[x + 1], 1);
        if (b0) v[x] = r;
        else v[x + 1] = r;
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const float r = __shfl_xor_sync(mask, b1 ? v[x] : v[x + 2], 2);
        if (b1) v[x] = r;
        else v[x + 2] = r;
    }
}

template <int VISC, bool ACC, bool DU, int LPP>
__global__ void __launch_bounds__(128, 7) k_hydro_list(LArgs A) {
    static_assert(LPP == 1 || LPP == 4, "lanes per particle");
    unsigned long long pairs = 0;
    const float alpha = A.alpha, beta = A.beta, eta2 = A.eta2;
    const int sub = threadIdx.x & (LPP - 1);
    const unsigned gm = ((1u << LPP) - 1u) << (threadIdx.x & 31 & ~(LPP - 1));
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LPP; i < A.n;
         i += (int64_t)gridDim.x * blockDim.x / LPP) {
        const int cnt = A.nlist[i];
        if (cnt > A.list_cap) continue;  // walked instead
        const float s10 = A.clouds[(int)(A.key[i] >> A.cloud_shift)].s10;
        const float4 *self = A.hrec + 3 * i;
        const float4 pi = self[0], tv = self[1], tt = self[2];  // tt = {rho, P/rho^2, c, h}
        const int ref = __float_as_int(pi.w);
        const float3 t = rel_to(pi, ref, s10);
        const float th = tt.w;
        const float tf = VISC == SPH3_VISC_BALSARA ? A.pk_thm[i].w : 0.f;
        // source records {pos}, {vx, vy, vz, m}, {rho, P/rho^2, c, h}, and f
        float4 q0, q1, q2;
        float qf = 0.f;
        auto fetch = [&](int j) {
            const float4 *r = A.hrec + 3 * (size_t)j;
            q0 = r[0];
            q1 = r[1];
            q2 = r[2];
            if (VISC == SPH3_VISC_BALSARA) qf = A.pk_thm[j].w;
        };
        auto pair = [&](float4 r0, float4 r1, float4 r2, float fj) {
            const float3 p = rel_to(r0, ref, s10);
            float dx = t.x - p.x, dy = t.y - p.y, dz = t.z - p.z;
            if (A.periodic) {
                dx = min_image(dx, A.box[0]);
                dy = min_image(dy, A.box[1]);
                dz = min_image(dz, A.box[2]);
            }
            const float d2 = dx * dx + dy * dy + dz * dz;
            const float hs = th + r2.w;
            const float rr = d2 > 0.f ? d2 * rsqrtf(d2) : 0.f;  // as the density pass computes |r|
            const float hij = 0.5f * hs;
            const float q = rr * __fdividef(1.0f, hij);
            const V4<float> sv{r1.x, r1.y, r1.z, r1.w};
            const V4<float> st{r2.x, r2.y, r2.z, fj};
            return hydro_terms<float, VISC, ACC, DU>(dx, dy, dz, rr, hij, q, tv.x, tv.y, tv.z, tt.x, tt.y, tt.z, tf, sv,
                                                     st, alpha, beta, eta2);
        };
        const int *row = A.list + (size_t)i * A.list_cap;
        float vmax = 0.f;
        if constexpr (LPP == 1) {
            // The row's indices come 4 at a time (16-byte loads, one chunk ahead:
            // a row holds list_cap slots, a multiple of 8, so whole chunks stay
            // inside it) and the next source's record is in flight while this
            // pair runs.
            float ax = 0.f, ay = 0.f, az = 0.f, du = 0.f;
            const int4 *row4 = reinterpret_cast<const int4 *>(row);
            int4 ids = cnt > 0 ? row4[0] : make_int4(0, 0, 0, 0);
            int4 ids_next = cnt > 4 ? row4[1] : ids;
            if (cnt > 0) fetch(ids.x);
            for (int k = 0; k < cnt; ++k) {
                const float4 r0 = q0, r1 = q1, r2 = q2;
                const float rf = qf;
                const int kn = k + 1;
                if (kn < cnt) {
                    const int x = kn & 3;
                    if (x == 0) {
                        ids = ids_next;
                        if (kn + 4 < cnt) ids_next = row4[(kn >> 2) + 1];
                    }
                    fetch(x == 0 ? ids.x : (x == 1 ? ids.y : (x == 2 ? ids.z : ids.w)));
                }
                hydro_add<float, ACC, DU>(pair(r0, r1, r2, rf), ax, ay, az, du, vmax);
            }
            pairs += (unsigned long long)cnt;
            if (ACC) {
                A.acc_sph[i] = (double)ax;
                A.acc_sph[A.n + i] = (double)ay;
                A.acc_sph[2 * A.n + i] = (double)az;
                A.vsig[i] = (double)vmax;
            }
            if (DU) A.dudt[i] = (double)du;
        } else {
            // consecutive lanes read consecutive indices; the index two pairs
            // ahead and the next record are in flight while a pair runs
            float sum = 0.f;  // this lane's component
            int jn = sub < cnt ? row[sub] : 0, jnn = sub + LPP < cnt ? row[sub + LPP] : 0;
            fetch(jn);
            for (int k0 = 0; k0 < cnt; k0 += LPP) {
                const int k = k0 + sub;
                const float4 r0 = q0, r1 = q1, r2 = q2;
                const float rf = qf;
                jn = jnn;
                if (k + 2 * LPP < cnt) jnn = row[k + 2 * LPP];
                if (k + LPP < cnt) fetch(jn);
                HydroTerms<float> p = {};
                if (k < cnt) {
                    p = pair(r0, r1, r2, rf);
                    if (ACC && p.vsig > vmax) vmax = p.vsig;
                }
                // lane c gets the c-th factors of all four pairs
                float f[4] = {-p.pt, -p.pt, -p.pt, p.ud}, g[4] = {p.gx, p.gy, p.gz, p.vg};
                transpose4(f, gm, sub);
                transpose4(g, gm, sub);
#pragma unroll
                for (int x = 0; x < 4; ++x)
                    if (k0 + x < cnt) sum = fma_rn(f[x], g[x], sum);
            }
            if (ACC) {
                vmax = fmaxf(vmax, __shfl_xor_sync(gm, vmax, 1));
                vmax = fmaxf(vmax, __shfl_xor_sync(gm, vmax, 2));
            }
            if (sub == 0) pairs += (unsigned long long)cnt;
            if (sub < 3) {
                if (ACC) A.acc_sph[sub * A.n + i] = (double)sum;
            } else {
                if (ACC) A.vsig[i] = (double)vmax;
                if (DU) A.dudt[i] = (double)sum;
            }
        }
    }
    pairs = warp_sum(pairs);
    if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(&A.counters[3], pairs);
}

// FP64 path over the same lists: the walk's FP64 pair arithmetic (the
// reference's operation order, correctly rounded predicates) with the periodic
// image the walk uses (source shifted by the FP32-rounded box length), and the
// pairs added in list order, so the results equal the walk's.
// kHydro64Lanes lanes share a particle: each computes every fourth pair, and all
// add the four pairs' terms in order.  The sources come as 96-byte records
// {x, y, z, h, vx, vy, vz, m, rho, P/rho^2, c, f}: three sectors a pair instead
// of one for each of twelve arrays.  131,072 particles: 246 us with a thread per
// particle on the arrays, 220 now; 10,000: 115 and 26.
constexpr int kHydro64Lanes = 4;

__global__ void k_pack_hrec_f64(LArgs A) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < A.n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double r = A.rho[i];
        double2 *o = reinterpret_cast<double2 *>(A.hrec) + 6 * i;
        o[0] = make_double2(A.pos[i], A.pos[A.n + i]);
        o[1] = make_double2(A.pos[2 * A.n + i], A.h[i]);
        o[2] = make_double2(A.vel[i], A.vel[A.n + i]);
        o[3] = make_double2(A.vel[2 * A.n + i], A.m[i]);
        o[4] = make_double2(r, A.P[i] / (r * r));
        o[5] = make_double2(A.c[i], A.bal[i]);
    }
}

template <int VISC>
__global__ void __launch_bounds__(128, 4) k_hydro_list_f64(LArgs A) {
    constexpr int LPP = kHydro64Lanes;
    unsigned long long pairs = 0;
    const int64_t n = A.n;
    const int sub = threadIdx.x & (LPP - 1);
    const unsigned gm = ((1u << LPP) - 1u) << (threadIdx.x & 31 & ~(LPP - 1));
    const double2 *rec = reinterpret_cast<const double2 *>(A.hrec);
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LPP; i < n;
         i += (int64_t)gridDim.x * blockDim.x / LPP) {
        const int cnt = A.nlist[i];
        if (cnt > A.list_cap) continue;  // walked instead
        const double2 t0 = rec[6 * i], t1 = rec[6 * i + 1], t2 = rec[6 * i + 2], t3 = rec[6 * i + 3],
                      t4 = rec[6 * i + 4], t5 = rec[6 * i + 5];
        const double ti[3] = {t0.x, t0.y, t1.x}, th = t1.y;
        double ax = 0, ay = 0, az = 0, du = 0, vmax = 0;
        const int *row = A.list + (size_t)i * A.list_cap;
        int jn = sub < cnt ? row[sub] : 0;
        for (int k0 = 0; k0 < cnt; k0 += LPP) {
            const int j = jn;
            if (k0 + LPP + sub < cnt) jn = row[k0 + LPP + sub];
            HydroTerms<double> t = {};
            if (k0 + sub < cnt) {
                const double2 s0 = rec[6 * j], s1 = rec[6 * j + 1], s2 = rec[6 * j + 2], s3 = rec[6 * j + 3],
                              s4 = rec[6 * j + 4], s5 = rec[6 * j + 5];
                double pj[3] = {s0.x, s0.y, s1.x};
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const double L = A.boxd[d];
                    if (L > 0.0) {
                        const double dd = ti[d] - pj[d];
                        if (dd > 0.5 * L) pj[d] += (double)(float)L;
                        else if (dd < -0.5 * L) pj[d] += (double)(-(float)L);
                    }
                }
                const double ddx = __dsub_rn(ti[0], pj[0]);
                const double ddy = __dsub_rn(ti[1], pj[1]);
                const double ddz = __dsub_rn(ti[2], pj[2]);
                const double drr = exact_dist(ddx, ddy, ddz);
                const double dh = __dmul_rn(0.5, __dadd_rn(th, s1.y));
                const double dq = __ddiv_rn(drr, dh);
                const V4<double> sv{s2.x, s2.y, s3.x, s3.y};
                const V4<double> st{s4.x, s4.y, s5.x, s5.y};
                t = hydro_terms<double, VISC, true, true>(ddx, ddy, ddz, drr, dh, dq, t2.x, t2.y, t3.x, t4.x, t4.y, t5.x,
                                                       t5.y, sv, st, A.alpha_d, A.beta_d, A.eta2_d);
            }
#pragma unroll
            for (int x = 0; x < LPP; ++x) {  // every lane, in list order
                HydroTerms<double> o;
                o.pt = __shfl_sync(gm, t.pt, x, LPP);
                o.gx = __shfl_sync(gm, t.gx, x, LPP);
                o.gy = __shfl_sync(gm, t.gy, x, LPP);
                o.gz = __shfl_sync(gm, t.gz, x, LPP);
                o.ud = __shfl_sync(gm, t.ud, x, LPP);
                o.vg = __shfl_sync(gm, t.vg, x, LPP);
                o.vsig = __shfl_sync(gm, t.vsig, x, LPP);
                if (k0 + x < cnt) hydro_add<double, true, true>(o, ax, ay, az, du, vmax);
            }
        }
        if (sub != 0) continue;
        pairs += (unsigned long long)cnt;
        if (A.acc_sph) {
            A.acc_sph[i] = ax;
            A.acc_sph[n + i] = ay;
            A.acc_sph[2 * n + i] = az;
            A.vsig[i] = vmax;
        }
        if (A.dudt) A.dudt[i] = du;
    }
    pairs = warp_sum(pairs);
    if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(&A.counters[3], pairs);
}

// ============================================================ neighbours
// Exact FP64 neighbour sets {j : q_ij <= 2} of selected particles; pass 0
// counts, pass 1 writes caller indices at the given offsets.  One warp per
// row, each lane testing its own staged candidate.
struct NArgs {
    WalkArgs w;
    const double *h;
    const int64_t *orig;
    const int64_t *rows;  // sorted indices
    int64_t nrows;
    int64_t *offsets;     // [nrows + 1]
    int64_t *out;
    int64_t cap;
    int *cursor;          // [nrows]
    int pass;
};

__global__ void __launch_bounds__(kWalkWarps * 32, kWalkMinBlocks) k_neighbours(NArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    const WalkArgs &a = A.w;
    using E = V4<double>;
    WarpMem wm = carve_warp_mem(smem, a.stack_cap, sizeof(E) * 64);
    E *tile = reinterpret_cast<E *>(wm.tile);
    const int lane = lane_id();
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int64_t r = gw; r < A.nrows; r += nw) {
        const int i = (int)A.rows[r];
        int cloud = 0;
        {
            int lo = 0, hi = a.ncloud - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (a.clouds[mid].begin <= i) lo = mid;
                else hi = mid - 1;
            }
            cloud = lo;
        }
        const Cloud &cl = a.clouds[cloud];
        const int ref = __float_as_int(a.pk_pos[i].w);
        const float3 prel = rel_to(a.pk_pos[i], ref, cl.s10);
        GroupBox gb = group_box(prel, lane == 0, ref, cl.s10);
        const double tx = a.pos[i], ty = a.pos[a.n + i], tz = a.pos[2 * a.n + i];
        const double th = A.h[i];
        int found = 0;
        const Images ims = group_images(gb, (float)th + a.box_h[cl.root].w, a.box, a.periodic);
        for (int im = 0; im < 27; ++im) {
            float3 s;
            if (!image_shift(ims, im, a.box, s)) continue;
            auto load = [&](int j) {
                const double dx = __dsub_rn(tx, a.pos[j] + (double)s.x);
                const double dy = __dsub_rn(ty, a.pos[a.n + j] + (double)s.y);
                const double dz = __dsub_rn(tz, a.pos[2 * a.n + j] + (double)s.z);
                const double rr = exact_dist(dx, dy, dz);
                const double hij = __dmul_rn(0.5, __dadd_rn(th, A.h[j]));
                if (__ddiv_rn(rr, hij) <= 2.0) {
                    ++found;
                    if (A.pass == 1) {
                        const int k = atomicAdd(&A.cursor[r], 1);
                        const int64_t at = A.offsets[r] + k;
                        if (at < A.cap) A.out[at] = A.orig[j];
                        else set_status(a.status, SPH3_STATUS_LIST_OVERFLOW);
                    }
                }
                return E{};
            };
            auto interact = [&](const E *t, int ne) {
                (void)t;
                (void)ne;
            };
            auto flush = [&](int nl) {
                flush_leaves(a.range, wm.leafq, nl, tile, load, interact);
            };
            collect_leaves(a, wm, cl.root, gb, (float)th, true, s, flush);
        }
        found = warp_sum(found);
        if (A.pass == 0 && lane == 0) A.offsets[r] = found;
    }
}

// ============================================================ launchers
static WalkArgs walk_args(State &S, const Params &P, int slot) {
    WalkArgs a;
    a.groups = S.groups;
    a.ngroups_dev = S.ngroups_dev;
    a.group_cloud = S.group_cloud;
    a.clouds = S.clouds;
    a.ncloud = S.ncloud;
    a.range = S.tree.range;
    a.child = S.tree.child;
    a.box_c = S.tree.box_c;
    a.box_h = S.tree.box_h;
    a.sw = S.tree.sw;
    a.pk_pos = S.pk_pos;
    a.pos = S.pos;
    a.n = S.n;
    a.stack_cap = P.stack_cap;
    a.max_depth = S.max_level + 1;
    a.node_cap = S.tree.cap;
    a.periodic = P.periodic;
    for (int d = 0; d < 3; ++d) a.box[d] = P.box[d];
    a.work = S.work + slot;
    a.status = S.status;
    a.counters = S.counters;
    // node-visit counters: boot h / h search / density / hydro / neighbours
    static const int kVisitSlot[5] = {kCntVisitsH, kCntVisitsH, kCntVisitsDensity, kCntVisitsHydro, kCntVisitsH};
    a.visit_slot = kVisitSlot[slot];
    return a;
}

// dynamic shared memory of a walk warp whose tile holds 64 entries E (double
// buffered) and `extra` bytes after them
template <typename E>
static size_t walk_smem(const Params &P, size_t extra = 0) {
    return warp_mem_bytes(P.stack_cap, sizeof(E) * 64 + extra);
}

template <typename Args>
static void run_walk(void (*kern)(Args), const Args &args, size_t warp_smem, State &S, cudaStream_t st, int slot,
                     int team = 1) {
    allow_smem((const void *)kern);
    cudaMemsetAsync(S.work + slot, 0, sizeof(int), st);
    // persistent grid: 32 warps' worth of blocks per SM; a team is a block
    const int warps = team > 1 ? team : warps_that_fit(S.walk_warps, warp_smem);
    kern<<<S.num_sms * (32 / warps), warps * 32, warp_smem * warps, st>>>(args);
}

void launch_boot_h(State &S, const Params &P, cudaStream_t st) {
    S.list_valid = false;
    if (S.n == 0) return;
    BootArgs A;
    A.w = walk_args(S, P, 0);
    A.h = S.h;
    A.pk_hme = S.pk_hme;
    A.k = P.n_boot;
    run_walk(k_boot_h, A, walk_smem<V4<double>>(P), S, st, 0);
}

// eps = h (the reference GPU driver's set_eps_of_gas_to_h)
__global__ void k_eps_from_h(int64_t n, const double *h, double *eps, float4 *pk_hme) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        eps[i] = h[i];
        pk_hme[i].z = (float)h[i];
    }
}

void launch_h_search(State &S, const Params &P, cudaStream_t st) {
    S.list_valid = false;  // new h: the supports change
    if (S.n == 0) return;
    HArgs A;
    A.w = walk_args(S, P, 1);
    A.h = S.h;
    A.pk_hme = S.pk_hme;
    A.nngb = S.nngb;
    A.n_ngb = P.n_ngb;
    A.tol = P.n_ngb_tol;
    A.max_iter = P.h_max_iter;
    const bool fp64 = P.precision == SPH3_PREC_FP64;
    auto run = [&](auto *alone, auto *shared, size_t tile, size_t counts) {
        const int team = warps_that_fit(kTeamH[fp64](S.n), tile + counts);
        run_walk(team > 1 ? shared : alone, A, tile + (team > 1 ? counts : 0), S, st, 1, team);
    };
    const size_t t64 = warp_mem_bytes(P.stack_cap, sizeof(float) * 64 * h_fields<double>());
    const size_t t32 = warp_mem_bytes(P.stack_cap, sizeof(float) * 64 * h_fields<float>());
    constexpr size_t cr = h_count_bytes<SPH3_H_REFSTEP>(), cn = h_count_bytes<SPH3_H_NEWTON>();
    if (fp64 && P.h_mode == SPH3_H_REFSTEP)
        run(k_h_search<double, SPH3_H_REFSTEP, false>, k_h_search<double, SPH3_H_REFSTEP, true>, t64, cr);
    else if (fp64)
        run(k_h_search<double, SPH3_H_NEWTON, false>, k_h_search<double, SPH3_H_NEWTON, true>, t64, cn);
    else if (P.h_mode == SPH3_H_REFSTEP)
        run(k_h_search<float, SPH3_H_REFSTEP, false>, k_h_search<float, SPH3_H_REFSTEP, true>, t32, cr);
    else
        run(k_h_search_f32_newton, k_h_search<float, SPH3_H_NEWTON, true>, t32, cn);
    if (P.eps_from_h) {
        const int blocks = (int)std::min<int64_t>((S.n + 255) / 256, (int64_t)S.num_sms * 8);
        k_eps_from_h<<<blocks, 256, 0, st>>>(S.n, S.h, S.eps, S.pk_hme);
    }
}

void launch_density(State &S, const Params &P, bool divcurl, cudaStream_t st, bool keep_rho, bool lists_only) {
    if (S.n == 0) return;
    DArgs A;
    A.keep_rho = keep_rho ? 1 : 0;
    A.w = walk_args(S, P, 2);
    A.pk_hme = S.pk_hme; A.pk_vel = S.pk_vel;
    A.h = S.h; A.m = S.m; A.vel = S.vel; A.u = S.u;
    A.rho = S.rho; A.P = S.P; A.c = S.c; A.divV = S.divV; A.curlV = S.curlV; A.bal = S.bal;
    A.pk_thm = S.pk_thm;
    A.gamma = P.gamma;
    A.list = S.list_cap > 0 ? S.list : nullptr;
    A.nlist = S.nlist;
    A.list_cap = S.list_cap;
    A.ovf = S.ovf;
    if (A.list) cudaMemsetAsync(S.ovf, 0, sizeof(int), st);
    // particles outside a restricted pass keep no pairs
    if (A.list && S.rows_only) cudaMemsetAsync(S.nlist, 0, sizeof(int) * (size_t)S.n, st);
    S.list_valid = A.list != nullptr;
    S.list_hidden = lists_only;
    const bool fp64 = P.precision == SPH3_PREC_FP64;
    auto run = [&](auto *alone, auto *shared, size_t tile) {
        const size_t warp_smem = warp_mem_bytes(P.stack_cap, tile);
        const int team = warps_that_fit((divcurl ? kTeamDivcurl : kTeamDensity)[fp64](S.n), warp_smem);
        run_walk(team > 1 ? shared : alone, A, warp_smem, S, st, 2, team);
    };
    if (lists_only)
        run(k_make_lists<false>, k_make_lists<true>, density_tile_bytes<double, false>());
    else if (fp64 && divcurl)
        run(k_density<double, true, false>, k_density<double, true, true>, density_tile_bytes<double, true>());
    else if (fp64)
        run(k_density<double, false, false>, k_density<double, false, true>, density_tile_bytes<double, false>());
    else if (divcurl)
        run(k_density_dc_f32, k_density<float, true, true>, density_tile_bytes<float, true>());
    else
        run(k_density_f32, k_density<float, false, true>, density_tile_bytes<float, false>());
}

template <typename R, int V>
static void hydro_dispatch(const YArgs &A, bool acc, bool du, const Params &P, State &S, cudaStream_t st) {
    const size_t sm = walk_smem<YE<R>>(P);
    if (acc && du) run_walk(k_hydro<R, V, true, true>, A, sm, S, st, 3);
    else if (acc) run_walk(k_hydro<R, V, true, false>, A, sm, S, st, 3);
    else run_walk(k_hydro<R, V, false, true>, A, sm, S, st, 3);
}

template <int V, int LPP>
static void list_launch_f32(const LArgs &L, int num_sms, cudaStream_t st) {
    // blocks of 128 threads, at most 32 a SM (7 resident, 28 warps, at <= 72 registers)
    const int blocks = (int)std::min<int64_t>((L.n * LPP + 127) / 128, (int64_t)num_sms * 32);
    if (L.acc_sph && L.dudt) k_hydro_list<V, true, true, LPP><<<blocks, 128, 0, st>>>(L);
    else if (L.acc_sph) k_hydro_list<V, true, false, LPP><<<blocks, 128, 0, st>>>(L);
    else k_hydro_list<V, false, true, LPP><<<blocks, 128, 0, st>>>(L);
}

// FP64: one kernel for the acceleration and du/dt, storing those whose arrays
// are set (instances for one of them alone: 382 and 665 us at 100,000 particles,
// 207 with both).
template <int V>
static void list_launch(const LArgs &L, bool fp64, int num_sms, cudaStream_t st) {
    if (fp64) {
        const int blocks = (int)std::min<int64_t>((L.n * kHydro64Lanes + 127) / 128, (int64_t)num_sms * 32);
        k_hydro_list_f64<V><<<blocks, 128, 0, st>>>(L);
    } else if (L.n <= kHydroLanes4) {
        list_launch_f32<V, 4>(L, num_sms, st);
    } else {
        list_launch_f32<V, 1>(L, num_sms, st);
    }
}

void launch_hydro(State &S, const Params &P, bool want_acc, bool want_dudt, cudaStream_t st) {
    if (S.n == 0 || (!want_acc && !want_dudt)) return;
    YArgs A;
    A.w = walk_args(S, P, 3);
    A.pk_hme = S.pk_hme; A.pk_vel = S.pk_vel; A.pk_thm = S.pk_thm;
    A.h = S.h; A.m = S.m; A.vel = S.vel; A.rho = S.rho; A.P = S.P; A.c = S.c; A.bal = S.bal;
    A.acc_sph = S.acc_sph; A.dudt = S.dudt; A.vsig = S.vsig;
    A.alpha = P.alpha; A.beta = P.beta; A.eta = P.eta;
    A.nlist = S.nlist;
    A.list_cap = S.list_cap;
    A.only_overflow = 0;
    A.ovf = S.ovf;
    // FP64 without lists (forces from given rho, P, c): make them first; the
    // list pass gives the walk's bits, and the two passes are far shorter than a
    // walk that runs every pair lane by lane (10,000 particles: 223 us walked, 68
    // for both).  Periodic boxes, whose given h may
    // exceed what a minimum image covers, walk.
    if (!S.list_valid && S.list_cap > 0 && P.precision == SPH3_PREC_FP64 && !P.periodic)
        launch_density(S, P, false, st, false, true);
    if (S.list_valid) {
        // the list pass, then a walk for the particles whose lists overflowed
        const bool fp64 = P.precision == SPH3_PREC_FP64;
        LArgs L;
        L.list = S.list; L.nlist = S.nlist; L.list_cap = S.list_cap;
        L.pk_pos = S.pk_pos; L.pk_hme = S.pk_hme; L.pk_vel = S.pk_vel; L.pk_thm = S.pk_thm;
        L.key = S.key; L.cloud_shift = 3 * S.max_level; L.clouds = S.clouds;
        L.n = S.n;
        L.periodic = P.periodic;
        for (int d = 0; d < 3; ++d) L.box[d] = (float)P.box[d];
        L.acc_sph = S.acc_sph; L.dudt = S.dudt; L.vsig = S.vsig;
        L.alpha = (float)P.alpha; L.beta = (float)P.beta; L.eta2 = (float)(P.eta * P.eta);
        L.counters = S.counters;
        L.hrec = S.hrec;
        L.pos = S.pos; L.vel = S.vel; L.h = S.h; L.m = S.m; L.rho = S.rho; L.P = S.P; L.c = S.c; L.bal = S.bal;
        for (int d = 0; d < 3; ++d) L.boxd[d] = P.box[d];
        L.alpha_d = P.alpha; L.beta_d = P.beta; L.eta2_d = P.eta * P.eta;
        const int blocks = (int)std::min<int64_t>((S.n + 255) / 256, (int64_t)S.num_sms * 16);
        if (fp64) k_pack_hrec_f64<<<blocks, 256, 0, st>>>(L);
        else k_pack_hrec<<<blocks, 256, 0, st>>>(L);
        if (!want_acc) L.acc_sph = nullptr;
        if (!want_dudt) L.dudt = nullptr;
        if (P.visc == SPH3_VISC_MG83) list_launch<SPH3_VISC_MG83>(L, fp64, S.num_sms, st);
        else if (P.visc == SPH3_VISC_BALSARA) list_launch<SPH3_VISC_BALSARA>(L, fp64, S.num_sms, st);
        else list_launch<SPH3_VISC_SIGNAL>(L, fp64, S.num_sms, st);
        A.only_overflow = 1;
    }
    if (P.precision == SPH3_PREC_FP64) {
        if (P.visc == SPH3_VISC_MG83) hydro_dispatch<double, SPH3_VISC_MG83>(A, want_acc, want_dudt, P, S, st);
        else if (P.visc == SPH3_VISC_BALSARA) hydro_dispatch<double, SPH3_VISC_BALSARA>(A, want_acc, want_dudt, P, S, st);
        else hydro_dispatch<double, SPH3_VISC_SIGNAL>(A, want_acc, want_dudt, P, S, st);
    } else {
        if (P.visc == SPH3_VISC_MG83) hydro_dispatch<float, SPH3_VISC_MG83>(A, want_acc, want_dudt, P, S, st);
        else if (P.visc == SPH3_VISC_BALSARA) hydro_dispatch<float, SPH3_VISC_BALSARA>(A, want_acc, want_dudt, P, S, st);
        else hydro_dispatch<float, SPH3_VISC_SIGNAL>(A, want_acc, want_dudt, P, S, st);
    }
}

// P and c from the stored rho and u (getPressure, sph_serial.py:116), plus
// the Balsara factor from the stored div/curl (shear.py:212-213)
__global__ void k_eos(int64_t n, double gamma, const double *rho, const double *u, const double *divV,
                      const double *curlV, const double *h, double *P, double *c, double *bal,
                      float4 *pk_thm) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double r = rho[i];
        const double p = (gamma - 1.0) * r * u[i];
        const double cc = sqrt(gamma * (gamma - 1.0) * u[i]);
        P[i] = p;
        c[i] = cc;
        const double f = divV[i] / (divV[i] + curlV[i] + 0.0001 * cc / h[i]);
        bal[i] = f;
        pk_thm[i] = make_float4((float)r, (float)(r > 0 ? p / (r * r) : 0.0), (float)cc, (float)f);
    }
}

void launch_eos(State &S, const Params &P, cudaStream_t st) {
    if (S.n == 0) return;
    int blocks = (int)std::min<int64_t>((S.n + 255) / 256, (int64_t)S.num_sms * 8);
    k_eos<<<blocks, 256, 0, st>>>(S.n, P.gamma, S.rho, S.u, S.divV, S.curlV, S.h, S.P, S.c, S.bal, S.pk_thm);
}

__global__ void k_balsara(int64_t n, const double *divV, const double *curlV, const double *c,
                          const double *h, double *bal, float4 *pk_thm) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double f = divV[i] / (divV[i] + curlV[i] + 0.0001 * c[i] / h[i]);
        bal[i] = f;
        pk_thm[i].w = (float)f;
    }
}

void launch_balsara(State &S, cudaStream_t st) {
    if (S.n == 0) return;
    int blocks = (int)std::min<int64_t>((S.n + 255) / 256, (int64_t)S.num_sms * 8);
    k_balsara<<<blocks, 256, 0, st>>>(S.n, S.divV, S.curlV, S.c, S.h, S.bal, S.pk_thm);
}

int launch_neighbours(State &S, const Params &P, const int64_t *rows_sorted_dev, int64_t nrows,
                      int64_t *offsets_dev, int64_t *idx_dev, int64_t cap, cudaStream_t st) {
    if (nrows == 0) return 0;
    NArgs A;
    A.w = walk_args(S, P, 4);
    A.h = S.h;
    A.orig = S.orig;
    A.rows = rows_sorted_dev;
    A.nrows = nrows;
    A.offsets = offsets_dev;
    A.out = idx_dev;
    A.cap = cap;
    A.cursor = nullptr;
    const size_t sm = walk_smem<V4<double>>(P) * P.walk_warps;
    allow_smem((const void *)k_neighbours);
    int blocks = (int)std::min<int64_t>((nrows + S.walk_warps - 1) / S.walk_warps, (int64_t)S.num_sms * 8);
    // pass 0: counts into offsets[0..nrows)
    A.pass = 0;
    k_neighbours<<<blocks, S.walk_warps * 32, sm, st>>>(A);
    // exclusive scan on the host (few rows)
    std::vector<int64_t> hv(nrows + 1);
    cudaMemcpyAsync(hv.data(), offsets_dev, sizeof(int64_t) * nrows, cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    int64_t run = 0;
    for (int64_t r = 0; r < nrows; ++r) {
        const int64_t v = hv[r];
        hv[r] = run;
        run += v;
    }
    hv[nrows] = run;
    cudaMemcpyAsync(offsets_dev, hv.data(), sizeof(int64_t) * (nrows + 1), cudaMemcpyHostToDevice, st);
    int *cursor = nullptr;
    cudaMallocAsync(&cursor, sizeof(int) * nrows, st);
    cudaMemsetAsync(cursor, 0, sizeof(int) * nrows, st);
    A.cursor = cursor;
    A.pass = 1;
    k_neighbours<<<blocks, S.walk_warps * 32, sm, st>>>(A);
    cudaFreeAsync(cursor, st);
    cudaStreamSynchronize(st);
    return 0;
}

}  // namespace sph3
