// Weight generation on the device.
//
// Conservative (Conservative1stOrder, GreatCircle) replaces
// generate_conservative_impl<3> (libs/axis/src/solver/weight_generator.cpp:
// 3304-3770):
//   1. cell prep per mesh (prep.cu);
//   2. an LBVH over the source cells' bounding caps: 30-bit Morton codes of
//      the cap centroids, radix-sorted leaves, Karras hierarchy, bottom-up
//      refit of FP32 boxes padded outward, and per-node ropes (escape
//      links) for stackless traversal;
//   3. one thread per destination cell walks the ropes; every leaf hit goes
//      through the reference's exact gates (source mask / degenerate /
//      area > 0, the reference's float AABB test, the FP64 cap test) and is
//      kept, grouped by row in traversal order, so the candidate list is
//      deterministic;
//   4. pairs that an edge separates are settled in FP32; for the others one
//      thread runs the FP64 great-circle clip and the spherical area
//      (geom.cuh, --fmad=false), pairs that are not convex or exceed 12
//      vertices with the reference's 32-vertex general clipper;
//   5. kept pairs (overlap > 0, the reference threshold at :3682) are placed
//      in CSR by their rank in the row (long rows: radix sort), and the weights,
//      frac_b (row order) and frac_a (column order, rows ascending) sums are
//      formed.
// Bilinear with a rectilinear source replaces
// generate_bilinear_rect_nonuniform
// (src/solver/weight_generator_bilinear_rect_nonuniform.cpp:22-149).
#include <chrono>

#include "geom.cuh"
#include "internal.hpp"
#include "lbvh.cuh"

namespace axgb {
namespace {

constexpr unsigned char kExcluded = 1 | 2 | 4;  // degenerate | masked | area <= 0

// ─── LBVH (lbvh.cuh) ───────────────────────────────────────────────────────

// Chord radius of a cap of angular radius r, rounded up into float with
// slack for the float rounding of the centre (|dc| <= 2^-24 per axis).
__device__ __forceinline__ float ball_radius(double r) {
    double rho = 2.0 * sin(0.5 * fmin(r, 3.141592653589793));
    return __double2float_ru(rho * (1.0 + 1e-6) + 1e-6);
}

__global__ void k_leaf_keys(MeshView S, unsigned *keys, int *vals) {
    i64 i = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= S.n_cells) return;
    DCap c = S.cap[i];
    keys[i] = morton30(c.x, c.y, c.z);
    vals[i] = static_cast<int>(i);
}

__global__ void k_leaves(Bvh t, MeshView S, const int *vals) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= t.n) return;
    int cell = vals[q];
    DCap c = S.cap[cell];
    float r = ball_radius(c.r);
    float4 lo, hi;
    lo.x = __fsub_rd(__double2float_rd(c.x), r);
    lo.y = __fsub_rd(__double2float_rd(c.y), r);
    lo.z = __fsub_rd(__double2float_rd(c.z), r);
    hi.x = __fadd_ru(__double2float_ru(c.x), r);
    hi.y = __fadd_ru(__double2float_ru(c.y), r);
    hi.z = __fadd_ru(__double2float_ru(c.z), r);
    lo.w = __int_as_float(cell);
    hi.w = __int_as_float(-1);
    t.lo[t.n - 1 + q] = lo;
    t.hi[t.n - 1 + q] = hi;
}

// ─── candidate search ──────────────────────────────────────────────────────

__device__ __forceinline__ bool fbox_meet(const float *a, const float *b) {
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if (a[d] > b[3 + d] || a[3 + d] < b[d]) return false;
    return true;
}

// The cap test acos(clamp(dot(c_s, c_d))) > r_s + r_d is taken in FP64 as
// the reference takes it (spherical_cap_filter.hpp:190-197), but most pairs
// are decided in FP32 first. On unit vectors the angle exceeds R exactly
// when the chord |c_s - c_d| exceeds 2 sin(R/2) (for R below pi, where
// both sides are monotone). From the float copies of the centroids and
// radii (rounding 6e-8 relative each) the float chord lies within 1.1e-6
// of the chord of the double centroids, and 2 sinf(R/2) within 0.6e-6 of
// its double value; the FP64 acos and sum differ from the exact angle and
// sum by less than 2e-8. So when the float sides differ by more than
// kCapMargin, the FP64 test returns the same answer. Nearer pairs, and sums
// above 3, take the FP64 test.
constexpr float kCapMargin = 4.0e-6f;

// Exact reference gates for a pair that the LBVH admitted.
__device__ __forceinline__ bool gate(const MeshView &S, int i, const float *dbox, const DCap &dc, const float4 &dcf) {
    if (S.flags[i] & kExcluded) return false;
    if (!fbox_meet(S.box + 6 * static_cast<i64>(i), dbox)) return false;
    const float4 sf = S.capf[i];
    const float rs = sf.w + dcf.w;
    if (rs < 3.0f) {
        const float ex = sf.x - dcf.x, ey = sf.y - dcf.y, ez = sf.z - dcf.z;
        const float ch = sqrtf(ex * ex + ey * ey + ez * ez);
        const float t = 2.0f * sinf(0.5f * rs);
        if (ch > t + kCapMargin) return false;
        if (ch < t - kCapMargin) return true;
    }
    DCap sc = S.cap[i];
    double cd = sc.x * dc.x + sc.y * dc.y + sc.z * dc.z;  // dot(centroid_s, centroid_d)
    cd = fmin(1.0, fmax(-1.0, cd));
    return !(acos(cd) > (sc.r + dc.r));
}

// One thread a row walks the ropes; the first cap candidates go to slots
// ([cap][rows]). A row that meets more, or visits more than kWalkSteps nodes,
// gives up (slots row 0 = -1) and is listed for k_search_wide: the polar rows
// of a lat-lon source have over a thousand candidates, and as one thread's
// chain of dependent loads they were the length of the whole search.
// 0.25 deg -> C384: 0.76 ms and 0.54 for the wide rows, against 2 x 2.97 ms for
// one thread a row, counting and then writing.
constexpr int kWalkSteps = 256;

__device__ __forceinline__ bool node_meets(const float4 &lo, const float4 &hi, float qx, float qy, float qz, float rq2) {
    const float dx = fmaxf(fmaxf(lo.x - qx, 0.f), qx - hi.x);
    const float dy = fmaxf(fmaxf(lo.y - qy, 0.f), qy - hi.y);
    const float dz = fmaxf(fmaxf(lo.z - qz, 0.f), qz - hi.z);
    return dx * dx + dy * dy + dz * dz <= rq2;
}

// A destination cell's query: its gates' operands, and the ball the nodes meet.
struct Query {
    DCap dc;
    float4 dcf;
    float dbox[6];
    float qx, qy, qz, rq2;
    __device__ __forceinline__ Query(const MeshView &D, i64 j) : dc(D.cap[j]), dcf(D.capf[j]) {
#pragma unroll
        for (int d = 0; d < 6; ++d) dbox[d] = D.box[6 * j + d];
        qx = static_cast<float>(dc.x);
        qy = static_cast<float>(dc.y);
        qz = static_cast<float>(dc.z);
        const float rq = ball_radius(dc.r);
        rq2 = __fmul_ru(rq, rq) * 1.000001f + 1e-12f;
    }
};

__global__ void k_search(MeshView S, MeshView D, const float4 *__restrict__ nlo, const float4 *__restrict__ nhi,
                         int root, int n_leaf_base, int *counts, int *slots, int cap, int *wide, int *n_wide,
                         unsigned long long *raw_hits) {
    i64 j = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    unsigned long long hits = 0;
    if (j < D.n_cells) {
        int cnt = 0;
        if (!(D.flags[j] & kExcluded) && root >= 0) {
            const Query q(D, j);
            int node = root;
            for (int steps = 0; node >= 0; ++steps) {
                if (steps == kWalkSteps) {
                    cnt = cap + 1;
                    break;
                }
                float4 lo = nlo[node], hi = nhi[node];
                if (node_meets(lo, hi, q.qx, q.qy, q.qz, q.rq2)) {
                    if (node >= n_leaf_base) {
                        int cell = __float_as_int(lo.w);
                        ++hits;
                        if (gate(S, cell, q.dbox, q.dc, q.dcf)) {
                            if (cnt < cap) slots[static_cast<i64>(cnt) * D.n_cells + j] = cell;
                            if (++cnt > cap) break;
                        }
                        node = __float_as_int(hi.w);
                    } else {
                        node = __float_as_int(lo.w);
                    }
                } else {
                    node = __float_as_int(hi.w);
                }
            }
        }
        if (cnt > cap) {
            slots[j] = -1;
            wide[atomicAdd(n_wide, 1)] = static_cast<int>(j);
            cnt = 0;
            hits = 0;  // counted by k_search_wide
        }
        counts[j] = cnt;
    }
    // warp-aggregated counter of raw leaf hits
    for (int o = 16; o > 0; o >>= 1) hits += __shfl_down_sync(0xffffffffu, hits, o);
    if ((threadIdx.x & 31) == 0 && hits) atomicAdd(raw_hits, hits);
}

// The listed rows, a warp each: the lanes test the 32 nodes on top of a stack
// and push the children of those that meet the query. Popping 32 and pushing
// up to 64 leaves at most 32 more; above kWideHigh entries one node is popped
// at a time, which adds one a level of the tree (at most 62), so the stack
// cannot overflow. Counts (FILL = false), then writes (the order of a row's
// candidates does not matter: the rows are sorted by column in the end).
constexpr int kWideStack = 1024, kWideHigh = kWideStack - 64 - 64, kWideWarps = 4;

template <bool FILL>
__global__ void __launch_bounds__(32 * kWideWarps) k_search_wide(MeshView S, MeshView D, const float4 *__restrict__ nlo,
                                                                const float4 *__restrict__ nhi,
                                                                const int *__restrict__ right, int root,
                                                                int n_leaf_base, const int *wide, const int *n_wide,
                                                                int *counts, const i64 *offs, int *out_src,
                                                                unsigned long long *raw_hits, int *err) {
    __shared__ int stacks[kWideWarps][kWideStack];
    const int lane = threadIdx.x & 31;
    int *st = stacks[threadIdx.x >> 5];
    const int n = *n_wide;
    unsigned long long hits = 0;
    for (int i = blockIdx.x * kWideWarps + (threadIdx.x >> 5); i < n; i += gridDim.x * kWideWarps) {
        const i64 j = wide[i];
        const Query q(D, j);
        const i64 at = FILL ? offs[j] : 0;
        int sp = 1, cnt = 0;
        i64 seen = 0;
        __syncwarp();
        if (lane == 0) st[0] = root;
        while (sp > 0) {
            __syncwarp();
            const int take = sp > kWideHigh ? 1 : min(sp, 32);
            const int node = lane < take ? st[sp - take + lane] : -1;
            sp -= take;
            // every node is reached once; more means a malformed tree: flag it and stop
            if ((seen += take) > 2 * static_cast<i64>(n_leaf_base) + 1) {
                if (lane == 0) atomicOr(err, 1);
                break;
            }
            bool inner = false, keep = false;
            int cell = -1, left = -1;
            if (node >= 0) {
                const float4 lo = nlo[node], hi = nhi[node];
                if (node_meets(lo, hi, q.qx, q.qy, q.qz, q.rq2)) {
                    if (node >= n_leaf_base) {
                        cell = __float_as_int(lo.w);
                        ++hits;
                        keep = gate(S, cell, q.dbox, q.dc, q.dcf);
                    } else {
                        inner = true;
                        left = __float_as_int(lo.w);
                    }
                }
            }
            const unsigned below = (1u << lane) - 1u;
            const unsigned who = __ballot_sync(0xffffffffu, inner), got = __ballot_sync(0xffffffffu, keep);
            if (inner) {
                const int p = sp + 2 * __popc(who & below);
                st[p] = left;
                st[p + 1] = right[node];
            }
            sp += 2 * __popc(who);
            if (FILL && keep) out_src[at + cnt + __popc(got & below)] = cell;
            cnt += __popc(got);
        }
        if (!FILL && lane == 0) counts[j] = cnt;
    }
    if (!FILL) {
        for (int o = 16; o > 0; o >>= 1) hits += __shfl_down_sync(0xffffffffu, hits, o);
        if (lane == 0 && hits) atomicAdd(raw_hits, hits);
    }
}

// Candidates kept by k_search, the row of every candidate.
__global__ void k_take_slots(const int *counts, const i64 *offs, const int *slots, i64 n_dst, int *out_src,
                             int *out_dst) {
    const i64 j = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= n_dst) return;
    const int n = counts[j];
    if (n == 0) return;
    const i64 b = offs[j];
    if (slots[j] >= 0)
        for (int q = 0; q < n; ++q) out_src[b + q] = slots[q * n_dst + j];
    for (int q = 0; q < n; ++q) out_dst[b + q] = static_cast<int>(j);
}

// ─── clipping ──────────────────────────────────────────────────────────────

template <int CAP>
__device__ __forceinline__ void load_poly(const MeshView &m, i64 c, DPoly<CAP> &p) {
    p.clear();
    if (m.regular) {
        // node trig cache (trig_cache.hpp:284-289, weight_generator.cpp:492-520)
        const int ni = m.ni, nj = m.nj;
        const double *slon = m.trig, *clon = m.trig + (ni + 1), *slat = m.trig + 2 * (ni + 1),
                     *clat = m.trig + 2 * (ni + 1) + (nj + 1);
        i64 ci = c % ni, cj = c / ni;
        auto at = [&](i64 i, i64 j) {
            double cl = clat[j];
            p.push({cl * clon[i], cl * slon[i], slat[j]});
        };
        at(ci, cj);
        at(ci + 1, cj);
        at(ci + 1, cj + 1);
        at(ci, cj + 1);
    } else {
        const int b = m.off[c], e = m.off[c + 1];
        for (int k = b; k < e && k < b + 32; ++k) {
            const double *q = m.xyz + 3 * static_cast<i64>(m.idx[k]);
            p.push({q[0], q[1], q[2]});
        }
    }
}

// The first 32 vertices of a cell, as load_poly has them.
struct CellRef {
    int n, b;  // vertices; first connectivity entry (regular: unused)
    int i, j;  // regular grids: column and row
    __device__ __forceinline__ CellRef(const MeshView &m, int c) : n(4), b(0), i(0), j(0) {
        if (m.regular) {
            j = c / m.ni;
            i = c - j * m.ni;
        } else {
            b = m.off[c];
            n = min(32, m.off[c + 1] - b);
        }
    }
    __device__ __forceinline__ DV3 at(const MeshView &m, int k) const {
        if (m.regular) {
            const int ci = i + (k == 1 || k == 2 ? 1 : 0), cj = j + (k >= 2 ? 1 : 0);
            const double *slon = m.trig, *clon = slon + (m.ni + 1), *slat = clon + (m.ni + 1), *clat = slat + (m.nj + 1);
            const double cl = clat[cj];
            return {cl * clon[ci], cl * slon[ci], slat[cj]};
        }
        const double *q = m.xyz + 3 * static_cast<i64>(m.idx[b + k]);
        return {q[0], q[1], q[2]};
    }
};

// What decides most side tests in FP32: per connectivity entry of the
// destination, the unit normal of the edge from that vertex to the next (w:
// below 0, an edge that is skipped; else the margin), and per entry of the
// source its vertex. The clipper's test is d = fl(n.p) >= -1e-14 in FP64 with
// n = ea x eb; the float value is off from n.p / |n| by less than 6e-7, so
// beyond kSideMargin it has the sign of d and, with |n| > 1e-7, d is clear of
// -1e-14. Shorter edges have an infinite margin: every test in FP64.
constexpr float kSideMargin = 2.0e-6f;

__global__ void k_edge_normals(MeshView D, float4 *en) {
    const int c = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (c >= D.n_cells) return;
    const CellRef E(D, c);
    const int b = D.off[c];
    if (E.n < 1) return;
    const DV3 first = E.at(D, 0);
    DV3 ea = first;
    for (int k = 0; k < E.n; ++k) {
        const DV3 eb = k + 1 == E.n ? first : E.at(D, k + 1);
        const DV3 n = d_cross(ea, eb);
        const double l2 = d_lensq(n), inv = rsqrt(l2);
        const float w = l2 < 1.0e-30 ? -1.0f : l2 < 1.0e-14 ? INFINITY : kSideMargin;
        en[b + k] = make_float4(static_cast<float>(n.x * inv), static_cast<float>(n.y * inv),
                                static_cast<float>(n.z * inv), w);
        ea = eb;
    }
}

__global__ void k_vertices_f(MeshView S, float4 *vf) {
    const int c = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (c >= S.n_cells) return;
    const CellRef C(S, c);
    const int b = S.off[c];
    for (int k = 0; k < C.n; ++k) {
        const DV3 p = C.at(S, k);
        vf[b + k] = make_float4(static_cast<float>(p.x), static_cast<float>(p.y), static_cast<float>(p.z), 0.0f);
    }
}

__device__ __forceinline__ float side_f(const float4 &n, float x, float y, float z) {
    return fmaf(n.x, x, fmaf(n.y, y, n.z * z));
}

// Pairs that an edge of the destination cell separates are settled here: all
// vertices of the source cell are outside it, and so is every point the
// clipper can put on an arc between them, so its polygon ends there with
// overlap 0. The others are listed for the clipper, whose warps are then full
// (two fifths of the candidates of 0.25 deg -> C384 are such pairs). The list's
// order varies; the overlaps do not depend on it.
__global__ void k_separate(MeshView S, MeshView D, const float4 *__restrict__ en, const float4 *__restrict__ vf,
                           const int *__restrict__ cs, const int *__restrict__ cd, i64 n, double *ov, int *list,
                           int *n_list) {
    const i64 k = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    bool meet = false;
    if (k < n) {
        const int c = cs[k], d = cd[k];
        const int sb = S.off[c], ns = min(32, S.off[c + 1] - sb), db = D.off[d], nd = min(32, D.off[d + 1] - db);
        meet = ns >= 3 && nd >= 3;
        for (int e = 0; e < nd && meet; ++e) {
            const float4 nf = en[db + e];
            if (nf.w < 0.0f) continue;
            bool outside = true;
            for (int i = 0; i < ns && outside; ++i) {
                const float4 p = vf[sb + i];
                outside = side_f(nf, p.x, p.y, p.z) < -nf.w;
            }
            meet = !outside;
        }
        if (!meet) ov[k] = 0.0;
    }
    const unsigned who = __ballot_sync(0xffffffffu, meet);
    const int lane = threadIdx.x & 31;
    int at = 0;
    if (lane == 0 && who) at = atomicAdd(n_list, __popc(who));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (meet) list[at + __popc(who & ((1u << lane) - 1u))] = static_cast<int>(k);
}

// Overlap areas of the listed pairs, a thread each: d_overlap_area for convex
// cells. A half space cuts a convex polygon in at most one run of vertices,
// so an edge of the clip cell has at most one crossing into and one out of
// it. Each lane goes on to its next edge that cuts (side tests, FP32), then
// the warp forms both crossings of all its lanes together in straight-line
// code. (In the vertex loop of d_overlap_area some lane of a warp has a
// crossing at nearly every vertex, and all of them pay.) The polygon stays in
// shared memory, a column a thread: a lane's vertex index does not change its
// bank. Pairs with more crossings or more than kClipCap vertices go to the
// general kernel through over_list.
// Bound by the FP64 pipe, which takes a warp's instruction in 64 cycles
// however many lanes are active; comparisons are made on the bits. 0.25 deg ->
// C384, 6.9 M candidates: 4.3 ms with k_separate; 10.2 ms with the side
// tests in FP64, edge by edge, on all candidates; 24.2 ms with the vertex
// loop, polygons in local memory, normalised midpoints and atan2.
constexpr int kClipCap = 12, kClipT = 64;
__global__ void __launch_bounds__(kClipT) k_clip_convex(MeshView S, MeshView D, const float4 *__restrict__ en,
                                                        const float4 *__restrict__ vf, const int *__restrict__ cs,
                                                        const int *__restrict__ cd, const int *__restrict__ list,
                                                        const int *n_list, double *ov, int *over_list, int *n_over) {
    __shared__ double P[3 * kClipCap][kClipT];
    __shared__ float F[3 * kClipCap][kClipT];
    const int n = *n_list;
    if (blockIdx.x * kClipT >= n) return;
    const int tid = threadIdx.x, t = static_cast<int>(blockIdx.x) * kClipT + tid;
    const int k = list[min(t, n - 1)];
    auto get = [&](int i) { return DV3{P[3 * i][tid], P[3 * i + 1][tid], P[3 * i + 2][tid]}; };
    auto put = [&](int i, const DV3 &v) {
        P[3 * i][tid] = v.x;
        P[3 * i + 1][tid] = v.y;
        P[3 * i + 2][tid] = v.z;
    };
    auto putf = [&](int i, float x, float y, float z) {
        F[3 * i][tid] = x;
        F[3 * i + 1][tid] = y;
        F[3 * i + 2][tid] = z;
    };
    auto move = [&](int to, int from) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            P[3 * to + q][tid] = P[3 * from + q][tid];
            F[3 * to + q][tid] = F[3 * from + q][tid];
        }
    };
    const int c = cs[k];
    const CellRef C(S, c), E(D, cd[k]);
    const int sb = S.off[c], db = D.off[cd[k]];
    const bool small = S.capf[c].w < 1.0f;  // no arc of the source cell reaches 120 degrees
    bool over = C.n > kClipCap;
    int m = t >= n || over ? 0 : C.n;
    for (int i = 0; i < m; ++i) {
        put(i, C.at(S, i));
        const float4 p = vf[sb + i];
        putf(i, p.x, p.y, p.z);
    }
    int e = m > 0 ? 0 : E.n;
    while (true) {
        bool cut = false, unsure = false;
        unsigned in = 0;
        while (e < E.n) {  // the next edge that cuts
            const float4 nf = en[db + e];
            if (nf.w >= 0.0f) {
                in = 0;
                unsure = !small;
                for (int i = 0; i < m; ++i) {
                    const float f = side_f(nf, F[3 * i][tid], F[3 * i + 1][tid], F[3 * i + 2][tid]);
                    bool inside = f > 0.0f;
                    if (fabsf(f) <= nf.w) {
                        unsure = true;
                        inside = d_dot(d_cross(E.at(D, e), E.at(D, e + 1 == E.n ? 0 : e + 1)), get(i)) >= -1.0e-14;
                    }
                    in |= inside ? 1u << i : 0u;
                }
                if (in == 0) {
                    m = 0;
                    e = E.n;
                    break;
                }
                if (in != (1u << m) - 1u) {
                    cut = true;
                    break;
                }
            }
            ++e;
        }
        if (!__any_sync(0xffffffffu, cut)) break;
        if (!cut) continue;
        const unsigned all = (1u << m) - 1u;
        const unsigned prev = ((in << 1) | (in >> (m - 1))) & all;  // bit i: vertex before i inside
        const unsigned enter = in & ~prev, leave = ~in & prev;
        const int kept = __popc(in);
        if (__popc(enter) > 1 || kept + 2 > kClipCap) {
            over = true;
            m = 0;
            e = E.n;
            continue;
        }
        const DV3 nrm = d_cross(E.at(D, e), E.at(D, e + 1 == E.n ? 0 : e + 1));
        const int a = __ffs(enter) - 1, b = __ffs(leave) - 1;
        const DV3 a0 = get(a == 0 ? m - 1 : a - 1), a1 = get(a), b0 = get(b == 0 ? m - 1 : b - 1), b1 = get(b);
        DV3 xa, xb;
        if (unsure) {
            xa = d_arc_cross_fast(a0, a1, nrm);
            xb = d_arc_cross_fast(b0, b1, nrm);
        } else {
            xa = d_arc_cross_known(a0, a1, nrm, false);
            xb = d_arc_cross_known(b0, b1, nrm, true);
        }
        // in vertex order: xa before vertex a, xb in place of vertex b
        int ia = 0, ib = kept + 1;
        if (a < b) {  // xa, [a, b), xb
            if (a == 0)
                for (int i = kept - 1; i >= 0; --i) move(i + 1, i);
            else if (a > 1)
                for (int i = 0; i < kept; ++i) move(i + 1, a + i);
        } else {  // the run passes the end: [0, b), xb, xa, [a, m)
            const int tail = m - a;
            if (a < b + 2)
                for (int i = tail - 1; i >= 0; --i) move(b + 2 + i, a + i);
            else if (a > b + 2)
                for (int i = 0; i < tail; ++i) move(b + 2 + i, a + i);
            ib = b;
            ia = b + 1;
        }
        put(ia, xa);
        putf(ia, static_cast<float>(xa.x), static_cast<float>(xa.y), static_cast<float>(xa.z));
        put(ib, xb);
        putf(ib, static_cast<float>(xb.x), static_cast<float>(xb.y), static_cast<float>(xb.z));
        m = kept + 2;
        ++e;
    }
    if (t >= n) return;
    if (over) {
        over_list[atomicAdd(n_over, 1)] = k;
        ov[k] = 0.0;
        return;
    }
    // fan from vertex 0, as d_poly_area
    double total = 0.0;
    if (m >= 3) {
        const DV3 a = get(0);
        DV3 b = get(1);
        double ab = d_dot(a, b);
        for (int i = 2; i < m; ++i) {
            const DV3 q = get(i);
            const double aq = d_dot(a, q), bq = d_dot(b, q);
            total += d_twice_atan(d_dot(a, d_cross(b, q)), 1.0 + ab + aq + bq);
            b = q;
            ab = aq;
        }
    }
    ov[k] = fabs(total);
}

// The pairs of list by the general clipper.
template <int CAP>
__global__ void __launch_bounds__(64) k_clip(MeshView S, MeshView D, const int *__restrict__ cs,
                                             const int *__restrict__ cd, i64 n, const int *list, double *ov) {
    i64 t = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    i64 k = list[t];
    DPoly<CAP> sp, dp, ba, bb;
    load_poly(S, cs[k], sp);
    load_poly(D, cd[k], dp);
    bool over = false;
    ov[k] = d_overlap_area(sp, dp, ba, bb, &over);
}

// ─── assembly ──────────────────────────────────────────────────────────────

// The kept pairs (overlap > 0) of the candidate list go into CSR, columns
// ascending. The list is grouped by row, so an entry's place is its row's
// start plus the kept candidates of the row that come before it in column
// order. That is counted directly, a thread an entry, where the rows are short
// (the squares of their lengths sum to at most kRankWork per candidate: 8
// for 0.25 deg -> C384); otherwise a stable radix sort by (row, column) gives
// it.
constexpr i64 kRankWork = 64;

// Kept candidates per row; key = the column of a kept candidate, else -1.
__global__ void k_row_kept(const double *ov, const int *cs, const int *cd, i64 n, int *kept, int *key) {
    const i64 k = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const bool keep = ov[k] > 0.0;
    key[k] = keep ? cs[k] : -1;
    if (keep) atomicAdd(&kept[cd[k]], 1);
}

__global__ void k_row_squares(const i64 *offs, i64 n_dst, unsigned long long *squares) {
    const i64 j = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    const unsigned long long m = j < n_dst ? static_cast<unsigned long long>(offs[j + 1] - offs[j]) : 0;
    unsigned long long sq = m * m;
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0 && sq) atomicAdd(squares, sq);
}

__global__ void k_reciprocal(const double *a, i64 n, double *y) {
    const i64 k = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < n) y[k] = __drcp_rn(a[k]);
}

// What an entry carries out of the candidate list (weight_generator.cpp:
// 3684-3716): w = overlap / destination area; fa = its contribution to
// frac_a, overlap / source area or the one the generator gives. The
// divisors repeat, so their reciprocals are formed once a cell (d_div_by).
struct EntryArgs {
    const double *ov, *fac;
    const int *cs, *cd;
    const double *area_src, *area_dst, *rcp_src, *rcp_dst;
    const int *row_ptr;
    int *col;
    double *w, *fa;
    unsigned *ckey;  // column and CSR index, for the column sums
    int *cval;
    int *gen;  // position among the kept candidates, or null
};

__device__ __forceinline__ void write_entry(const EntryArgs &a, i64 k, int at, int before) {
    const int c = a.cs[k], j = a.cd[k];
    const double o = a.ov[k];
    a.col[at] = c;
    a.w[at] = d_div_by(o, a.area_dst[j], a.rcp_dst[j]);
    a.fa[at] = a.fac ? a.fac[k] : d_div_by(o, a.area_src[c], a.rcp_src[c]);
    a.ckey[at] = static_cast<unsigned>(c);
    a.cval[at] = at;
    if (a.gen) a.gen[at] = before;
}

__global__ void k_place(EntryArgs a, const i64 *offs, const int *__restrict__ key, int n) {
    const int k = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (k >= n) return;
    const int c = key[k];
    if (c < 0) return;
    const int j = a.cd[k], b = static_cast<int>(offs[j]), e = static_cast<int>(offs[j + 1]);
    int rank = 0, before = 0;
    for (int q = b; q < e; ++q) {
        const int cq = key[q];
        rank += static_cast<unsigned>(cq) < static_cast<unsigned>(c) || (cq == c && q < k) ? 1 : 0;
        before += cq >= 0 && q < k ? 1 : 0;
    }
    write_entry(a, k, a.row_ptr[j] + rank, a.row_ptr[j] + before);
}

// The radix path: kept candidates compacted (pos), sorted, written.
__global__ void k_keep_flags(const double *ov, i64 n, int *keep) {
    i64 k = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < n) keep[k] = ov[k] > 0.0 ? 1 : 0;
}

__global__ void k_compact(const double *ov, const int *cs, const int *cd, const i64 *pos, i64 n, std::uint64_t *key,
                          int *vals, int *cand) {
    i64 k = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= n || !(ov[k] > 0.0)) return;
    const i64 p = pos[k];
    key[p] = (static_cast<unsigned long long>(cd[k]) << 32) | static_cast<unsigned>(cs[k]);
    vals[p] = static_cast<int>(p);
    cand[p] = static_cast<int>(k);
}

__global__ void k_write_sorted(EntryArgs a, const int *perm, const int *cand, i64 nnz) {
    const i64 at = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (at < nnz) write_entry(a, cand[perm[at]], static_cast<int>(at), perm[at]);
}

__global__ void k_count_keys(const unsigned *key, i64 n, int *cnt) {
    i64 k = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < n) atomicAdd(&cnt[key[k]], 1);
}

// Per row: frac_b, the sum of overlap / area in column order, or fb_pre, the
// row sums already taken in the generator's own order; weights clamped at 0
// and divided by the row's fraction under FracArea.
__global__ void k_rows(const int *row_ptr, const double *fb_pre, i64 n_dst, int fracarea, double *w, double *frac_b) {
    i64 j = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= n_dst) return;
    const int b = row_ptr[j], e = row_ptr[j + 1];
    double fb = 0.0;
    for (int k = b; k < e; ++k) {
        const double q = w[k];
        if (!(q >= 0.0)) w[k] = fmax(q, 0.0);
        fb += q;
    }
    if (fb_pre) fb = fb_pre[j];
    if (fracarea && fb > 0.0)
        for (int k = b; k < e; ++k) w[k] /= fb;
    frac_b[j] = fmin(fb, 1.0);
}

// frac_a per source cell, contributions in ascending row order.
__global__ void k_cols(const int *col_ptr, const int *perm, const double *fa, i64 n_src, double *frac_a) {
    i64 i = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_src) return;
    double s = 0.0;
    for (int k = col_ptr[i]; k < col_ptr[i + 1]; ++k) s += fa[perm[k]];
    frac_a[i] = fmin(s, 1.0);
}

__global__ void k_unmapped(MeshView D, const int *row_ptr, int *bad) {
    i64 j = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= D.n_cells) return;
    unsigned char f = D.flags[j];
    if (f & (1 | 2)) return;  // degenerate or masked
    if ((f & 4) || row_ptr[j + 1] == row_ptr[j]) atomicAdd(bad, 1);
}

// ─── bilinear (rectilinear source) ─────────────────────────────────────────

__device__ int upper_bound_d(const double *a, int n, double v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (!(v < a[mid])) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__global__ void k_bilinear(MeshView D, const double *clon, int ni, const double *clat, int nj, int *row_ptr, int *col,
                           double *w) {
    i64 c = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c > D.n_cells) return;
    row_ptr[c] = static_cast<int>(4 * c);
    if (c == D.n_cells) return;
    int b = D.off[c], e = D.off[c + 1];
    double ls = 0.0, ts = 0.0;
    for (int k = b; k < e; ++k) {
        i64 n = D.idx[k];
        ls += D.lonlat[n];
        ts += D.lonlat[n + D.n_nodes];
    }
    double ld = ls / static_cast<double>(e - b);
    double td = ts / static_cast<double>(e - b);
    int i = upper_bound_d(clon, ni, ld) - 1;
    int j = upper_bound_d(clat, nj, td) - 1;
    if (i < 0) i = 0;
    if (i >= ni - 1) i = ni - 2;
    if (i < 0) i = 0;
    if (j < 0) j = 0;
    if (j >= nj - 1) j = nj - 2;
    if (j < 0) j = 0;
    double x0 = clon[i], x1 = clon[i + 1], y0 = clat[j], y1 = clat[j + 1];
    double tx = (ld - x0) / (x1 - x0);
    double ty = (td - y0) / (y1 - y0);
    tx = fmax(0.0, fmin(1.0, tx));
    ty = fmax(0.0, fmin(1.0, ty));
    i64 o = 4 * c;
    col[o] = j * ni + i;
    col[o + 1] = j * ni + i + 1;
    col[o + 2] = (j + 1) * ni + i;
    col[o + 3] = (j + 1) * ni + i + 1;
    w[o] = (1.0 - tx) * (1.0 - ty);
    w[o + 1] = tx * (1.0 - ty);
    w[o + 2] = (1.0 - tx) * ty;
    w[o + 3] = tx * ty;
}

// Regular x regular bilinear: generate_bilinear_rect
// (src/solver/weight_generator_bilinear_rect.cpp:31-320), one thread per
// destination cell. The point is the mean of the cell's vertex (lon, lat)
// degrees, wrapped into [lon_min, lon_min + 360) on a periodic source; its
// fractional cell-centre index is bounds-tested with a 1e-9 slack, floored,
// clamped (wrapped in longitude when periodic), and the four weights are
// written column-ascending (ties in emission order, as a stable to_csr).
// cnt = 4 for a mapped row, 0 otherwise.
struct BilRegArgs {
    double lon_min, lat_min, dlon, dlat;
    int ni, nj;
    bool periodic;
};

__global__ void k_bilinear_reg(MeshView D, BilRegArgs g, int *cnt, int *col4, double *w4, int *gen4,
                               int *n_unmapped) {
    const i64 c = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= D.n_cells) return;
    const int b = D.off[c], e = D.off[c + 1];
    double ls = 0.0, ts = 0.0;
    for (int k = b; k < e; ++k) {
        const i64 n = D.idx[k];
        ls += D.lonlat[n];
        ts += D.lonlat[n + D.n_nodes];
    }
    double ld = ls / static_cast<double>(e - b);
    const double td = ts / static_cast<double>(e - b);
    if (g.periodic) {
        double off = ld - g.lon_min;
        off = off - floor(off / 360.0) * 360.0;
        ld = g.lon_min + off;
    }
    const double fi = (ld - g.lon_min) / g.dlon - 0.5, fj = (td - g.lat_min) / g.dlat - 0.5;
    const double tol = 1.0e-9;
    bool inside = fj >= -0.5 - tol && fj <= static_cast<double>(g.nj) - 0.5 + tol;
    if (!g.periodic) inside = inside && fi >= -0.5 - tol && fi <= static_cast<double>(g.ni) - 0.5 + tol;
    if (!inside) {
        cnt[c] = 0;
        atomicAdd(n_unmapped, 1);
        return;
    }
    int i = static_cast<int>(floor(fi)), j = static_cast<int>(floor(fj));
    j = max(0, min(j, g.nj - 2));
    i = g.periodic ? ((i % g.ni) + g.ni) % g.ni : max(0, min(i, g.ni - 2));
    const double tx = fmin(1.0, fmax(0.0, fi - static_cast<double>(i)));
    const double ty = fmin(1.0, fmax(0.0, fj - static_cast<double>(j)));
    int i1 = i + 1;
    if (i1 >= g.ni) i1 = g.periodic ? 0 : g.ni - 1;
    const int j1 = min(j + 1, g.nj - 1);
    int cc[4] = {j * g.ni + i, j * g.ni + i1, j1 * g.ni + i, j1 * g.ni + i1};
    double ww[4] = {(1.0 - tx) * (1.0 - ty), tx * (1.0 - ty), (1.0 - tx) * ty, tx * ty};
    int rk[4] = {0, 1, 2, 3};  // corner = place in the generation order
    for (int a = 1; a < 4; ++a)  // stable insertion sort by column
        for (int q = a; q > 0 && cc[q - 1] > cc[q]; --q) {
            const int tc = cc[q];
            cc[q] = cc[q - 1];
            cc[q - 1] = tc;
            const double tw = ww[q];
            ww[q] = ww[q - 1];
            ww[q - 1] = tw;
            const int tr = rk[q];
            rk[q] = rk[q - 1];
            rk[q - 1] = tr;
        }
    cnt[c] = 4;
    for (int k = 0; k < 4; ++k) {
        col4[4 * c + k] = cc[k];
        w4[4 * c + k] = ww[k];
        gen4[4 * c + k] = rk[k];
    }
}

__global__ void k_bilinear_reg_pack(const int *row_ptr, const int *cnt, const int *col4, const double *w4,
                                    const int *gen4, i64 n_dst, int *col, double *w, int *gen, double *frac_b) {
    const i64 c = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= n_dst) return;
    const int p = row_ptr[c];
    for (int k = 0; k < cnt[c]; ++k) {
        col[p + k] = col4[4 * c + k];
        w[p + k] = w4[4 * c + k];
        gen[p + k] = gen4[4 * c + k];
    }
    frac_b[c] = cnt[c] ? 1.0 : 0.0;
}

__global__ void k_fill(double *a, i64 n, double v) {
    i64 k = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < n) a[k] = v;
}

inline unsigned nblk(i64 n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

// ─── regular x regular conservative fast path ──────────────────────────────
// generate_conservative_rect (src/solver/weight_generator_conservative_rect.cpp
// :87-415): per destination cell the overlapping source cells by index
// arithmetic and their exact spherical-rectangle overlap (:50-66), one thread
// per destination cell, counted (pass 1) then written (pass 2) in the
// reference's (js, is) loop order.
struct RectGrid {
    i64 ni, nj;
    double lon_min, dlon, lat_min, dlat;
};
struct RectArgs {
    RectGrid sg, dg;
    bool src_global;
    const double *sa, *da;  // cell areas
    const int *smask, *dmask;
    i64 n_src, n_dst;
};

__device__ __forceinline__ double band_area(double lo, double dlat, double dlon) {
    constexpr double d2r = 3.14159265358979323846 / 180.0;
    const double hi = lo + dlat;
    return (dlon * d2r) * (sin(hi * d2r) - sin(lo * d2r));
}

__global__ void k_band_area(RectGrid g, const double *user, i64 n, double *area) {
    const i64 c = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= n) return;
    area[c] = user ? user[c] : band_area(g.lat_min + static_cast<double>(c / g.ni) * g.dlat, g.dlat, g.dlon);
}

template <bool FILL>
__global__ void k_rect(RectArgs a, int *count, const i64 *offs, int *cs, int *cd, double *ov, double *fb) {
    const i64 j = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= a.n_dst) return;
    int n = 0;
    double fbj = 0.0;  // frac_b in the reference's emission order
    i64 at = FILL ? offs[j] : 0;
    const i64 jd = j / a.dg.ni, id = j - jd * a.dg.ni;
    if (!(a.dmask && a.dmask[j] == 0) && a.da[j] > 0.0) {
        const double d_lo_x = a.dg.lon_min + static_cast<double>(id) * a.dg.dlon, d_hi_x = d_lo_x + a.dg.dlon;
        const double d_lo_y = a.dg.lat_min + static_cast<double>(jd) * a.dg.dlat, d_hi_y = d_lo_y + a.dg.dlat;
        double dlx = d_lo_x, dhx = d_hi_x;
        if (a.src_global) {
            const double shift = 360.0 * floor((d_lo_x - a.sg.lon_min) / 360.0);
            dlx = d_lo_x - shift;
            dhx = d_hi_x - shift;
        }
        const int sni = static_cast<int>(a.sg.ni), snj = static_cast<int>(a.sg.nj);
        int is_lo = static_cast<int>(floor((dlx - a.sg.lon_min) / a.sg.dlon));
        int is_hi = static_cast<int>(floor((dhx - a.sg.lon_min) / a.sg.dlon));
        int js_lo = static_cast<int>(floor((d_lo_y - a.sg.lat_min) / a.sg.dlat));
        int js_hi = static_cast<int>(floor((d_hi_y - a.sg.lat_min) / a.sg.dlat));
        if (!a.src_global) {
            is_lo = max(0, is_lo);
            is_hi = min(sni - 1, is_hi);
        }
        js_lo = max(0, js_lo);
        js_hi = min(snj - 1, js_hi);
        constexpr double d2r = 3.14159265358979323846 / 180.0;
        if (is_lo <= is_hi && js_lo <= js_hi) {
            for (int js = js_lo; js <= js_hi; ++js)
                for (int is = is_lo; is <= is_hi; ++is) {
                    const int ia = a.src_global ? ((is % sni) + sni) % sni : is;
                    const i64 c = static_cast<i64>(js) * sni + ia;
                    if (c >= a.n_src || (a.smask && a.smask[c] == 0) || a.sa[c] <= 0.0) continue;
                    const double s_lo_x = a.sg.lon_min + static_cast<double>(is) * a.sg.dlon, s_hi_x = s_lo_x + a.sg.dlon;
                    const double s_lo_y = a.sg.lat_min + static_cast<double>(js) * a.sg.dlat, s_hi_y = s_lo_y + a.sg.dlat;
                    const double dx = fmax(0.0, fmin(s_hi_x, dhx) - fmax(s_lo_x, dlx));
                    const double lo_y = fmax(s_lo_y, d_lo_y), hi_y = fmin(s_hi_y, d_hi_y);
                    if (hi_y <= lo_y || dx <= 0.0) continue;
                    const double o = (dx * d2r) * (sin(hi_y * d2r) - sin(lo_y * d2r));
                    if (o <= 0.0) continue;
                    if (FILL) {
                        cs[at] = static_cast<int>(c);
                        cd[at] = static_cast<int>(j);
                        ov[at] = o;
                        fbj += o / a.da[j];
                        ++at;
                    } else {
                        ++n;
                    }
                }
        }
    }
    if (!FILL) count[j] = n;
    if (FILL) fb[j] = fbj;
}

// Non-uniform rectilinear grids: generate_conservative_rect_nonuniform
// (src/solver/weight_generator_conservative_rect_nonuniform.cpp:52-311). Cell
// c is (c % ni, c / ni) on the sorted unique edge coordinates ulon/ulat.
struct RectNuGrid {
    int ni, nj;
    const double *ulon, *ulat;  // ni+1, nj+1 edges
};
struct RectNuArgs {
    RectNuGrid sg, dg;
    bool src_global;
    double s_lon_min, s_lon_max;
    const double *s_user, *d_user;  // mesh cell areas, or null
    const int *smask, *dmask;
    i64 n_src, n_dst;
};

__device__ __forceinline__ double band_area_edges(double lo_x, double hi_x, double lo_y, double hi_y) {
    constexpr double d2r = 3.14159265358979323846 / 180.0;
    double dlon = hi_x - lo_x;
    dlon *= d2r;
    return dlon * (sin(hi_y * d2r) - sin(lo_y * d2r));
}

__device__ __forceinline__ int lower_bound_d(const double *a, int n, double v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ int upper_bound_e(const double *a, int n, double v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (!(v < a[mid])) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Reported areas from the unshifted edges (:251-300).
__global__ void k_edge_area(RectNuGrid g, const double *user, i64 n, double *area) {
    const i64 c = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const i64 ci = c % g.ni, cj = c / g.ni;
    area[c] = user ? user[c] : band_area_edges(g.ulon[ci], g.ulon[ci + 1], g.ulat[cj], g.ulat[cj + 1]);
}

// One thread per destination cell, in the reference's loop order: the
// destination box (shifted by whole turns onto a global source), its area
// from those shifted edges, binary searches for the source index ranges
// (:140-156), then every (js, is) with overlap > 1e-12 and a positive source
// area, that area taken from the source edges as placed (+360 past the last
// column). FILL writes the pairs, the overlap, the frac_a contribution, the
// row's frac_b (emission order) and the area the weights divide by.
template <bool FILL>
__global__ void k_rect_nu(RectNuArgs a, int *count, const i64 *offs, int *cs, int *cd, double *ov, double *fac,
                          double *fb, double *da_w) {
    const i64 j = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= a.n_dst) return;
    int n = 0;
    i64 at = FILL ? offs[j] : 0;
    double fbj = 0.0, area_dst = 0.0;
    const int sni = a.sg.ni, snj = a.sg.nj;
    const i64 jd = j / a.dg.ni, id = j - jd * a.dg.ni;
    if (!(a.dmask && a.dmask[j] == 0)) {
        const double d_lo_y = a.dg.ulat[jd], d_hi_y = a.dg.ulat[jd + 1];
        double dlx = a.dg.ulon[id], dhx = a.dg.ulon[id + 1];
        if (a.src_global) {
            const double shift = 360.0 * floor((dlx - a.s_lon_min) / 360.0);
            dlx = dlx - shift;
            dhx = dhx - shift;
        }
        area_dst = a.d_user ? a.d_user[j] : band_area_edges(dlx, dhx, d_lo_y, d_hi_y);
        if (area_dst > 0.0) {
            const int is0 = max(0, lower_bound_d(a.sg.ulon, sni + 1, dlx) - 1);
            int is1 = upper_bound_e(a.sg.ulon, sni + 1, dhx);
            if (!a.src_global || dhx <= a.s_lon_max) is1 = min(sni - 1, is1);
            const int js0 = max(0, lower_bound_d(a.sg.ulat, snj + 1, d_lo_y) - 1);
            const int js1 = min(snj - 1, upper_bound_e(a.sg.ulat, snj + 1, d_hi_y));
            constexpr double d2r = 3.14159265358979323846 / 180.0;
            for (int js = js0; js <= js1; ++js)
                for (int is = is0; is <= is1; ++is) {
                    const int ia = a.src_global ? ((is % sni) + sni) % sni : is;
                    const i64 c = ia + static_cast<i64>(js) * sni;
                    if (a.smask && a.smask[c] == 0) continue;
                    double s_lo_x = a.sg.ulon[ia], s_hi_x = a.sg.ulon[ia + 1];
                    if (a.src_global && is >= sni) {
                        s_lo_x += 360.0;
                        s_hi_x += 360.0;
                    }
                    const double s_lo_y = a.sg.ulat[js], s_hi_y = a.sg.ulat[js + 1];
                    const double dx = fmax(0.0, fmin(s_hi_x, dhx) - fmax(s_lo_x, dlx));
                    const double lo_y = fmax(s_lo_y, d_lo_y), hi_y = fmin(s_hi_y, d_hi_y);
                    if (hi_y <= lo_y || dx <= 0.0) continue;
                    const double o = (dx * d2r) * (sin(hi_y * d2r) - sin(lo_y * d2r));
                    if (!(o > 1e-12)) continue;
                    const double area_src = a.s_user ? a.s_user[c] : band_area_edges(s_lo_x, s_hi_x, s_lo_y, s_hi_y);
                    if (area_src <= 0.0) continue;
                    if (FILL) {
                        cs[at] = static_cast<int>(c);
                        cd[at] = static_cast<int>(j);
                        ov[at] = o;
                        fac[at] = o / area_src;
                        fbj += o / area_dst;
                        ++at;
                    } else {
                        ++n;
                    }
                }
        }
    }
    if (!FILL) count[j] = n;
    if (FILL) {
        fb[j] = fbj;
        da_w[j] = area_dst;
    }
}

using Clock = std::chrono::steady_clock;
inline double ms_since(Clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(Clock::now() - t0).count();
}

}  // namespace

// What a fast path hands the assembly besides (cs, cd, ov).
struct AssembleOpts {
    const double *fac = nullptr;         // per-pair frac_a contribution (instead of ov / area_src)
    const double *fb_pre = nullptr;      // per-row frac_b, summed in the generator's order
    const double *area_a_out = nullptr;  // reported areas, when not the ones the weights divide by
    const double *area_b_out = nullptr;
    bool check_unmapped = true;          // the general path's UnmappedAction::Error check
    bool keep_gen = false;               // keep each entry's candidate position (generation order)
};

// Kept pairs (overlap > 0, weight_generator.cpp:3682) of the candidate list
// (cs, cd, ov) into the CSR of out: weights, frac_b per row and frac_a per
// column (the steps of :3684-3724), areas copied from area_src / area_dst.
static void assemble(const int *cs, const int *cd, const double *ov, const i64 *offs, i64 n_cand,
                     const double *area_src, const double *area_dst, const MeshView &D, const axgb_regrid_config &cfg,
                     Matrix &out, cudaStream_t s, const AssembleOpts &o = AssembleOpts{}) {
    const i64 n_src = out.n_src, n_dst = out.n_dst;
    Scratch<int> kept(n_dst, s), ccnt(n_src, s), col_ptr(n_src + 1, s);
    Scratch<unsigned long long> squares(1, s);
    Scratch<double> rcp_src(o.fac ? 0 : n_src, s), rcp_dst(n_dst, s);
    Scratch<int> key(n_cand, s);
    squares.zero();
    ccnt.zero();
    kept.zero();
    out.row_ptr.alloc(n_dst + 1);
    if (n_cand > 0) {
        k_row_kept<<<nblk(n_cand, 256), 256, 0, s>>>(ov, cs, cd, n_cand, kept.p, key.p);
        k_row_squares<<<nblk(n_dst, 256), 256, 0, s>>>(offs, n_dst, squares.p);
        k_reciprocal<<<nblk(n_dst, 256), 256, 0, s>>>(area_dst, n_dst, rcp_dst.p);
        if (!o.fac) k_reciprocal<<<nblk(n_src, 256), 256, 0, s>>>(area_src, n_src, rcp_src.p);
    }
    AXGB_CUDA(cudaGetLastError());
    scan_exclusive_i32(kept.p, out.row_ptr.p, n_dst, s);
    int h_nnz = 0;
    unsigned long long h_squares = 0;
    AXGB_CUDA(cudaMemcpyAsync(&h_nnz, out.row_ptr.p + n_dst, sizeof(int), cudaMemcpyDeviceToHost, s));
    AXGB_CUDA(cudaMemcpyAsync(&h_squares, squares.p, sizeof(h_squares), cudaMemcpyDeviceToHost, s));
    AXGB_CUDA(cudaStreamSynchronize(s));
    const i64 nnz = h_nnz;
    out.col.alloc(nnz);
    out.val.alloc(nnz);
    out.frac_a.alloc(n_src);
    out.frac_b.alloc(n_dst);
    out.area_a.alloc(n_src);
    out.area_b.alloc(n_dst);
    if (o.keep_gen) out.gen_rank.alloc(nnz);
    Scratch<double> fa(nnz, s);
    Scratch<unsigned> ckey(nnz, s);
    Scratch<int> cval(nnz, s);
    if (nnz > 0) {
        EntryArgs a{};
        a.ov = ov;
        a.fac = o.fac;
        a.cs = cs;
        a.cd = cd;
        a.area_src = area_src;
        a.area_dst = area_dst;
        a.rcp_src = rcp_src.p;
        a.rcp_dst = rcp_dst.p;
        a.row_ptr = out.row_ptr.p;
        a.col = out.col.p;
        a.w = out.val.p;
        a.fa = fa.p;
        a.ckey = ckey.p;
        a.cval = cval.p;
        a.gen = o.keep_gen ? out.gen_rank.p : nullptr;
        if (h_squares <= static_cast<unsigned long long>(kRankWork * n_cand)) {
            k_place<<<nblk(n_cand, 256), 256, 0, s>>>(a, offs, key.p, static_cast<int>(n_cand));
        } else {
            Scratch<int> keep(n_cand, s), vals(nnz, s), cand(nnz, s);
            Scratch<i64> pos(n_cand + 1, s);
            Scratch<std::uint64_t> rc(nnz, s);
            k_keep_flags<<<nblk(n_cand, 256), 256, 0, s>>>(ov, n_cand, keep.p);
            scan_exclusive_i32_to_i64(keep.p, pos.p, n_cand, s);
            k_compact<<<nblk(n_cand, 256), 256, 0, s>>>(ov, cs, cd, pos.p, n_cand, rc.p, vals.p, cand.p);
            int rbits = 32;
            while (rbits < 64 && (static_cast<unsigned long long>(n_dst) >> (rbits - 32)) > 0) ++rbits;
            radix_sort_pairs_u64(rc.p, vals.p, nnz, rbits, s);
            k_write_sorted<<<nblk(nnz, 256), 256, 0, s>>>(a, vals.p, cand.p, nnz);
        }
        AXGB_CUDA(cudaGetLastError());
        // entries by column, rows ascending: the CSR order sorted stably by column
        k_count_keys<<<nblk(nnz, 256), 256, 0, s>>>(ckey.p, nnz, ccnt.p);
        int cbits = 1;
        while (cbits < 32 && (static_cast<unsigned long long>(n_src) >> cbits) > 0) ++cbits;
        radix_sort_pairs_u32(ckey.p, cval.p, nnz, cbits, s);
        AXGB_CUDA(cudaGetLastError());
    }
    scan_exclusive_i32(ccnt.p, col_ptr.p, n_src, s);
    AXGB_CUDA(cudaMemcpyAsync(out.area_a.p, o.area_a_out ? o.area_a_out : area_src, sizeof(double) * n_src,
                              cudaMemcpyDeviceToDevice, s));
    AXGB_CUDA(cudaMemcpyAsync(out.area_b.p, o.area_b_out ? o.area_b_out : area_dst, sizeof(double) * n_dst,
                              cudaMemcpyDeviceToDevice, s));
    if (n_dst > 0)
        k_rows<<<nblk(n_dst, 256), 256, 0, s>>>(out.row_ptr.p, o.fb_pre, n_dst, cfg.norm_type == AXGB_FRACAREA ? 1 : 0,
                                                out.val.p, out.frac_b.p);
    if (n_src > 0) k_cols<<<nblk(n_src, 256), 256, 0, s>>>(col_ptr.p, cval.p, fa.p, n_src, out.frac_a.p);
    AXGB_CUDA(cudaGetLastError());
    if (o.check_unmapped && cfg.unmapped == AXGB_UNMAPPED_ERROR && n_dst > 0) {
        Scratch<int> bad(1, s);
        bad.zero();
        k_unmapped<<<nblk(n_dst, 256), 256, 0, s>>>(D, out.row_ptr.p, bad.p);
        int h_bad = 0;
        AXGB_CUDA(cudaMemcpy(&h_bad, bad.p, sizeof(int), cudaMemcpyDeviceToHost));
        if (h_bad > 0)
            throw Error(AXGB_ERR_UNMAPPED,
                        "generate_conservative: " + std::to_string(h_bad) + " unmapped destination cell(s)");
    }
    AXGB_CUDA(cudaStreamSynchronize(s));
    out.nnz = nnz;
    out.stats[3] = nnz;
}

void generate_conservative(Mesh &src, Mesh &dst, const axgb_regrid_config &cfg, Matrix &out) {
    cudaStream_t s = 0;
    auto t_all = Clock::now();
    auto t0 = Clock::now();
    mesh_prepare(src, s);
    mesh_prepare(dst, s);
    out.times_ms[0] = ms_since(t0);
    MeshView S = src.view(), D = dst.view();
    const i64 n_src = src.n_cells, n_dst = dst.n_cells;
    AXGB_REQUIRE(n_src < (i64(1) << 31) - 1 && n_dst < (i64(1) << 31) - 1, "meshes above 2^31 cells");
    out.n_src = n_src;
    out.n_dst = n_dst;

    // 2. LBVH
    t0 = Clock::now();
    const int n = static_cast<int>(n_src);
    Scratch<float4> nlo(n > 0 ? 2 * n - 1 : 1, s), nhi(n > 0 ? 2 * n - 1 : 1, s);
    Scratch<int> right(n > 1 ? n - 1 : 1, s);
    int root = -1;
    if (n > 0) {
        Scratch<unsigned> keys(n, s);
        Scratch<int> vals(n, s), parent(2 * n - 1, s), flag(n > 1 ? n - 1 : 1, s);
        k_leaf_keys<<<nblk(n, 256), 256, 0, s>>>(S, keys.p, vals.p);
        AXGB_CUDA(cudaGetLastError());
        radix_sort_pairs_u32(keys.p, vals.p, n, 30, s);
        Bvh t{n, n > 1 ? 0 : 0, nlo.p, nhi.p, parent.p, right.p, flag.p, keys.p};
        root = 0;  // internal node 0, or the single leaf (index n-1 = 0)
        AXGB_CUDA(cudaMemsetAsync(parent.p, 0xff, sizeof(int) * (2 * n - 1), s));
        flag.zero();
        k_leaves<<<nblk(n, 256), 256, 0, s>>>(t, S, vals.p);
        if (n > 1) {
            k_internal<<<nblk(n - 1, 256), 256, 0, s>>>(t);
            k_refit<<<nblk(n, 256), 256, 0, s>>>(t);
        }
        k_ropes<<<nblk(2 * n - 1, 256), 256, 0, s>>>(t);
        AXGB_CUDA(cudaGetLastError());
        AXGB_CUDA(cudaStreamSynchronize(s));
    }
    out.stats[4] = n > 0 ? 2 * n - 1 : 0;
    out.times_ms[1] = ms_since(t0);

    // 3. candidates
    t0 = Clock::now();
    Scratch<int> counts(n_dst, s);
    Scratch<i64> offs(n_dst + 1, s);
    Scratch<unsigned long long> raw(1, s);
    Scratch<int> wide(n_dst, s), n_wide(2, s);  // n_wide[1]: error flag
    raw.zero();
    n_wide.zero();
    const int n_leaf_base = n > 0 ? n - 1 : 0;
    // Two tilings of ns and nd cells meet in 1 + r^2 + 2.55 r pairs a row on
    // average (r^2 = ns / nd), and the gates admit about 1.6 times as many; a
    // row keeps up to 2.5 times that, at most 32 (longer ones go to
    // k_search_wide) and 1 GiB in all.
    const double r2 = n_dst > 0 ? static_cast<double>(n_src) / static_cast<double>(n_dst) : 0.0;
    const double room = std::min(32.0, std::max(16.0, 2.5 * 1.6 * (1.0 + r2 + 2.55 * std::sqrt(r2))));
    const int cap = static_cast<int>(std::max<i64>(1, std::min<i64>(static_cast<i64>(room),
                                                                   (i64(1) << 28) / std::max<i64>(1, n_dst))));
    Scratch<int> slots(cap * n_dst, s);
    const unsigned wide_grid = nblk(std::min<i64>(n_dst, 152 * 8 * kWideWarps), kWideWarps);
    if (n_dst > 0) {
        k_search<<<nblk(n_dst, 128), 128, 0, s>>>(S, D, nlo.p, nhi.p, root, n_leaf_base, counts.p, slots.p, cap, wide.p,
                                                 n_wide.p, raw.p);
        k_search_wide<false><<<wide_grid, 32 * kWideWarps, 0, s>>>(S, D, nlo.p, nhi.p, right.p, root, n_leaf_base, wide.p,
                                                                  n_wide.p, counts.p, nullptr, nullptr, raw.p, n_wide.p + 1);
    }
    AXGB_CUDA(cudaGetLastError());
    scan_exclusive_i32_to_i64(counts.p, offs.p, n_dst, s);
    i64 n_cand = 0;
    unsigned long long n_raw = 0;
    AXGB_CUDA(cudaMemcpyAsync(&n_cand, offs.p + n_dst, sizeof(i64), cudaMemcpyDeviceToHost, s));
    AXGB_CUDA(cudaMemcpyAsync(&n_raw, raw.p, sizeof(n_raw), cudaMemcpyDeviceToHost, s));
    int h_err = 0;
    AXGB_CUDA(cudaMemcpyAsync(&h_err, n_wide.p + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    AXGB_CUDA(cudaStreamSynchronize(s));
    if (h_err) throw Error(AXGB_ERROR, "LBVH traversal exceeded its step bound (malformed tree)");
    AXGB_REQUIRE(n_cand < (i64(1) << 31), "more than 2^31 candidate pairs");
    Scratch<int> cs(n_cand, s), cd(n_cand, s);
    if (n_cand > 0) {
        k_take_slots<<<nblk(n_dst, 256), 256, 0, s>>>(counts.p, offs.p, slots.p, n_dst, cs.p, cd.p);
        k_search_wide<true><<<wide_grid, 32 * kWideWarps, 0, s>>>(S, D, nlo.p, nhi.p, right.p, root, n_leaf_base, wide.p,
                                                                 n_wide.p, nullptr, offs.p, cs.p, nullptr, n_wide.p + 1);
        AXGB_CUDA(cudaGetLastError());
    }
    slots.release();
    out.stats[0] = static_cast<i64>(n_raw);
    out.stats[1] = n_cand;
    out.times_ms[2] = ms_since(t0);

    // 4. clip
    t0 = Clock::now();
    Scratch<double> ov(n_cand, s);
    Scratch<int> over_list(n_cand, s), n_over(2, s);  // n_over[1]: pairs for the clipper
    n_over.zero();
    int h_over = 0;
    if (n_cand > 0) {
        Scratch<float4> en(dst.n_conn, s), vf(src.n_conn, s);
        Scratch<int> list(n_cand, s);
        k_edge_normals<<<nblk(n_dst, 128), 128, 0, s>>>(D, en.p);
        k_vertices_f<<<nblk(n_src, 128), 128, 0, s>>>(S, vf.p);
        k_separate<<<nblk(n_cand, 256), 256, 0, s>>>(S, D, en.p, vf.p, cs.p, cd.p, n_cand, ov.p, list.p, n_over.p + 1);
        k_clip_convex<<<nblk(n_cand, kClipT), kClipT, 0, s>>>(S, D, en.p, vf.p, cs.p, cd.p, list.p, n_over.p + 1, ov.p,
                                                             over_list.p, n_over.p);
        AXGB_CUDA(cudaGetLastError());
        AXGB_CUDA(cudaMemcpy(&h_over, n_over.p, sizeof(int), cudaMemcpyDeviceToHost));
        if (h_over > 0) {
            k_clip<32><<<nblk(h_over, 64), 64, 0, s>>>(S, D, cs.p, cd.p, h_over, over_list.p, ov.p);
            AXGB_CUDA(cudaGetLastError());
        }
    }
    AXGB_CUDA(cudaStreamSynchronize(s));
    out.stats[2] = h_over;
    out.times_ms[3] = ms_since(t0);

    // 5. assembly
    t0 = Clock::now();
    assemble(cs.p, cd.p, ov.p, offs.p, n_cand, S.area, D.area, D, cfg, out, s);
    out.times_ms[4] = ms_since(t0);
    out.times_ms[5] = ms_since(t_all);
    slice_centroids(D, out, s);  // locality hint for the blocked apply layout (not timed)
}

bool generate_conservative_regular(Mesh &src, Mesh &dst, const axgb_regrid_config &cfg, Matrix &out) {
    const GridInfo &sg = src.grid, &dg = dst.grid;
    // decline non-global grids whose longitude ranges do not fit (:127-147)
    const bool src_global = static_cast<double>(sg.ni) * sg.dlon > 350.0;
    const bool dst_global = static_cast<double>(dg.ni) * dg.dlon > 350.0;
    if (!src_global && !dst_global &&
        (dg.lon_min < sg.lon_min - sg.dlon * 0.5 || dg.lon_max > sg.lon_max + sg.dlon * 0.5))
        return false;
    cudaStream_t s = 0;
    auto t_all = Clock::now();
    mesh_prepare(src, s);
    mesh_prepare(dst, s);
    MeshView D = dst.view();
    const i64 n_src = src.n_cells, n_dst = dst.n_cells;
    AXGB_REQUIRE(n_src < (i64(1) << 31) - 1 && n_dst < (i64(1) << 31) - 1, "meshes above 2^31 cells");
    out.n_src = n_src;
    out.n_dst = n_dst;
    RectArgs a;
    a.sg = {sg.ni, sg.nj, sg.lon_min, sg.dlon, sg.lat_min, sg.dlat};
    a.dg = {dg.ni, dg.nj, dg.lon_min, dg.dlon, dg.lat_min, dg.dlat};
    a.src_global = src_global;
    a.n_src = n_src;
    a.n_dst = n_dst;
    a.smask = src.has_mask ? src.d_mask.p : nullptr;
    a.dmask = dst.has_mask ? dst.d_mask.p : nullptr;
    Scratch<double> sa(n_src, s), da(n_dst, s);
    if (n_src) k_band_area<<<nblk(n_src, 256), 256, 0, s>>>(a.sg, src.has_area ? src.d_user_area.p : nullptr, n_src, sa.p);
    if (n_dst) k_band_area<<<nblk(n_dst, 256), 256, 0, s>>>(a.dg, dst.has_area ? dst.d_user_area.p : nullptr, n_dst, da.p);
    a.sa = sa.p;
    a.da = da.p;
    Scratch<int> counts(n_dst, s);
    Scratch<i64> offs(n_dst + 1, s);
    if (n_dst) k_rect<false><<<nblk(n_dst, 128), 128, 0, s>>>(a, counts.p, nullptr, nullptr, nullptr, nullptr, nullptr);
    AXGB_CUDA(cudaGetLastError());
    scan_exclusive_i32_to_i64(counts.p, offs.p, n_dst, s);
    i64 n_cand = 0;
    AXGB_CUDA(cudaMemcpy(&n_cand, offs.p + n_dst, sizeof(i64), cudaMemcpyDeviceToHost));
    AXGB_REQUIRE(n_cand < (i64(1) << 31), "more than 2^31 overlapping pairs");
    if (cfg.unmapped == AXGB_UNMAPPED_ERROR && n_cand == 0) return false;  // the general path diagnoses it
    Scratch<int> cs(n_cand, s), cd(n_cand, s);
    Scratch<double> ov(n_cand, s), fb(n_dst, s);
    fb.zero();
    if (n_cand) k_rect<true><<<nblk(n_dst, 128), 128, 0, s>>>(a, nullptr, offs.p, cs.p, cd.p, ov.p, fb.p);
    AXGB_CUDA(cudaGetLastError());
    out.stats[0] = out.stats[1] = n_cand;
    auto t0 = Clock::now();
    AssembleOpts o;
    o.keep_gen = true;  // rows generated in the reference's (js, is) loop order
    o.fb_pre = fb.p;
    o.check_unmapped = false;  // the fast path returns its matrix as it is (:380-415)
    assemble(cs.p, cd.p, ov.p, offs.p, n_cand, sa.p, da.p, D, cfg, out, s, o);
    AXGB_CUDA(cudaStreamSynchronize(s));
    out.times_ms[4] = ms_since(t0);
    out.times_ms[5] = ms_since(t_all);
    slice_centroids(D, out, s);
    return true;
}

bool generate_conservative_rectilinear(Mesh &src, Mesh &dst, const axgb_regrid_config &cfg, Matrix &out) {
    const GridInfo &sg = src.grid, &dg = dst.grid;
    cudaStream_t s = 0;
    auto t_all = Clock::now();
    mesh_prepare(src, s);
    mesh_prepare(dst, s);
    MeshView D = dst.view();
    const i64 n_src = src.n_cells, n_dst = dst.n_cells;
    AXGB_REQUIRE(n_src < (i64(1) << 31) - 1 && n_dst < (i64(1) << 31) - 1, "meshes above 2^31 cells");
    out.n_src = n_src;
    out.n_dst = n_dst;
    DBuf<double> sl, st, dl, dt;
    sl.upload(sg.ulon.data(), sg.ulon.size(), s);
    st.upload(sg.ulat.data(), sg.ulat.size(), s);
    dl.upload(dg.ulon.data(), dg.ulon.size(), s);
    dt.upload(dg.ulat.data(), dg.ulat.size(), s);
    RectNuArgs a;
    a.sg = {static_cast<int>(sg.ni), static_cast<int>(sg.nj), sl.p, st.p};
    a.dg = {static_cast<int>(dg.ni), static_cast<int>(dg.nj), dl.p, dt.p};
    a.s_lon_min = sg.ulon.front();
    a.s_lon_max = sg.ulon.back();
    a.src_global = (a.s_lon_max - a.s_lon_min) > 350.0;  // degrees (:81-83)
    a.s_user = src.has_area ? src.d_user_area.p : nullptr;
    a.d_user = dst.has_area ? dst.d_user_area.p : nullptr;
    a.smask = src.has_mask ? src.d_mask.p : nullptr;
    a.dmask = dst.has_mask ? dst.d_mask.p : nullptr;
    a.n_src = n_src;
    a.n_dst = n_dst;
    Scratch<int> counts(n_dst, s);
    Scratch<i64> offs(n_dst + 1, s);
    if (n_dst)
        k_rect_nu<false><<<nblk(n_dst, 128), 128, 0, s>>>(a, counts.p, nullptr, nullptr, nullptr, nullptr, nullptr,
                                                          nullptr, nullptr);
    AXGB_CUDA(cudaGetLastError());
    scan_exclusive_i32_to_i64(counts.p, offs.p, n_dst, s);
    i64 n_cand = 0;
    AXGB_CUDA(cudaMemcpy(&n_cand, offs.p + n_dst, sizeof(i64), cudaMemcpyDeviceToHost));
    AXGB_REQUIRE(n_cand < (i64(1) << 31), "more than 2^31 overlapping pairs");
    // under UnmappedAction::Error an empty matrix goes on to the general path (weight_generator.cpp:3286-3295)
    if (n_dst == 0 || (cfg.unmapped == AXGB_UNMAPPED_ERROR && n_cand == 0)) return false;
    Scratch<int> cs(n_cand, s), cd(n_cand, s);
    Scratch<double> ov(n_cand, s), fac(n_cand, s), fb(n_dst, s), da_w(n_dst, s), sa(n_src, s), da(n_dst, s);
    k_rect_nu<true><<<nblk(n_dst, 128), 128, 0, s>>>(a, nullptr, offs.p, cs.p, cd.p, ov.p, fac.p, fb.p, da_w.p);
    if (n_src) k_edge_area<<<nblk(n_src, 256), 256, 0, s>>>(a.sg, a.s_user, n_src, sa.p);
    k_edge_area<<<nblk(n_dst, 256), 256, 0, s>>>(a.dg, a.d_user, n_dst, da.p);
    AXGB_CUDA(cudaGetLastError());
    out.stats[0] = out.stats[1] = n_cand;
    auto t0 = Clock::now();
    AssembleOpts o;
    o.keep_gen = true;  // rows generated in the reference's (js, is) loop order
    o.fac = fac.p;
    o.fb_pre = fb.p;
    o.area_b_out = da.p;
    o.check_unmapped = false;
    assemble(cs.p, cd.p, ov.p, offs.p, n_cand, sa.p, da_w.p, D, cfg, out, s, o);
    AXGB_CUDA(cudaStreamSynchronize(s));
    out.times_ms[4] = ms_since(t0);
    out.times_ms[5] = ms_since(t_all);
    slice_centroids(D, out, s);
    return true;
}

bool generate_bilinear_regular(Mesh &src, Mesh &dst, const axgb_regrid_config &cfg, Matrix &out) {
    const GridInfo &g = src.grid;
    const i64 n_src = src.n_cells, n_dst = dst.n_cells;
    if (n_dst == 0 || g.ni == 0 || g.nj == 0) return false;  // the reference's fall-through signal
    cudaStream_t s = 0;
    auto t_all = Clock::now();
    mesh_prepare(dst, s);
    AXGB_REQUIRE(4 * n_dst < (i64(1) << 31) && n_src < (i64(1) << 31), "bilinear: meshes too large");
    BilRegArgs a{g.lon_min, g.lat_min, g.dlon, g.dlat, static_cast<int>(g.ni), static_cast<int>(g.nj),
                 std::abs((g.lon_max - g.lon_min) - 360.0) < 1.0e-10 * g.dlon};
    Scratch<int> cnt(n_dst, s), col4(4 * n_dst, s), gen4(4 * n_dst, s), bad(1, s);
    Scratch<double> w4(4 * n_dst, s);
    bad.zero();
    k_bilinear_reg<<<nblk(n_dst, 128), 128, 0, s>>>(dst.view(), a, cnt.p, col4.p, w4.p, gen4.p, bad.p);
    AXGB_CUDA(cudaGetLastError());
    int h_bad = 0;
    AXGB_CUDA(cudaMemcpy(&h_bad, bad.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (h_bad > 0 && cfg.unmapped == AXGB_UNMAPPED_ERROR)
        throw Error(AXGB_ERR_UNMAPPED, "bilinear: " + std::to_string(h_bad) +
                                           " unmapped destination cell(s) in the regular-grid fast path");
    out.n_src = n_src;
    out.n_dst = n_dst;
    out.row_ptr.alloc(n_dst + 1);
    scan_exclusive_i32(cnt.p, out.row_ptr.p, n_dst, s);
    int nnz = 0;
    AXGB_CUDA(cudaMemcpy(&nnz, out.row_ptr.p + n_dst, sizeof(int), cudaMemcpyDeviceToHost));
    out.nnz = nnz;
    out.col.alloc(std::max(1, nnz));
    out.val.alloc(std::max(1, nnz));
    out.gen_rank.alloc(std::max(1, nnz));
    out.frac_a.alloc(n_src);
    out.frac_b.alloc(n_dst);
    out.area_a.alloc(n_src);
    out.area_b.alloc(n_dst);
    k_bilinear_reg_pack<<<nblk(n_dst, 256), 256, 0, s>>>(out.row_ptr.p, cnt.p, col4.p, w4.p, gen4.p, n_dst,
                                                         out.col.p, out.val.p, out.gen_rank.p, out.frac_b.p);
    if (n_src) k_fill<<<nblk(n_src, 256), 256, 0, s>>>(out.frac_a.p, n_src, 1.0);
    out.area_a.zero(s);
    out.area_b.zero(s);
    AXGB_CUDA(cudaGetLastError());
    AXGB_CUDA(cudaStreamSynchronize(s));
    out.stats[3] = nnz;
    out.times_ms[5] = ms_since(t_all);
    slice_centroids(dst.view(), out, s);
    return true;
}

void generate_bilinear(Mesh &src, Mesh &dst, const axgb_regrid_config &cfg, Matrix &out) {
    (void)cfg;
    cudaStream_t s = 0;
    auto t_all = Clock::now();
    const GridInfo &g = src.grid;
    const i64 ni = g.ni, nj = g.nj, n_dst = dst.n_cells, n_src = src.n_cells;
    AXGB_REQUIRE(ni >= 2 && nj >= 2, "bilinear: rectilinear source needs at least 2x2 cells");
    std::vector<double> cl(ni), ct(nj);
    for (i64 i = 0; i < ni; ++i) cl[i] = 0.5 * (g.ulon[i] + g.ulon[i + 1]);
    for (i64 j = 0; j < nj; ++j) ct[j] = 0.5 * (g.ulat[j] + g.ulat[j + 1]);
    DBuf<double> dcl, dct;
    dcl.upload(cl.data(), cl.size(), s);
    dct.upload(ct.data(), ct.size(), s);
    AXGB_REQUIRE(4 * n_dst < (i64(1) << 31), "bilinear: too many destination cells");
    out.n_src = n_src;
    out.n_dst = n_dst;
    out.nnz = 4 * n_dst;
    out.row_ptr.alloc(n_dst + 1);
    out.col.alloc(4 * n_dst);
    out.val.alloc(4 * n_dst);
    out.frac_a.alloc(n_src);
    out.frac_b.alloc(n_dst);
    out.area_a.alloc(n_src);
    out.area_b.alloc(n_dst);
    k_bilinear<<<nblk(n_dst + 1, 128), 128, 0, s>>>(dst.view(), dcl.p, static_cast<int>(ni), dct.p,
                                                   static_cast<int>(nj), out.row_ptr.p, out.col.p, out.val.p);
    k_fill<<<nblk(n_src, 256), 256, 0, s>>>(out.frac_a.p, n_src, 1.0);
    k_fill<<<nblk(n_dst, 256), 256, 0, s>>>(out.frac_b.p, n_dst, 1.0);
    out.area_a.zero(s);
    out.area_b.zero(s);
    AXGB_CUDA(cudaGetLastError());
    AXGB_CUDA(cudaStreamSynchronize(s));
    out.stats[3] = out.nnz;
    out.times_ms[5] = ms_since(t_all);
    mesh_prepare(dst, s);
    slice_centroids(dst.view(), out, s);
}

}  // namespace axgb
