// Sparse weight apply on the device: y[f] = S x[f] for fields f < nrhs,
// fields laid out [f][cell] (the LayoutLeft (n_cells, n_vars) of
// batch_apply, libs/axis/include/axis/solver/apply.hpp:275-343).
//
// Layout: 32-row sliced ELL built once per matrix from the CSR. One warp
// owns one slice (one row per lane) and a tile of fields, several of them side
// by side; it reads the row's entries (column, FP64 weight or FP32 hi+lo pair)
// a few ahead, and again (from L1) for the tile's next fields. Rows of more
// than 32 entries are taken by a warp each, from a row-contiguous copy, in the
// same launch, first in the grid.
//
// Split FP32 path: weights w = hi + lo (hi = fp32(w), lo = fp32(w - hi));
// per entry the product hi*x is split exactly (fma), lo*x is added to the
// error term, and the running sum is carried with Knuth's TwoSum, so each
// output is the compensated sum rounded once to FP32. Two fields are
// processed together with packed f32x2 instructions.
//
// Tiles come one after another: all warps sweep the same tile of fields at once,
// so the source values they gather stay in L2 between neighbouring slices.
#include <algorithm>
#include <type_traits>

#include "fp32x2.cuh"
#include "internal.hpp"
#include "row_items.hpp"

namespace axgb {

// Arguments of the source gather of a batch member (renumbered sources).
struct GatherDesc {
    const float *x;
    i64 ldx;
    const int *inv;
    const int2 *span;
    i64 n, nrhs;
    float *xr;
    i64 ldr;
};

struct Batch {
    // One descriptor per (matrix, kind): slice items (lane per row of at most 32
    // entries, items = tile of kBatchTile fields x slice), or long-row items
    // (rows of more than 32 entries, lane = leaf, items = kBatchLongF fields x row).
    struct Desc {
        const int *base, *rlen, *col;
        const float2 *hl;
        const int *lrow, *lptr, *lcol;  // long rows, row-contiguous
        const float2 *lhl;
        const int *ids;  // slice ids (null: all slices)
        i64 n_ids;       // slices or long rows
        int mat;  // index of the matrix in the batch
        i64 n_rows;
        const float *x;
        i64 ldx;
        float *y;
        i64 ldy;
        i64 nrhs;
        i64 item_begin;  // first global item of this matrix
    };
    std::vector<std::shared_ptr<Matrix>> mats;
    std::vector<i64> nrhs;
    // descriptors: the slice items first, then the long-row items; each group
    // has its own persistent kernel and counter
    std::vector<Desc> desc;
    DBuf<Desc> d_desc;
    DBuf<unsigned long long> counter;  // [0]: slice items, [1]: row items
    i64 total_slice_items = 0, total_row_items = 0;
    int n_slice_desc = 0;
    int blocks_slices = 0, blocks_rows = 0;
    // matrices whose fields take the persistent staged kernels (blocked
    // layout) in the current plan, and that plan
    std::vector<char> use;
    bool planned = false;
    std::shared_ptr<BlkBatch> blk;
    // members with renumbered sources: fields gathered into xr first
    std::vector<DBuf<float>> xr;
    std::vector<GatherDesc> gdesc;
    DBuf<GatherDesc> d_gdesc;
    // graph per stream, replayed while descriptors are updated in place
    std::map<cudaStream_t, std::pair<cudaGraph_t, cudaGraphExec_t>> graphs;
    std::vector<const void *> last_ptrs;
    // Every graph shares the work counters, descriptors and gather scratch
    // above, so a call on another stream than the previous call's first waits
    // for the previous call's work (event `done`, recorded after each launch).
    cudaEvent_t done = nullptr;
    cudaStream_t last_stream = nullptr;
    bool launched = false;
    // side streams and events of the captured fork/join (kernels of the graph
    // that may run concurrently)
    static constexpr int kSide = 5;
    cudaStream_t side[kSide] = {};
    cudaEvent_t fork = nullptr, join[kSide] = {};
    std::mutex mu;
    ~Batch() {
        for (auto &g : graphs) {
            cudaGraphExecDestroy(g.second.second);
            cudaGraphDestroy(g.second.first);
        }
        if (done) cudaEventDestroy(done);
        for (int q = 0; q < kSide; ++q) {
            if (side[q]) cudaStreamDestroy(side[q]);
            if (join[q]) cudaEventDestroy(join[q]);
        }
        if (fork) cudaEventDestroy(fork);
    }
};

namespace {

inline unsigned nblk(i64 n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

struct SellArgs {
    const int *ids;
    const int *base, *rlen, *col;
    const float2 *hl;  // (hi, lo)
    const double *w64;
    i64 n_rows;
    float *ylo;  // split kernels: low parts of the outputs (hi+lo form), or null
    i64 ldylo;
};

__device__ __forceinline__ float ldg_f(const float *p) { return __ldg(p); }

// ─── long rows ─────────────────────────────────────────────────────────────
// Rows of more than 32 entries (coarse destination cells over a fine source,
// e.g. polar cells over a lat-lon source): one warp per (row, F fields), lane =
// leaf of the order in fp32x2.cuh, the F fields carried side by side, entries
// read row-contiguous (Sell::lcol/lhl), shuffle tree at the end.
constexpr int kF64F = 4;          // fields an FP64 row carries side by side
constexpr int kOrdGain = 16;       // twentieths, see rows_by_length
constexpr int kOrdPlain = static_cast<int>(0x80000000u);  // in Sell::ord: the group gains little
constexpr int kFusedK = 4;        // entries a row of the fused kernels loads before gathering
constexpr int kF64K = 2;          // the same of the FP64 kernel from three fields up

struct LongRows {
    const int *row, *ptr, *col;
    const float2 *hl;
    const double *w64;
    i64 n;
    float *ylo;  // split: low parts of the outputs (hi+lo form), or null
    i64 ldylo;
};
constexpr int kLongF = 8;  // fields per warp in the long-row kernels
constexpr int kLongQ1 = 12;  // entries a lane loads ahead in a single-field long row
constexpr int kLongQ1D = 8;  // the same in FP64
constexpr int kLongQ = 4;   // the same with several fields
constexpr int kBatchLongF = 8;  // fields per long-row item of the persistent batch kernel (k_batch<true>)

// In-order pairwise tree over the 32 leaves (lane = leaf) for F values a
// lane, F a power of two up to 32. While a lane holds more than one value,
// the two lanes of a pair split them: each sends the half it gives up and
// combines the half it keeps, so the five levels cost F/2 + F/4 + ... + 1
// combinations (and one more a level once a single value is left) instead of
// 5 F. combine() is the same in either operand order. Afterwards lane l
// holds the root of value tree_value<F>(l) in v[0], the lanes that agree in
// their low log2(F) bits the same one.
template <int F, class V, class X, class C>
__device__ __forceinline__ void tree_combine(V (&v)[F], X shfl, C combine) {
    const int lane = threadIdx.x & 31;
    int n = F;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = (lane & off) != 0;
#pragma unroll
            for (int i = 0; i < F / 2; ++i)
                if (i < n) {
                    const V keep = up ? v[i + n] : v[i], give = up ? v[i] : v[i + n];
                    v[i] = combine(keep, shfl(give, off));
                }
        } else {
            v[0] = combine(v[0], shfl(v[0], off));
        }
    }
}
template <int F>
__device__ __forceinline__ int tree_value(int lane) {
    int f = 0;
#pragma unroll
    for (int h = F / 2, b = 1; h > 0; h >>= 1, b <<= 1)
        if (lane & b) f += h;
    return f;
}

struct Leaf {
    float s, c;
};

// One warp: long row i, fields [F*fc, ...). Lane j sums entries
// j, j+32, ... of the row for each of the F fields (leaves), two fields at a
// time in packed arithmetic, then the leaves go through tree_combine.
// Bound by instruction issue (0.25 deg -> C48, 45 fields, rows of 110 entries
// on average). Fields the call does not have (f >= nf) are summed as zeros
// and not stored.
template <int F = kLongF>
__device__ __forceinline__ void split_long_row(const LongRows &L, i64 i, i64 fc, const float *x, i64 ldx, float *y,
                                               i64 ldy, i64 nrhs) {
    const int lane = threadIdx.x & 31;
    const i64 row = L.row[i];
    const int b = L.ptr[i], n = L.ptr[i + 1] - b;
    const i64 f0 = fc * F;
    const int nf = static_cast<int>(nrhs - f0 < F ? nrhs - f0 : F);
    x += f0 * ldx;
    Leaf v[F];
    int k = lane;
    if constexpr (F == 1) {
        // kLongQ1 of the leaf's entries per step: their loads are issued
        // together (memory-level parallelism for rows of hundreds of
        // entries), then summed in order, as one entry per step would. The
        // last step is partial.
        v[0] = {0.f, 0.f};
        for (; k - lane < n; k += 32 * kLongQ1) {
            int cq[kLongQ1];
            float2 wq[kLongQ1];
            float xq[kLongQ1];
#pragma unroll
            for (int q = 0; q < kLongQ1; ++q)
                if (k + 32 * q < n) {
                    cq[q] = L.col[b + k + 32 * q];
                    wq[q] = L.hl[b + k + 32 * q];
                }
#pragma unroll
            for (int q = 0; q < kLongQ1; ++q)
                if (k + 32 * q < n) xq[q] = ldg_f(x + cq[q]);
#pragma unroll
            for (int q = 0; q < kLongQ1; ++q)
                if (k + 32 * q < n) csum1(v[0].s, v[0].c, wq[q].x, wq[q].y, xq[q]);
        }
    } else {
        F2 s[F / 2], c[F / 2];
#pragma unroll
        for (int f = 0; f < F / 2; ++f) s[f] = c[f] = pk(0.f, 0.f);
        // Q rounds of 32 entries, their loads issued together; only the last
        // round of a row is partial (its missing entries are steps of weight
        // 0 on 0, which leave both sums as they are)
        auto rounds = [&](auto q_tag, bool partial) {
            constexpr int Q = decltype(q_tag)::value;
            int cq[Q];
            float2 wq[Q];
            float xq[Q][F];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const bool on = q < Q - 1 || !partial || k + 32 * q < n;
                cq[q] = on ? L.col[b + k + 32 * q] : -1;
                wq[q] = on ? L.hl[b + k + 32 * q] : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int f = 0; f < F; ++f) xq[q][f] = f < nf && cq[q] >= 0 ? ldg_f(x + f * ldx + cq[q]) : 0.f;
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const F2 hp = pk(wq[q].x, wq[q].x), lp = pk(wq[q].y, wq[q].y);
#pragma unroll
                for (int f = 0; f < F / 2; ++f) csum2(s[f], c[f], wq[q].x, hp, lp, xq[q][2 * f], xq[q][2 * f + 1]);
            }
            k += 32 * Q;
        };
        int left = n;  // warp-uniform
        for (; left >= 32 * kLongQ; left -= 32 * kLongQ) rounds(std::integral_constant<int, kLongQ>{}, false);
        if (left > 96)
            rounds(std::integral_constant<int, 4>{}, true);
        else if (left > 64)
            rounds(std::integral_constant<int, 3>{}, true);
        else if (left > 32)
            rounds(std::integral_constant<int, 2>{}, true);
        else if (left > 0)
            rounds(std::integral_constant<int, 1>{}, true);
#pragma unroll
        for (int f = 0; f < F / 2; ++f) {
            upk(s[f], v[2 * f].s, v[2 * f + 1].s);
            upk(c[f], v[2 * f].c, v[2 * f + 1].c);
        }
    }
    __syncwarp();
    tree_combine<F>(
        v,
        [](Leaf a, int off) {
            return Leaf{__shfl_xor_sync(0xffffffffu, a.s, off), __shfl_xor_sync(0xffffffffu, a.c, off)};
        },
        [](Leaf a, Leaf o) {
            lcombine(a.s, a.c, o.s, o.c);
            return a;
        });
    const int f = tree_value<F>(lane);
    if (lane < F && f < nf) {
        const float r = __fadd_rn(v[0].s, v[0].c);
        y[(f0 + f) * ldy + row] = r;
        if (L.ylo) L.ylo[(f0 + f) * L.ldylo + row] = sum_err(v[0].s, v[0].c, r);
    }
}

// Three blocks an SM (80 registers): 128 us for 45 fields of 0.25 deg -> C48,
// against 170 us at two blocks (92 registers, what the compiler takes by
// itself), 158 us at four (64), and 140 us at four with two rounds a step.
// 292 us with every lane combining every field's tree.
__global__ void __launch_bounds__(256, 3) k_split_long(LongRows L, const float *__restrict__ x, i64 ldx,
                                                    float *__restrict__ y, i64 ldy, i64 nrhs) {
    const i64 i = (static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (i >= L.n) return;
    for (i64 fc = blockIdx.y; fc * kLongF < nrhs; fc += gridDim.y) split_long_row(L, i, fc, x, ldx, y, ldy, nrhs);
}

// FP64 form of split_long_row: leaves summed with fma in entry order, then
// tree_combine with plain additions.
template <int F = kLongF>
__device__ __forceinline__ void f64_long_row(const LongRows &L, i64 i, i64 fc, const double *x, i64 ldx, double *y,
                                             i64 ldy, i64 nrhs) {
    const int lane = threadIdx.x & 31;
    const i64 row = L.row[i];
    const int b = L.ptr[i], n = L.ptr[i + 1] - b;
    const i64 f0 = fc * F;
    const int nf = static_cast<int>(nrhs - f0 < F ? nrhs - f0 : F);
    x += f0 * ldx;
    double s[F];
#pragma unroll
    for (int f = 0; f < F; ++f) s[f] = 0.0;
    int k = lane;
    // Q rounds, as split_long_row (a missing entry is an FMA of 0 and 0)
    auto rounds = [&](auto q_tag, bool partial) {
        constexpr int Q = decltype(q_tag)::value;
        int cq[Q];
        double wq[Q], xq[Q][F];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const bool on = q < Q - 1 || !partial || k + 32 * q < n;
            cq[q] = on ? L.col[b + k + 32 * q] : -1;
            wq[q] = on ? L.w64[b + k + 32 * q] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int f = 0; f < F; ++f) xq[q][f] = f < nf && cq[q] >= 0 ? __ldg(x + f * ldx + cq[q]) : 0.0;
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int f = 0; f < F; ++f)
                if (f < nf) s[f] = fma(wq[q], xq[q][f], s[f]);
        k += 32 * Q;
    };
    constexpr int kQ = F == 1 ? kLongQ1D : kLongQ;
    int left = n;  // warp-uniform
    for (; left >= 32 * kQ; left -= 32 * kQ) rounds(std::integral_constant<int, kQ>{}, false);
    if (kQ > 4 && left >= 128) {
        rounds(std::integral_constant<int, 4>{}, false);
        left -= 128;
    }
    if (left > 96)
        rounds(std::integral_constant<int, 4>{}, true);
    else if (left > 64)
        rounds(std::integral_constant<int, 3>{}, true);
    else if (left > 32)
        rounds(std::integral_constant<int, 2>{}, true);
    else if (left > 0)
        rounds(std::integral_constant<int, 1>{}, true);
    __syncwarp();
    tree_combine<F>(
        s, [](double a, int off) { return __shfl_xor_sync(0xffffffffu, a, off); },
        [](double a, double o) { return a + o; });
    const int f = tree_value<F>(lane);
    if (lane < F && f < nf) y[(f0 + f) * ldy + row] = s[0];
}

// ─── direct split kernel: one launch over the whole matrix ───────────────
// One field (k_split_fused is the form for several). There is too little work in
// a row to hide its chain of dependent loads (length, entries, source values)
// behind other warps: the short rows' warps stay and take slice after slice, with the lengths read
// two slices ahead and the first kOneK entries one slice ahead, so that only
// the gathers are waited for. The first blocks take the long rows, a warp
// each. 0.25 deg -> C384: 16.7 us, against 23 us with a warp a slice.
constexpr int kOneK = 5;
constexpr int kOneBlocks = 3;  // an SM
__global__ void __launch_bounds__(256, kOneBlocks) k_split_one(SellArgs a, LongRows L, int n_long, int long_blocks,
                                                               int n_slices, const float *__restrict__ x,
                                                               float *__restrict__ y) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    if (static_cast<int>(blockIdx.x) < long_blocks) {
        const int i = static_cast<int>(blockIdx.x) * 8 + wp;
        if (i < n_long) split_long_row<1>(L, i, 0, x, 0, y, 0, 1);
        return;
    }
    const int step = static_cast<int>(gridDim.x - long_blocks) * 8;
    int sid = static_cast<int>(blockIdx.x - long_blocks) * 8 + wp;
    // entries (-1: a long row or none to store) and first entry of the lane's row
    auto meta = [&](int s, int &n, int &e) {
        n = -1;
        e = 0;
        const i64 row = static_cast<i64>(s) * 32 + lane;
        if (s < n_slices && row < a.n_rows) {
            n = a.rlen[row];
            e = a.base[s] + lane;
        }
        if (n > 32) n = -1;
    };
    int n0, e0, n1, e1;
    int c0[kOneK];
    float2 w0[kOneK];
    meta(sid, n0, e0);
    meta(sid + step, n1, e1);
#pragma unroll
    for (int j = 0; j < kOneK; ++j)
        if (j < n0) {
            c0[j] = a.col[e0 + 32 * j];
            w0[j] = a.hl[e0 + 32 * j];
        }
    for (; sid < n_slices; sid += step) {
        int n2, e2, c1[kOneK];
        float2 w1[kOneK];
        float xv[kOneK];
        meta(sid + 2 * step, n2, e2);
#pragma unroll
        for (int j = 0; j < kOneK; ++j)
            if (j < n0) xv[j] = ldg_f(x + c0[j]);
#pragma unroll
        for (int j = 0; j < kOneK; ++j)
            if (j < n1) {
                c1[j] = a.col[e1 + 32 * j];
                w1[j] = a.hl[e1 + 32 * j];
            }
        float s = 0.f, c = 0.f;
#pragma unroll
        for (int j = 0; j < kOneK; ++j)
            if (j < n0) csum1(s, c, w0[j].x, w0[j].y, xv[j]);
        for (int k0 = kOneK; k0 < n0; k0 += kFusedK) {
            int cl[kFusedK];
            float2 w[kFusedK];
            float xr[kFusedK];
#pragma unroll
            for (int j = 0; j < kFusedK; ++j)
                if (k0 + j < n0) {
                    cl[j] = a.col[e0 + 32 * (k0 + j)];
                    w[j] = a.hl[e0 + 32 * (k0 + j)];
                }
#pragma unroll
            for (int j = 0; j < kFusedK; ++j)
                if (k0 + j < n0) xr[j] = ldg_f(x + cl[j]);
#pragma unroll
            for (int j = 0; j < kFusedK; ++j)
                if (k0 + j < n0) csum1(s, c, w[j].x, w[j].y, xr[j]);
        }
        if (n0 >= 0) {
            const i64 row = static_cast<i64>(sid) * 32 + lane;
            const float r = __fadd_rn(s, c);
            y[row] = r;
            if (a.ylo) a.ylo[row] = sum_err(s, c, r);
        }
        n0 = n1;
        e0 = e1;
        n1 = n2;
        e1 = e2;
#pragma unroll
        for (int j = 0; j < kOneK; ++j) {
            c0[j] = c1[j];
            w0[j] = w1[j];
        }
    }
}

// A lane's row of at most 32 entries for fields f .. f + nf - 1, F side by side: K
// entries' loads, then their gathers, then the compensated steps in entry order.
template <int F, int K, bool ALL>
__device__ __forceinline__ void short_rows(const SellArgs &a, int n, int e0, i64 row, const float *__restrict__ x,
                                           i64 ldx, float *__restrict__ y, i64 ldy, i64 f, int nf) {
    const float *xf = x + f * ldx;
    F2 s[F / 2], c[F / 2];
#pragma unroll
    for (int u = 0; u < F / 2; ++u) s[u] = c[u] = pk(0.f, 0.f);
    for (int k0 = 0; k0 < n; k0 += K) {
        int cl[K];
        float2 w[K];
        float xv[K][F];
#pragma unroll
        for (int j = 0; j < K; ++j)
            if (k0 + j < n) {
                cl[j] = a.col[e0 + 32 * (k0 + j)];
                w[j] = a.hl[e0 + 32 * (k0 + j)];
            }
#pragma unroll
        for (int j = 0; j < K; ++j)
            if (k0 + j < n) {
#pragma unroll
                for (int u = 0; u < F; ++u) xv[j][u] = ALL || u < nf ? ldg_f(xf + u * ldx + cl[j]) : 0.f;
            }
#pragma unroll
        for (int j = 0; j < K; ++j)
            if (k0 + j < n) {
                const F2 hp = pk(w[j].x, w[j].x), lp = pk(w[j].y, w[j].y);
#pragma unroll
                for (int u = 0; u < F / 2; ++u) csum2(s[u], c[u], w[j].x, hp, lp, xv[j][2 * u], xv[j][2 * u + 1]);
            }
    }
    float *yf = y + f * ldy + row;
#pragma unroll
    for (int u = 0; u < F; ++u) {
        if (!ALL && u >= nf) break;
        float sv, cv, o;
        if (u & 1) {
            upk(s[u / 2], o, sv);
            upk(c[u / 2], o, cv);
        } else {
            upk(s[u / 2], sv, o);
            upk(c[u / 2], cv, o);
        }
        const float r = __fadd_rn(sv, cv);
        yf[u * ldy] = r;
        if (a.ylo) a.ylo[(f + u) * a.ldylo + row] = sum_err(sv, cv, r);
    }
}

// blockIdx.y: a tile of fields. Warps [0, n_long): a row of more than 32
// entries (split_long_row; the chunks of F fields shared out over blockIdx.y);
// the others: lane per row of one slice (of ids, or all), rows of at most 32
// entries, F fields side by side (short_rows: two memory round trips for K
// entries instead of two an entry). The entries are read again for the tile's next F fields, from L1. Nothing is
// asked of the fields' alignment. Bound by the latency of its dependent round
// trips and by instruction issue: it is the kernel for few fields, small
// matrices (the rule is default_split_params in api.cpp) and unaligned
// fields. 45 unaligned fields of a 361 x 271 ocean grid -> 1 deg: 30 us, against
// 184 us for a launch per length class whose warps walked all fields; 7 fields
// of C192 -> 0.5 deg with hi+lo outputs 16.4 us, against 20 staged.
template <int F, int K>
__global__ void __launch_bounds__(256, F <= 4 ? 4 : 3) k_split_fused(SellArgs a, LongRows L, int n_long, int n_slices,
                                                                    const float *__restrict__ x, i64 ldx,
                                                                    float *__restrict__ y, i64 ldy, i64 nrhs, int tile) {
    const int lane = threadIdx.x & 31;
    int w = static_cast<int>(blockIdx.x * 8 + (threadIdx.x >> 5));
    // the long rows' warps come first in the grid: each is a long chain of
    // dependent loads, and starting them with the first wave overlaps them
    // with the short rows instead of leaving them as the tail
    if (w < n_long) {
        for (i64 fc = blockIdx.y; fc * F < nrhs; fc += gridDim.y) split_long_row<F>(L, w, fc, x, ldx, y, ldy, nrhs);
        return;
    }
    w -= n_long;
    if (w >= n_slices) return;
    const int sid = a.ids ? a.ids[w] : w;
    const i64 row = static_cast<i64>(sid) * 32 + lane;
    if (row >= a.n_rows) return;
    const int n = a.rlen[row];
    if (n > 32) return;  // a long row: its own warp above
    const int e0 = a.base[sid] + lane;
    const i64 fa = static_cast<i64>(blockIdx.y) * tile, fb = min(fa + tile, nrhs);
    i64 f = fa;
    for (; f + F <= fb; f += F) short_rows<F, K, true>(a, n, e0, row, x, ldx, y, ldy, f, F);
    if (f < fb) short_rows<F, K, false>(a, n, e0, row, x, ldx, y, ldy, f, static_cast<int>(fb - f));
}

// FP64 apply in one launch. Warps [0, L.n * ceil(nrhs / F)): a long row and F
// fields; the others: lane per row (rows of at most 32 entries, in the order
// of Sell::ord from three fields up) and a tile of fields, F side by side,
// K entries at a time (their loads, then their gathers, then the FMAs in
// entry order; entries past the row's end and fields past the last load the
// last one again, since a load under a condition of its own waits: 10 fields
// of 0.25 deg -> C384 159 -> 143 us). The entries are read again for the next
// F fields (from L1), so rows of every length run in one launch without a
// register array for the longest. The bound is the FP64 pipe (half a lane an SM
// sub-partition and cycle). 64 fields of C192 -> 0.5 deg: 169 us, against
// 297 us for one launch per length class with the entries in registers, the
// last launches on a few blocks (three blocks an SM and four entries ahead:
// 210 us; eight fields side by side: 223).
template <int F, int K, bool BY_LENGTH>
__global__ void __launch_bounds__(256, 4)
    k_f64_fused(SellArgs a, LongRows L, const int *__restrict__ ord, i64 n_slices, const double *__restrict__ x, i64 ldx,
                double *__restrict__ y, i64 ldy, i64 nrhs, i64 tile) {
    constexpr bool kAll = F <= 2;  // nrhs == F
    const int lane = threadIdx.x & 31;
    const i64 w = (static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    // the long rows' warps come first in the grid, as in k_split_fused
    const i64 n_long = kAll ? L.n : L.n * ((nrhs + F - 1) / F);
    if (w < n_long) {
        const i64 fc = nrhs <= F ? 0 : w / L.n;
        f64_long_row<F>(L, w - fc * L.n, fc, x, ldx, y, ldy, nrhs);
        return;
    }
    // the grid's surplus warps leave before ord is read
    const RowItem it = row_item(w - n_long, n_slices, kAll ? F : nrhs, kAll ? F : tile);
    if (!it.on) return;
    const i64 pos = it.slice * 32 + lane;
    const i64 fa = kAll ? 0 : it.tile * tile, fb = kAll ? F : min(fa + tile, nrhs);
    const int o = BY_LENGTH ? ord[pos] : kOrdPlain;
    const i64 row = o & kOrdPlain ? pos : o;
    if (row >= a.n_rows) return;
    const int n = a.rlen[row];
    if (n > 32) return;
    const int e0 = a.base[row >> 5] + static_cast<int>(row & 31);
    if (!kAll && __all_sync(__activemask(), n <= 1)) {
        // Rows of one entry (nearest neighbour, a destination within the source's
        // cells): it is loaded once, eight fields side by side. 100 fields of 1 -> 0.25
        // deg: 218 us, 389 with two entries' loads for every four fields.
        constexpr int U = 8;
        const int c = n == 1 ? a.col[e0] : 0;
        const double w = n == 1 ? a.w64[e0] : 0.0;
        for (i64 f = fa; f < fb; f += U) {
            const int nf = static_cast<int>(min(static_cast<i64>(U), fb - f));
            const double *xf = x + f * ldx + c;
            double *yf = y + f * ldy + row;
            double v[U];
            if (n == 1) {
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = fma(w, __ldg(xf + min(u, nf - 1) * ldx), 0.0);
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (u < nf) yf[u * ldy] = v[u];
        }
        return;
    }
    for (i64 f = fa; f < fb; f += F) {
        const int nf = kAll ? F : static_cast<int>(min(static_cast<i64>(F), fb - f));
        const double *xf = x + f * ldx;
        double s[F];
#pragma unroll
        for (int u = 0; u < F; ++u) s[u] = 0.0;
        for (int k0 = 0; k0 < n; k0 += K) {
            int cl[K];
            double wv[K], xv[K][F];
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const int e = e0 + 32 * min(k0 + j, n - 1);
                cl[j] = a.col[e];
                wv[j] = a.w64[e];
            }
#pragma unroll
            for (int j = 0; j < K; ++j)
#pragma unroll
                for (int u = 0; u < F; ++u) xv[j][u] = __ldg(xf + min(u, nf - 1) * ldx + cl[j]);
#pragma unroll
            for (int j = 0; j < K; ++j)
                if (k0 + j < n) {
#pragma unroll
                    for (int u = 0; u < F; ++u) s[u] = fma(wv[j], xv[j][u], s[u]);
                }
        }
#pragma unroll
        for (int u = 0; u < F; ++u)
            if (u < nf) y[(f + u) * ldy + row] = s[u];
    }
}

// Row-contiguous copy of the long rows' entries (in the layout's order).
__global__ void k_long_fill(const int *rp, const int *ccol, const double *val, const int *perm, const int *lrow,
                            const int *lptr, i64 n_lrows, int *lcol, float2 *lhl, double *lw64) {
    const i64 i = blockIdx.x;
    if (i >= n_lrows) return;
    const int r = lrow[i], r0 = rp[r], b = lptr[i], n = lptr[i + 1] - b;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int src = perm ? perm[r0 + k] : r0 + k;
        const double w = val[src];
        lcol[b + k] = ccol[src];
        if (lhl) {
            const float h = __double2float_rn(w);
            lhl[b + k] = make_float2(h, __double2float_rn(w - static_cast<double>(h)));
        }
        if (lw64) lw64[b + k] = w;
    }
}

// ─── layout build ──────────────────────────────────────────────────────────

__global__ void k_slice_len(const int *rp, i64 n_rows, i64 n_slices, int *len) {
    i64 s = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= n_slices) return;
    int m = 0;
    for (int q = 0; q < 32; ++q) {
        i64 r = s * 32 + q;
        if (r < n_rows) m = max(m, rp[r + 1] - rp[r]);
    }
    len[s] = m * 32;  // entries of the slice; scanned into base
}

// perm (optional): CSR index of the k-th entry of each row (split layouts).
__global__ void k_sell_fill(const int *rp, const int *ccol, const double *val, const int *perm, i64 n_rows,
                            i64 n_slices, const int *base, const int *slen32, int *rlen, int *col, float2 *hl,
                            double *w64, double *total) {
    i64 r = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= n_slices * 32) return;
    i64 s = r >> 5;
    int lane = static_cast<int>(r & 31);
    int L = slen32[s] / 32;
    int b = base[s];
    int n = 0, r0 = 0;
    if (r < n_rows) {
        r0 = rp[r];
        n = rp[r + 1] - r0;
    }
    rlen[r] = n;
    int last = n > 0 ? ccol[r0 + n - 1] : 0;
    double tot = 0.0;
    for (int k = 0; k < L; ++k) {
        int e = b + k * 32 + lane;
        if (k < n) {
            const int src = perm ? perm[r0 + k] : r0 + k;
            double w = val[src];
            tot = __dadd_rn(tot, w);
            col[e] = ccol[src];
            if (hl) {
                float h = __double2float_rn(w);
                hl[e] = make_float2(h, __double2float_rn(w - static_cast<double>(h)));
            }
            if (w64) w64[e] = w;
        } else {
            col[e] = last;
            if (hl) hl[e] = make_float2(0.f, 0.f);
            if (w64) w64[e] = 0.0;
        }
    }
    if (total && r < n_rows) total[r] = tot;
}

// Rows of every 128 consecutive ones, longest first, rows of more than 32
// entries (which have their own kernels) as if empty; positions past n_rows
// keep themselves. The FP64 kernels take a lane's row from here: a warp's
// FP64 instructions cost the same with any number of lanes active, and
// consecutive rows differ enough in length (C192 -> 0.5 deg: 3 to 9 entries)
// to leave a quarter of the lanes idle. Groups of 128 measured best or within
// 1% of 256 (16 NaN fields of 0.25 deg -> C384 651 / 646 us, 20 FP64 fields of
// C384 -> 1 deg 121 / 125, 300 of C384 -> 0.25 deg 2836 / 2867); 64 is slower
// on the first (665).
//
// Out of row order a warp's entries, gathers and stores touch more sectors, which
// the plain FP64 kernel (one operation an entry) notices: where the order
// leaves more than 0.8 of a group's steps, the group is flagged kOrdPlain and
// that kernel keeps its row order. 64 fields of a 2.6 M-cell Voronoi mesh (in a
// numbering that is not local) -> 0.1 deg: 3.13 ms, 3.78 with every group in
// order of length; 1016 of C768 -> 0.25 deg 21.1 against 24.2. With the line at
// 0.75 the first is another 5% faster, but 64 fields of C192 -> 0.5 deg take
// 183 us instead of 171.
std::vector<int> rows_by_length(const std::vector<int> &rp, i64 n_rows, i64 n_pos) {
    std::vector<int> ord(n_pos);
    for (i64 g = 0; g < n_pos; g += 128) {
        const i64 e = std::min<i64>(n_pos, g + 128);
        auto len = [&](i64 r) {
            const int n = r < n_rows ? rp[r + 1] - rp[r] : 0;
            return n > 32 ? 0 : n;
        };
        int at[34] = {};  // at[32 - n + 1]: rows of length n, then their first position
        for (i64 r = g; r < e; ++r) ++at[33 - len(r)];
        for (int k = 1; k < 34; ++k) at[k] += at[k - 1];
        for (i64 r = g; r < e; ++r) ord[g + at[32 - len(r)]++] = static_cast<int>(r);
        int plain = 0, sorted = 0;  // steps of the four warps in either order
        for (i64 q = g; q < e; q += 32) {
            int lp = 0, ls = 0;
            for (i64 r = q; r < q + 32; ++r) {
                lp = std::max(lp, len(r));
                ls = std::max(ls, len(ord[r]));
            }
            plain += lp;
            sorted += ls;
        }
        if (sorted * 20 > plain * kOrdGain)
            for (i64 r = g; r < e; ++r) ord[r] |= kOrdPlain;
    }
    return ord;
}

// Rows of more than 32 entries in the order their kernels take them. Rows of
// hundreds to thousands of entries (polar cells) are the kernels' length where
// they are begun in the last wave, and slow one another on one SM: they come
// first, the longest at the front, with others between them (a block of k_nan
// takes up to 80 rows). The others keep their order, as neighbours share
// sources. 0.25 deg -> C48 (rows of 33 to 4300), in row order and in this one: one
// field 18.8 and 14.7 us, FP64 24.5 and 21.0, NaN-aware 630 and 593 (679 with the heavy rows
// next to one another), 8 fields 38.7 and 31.6.
std::vector<int> long_row_order(const std::vector<int> &rp, i64 n_rows) {
    std::vector<int> rows, heavy, out;
    for (i64 r = 0; r < n_rows; ++r) {
        const int n = rp[r + 1] - rp[r];
        if (n > 32) (n > 256 ? heavy : rows).push_back(static_cast<int>(r));
    }
    std::stable_sort(heavy.begin(), heavy.end(),
                     [&](int a, int b) { return rp[a + 1] - rp[a] > rp[b + 1] - rp[b]; });
    const size_t gap = heavy.empty() ? 0 : std::min<size_t>(79, rows.size() / heavy.size());
    size_t at = 0;
    for (int h : heavy) {
        out.push_back(h);
        for (size_t k = 0; k < gap; ++k) out.push_back(rows[at++]);
    }
    out.insert(out.end(), rows.begin() + at, rows.end());
    return out;
}

void build_sell(Matrix &m, int fmt, cudaStream_t s) {
    Sell &S = fmt == 0 ? m.sell64 : m.sell32;
    if (S.built) return;
    const i64 n_rows = m.n_dst;
    const i64 n_slices = (n_rows + 31) / 32;
    DBuf<int> slen32(n_slices), base(n_slices + 1);
    if (n_slices > 0) {
        k_slice_len<<<nblk(n_slices, 256), 256, 0, s>>>(m.row_ptr.p, n_rows, n_slices, slen32.p);
        AXGB_CUDA(cudaGetLastError());
    }
    scan_exclusive_i32(slen32.p, base.p, n_slices, s);
    int total = 0;
    AXGB_CUDA(cudaMemcpyAsync(&total, base.p + n_slices, sizeof(int), cudaMemcpyDeviceToHost, s));
    AXGB_CUDA(cudaStreamSynchronize(s));
    S.n_slices = n_slices;
    S.n_entries = total;
    S.col.alloc(total);
    S.len.alloc(n_slices);
    S.base = std::move(base);
    DBuf<int> rlen(n_slices * 32);
    if (fmt == 1) {
        S.hl.alloc(total);
    } else {
        S.w64.alloc(total);
        S.total.alloc(n_rows);
    }
    if (n_slices > 0) {
        const int *perm = (fmt == 1 && m.split_perm.p) ? m.split_perm.p : nullptr;
        const int *ccol = (fmt == 1 && m.src_renum) ? m.split_col.p : m.col.p;
        k_sell_fill<<<nblk(n_slices * 32, 256), 256, 0, s>>>(m.row_ptr.p, ccol, m.val.p, perm, n_rows, n_slices,
                                                            S.base.p, slen32.p, rlen.p, S.col.p,
                                                            fmt == 1 ? S.hl.p : nullptr,
                                                            fmt == 0 ? S.w64.p : nullptr, fmt == 0 ? S.total.p : nullptr);
        AXGB_CUDA(cudaGetLastError());
    }
    // rows of more than 32 entries, row-contiguous
    {
        std::vector<int> rp(n_rows + 1);
        AXGB_CUDA(cudaMemcpy(rp.data(), m.row_ptr.p, sizeof(int) * (n_rows + 1), cudaMemcpyDeviceToHost));
        std::vector<int> lptr(1, 0);
        const std::vector<int> lrow = long_row_order(rp, n_rows);
        for (int r : lrow) lptr.push_back(lptr.back() + rp[r + 1] - rp[r]);
        if (fmt == 0) S.ord.upload_vec(rows_by_length(rp, n_rows, n_slices * 32), s);
        S.n_lrows = static_cast<i64>(lrow.size());
        S.n_lentries = lptr.back();
        S.lrow.upload_vec(lrow, s);
        S.lptr.upload_vec(lptr, s);
        const size_t ne = std::max<size_t>(1, lptr.back());
        S.lcol.alloc(ne);
        if (fmt == 1) {
            S.lhl.alloc(ne);
        } else {
            S.lw64.alloc(ne);
        }
        if (S.n_lrows > 0) {
            const int *perm = (fmt == 1 && m.split_perm.p) ? m.split_perm.p : nullptr;
            const int *ccol = (fmt == 1 && m.src_renum) ? m.split_col.p : m.col.p;
            k_long_fill<<<static_cast<unsigned>(S.n_lrows), 128, 0, s>>>(
                m.row_ptr.p, ccol, m.val.p, perm, S.lrow.p, S.lptr.p, S.n_lrows, S.lcol.p,
                fmt == 1 ? S.lhl.p : nullptr, fmt == 0 ? S.lw64.p : nullptr);
            AXGB_CUDA(cudaGetLastError());
        }
    }
    // keep row lengths in the len buffer's companion: store rlen in 'len' slot
    S.len = std::move(rlen);
    AXGB_CUDA(cudaStreamSynchronize(s));
    S.built = true;
}

SellArgs sell_args(const Matrix &m, const Sell &S, float *ylo = nullptr, i64 ldylo = 0) {
    SellArgs a{};
    a.ylo = ylo;
    a.ldylo = ldylo;
    a.base = S.base.p;
    a.rlen = S.len.p;
    a.col = S.col.p;
    a.hl = S.hl.p;
    a.w64 = S.w64.p;
    a.n_rows = m.n_dst;
    return a;
}

LongRows long_rows(const Sell &S) {
    LongRows L{};
    L.row = S.lrow.p;
    L.ptr = S.lptr.p;
    L.col = S.lcol.p;
    L.hl = S.lhl.p;
    L.w64 = S.lw64.p;
    L.n = S.n_lrows;
    return L;
}

// Grid of the long-row kernels: a warp per row along x, chunks of kLongF
// fields along y (all rows of one chunk of fields are in flight together, so
// the chunk's source values stay in L2).
dim3 long_grid(i64 rows, i64 nrhs) {
    return dim3(nblk(rows * 32, 256), static_cast<unsigned>(std::min<i64>(65535, (nrhs + kLongF - 1) / kLongF)));
}

// Every row of more than 32 entries (the staged applies leave them out).
void launch_split_long(const Sell &S, const float *x, i64 ldx, float *y, i64 ldy, i64 nrhs, cudaStream_t s,
                       float *ylo = nullptr, i64 ldylo = 0) {
    if (S.n_lrows == 0 || nrhs == 0) return;
    LongRows L = long_rows(S);
    L.ylo = ylo;
    L.ldylo = ldylo;
    k_split_long<<<long_grid(L.n, nrhs), 256, 0, s>>>(L, x, ldx, y, ldy, nrhs);
}
}  // namespace

// Rows of more than 32 entries given row-contiguous (the segmented layout's
// own copy, original source numbering): k_split_long, same summation order.
void launch_long_rows(const int *row, const int *ptr, const int *col, const float2 *hl, i64 n, const float *x, i64 ldx, float *y, i64 ldy, i64 nrhs, cudaStream_t s, float *ylo, i64 ldylo) {
    if (n == 0 || nrhs == 0) return;
    LongRows L{};
    L.row = row;
    L.ptr = ptr;
    L.col = col;
    L.hl = hl;
    L.n = n;
    L.ylo = ylo;
    L.ldylo = ldylo;
    k_split_long<<<long_grid(n, nrhs), 256, 0, s>>>(L, x, ldx, y, ldy, nrhs);
}

namespace {

// F fields side by side (0: by the count), tile fields a warp (0: by the
// size, as launch_f64_fused); ids / n_ids: these slices only, without the
// long rows.
void launch_split_fused(const Matrix &m, const Sell &S, const float *x, i64 ldx, float *y, i64 ldy, i64 nrhs,
                        cudaStream_t s, float *ylo, i64 ldylo, int F = 0, i64 tile = 0, const int *ids = nullptr,
                        i64 n_ids = 0) {
    LongRows L = long_rows(S);
    L.ylo = ylo;
    L.ldylo = ldylo;
    SellArgs a = sell_args(m, S, ylo, ldylo);
    a.ids = ids;
    const i64 n_slices = ids ? n_ids : S.n_slices;
    const int n_long = ids ? 0 : static_cast<int>(L.n);
    if (n_slices + n_long == 0 || nrhs == 0) return;
    if (nrhs == 1 && !ids) {
        const int long_blocks = static_cast<int>(nblk(n_long, 8));
        const int room = std::max(152 * 2, 152 * kOneBlocks - long_blocks);
        const int blocks = std::min<int>(static_cast<int>(nblk(n_slices, 8)), room);
        k_split_one<<<long_blocks + blocks, 256, 0, s>>>(a, L, n_long, long_blocks, static_cast<int>(n_slices), x, y);
        return;
    }
    if (F == 0) F = nrhs == 2 ? 2 : nrhs <= 4 ? 4 : 8;
    if (tile <= 0) tile = std::min<i64>(64, n_slices * nrhs / (152 * 24 * 4));
    tile = std::max<i64>(tile, (nrhs + 65534) / 65535);
    F = std::max(F, 2);
    tile = (tile + F - 1) / F * F;
    const dim3 g(nblk(n_long + n_slices, 8), static_cast<unsigned>((nrhs + tile - 1) / tile));
    auto launch = [&](auto kernel) {
        kernel<<<g, 256, 0, s>>>(a, L, n_long, static_cast<int>(n_slices), x, ldx, y, ldy, nrhs, static_cast<int>(tile));
    };
    if (F <= 2)
        launch(k_split_fused<2, 4>);
    else if (F <= 4)
        launch(k_split_fused<4, 4>);
    else
        launch(k_split_fused<8, 2>);
}
void launch_f64_fused(const Matrix &m, const Sell &S, const double *x, i64 ldx, double *y, i64 ldy, i64 nrhs,
                      cudaStream_t s) {
    const i64 warps = S.n_slices + S.n_lrows;
    if (warps == 0 || nrhs == 0) return;
    const SellArgs a = sell_args(m, S);
    const LongRows L = long_rows(S);
    // Fields of a short row's warp: up to 64, so that its entries are read once
    // from L2 and the tile's other passes find them in L1; fewer, down to 8,
    // where that would leave less than about four waves of warps. With all rows
    // in row order, 300 fields of C384 -> 0.25 deg: 3.58 ms with 64, 3.91 with 16,
    // 4.70 with all; 20 fields of C384 -> 1 deg: 148 us with 8, 191 with 16 (2.80
    // ms and 114 us with rows by length).
    // Four where eight would not fill the chip once: 10 fields of C384 -> 41 k
    // Voronoi cells 122 -> 103 us, 20 of C48 -> 2 deg 13.5 -> 11.1.
    const i64 fit = S.n_slices * nrhs / (152 * 24 * 4) / kF64F * kF64F;
    const i64 least = S.n_slices * nrhs < 152 * 32 * 8 ? kF64F : 2 * kF64F;
    const i64 tile = std::min<i64>(64, std::max<i64>(least, fit));
    auto launch = [&](auto kernel, int F) {
        const i64 warps = row_item_warps(L.n, F, S.n_slices, nrhs, tile);
        kernel<<<nblk(warps * 32, 256), 256, 0, s>>>(a, L, S.ord.p, S.n_slices, x, ldx, y, ldy, nrhs, tile);
    };
    if (nrhs == 1)
        launch(k_f64_fused<1, kFusedK, false>, 1);
    else if (nrhs == 2)
        launch(k_f64_fused<2, kFusedK, false>, 2);
    else
        launch(k_f64_fused<kF64F, kF64K, true>, kF64F);
}

// ─── NaN-aware and masked FP64 applies ────────────────────────────────────
// nan_batch_apply of include/axis/solver/apply.hpp:359-437 on the FP64
// layout (each row's entries in CSR order): per row the total weight
// (Sell::total), per field the weighted sum and the valid weight, with
// unfused multiply and add in entry order, so the NaN decisions and the
// values match the reference loop bit for bit.
//
// The bound is the FP64 pipe (half a lane an SM sub-partition and cycle), so
// FP64 work is what is left out: NaN is tested on the bits, the valid weight
// is summed only in rows that have a NaN (else it is the total, the same
// additions), and the divisions are shortened (NanRow). 16 fields of 0.25 deg -> C384 with a third of the cells missing:
// 617 us, against 2485 us with three FP64 operations an entry, two
// divisions an output, and a lane walking each long row.
constexpr int kNanG = 16;  // fields a warp
constexpr int kNanU = 4;   // fields of a short row carried side by side
constexpr int kNanK = 4;   // entries loaded ahead in a short row

__device__ __forceinline__ bool nan_bits(double x) {
    return (static_cast<unsigned long long>(__double_as_longlong(x)) & 0x7fffffffffffffffull) > 0x7ff0000000000000ull;
}

__device__ __forceinline__ double nan_result(double total, double wsum, double valid, double thres) {
    if (valid == 0.0 || total == 0.0) return __longlong_as_double(0x7ff8000000000000ll);
    return __ddiv_rn(valid, total) < thres ? __longlong_as_double(0x7ff8000000000000ll) : __ddiv_rn(wsum, valid);
}

// What the outputs of one row share. A row without a NaN has valid = total,
// its fraction total / total is 1 unless total is not finite, and its outputs
// are quotients by one divisor: from the correctly rounded reciprocal y,
// Markstein's two corrections with exact FMA residuals (IBM J. Res. Dev. 34,
// 1990) give the correctly rounded quotient in five operations, where
// __ddiv_rn takes about 25. It holds away from over- and underflow: operands
// outside 2^+-500 take __ddiv_rn.
struct NanRow {
    double total, thres, p, y;  // p = thres * total
    bool none;  // every output without a NaN is NaN
    bool safe;  // total within 2^+-500
    static __device__ __forceinline__ bool mid(double v) {
        return static_cast<unsigned>(((__double2hiint(v) >> 20) & 0x7ff) - 523) <= 1000u;
    }
    __device__ __forceinline__ NanRow(double t, double th) : total(t), thres(th) {
        none = t == 0.0 || (1.0 < th && fabs(t) <= 1.7976931348623157e308);
        p = __dmul_rn(th, t);
        safe = mid(t);
        y = safe ? __drcp_rn(t) : 0.0;
    }
    __device__ __forceinline__ double all(double wsum) const {
        if (none) return __longlong_as_double(0x7ff8000000000000ll);
        if (!safe || !mid(wsum)) return __ddiv_rn(wsum, total);
        const double q0 = __dmul_rn(wsum, y);
        const double q1 = __fma_rn(__fma_rn(-total, q0, wsum), y, q0);
        return __fma_rn(__fma_rn(-total, q1, wsum), y, q1);
    }
    // Some sources NaN, valid weight above 0 possible. The fraction is divided
    // out only where it lies within 2^-48 of the threshold: the rounded product
    // and quotient are off by 2^-52 at most. Positive doubles order as integers.
    __device__ __forceinline__ double some(double wsum, double valid) const {
        if (safe && mid(p) && mid(valid) && (__double2hiint(total) | __double2hiint(p) | __double2hiint(valid)) >= 0) {
            const long long v = __double_as_longlong(valid), q = __double_as_longlong(p);
            if (v < q - 32) return __longlong_as_double(0x7ff8000000000000ll);
            if (v > q + 32) return __ddiv_rn(wsum, valid);
        }
        return nan_result(total, wsum, valid, thres);
    }
};

// The first warps: rows_w rows of more than 32 entries each. The lanes multiply 32
// entries of each (row, field) side by side; then lane q < 16 adds the products
// of the q-th (row, field) in entry order and lane 16 + q the valid weights.
// rows_w is one from nine fields up and more with fewer, so that the additions,
// which cost the same with any number of lanes, have lanes to serve (one
// field of C384 -> 41 k Voronoi cells, most rows long: 249 -> 42 us; 5
// fields: 324 -> 183).
// The warps after them: lane per row (Sell::ord), U fields side by side and K
// entries ahead, loads past a row's end or the last field repeated, not left
// out (k_f64_fused). blockIdx.y: 16 fields. The long rows come
// first in the grid: their additions are chains of up to some thousand. The
// outputs of short rows with some sources NaN need a second sum and a
// division of their own; a warp with a coast has a few such lanes for every
// field, so they are put aside and worked off 32 at a time, a lane each.
struct NanItem {
    double wsum;
    unsigned mask;  // entries of the row whose source is NaN
    unsigned short lane, field;
};
constexpr int kNanPs = 33;  // products a field (32, and one against bank conflicts)
constexpr int kNanRows = kNanG + 4;  // rows of products and of weights a warp holds
// Long rows a warp takes side by side.
__host__ __device__ inline int nan_rows_w(i64 nrhs) {
    const int g = static_cast<int>(nrhs < kNanG ? nrhs : kNanG);
    return kNanG / g < kNanRows / (g + 1) ? kNanG / g : kNanRows / (g + 1);
}
static_assert(sizeof(NanItem) * (31 + 32 * kNanU) <= sizeof(double) * kNanG * kNanPs, "items put aside fit a warp's ps");
template <int U, int K>
__global__ void __launch_bounds__(256, U == 1 ? 4 : 2)
    k_nan(SellArgs a, LongRows L, const double *__restrict__ totals, const int *__restrict__ ord, i64 n_slices,
          const double *__restrict__ x, i64 ldx, double *__restrict__ y, i64 ldy, i64 nrhs, int rows_w,
          double na_thres) {
    __shared__ double ps[8][kNanRows][kNanPs];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const i64 wg = static_cast<i64>(blockIdx.x) * 8 + wp;
    const double thres = __dsub_rn(__dsub_rn(1.0, na_thres), 1e-6);
    const i64 n_long = (L.n + rows_w - 1) / rows_w;
    if (wg < n_long && (U == 1 || rows_w > 1)) {  // one chunk of fewer than kNanG fields
        const int G = static_cast<int>(nrhs), R = static_cast<int>(min(static_cast<i64>(rows_w), L.n - wg * rows_w));
        const int q = lane & 15, qr = q / G, qf = q - qr * G;
        const bool has = qr < R;  // the lane serves a (row, field)
        const i64 at = wg * rows_w + min(lane, R - 1);
        const int b = L.ptr[at], n = lane < R ? L.ptr[at + 1] - b : 0;
        const int from = has ? qr : 0;
        const int qn = __shfl_sync(0xffffffffu, n, from);
        const double *const src = ps[wp][has ? (lane < 16 ? q : R * G + qr) : 0];
        int most = n;
        for (int d = 16; d > 0; d >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, d));
        double acc = 0.0;
        for (int k0 = 0; k0 < most; k0 += 32) {
            double xv[kNanG];
            int r = 0, f = 0, e = 0, c = 0;
            bool on = false;
#pragma unroll
            for (int j = 0; j < kNanG; ++j) {
                xv[j] = 0.0;
                if (r < R) {  // warp-uniform, as r and f are
                    if (f == 0) {
                        const int nr = __shfl_sync(0xffffffffu, n, r);
                        e = __shfl_sync(0xffffffffu, b, r) + k0 + lane;
                        on = k0 + lane < nr;
                        c = on ? L.col[e] : 0;
                        ps[wp][R * G + r][lane] = on ? L.w64[e] : 0.0;
                    }
                    if (on) xv[j] = __ldg(x + f * ldx + c);
                    if (++f == G) {
                        f = 0;
                        ++r;
                    }
                }
            }
            const int left = max(0, qn - k0);
            unsigned skip = left >= 32 ? 0u : ~0u << left;  // the entries the lane leaves out
            r = f = 0;
#pragma unroll
            for (int j = 0; j < kNanG; ++j)
                if (r < R) {
                    const unsigned nan_mask = __ballot_sync(0xffffffffu, nan_bits(xv[j]));
                    if (q == j) skip |= nan_mask;
                    ps[wp][j][lane] = __dmul_rn(ps[wp][R * G + r][lane], xv[j]);
                    if (++f == G) {
                        f = 0;
                        ++r;
                    }
                }
            __syncwarp();
            const int m = min(32, most - k0);
#pragma unroll 8
            for (int k = 0; k < m; ++k) {
                const double t = __dadd_rn(acc, src[k]);
                if (!((skip >> k) & 1u)) acc = t;
            }
            __syncwarp();
        }
        const double valid = __shfl_down_sync(0xffffffffu, acc, 16);
        if (has && lane < 16) {
            const i64 row = L.row[wg * rows_w + qr];
            y[qf * ldy + row] = nan_result(totals[row], acc, valid, thres);
        }
        return;
    }
    if (U > 1 && wg < n_long) {  // rows_w 1
        const i64 row = L.row[wg];
        const int b = L.ptr[wg], n = L.ptr[wg + 1] - b;
        const double total = totals[row];
        double *const wsh = ps[wp][kNanG];
        {
            const i64 f0 = static_cast<i64>(blockIdx.y) * kNanG;
            const int nf = static_cast<int>(min(static_cast<i64>(kNanG), nrhs - f0));
            const double *xf = x + f0 * ldx;
            double acc = 0.0;  // lanes 0..15: weighted sum of field lane; lanes 16..31: its valid weight
            for (int k0 = 0; k0 < n; k0 += 32) {
                const bool on = k0 + lane < n;
                const int c = on ? L.col[b + k0 + lane] : 0;
                const double w = on ? L.w64[b + k0 + lane] : 0.0;
                double xv[kNanG];
#pragma unroll
                for (int f = 0; f < kNanG; ++f) xv[f] = on && f < nf ? __ldg(xf + f * ldx + c) : 0.0;
                unsigned skip = 0;
                wsh[lane] = w;
#pragma unroll
                for (int f = 0; f < kNanG; ++f) {
                    if (f >= nf) break;  // what the lanes without a field add up is not stored
                    const unsigned nan_mask = __ballot_sync(0xffffffffu, nan_bits(xv[f]));
                    if ((lane & 15) == f) skip = nan_mask;
                    ps[wp][f][lane] = __dmul_rn(w, xv[f]);
                }
                __syncwarp();
                const int m = min(32, n - k0);
                const double *src = lane < kNanG ? ps[wp][lane] : wsh;
#pragma unroll 8
                for (int k = 0; k < m; ++k) {
                    const double t = __dadd_rn(acc, src[k]);
                    if (!((skip >> k) & 1u)) acc = t;
                }
                __syncwarp();
            }
            const double valid = __shfl_down_sync(0xffffffffu, acc, 16);
            if (lane < nf) y[(f0 + lane) * ldy + row] = nan_result(total, acc, valid, thres);
        }
        return;
    }
    const i64 sid = wg - n_long;
    if (sid >= n_slices) return;
    const i64 row = ord[sid * 32 + lane] & ~kOrdPlain;
    const bool live = row < a.n_rows && a.rlen[row] <= 32;
    const int n = live ? a.rlen[row] : 0;
    const int base = a.base[row >> 5] + static_cast<int>(row & 31);
    const NanRow R(live ? totals[row] : 0.0, thres);
    const unsigned full = n == 32 ? 0xffffffffu : (1u << n) - 1u;
    // outputs of rows with some sources NaN, put aside
    NanItem *list = reinterpret_cast<NanItem *>(&ps[wp][0][0]);
    int held = 0;  // warp-uniform
    auto drain = [&](int at_least) {
        while (held >= at_least && held > 0) {
            const int take = min(held, 32);
            __syncwarp();
            const int i = held - take + lane;
            NanItem it{0.0, 0, 0, 0};
            if (lane < take) it = list[i];
            held -= take;
            // the row's constants by its lane
            NanRow Q = R;
            Q.total = __shfl_sync(0xffffffffu, R.total, it.lane);
            Q.p = __shfl_sync(0xffffffffu, R.p, it.lane);
            Q.safe = __shfl_sync(0xffffffffu, static_cast<int>(R.safe), it.lane) != 0;
            const int qn = __shfl_sync(0xffffffffu, n, it.lane), qb = __shfl_sync(0xffffffffu, base, it.lane);
            const i64 qrow = __shfl_sync(0xffffffffu, row, it.lane);
            if (lane < take) {
                double valid = 0.0;
                for (int k = 0; k < qn; ++k)
                    if (!((it.mask >> k) & 1u)) valid = __dadd_rn(valid, a.w64[qb + 32 * k]);
                y[(static_cast<i64>(blockIdx.y) * kNanG + it.field) * ldy + qrow] = Q.some(it.wsum, valid);
            }
            __syncwarp();
        }
    };
    {
        const i64 f0 = static_cast<i64>(blockIdx.y) * kNanG;
        const int nf = static_cast<int>(min(static_cast<i64>(kNanG), nrhs - f0));
        for (int g = 0; g < nf; g += U) {
            const double *xf = x + (f0 + g) * ldx;
            double ws[U];
            unsigned nm[U];  // the row's entries whose source is NaN
#pragma unroll
            for (int u = 0; u < U; ++u) {
                ws[u] = 0.0;
                nm[u] = 0;
            }
            for (int k0 = 0; k0 < n; k0 += K) {
                int c[K];
                double w[K], xv[K][U];
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    const int e = base + 32 * min(k0 + j, n - 1);
                    c[j] = a.col[e];
                    w[j] = a.w64[e];
                }
#pragma unroll
                for (int j = 0; j < K; ++j)
#pragma unroll
                    for (int u = 0; u < U; ++u) xv[j][u] = __ldg(xf + min(u, nf - g - 1) * ldx + c[j]);
#pragma unroll
                for (int j = 0; j < K; ++j)
                    if (k0 + j < n) {
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            if (g + u < nf) {
                                const bool bad = nan_bits(xv[j][u]);
                                const double t = __dadd_rn(ws[u], __dmul_rn(w[j], xv[j][u]));
                                ws[u] = bad ? ws[u] : t;
                                nm[u] |= static_cast<unsigned>(bad) << (k0 + j);
                            }
                    }
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (g + u >= nf) break;
                const bool aside = live && nm[u] != 0 && nm[u] != full;
                const unsigned who = __ballot_sync(0xffffffffu, aside);
                if (aside)
                    list[held + __popc(who & ((1u << lane) - 1u))] =
                        NanItem{ws[u], nm[u], static_cast<unsigned short>(lane), static_cast<unsigned short>(g + u)};
                else if (live)
                    y[(f0 + g + u) * ldy + row] =
                        nm[u] == 0 ? R.all(ws[u]) : __longlong_as_double(0x7ff8000000000000ll);
                held += __popc(who);
            }
            drain(32);
        }
        drain(1);
    }
}

// Masked apply of include/axis/solver/apply.hpp:458-532: rows with mask 0
// are not written; the others get the row sum in CSR order.
__global__ void k_masked_apply(const int *__restrict__ rp, const int *__restrict__ col,
                               const double *__restrict__ val, i64 n_dst, const double *__restrict__ x,
                               const int *__restrict__ mask, double *__restrict__ y) {
    const i64 j = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= n_dst || (mask && mask[j] == 0)) return;
    double s = 0.0;
    for (int k = rp[j]; k < rp[j + 1]; ++k) s = __dadd_rn(s, __dmul_rn(val[k], __ldg(x + col[k])));
    y[j] = s;
}

// ─── conservation ──────────────────────────────────────────────────────────

template <class T>
__global__ void k_integral(const T *f, const double *area, const double *frac, i64 n, int mode, double *partial) {
    // mode 0: sum f*area*frac; 1: sum over frac != 0 of f*area (DstArea)
    __shared__ double sh[256];
    double acc = 0.0;
    for (i64 i = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<i64>(gridDim.x) * blockDim.x) {
        double v = static_cast<double>(f[i]);
        if (mode == 0)
            acc += v * area[i] * frac[i];
        else if (frac[i] != 0.0)
            acc += v * area[i];
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

template <class T>
double integral(const T *f, const double *area, const double *frac, i64 n, int mode, cudaStream_t s) {
    const int blocks = 1024;
    DBuf<double> part(blocks);
    k_integral<T><<<blocks, 256, 0, s>>>(f, area, frac, n, mode, part.p);
    AXGB_CUDA(cudaGetLastError());
    std::vector<double> h(blocks);
    AXGB_CUDA(cudaMemcpyAsync(h.data(), part.p, sizeof(double) * blocks, cudaMemcpyDeviceToHost, s));
    AXGB_CUDA(cudaStreamSynchronize(s));
    double acc = 0.0;
    for (double v : h) acc += v;
    return acc;
}

// ─── FP64 FMA rate probe ──────────────────────────────────────────────────
// Eight independent dependent-FMA chains per thread (enough to cover the FP64
// pipe's latency), four resident blocks of 256 threads per SM: the FP64 FMA
// throughput the FP64 apply and the clipper are compared against. The
// result is written so the chains are not removed.
__global__ void __launch_bounds__(256) k_fp64_fma(double *out, i64 iters, double b, double c) {
    const double x = 1.0 + 1e-3 * threadIdx.x;
    double a0 = x, a1 = x + 1, a2 = x + 2, a3 = x + 3, a4 = x + 4, a5 = x + 5, a6 = x + 6, a7 = x + 7;
    for (i64 i = 0; i < iters; ++i) {
        a0 = fma(a0, b, c);
        a1 = fma(a1, b, c);
        a2 = fma(a2, b, c);
        a3 = fma(a3, b, c);
        a4 = fma(a4, b, c);
        a5 = fma(a5, b, c);
        a6 = fma(a6, b, c);
        a7 = fma(a7, b, c);
    }
    const double r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (r == 12345.678) out[0] = r;  // never true for these inputs; keeps the chains live
}

}  // namespace

double fp64_fma_tflops(i64 iters) {
    int dev = 0, sms = 0;
    AXGB_CUDA(cudaGetDevice(&dev));
    AXGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    DBuf<double> out(1);
    cudaEvent_t e0, e1;
    AXGB_CUDA(cudaEventCreate(&e0));
    AXGB_CUDA(cudaEventCreate(&e1));
    const unsigned blocks = static_cast<unsigned>(4 * sms);
    k_fp64_fma<<<blocks, 256>>>(out.p, iters / 8 + 1, 0.999999, 1e-7);  // warm-up
    AXGB_CUDA(cudaEventRecord(e0));
    k_fp64_fma<<<blocks, 256>>>(out.p, iters, 0.999999, 1e-7);
    AXGB_CUDA(cudaEventRecord(e1));
    AXGB_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    AXGB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    const double flops = 2.0 * 8.0 * static_cast<double>(iters) * blocks * 256.0;
    return flops / (static_cast<double>(ms) * 1e-3) / 1e12;
}

namespace {

// ─── conservation report without allocation ───────────────────────────────
// For callers that cannot allocate device memory while they run (a model
// whose device memory is owned by its own pool, or code between
// allocation-free phases): the per-block partial sums live in a fixed
// file-scope device array instead of cudaMalloc'd scratch. The call copies
// its two results to the host and synchronises its stream, so it is made
// before or between stream captures, never inside one.
// Each block reduces a fixed span of 2048 cells; the partials are then
// reduced by one block in a fixed order, so results are deterministic.

constexpr int kNaThreads = 256;
constexpr i64 kNaCellsPerBlock = 2048;                      // 8 cells per thread
constexpr int kNaMaxBlocks = 8192;                          // per integral
constexpr i64 kNaMaxCells = kNaCellsPerBlock * kNaMaxBlocks;  // 16,777,216 cells per side
// [0, K): source partials, [K, 2K): destination partials, [2K, 2K+2): results.
// Every slot a call reads is written earlier in the same call.
static __device__ __align__(256) double g_noalloc_scratch[2 * kNaMaxBlocks + 2];

template <class T>
__global__ void k_integral_span(const T *f, const double *area, const double *frac, i64 n, int mode, double *partial) {
    __shared__ double sh[kNaThreads];
    const i64 b0 = static_cast<i64>(blockIdx.x) * kNaCellsPerBlock;
    double acc = 0.0;
    for (int q = 0; q < kNaCellsPerBlock / kNaThreads; ++q) {
        const i64 i = b0 + q * kNaThreads + threadIdx.x;
        if (i < n) {
            double v = static_cast<double>(f[i]);
            if (mode == 0)
                acc += v * area[i] * frac[i];
            else if (frac[i] != 0.0)
                acc += v * area[i];
        }
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = kNaThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// One block: result[w] = sum of partial[w*K .. w*K + nb[w]) for w = 0, 1.
__global__ void k_sum_partials(const double *partial, int nb0, int nb1, double *result) {
    __shared__ double sh[kNaThreads];
    for (int w = 0; w < 2; ++w) {
        const int nb = w == 0 ? nb0 : nb1;
        const double *p = partial + static_cast<i64>(w) * kNaMaxBlocks;
        double acc = 0.0;
        for (int i = threadIdx.x; i < nb; i += kNaThreads) acc += p[i];
        sh[threadIdx.x] = acc;
        __syncthreads();
        for (int o = kNaThreads / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) result[w] = sh[0];
        __syncthreads();
    }
}

// Device address of g_noalloc_scratch for the current device, looked up
// once per device (the host-side name is not a device address). The cached
// address belongs to the device's current context: after cudaDeviceReset
// it is stale, as is every other handle of this library on that device.
double *noalloc_scratch() {
    static std::mutex mu;
    static double *ptr[256] = {};
    int dev = 0;
    AXGB_CUDA(cudaGetDevice(&dev));
    AXGB_REQUIRE(dev >= 0 && dev < 256, "conservation_noalloc: device ordinal out of range");
    std::lock_guard<std::mutex> lk(mu);
    if (!ptr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess)
            throw Error(AXGB_ERR_CUDA, std::string("cudaGetSymbolAddress(g_noalloc_scratch): ") + cudaGetErrorString(e));
        ptr[dev] = static_cast<double *>(p);
    }
    return ptr[dev];
}

// ─── persistent batch kernels ──────────────────────────────────────────────
// Items of all matrices are handed out by one atomic counter (no waiting).
// ROWS: the long-row items, else the slice items, with the row functions of
// the direct kernel: eight fields side by side in 80 registers, three blocks
// an SM (17-pair batch 1043 us, against 1096 us with four fields a long row in
// 64 registers). The long rows' form spills at 80 registers (32 bytes stored, 40
// loaded a thread).
constexpr int kBatchTile = 8;  // fields of a slice item
template <bool ROWS>
__global__ void __launch_bounds__(256, ROWS ? 3 : 2) k_batch(const Batch::Desc *__restrict__ desc, int n_desc, i64 total,
                                                  unsigned long long *counter) {
    const int lane = threadIdx.x & 31;
    while (true) {
        unsigned long long it = 0;
        if (lane == 0) it = atomicAdd(counter, 1ull);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (static_cast<i64>(it) >= total) return;
        int m = 0;
        while (m + 1 < n_desc && desc[m + 1].item_begin <= static_cast<i64>(it)) ++m;
        const Batch::Desc &d = desc[m];
        const i64 local = static_cast<i64>(it) - d.item_begin;
        const i64 t = local / d.n_ids, i = local - t * d.n_ids;
        if constexpr (ROWS) {
            LongRows L{};
            L.row = d.lrow;
            L.ptr = d.lptr;
            L.col = d.lcol;
            L.hl = d.lhl;
            L.n = d.n_ids;
            split_long_row<kBatchLongF>(L, i, t, d.x, d.ldx, d.y, d.ldy, d.nrhs);
        } else {
            const i64 sid = d.ids ? d.ids[i] : i;
            const i64 row = sid * 32 + lane;
            if (row < d.n_rows) {
                const int n = d.rlen[row];
                SellArgs a{};
                a.col = d.col;
                a.hl = d.hl;
                const i64 f = t * kBatchTile;
                const int nf = static_cast<int>(d.nrhs - f < kBatchTile ? d.nrhs - f : kBatchTile);
                if (n <= 32) {
                    if (nf == kBatchTile)
                        short_rows<kBatchTile, 2, true>(a, n, d.base[sid] + lane, row, d.x, d.ldx, d.y, d.ldy, f, nf);
                    else
                        short_rows<kBatchTile, 2, false>(a, n, d.base[sid] + lane, row, d.x, d.ldx, d.y, d.ldy, f, nf);
                }
            }
            __syncwarp();
        }
    }
}

}  // namespace

void matrix_prepare(Matrix &m, int format, cudaStream_t s) {
    std::lock_guard<std::mutex> lk(m.mu);
    if (format == 0) {
        build_sell(m, 0, s);
        return;
    }
    build_blocked(m, s);  // fixes the split entry order (split_perm) first
    if (format == 3) build_segmented(m, s);
    build_sell(m, 1, s);  // the direct kernels' and, for long rows and blocks that do not fit, the staged ones'
    if (format == 1) m.stats[5] = 1;  // the direct kernel is one launch
    if (format >= 2) m.stats[6] = blocked_launches(m);
}

namespace {

// xr[f][j] = x[f][inv[j]]: fields into the split layouts' source numbering. A
// block takes kGatherTile new cells and one field after another of its share.
// A numbering with some locality (cells in latitude bands, as along a spiral)
// keeps the tile's originals within a span a few times its length: the block
// then reads that span in order into shared memory and gathers from there. A
// gather from L2 moves a 32-byte sector for every 4-byte value. Tiles whose
// originals are spread wider gather from L2. 64 fields of 163,843 Voronoi cells:
// 23.8 us, against 38.6 us (cold).
constexpr int kGatherSpan = 11 * 1024;  // floats staged (44 KB)
constexpr int kGatherT = 512, kGatherPer = kGatherTile / kGatherT;

__device__ __forceinline__ void gather_tile(const float *__restrict__ x, i64 ldx, const int *__restrict__ inv,
                                            const int2 *__restrict__ span, i64 n, i64 nrhs, float *__restrict__ xr,
                                            i64 ldr, i64 tile, float *sh) {
    const i64 j0 = tile * kGatherTile;
    const int2 sp = span[tile];
    const int len = sp.y - sp.x + 1;
    int src[kGatherPer];
#pragma unroll
    for (int q = 0; q < kGatherPer; ++q) {
        const i64 j = j0 + q * kGatherT + threadIdx.x;
        src[q] = j < n ? inv[j] : -1;
    }
    for (i64 f = blockIdx.y; f < nrhs; f += gridDim.y) {
        const float *xf = x + f * ldx;
        float *o = xr + f * ldr + j0 + threadIdx.x;
        if (len <= kGatherSpan) {
            __syncthreads();  // the previous field's values have been read
            for (int k = threadIdx.x; k < len; k += kGatherT) sh[k] = __ldg(xf + sp.x + k);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kGatherPer; ++q)
                if (src[q] >= 0) o[q * kGatherT] = sh[src[q] - sp.x];
        } else {
            float v[kGatherPer];
#pragma unroll
            for (int q = 0; q < kGatherPer; ++q)
                if (src[q] >= 0) v[q] = __ldg(xf + src[q]);
#pragma unroll
            for (int q = 0; q < kGatherPer; ++q)
                if (src[q] >= 0) o[q * kGatherT] = v[q];
        }
    }
}

__global__ void __launch_bounds__(kGatherT) k_gather_src(const float *__restrict__ x, i64 ldx,
                                                         const int *__restrict__ inv, const int2 *__restrict__ span,
                                                         i64 n, i64 nrhs, float *__restrict__ xr, i64 ldr) {
    __shared__ float sh[kGatherSpan];
    gather_tile(x, ldx, inv, span, n, nrhs, xr, ldr, blockIdx.x, sh);
}

// Same for a batch member: arguments read from device memory, so a captured
// graph picks up new field pointers.
__global__ void __launch_bounds__(kGatherT) k_gather_desc(const GatherDesc *__restrict__ g) {
    __shared__ float sh[kGatherSpan];
    const GatherDesc d = *g;
    gather_tile(d.x, d.ldx, d.inv, d.span, d.n, d.nrhs, d.xr, d.ldr, blockIdx.x, sh);
}

// Blocks of a gather: the tiles, and so many of the fields side by side that
// there are about eight blocks an SM and a block keeps its indices for several
// fields.
dim3 gather_grid(i64 n, i64 nrhs) {
    const i64 tiles = (n + kGatherTile - 1) / kGatherTile;
    const i64 y = std::min<i64>(nrhs, std::max<i64>(1, 152 * 8 / tiles));
    return dim3(static_cast<unsigned>(tiles), static_cast<unsigned>(y));
}
}  // namespace

i64 renum_ld(const Matrix &m) { return (m.n_src + 3) / 4 * 4; }

void gather_source(const Matrix &m, const float *x, i64 ldx, i64 nrhs, float *xr, cudaStream_t s) {
    k_gather_src<<<gather_grid(m.n_src, nrhs), kGatherT, 0, s>>>(x, ldx, m.src_inv.p, m.src_span.p, m.n_src, nrhs, xr,
                                                                 renum_ld(m));
    AXGB_CUDA(cudaGetLastError());
}

int split_launches(const Matrix &m, i64 nrhs) {
    return static_cast<int>(staged_launches(m, nrhs).size()) + (m.blocked.n_fallback > 0 ? 1 : 0) + (m.sell32.n_lrows > 0 ? 1 : 0);
}

void apply_split_layouts(Matrix &m, const float *x, i64 ldx, float *y, i64 ldy, i64 nrhs, const SplitParams &p,
                         cudaStream_t s, float *ylo, i64 ldylo);

// A renumbered matrix first gathers the fields into stream-ordered scratch of
// the library's pool, given back on the same stream after the apply. (The
// default pool returns memory to the system whenever the stream is waited
// for: 379 us for a call of 96.)
void apply_split(Matrix &m, const float *x, i64 ldx, float *y, i64 ldy, i64 nrhs, const SplitParams &p,
                 cudaStream_t s, float *ylo, i64 ldylo) {
    if (nrhs <= 0) return;
    if (p.variant == 5) {  // segmented: cells staged by their own ids, no renumbering gather
        if (!m.seg.built) matrix_prepare(m, 3, s);
        apply_segmented(m, x, ldx, y, ldy, nrhs, s, ylo, ldylo, p.stages);
        return;
    }
    if (!m.split_ready()) matrix_prepare(m, 2, s);
    if (!m.src_renum) {
        apply_split_layouts(m, x, ldx, y, ldy, nrhs, p, s, ylo, ldylo);
        return;
    }
    const i64 ldr = renum_ld(m);
    Scratch<float> xr(static_cast<size_t>(ldr * nrhs), s);
    gather_source(m, x, ldx, nrhs, xr.p, s);
    apply_split_layouts(m, xr.p, ldr, y, ldy, nrhs, p, s, ylo, ldylo);
}

// The layouts are there (apply_split).
void apply_split_layouts(Matrix &m, const float *x, i64 ldx, float *y, i64 ldy, i64 nrhs, const SplitParams &p,
                         cudaStream_t s, float *ylo, i64 ldylo) {
    if (p.variant >= 1 && p.variant <= 3 && blocked_eligible(m, x, ldx, p.variant == 2)) {
        apply_blocked(m, x, ldx, y, ldy, nrhs, p.variant, p.unroll, p.stages, p.fields_per_pass, s, ylo, ldylo);
        const Blocked &B = m.blocked;
        if (B.n_fallback > 0) {
            launch_split_fused(m, m.sell32, x, ldx, y, ldy, nrhs, s, ylo, ldylo, 0, 0, B.fallback_slices.p,
                               B.n_fallback);
        }
        launch_split_long(m.sell32, x, ldx, y, ldy, nrhs, s, ylo, ldylo);
        AXGB_CUDA(cudaGetLastError());
        return;
    }
    const Sell &S = m.sell32;
    // direct kernel: with the caller's knobs (variant 0), else its own choice
    if (p.variant == 0)
        launch_split_fused(m, S, x, ldx, y, ldy, nrhs, s, ylo, ldylo, p.unroll,
                           p.fields_per_pass <= 0 || p.fields_per_pass > nrhs ? nrhs : p.fields_per_pass);
    else
        launch_split_fused(m, S, x, ldx, y, ldy, nrhs, s, ylo, ldylo);
    AXGB_CUDA(cudaGetLastError());
}

void apply_f64(Matrix &m, const double *x, i64 ldx, double *y, i64 ldy, i64 nrhs, cudaStream_t s) {
    if (!m.sell64.built) matrix_prepare(m, 0, s);
    const Sell &S = m.sell64;
    if (nrhs <= 0) return;
    launch_f64_fused(m, S, x, ldx, y, ldy, nrhs, s);
    AXGB_CUDA(cudaGetLastError());
}

void conservation(Matrix &m, const void *src, const void *dst, bool f32, int norm_type, double *out, cudaStream_t s) {
    double si, di;
    if (f32) {
        si = integral(static_cast<const float *>(src), m.area_a.p, m.frac_a.p, m.n_src, 0, s);
        di = integral(static_cast<const float *>(dst), m.area_b.p, m.frac_b.p, m.n_dst, norm_type == 0 ? 1 : 0, s);
    } else {
        si = integral(static_cast<const double *>(src), m.area_a.p, m.frac_a.p, m.n_src, 0, s);
        di = integral(static_cast<const double *>(dst), m.area_b.p, m.frac_b.p, m.n_dst, norm_type == 0 ? 1 : 0, s);
    }
    double ae = std::abs(si - di);
    double den = std::max({std::abs(si), std::abs(di), 2.220446049250313e-16});
    out[0] = si;
    out[1] = di;
    out[2] = ae;
    out[3] = ae / den;
}

void conservation_noalloc(Matrix &m, const double *src, const double *dst, int norm_type, double *out,
                          cudaStream_t s) {
    if (m.n_src > kNaMaxCells || m.n_dst > kNaMaxCells)
        throw Error(AXGB_ERR_INVALID, "conservation_noalloc: n_src (" + std::to_string(m.n_src) + ") or n_dst (" +
                                          std::to_string(m.n_dst) + ") exceeds the fixed scratch limit of " +
                                          std::to_string(kNaMaxCells) + " cells; use axgb_conservation_f64");
    double *scr = noalloc_scratch();
    const int nbs = static_cast<int>((m.n_src + kNaCellsPerBlock - 1) / kNaCellsPerBlock);
    const int nbd = static_cast<int>((m.n_dst + kNaCellsPerBlock - 1) / kNaCellsPerBlock);
    if (nbs > 0) k_integral_span<double><<<nbs, kNaThreads, 0, s>>>(src, m.area_a.p, m.frac_a.p, m.n_src, 0, scr);
    if (nbd > 0)
        k_integral_span<double><<<nbd, kNaThreads, 0, s>>>(dst, m.area_b.p, m.frac_b.p, m.n_dst,
                                                           norm_type == 0 ? 1 : 0, scr + kNaMaxBlocks);
    k_sum_partials<<<1, kNaThreads, 0, s>>>(scr, nbs, nbd, scr + 2 * kNaMaxBlocks);
    AXGB_CUDA(cudaGetLastError());
    double two[2] = {0.0, 0.0};
    AXGB_CUDA(cudaMemcpyAsync(two, scr + 2 * kNaMaxBlocks, sizeof(two), cudaMemcpyDeviceToHost, s));
    AXGB_CUDA(cudaStreamSynchronize(s));
    const double si = two[0], di = two[1];
    const double ae = std::abs(si - di);
    const double den = std::max({std::abs(si), std::abs(di), 2.220446049250313e-16});
    out[0] = si;
    out[1] = di;
    out[2] = ae;
    out[3] = ae / den;
}

void nan_batch_apply_f64(Matrix &m, const double *x, i64 ldx, double *y, i64 ldy, i64 nrhs, double na_thres,
                         cudaStream_t s) {
    if (nrhs <= 0 || m.n_dst == 0) return;
    if (!m.sell64.built) matrix_prepare(m, 0, s);
    const Sell &S = m.sell64;
    // One field alone: without others side by side, twice the blocks an SM (0.25
    // -> 0.5 deg: 35 -> 26 us; eight entries ahead instead of four 28).
    auto launch = [&](const double *xf, double *yf, i64 nf) {
        const auto kernel = nf == 1 ? k_nan<1, kNanK> : k_nan<kNanU, kNanK>;
        const int rows_w = nan_rows_w(nf);
        const i64 warps = (S.n_lrows + rows_w - 1) / rows_w + S.n_slices;
        const dim3 grid(nblk(warps, 8), nblk(nf, kNanG));
        kernel<<<grid, 256, 0, s>>>(sell_args(m, S), long_rows(S), S.total.p, S.ord.p, S.n_slices, xf, ldx, yf, ldy, nf,
                                    rows_w, na_thres);
    };
    // 9 to 11 fields leave the 16 lanes that add up a long row half empty: where long
    // rows are a good part of the rows and not much above 32 entries, eight fields
    // (two rows a warp) and then the others (five rows and more) are faster. C384 ->
    // 41 k Voronoi cells (rows of 35), 9 fields: 322 us, 370 in one launch. Longer rows
    // are chains whose length counts: 0.25 deg -> C48 815 us in one launch, 1665 in two.
    const bool split = nrhs > 8 && nrhs < 12 && S.n_lrows * 8 > m.n_dst && S.n_lentries <= 48 * S.n_lrows;
    const i64 most = split ? 8 : 65535 * kNanG;
    for (i64 f = 0; f < nrhs; f += most) launch(x + f * ldx, y + f * ldy, std::min<i64>(nrhs - f, most));
    AXGB_CUDA(cudaGetLastError());
}

void apply_masked_f64(Matrix &m, const double *x, const int *mask, double *y, cudaStream_t s) {
    if (m.n_dst == 0) return;
    k_masked_apply<<<nblk(m.n_dst, 256), 256, 0, s>>>(m.row_ptr.p, m.col.p, m.val.p, m.n_dst, x, mask, y);
    AXGB_CUDA(cudaGetLastError());
}

std::shared_ptr<Batch> batch_create(const std::vector<std::shared_ptr<Matrix>> &mats, const std::vector<i64> &nrhs) {
    auto b = std::make_shared<Batch>();
    b->mats = mats;
    b->nrhs = nrhs;
    for (auto &m : mats) matrix_prepare(*m, 2, 0);
    int dev = 0, sms = 0;
    AXGB_CUDA(cudaGetDevice(&dev));
    AXGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int per_sm = 0;
    AXGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<false>, 256, 0));
    b->blocks_slices = std::max(1, sms * std::max(1, per_sm));
    AXGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<true>, 256, 0));
    b->blocks_rows = std::max(1, sms * std::max(1, per_sm));
    b->counter.alloc(2);
    return b;
}

namespace {

// Work of the direct persistent kernels: for a matrix on the staged kernels,
// the slices the blocked layout leaves out, for the others all slices; and
// the rows of more than 32 entries.
void plan_direct(Batch &b) {
    b.desc.clear();
    for (int group = 0; group < 2; ++group) {  // slice items, then long-row items
        i64 items = 0;
        for (size_t q = 0; q < b.mats.size(); ++q) {
            Matrix &m = *b.mats[q];
            const Sell &S = m.sell32;
            const i64 k = b.nrhs[q];
            Batch::Desc d{};
            d.base = S.base.p;
            d.rlen = S.len.p;
            d.col = S.col.p;
            d.hl = S.hl.p;
            d.lrow = S.lrow.p;
            d.lptr = S.lptr.p;
            d.lcol = S.lcol.p;
            d.lhl = S.lhl.p;
            d.mat = static_cast<int>(q);
            d.n_rows = m.n_dst;
            d.nrhs = k;
            if (group == 1) {
                d.n_ids = S.n_lrows;
            } else if (b.use[q]) {
                d.ids = m.blocked.fallback_slices.p;
                d.n_ids = m.blocked.n_fallback;
            } else {
                d.n_ids = S.n_slices;
            }
            const i64 per = group == 0 ? kBatchTile : kBatchLongF;
            const i64 n_items = d.n_ids * ((k + per - 1) / per);
            if (n_items == 0) continue;
            d.item_begin = items;
            items += n_items;
            b.desc.push_back(d);
        }
        if (group == 0) {
            b.n_slice_desc = static_cast<int>(b.desc.size());
            b.total_slice_items = items;
        } else {
            b.total_row_items = items;
        }
    }
    b.d_desc.alloc(std::max<size_t>(1, b.desc.size()));
}

void drop_graphs(Batch &b) {
    for (auto &g : b.graphs) {
        cudaGraphExecDestroy(g.second.second);
        cudaGraphDestroy(g.second.first);
    }
    b.graphs.clear();
}

}  // namespace

// Ends a stream capture that an exception left open (dropping the partial
// graph) and destroys the private capture stream when there is one.
struct CaptureGuard {
    cudaStream_t st;
    bool own;
    bool open = true;
    ~CaptureGuard() {
        if (open) {
            cudaGraph_t g = nullptr;
            cudaStreamEndCapture(st, &g);
            if (g) cudaGraphDestroy(g);
        }
        if (own) cudaStreamDestroy(st);
    }
};

// Stream-ordered. The first call (and a call whose fields change which
// matrices can use the staged kernels) plans the work and captures a CUDA
// graph per stream; later calls update the field pointers in the device
// descriptors the graph reads and replay it. Calls on different streams are
// ordered after one another on the GPU (they share the batch's device
// buffers).
void batch_apply(Batch &b, const float *const *x, const i64 *ldx, float *const *y, const i64 *ldy, cudaStream_t s) {
    std::lock_guard<std::mutex> lk(b.mu);
    if (!b.done) AXGB_CUDA(cudaEventCreateWithFlags(&b.done, cudaEventDisableTiming));
    if (b.launched && b.last_stream != s) AXGB_CUDA(cudaStreamWaitEvent(s, b.done, 0));
    const size_t nm = b.mats.size();
    std::vector<const void *> ptrs;
    std::vector<char> use(nm, 0);
    // members with renumbered sources read their fields from b.xr (gathered first)
    if (b.xr.size() != nm) b.xr.resize(nm);
    std::vector<const float *> ex(nm);
    std::vector<i64> eld(nm);
    for (size_t q = 0; q < nm; ++q) {
        const Matrix &m = *b.mats[q];
        AXGB_REQUIRE(ldx[q] >= m.n_src && ldy[q] >= m.n_dst, "batch_apply: leading dimension");
        ptrs.push_back(x[q]);
        ptrs.push_back(y[q]);
        ptrs.push_back(reinterpret_cast<const void *>(ldx[q]));
        ptrs.push_back(reinterpret_cast<const void *>(ldy[q]));
        if (m.src_renum) {
            const size_t need = static_cast<size_t>(std::max<i64>(1, renum_ld(m) * b.nrhs[q]));
            if (b.xr[q].n < need) {
                b.xr[q].alloc(need);
                b.planned = false;  // new scratch address: re-plan and re-capture
            }
            ex[q] = b.xr[q].p;
            eld[q] = renum_ld(m);
        } else {
            ex[q] = x[q];
            eld[q] = ldx[q];
        }
        use[q] = (b.nrhs[q] > 0 && m.blocked.built && blocked_eligible(m, ex[q], eld[q], false)) ? 1 : 0;
    }
    if (!b.planned || use != b.use) {
        b.use = use;
        plan_direct(b);
        std::vector<Matrix *> raw;
        for (auto &m : b.mats) raw.push_back(m.get());
        b.blk = blk_batch_create(raw, b.nrhs, b.use);
        drop_graphs(b);
        b.last_ptrs.clear();
        b.planned = true;
    }
    if (ptrs != b.last_ptrs) {
        for (auto &d : b.desc) {
            d.x = ex[d.mat];
            d.ldx = eld[d.mat];
            d.y = y[d.mat];
            d.ldy = ldy[d.mat];
        }
        b.gdesc.clear();
        for (size_t q = 0; q < nm; ++q)
            if (b.mats[q]->src_renum && b.nrhs[q] > 0)
                b.gdesc.push_back({x[q], ldx[q], b.mats[q]->src_inv.p, b.mats[q]->src_span.p, b.mats[q]->n_src, b.nrhs[q], b.xr[q].p, eld[q]});
        if (b.d_gdesc.n < b.gdesc.size()) b.d_gdesc.alloc(b.gdesc.size());
        // stream-ordered update of the descriptors the graph reads
        if (!b.desc.empty())
            AXGB_CUDA(cudaMemcpyAsync(b.d_desc.p, b.desc.data(), sizeof(Batch::Desc) * b.desc.size(),
                                      cudaMemcpyHostToDevice, s));
        if (!b.gdesc.empty())
            AXGB_CUDA(cudaMemcpyAsync(b.d_gdesc.p, b.gdesc.data(), sizeof(GatherDesc) * b.gdesc.size(),
                                      cudaMemcpyHostToDevice, s));
        blk_batch_set_fields(*b.blk, ex.data(), eld.data(), y, ldy, s);
        AXGB_CUDA(cudaStreamSynchronize(s));
        b.last_ptrs = ptrs;
    }
    auto it = b.graphs.find(s);
    if (it == b.graphs.end()) {
        cudaStream_t cap = s;
        bool own = false;
        if (cap == 0) {  // legacy stream cannot be captured: capture on a private stream
            AXGB_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
            own = true;
        }
        CaptureGuard guard{cap, own};
        cudaGraph_t g;
        cudaGraphExec_t ge;
        AXGB_CUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
        for (size_t i = 0; i < b.gdesc.size(); ++i) {  // renumbered members: gather their fields first
            const GatherDesc &g = b.gdesc[i];
            k_gather_desc<<<gather_grid(g.n, g.nrhs), kGatherT, 0, cap>>>(b.d_gdesc.p + i);
        }
        // fork: the direct persistent kernel on its own side stream, the staged
        // class kernels over the others, joined back before the capture ends
        if (!b.fork) {
            AXGB_CUDA(cudaEventCreateWithFlags(&b.fork, cudaEventDisableTiming));
            for (int q = 0; q < Batch::kSide; ++q) {
                AXGB_CUDA(cudaStreamCreateWithFlags(&b.side[q], cudaStreamNonBlocking));
                AXGB_CUDA(cudaEventCreateWithFlags(&b.join[q], cudaEventDisableTiming));
            }
        }
        AXGB_CUDA(cudaEventRecord(b.fork, cap));
        for (int q = 0; q < Batch::kSide; ++q) AXGB_CUDA(cudaStreamWaitEvent(b.side[q], b.fork, 0));
        if (b.total_row_items > 0) {  // the row items (long chains of gathers) on their own side stream
            AXGB_CUDA(cudaMemsetAsync(b.counter.p + 1, 0, sizeof(unsigned long long), b.side[0]));
            k_batch<true><<<b.blocks_rows, 256, 0, b.side[0]>>>(
                b.d_desc.p + b.n_slice_desc, static_cast<int>(b.desc.size()) - b.n_slice_desc, b.total_row_items,
                b.counter.p + 1);
        }
        if (b.total_slice_items > 0) {
            AXGB_CUDA(cudaMemsetAsync(b.counter.p, 0, sizeof(unsigned long long), b.side[1]));
            k_batch<false><<<b.blocks_slices, 256, 0, b.side[1]>>>(b.d_desc.p, b.n_slice_desc, b.total_slice_items,
                                                                   b.counter.p);
        }
        blk_batch_launch(*b.blk, b.side + 2, Batch::kSide - 2);
        for (int q = 0; q < Batch::kSide; ++q) {
            AXGB_CUDA(cudaEventRecord(b.join[q], b.side[q]));
            AXGB_CUDA(cudaStreamWaitEvent(cap, b.join[q], 0));
        }
        guard.open = false;
        AXGB_CUDA(cudaStreamEndCapture(cap, &g));
        cudaError_t e = cudaGraphInstantiate(&ge, g, 0);
        if (e != cudaSuccess) {
            cudaGraphDestroy(g);
            AXGB_CUDA(e);
        }
        it = b.graphs.emplace(s, std::make_pair(g, ge)).first;
    }
    AXGB_CUDA(cudaGraphLaunch(it->second.second, s));
    AXGB_CUDA(cudaEventRecord(b.done, s));
    b.last_stream = s;
    b.launched = true;
}

}  // namespace axgb
