// ilu.cu -- ILU(0) on the device (ILUPreconditioner, ilu.cpp:41-89 and :225-271).
//
// Setup, all on the device:
//   1. level sets of the lower and upper triangles: level(i) = 1 + max level(j) over the
//      strictly lower (upper) columns j of row i.  k_levels_chain takes the rows in index
//      order, a block of them at a time, with a prefix scan for the dependence of each row
//      on its neighbour; patterns it does not suit go to a frontier sweep (k_levels, Kahn's
//      order, one grid barrier per level).
//   2. the factorisation, level by level of the lower sets: each row runs the reference's
//      IKJ elimination (same pivots, same update order, separate multiply and subtract),
//      so the factor values equal the reference's lu_val_ bit for bit.  Where a lower entry
//      updates only its row's diagonal (five-point grids) that is a sweep over the diagonals
//      (TriOp::FACTOR); other short rows run from an operation list worked out beforehand for
//      all rows at once (k_ilu_factor_ops).
//   3. level-ordered copies of L (strictly lower part) and U (diagonal + upper part), so
//      the rows of one level are contiguous in memory.
// Apply: forward then backward sweep, each by the kernel its triangle's shape asks for
// (tri_mode, rules.hpp).  The arithmetic per row is the reference's (ilu.cpp:230-237, :249-260),
// so z is bit-identical to ILUPreconditioner::apply.
#include <cooperative_groups.h>

#include <climits>
#include <cmath>
#include <tuple>
#include <cstring>

#include "ilu_row.cuh"
#include "ilu_sweep.cuh"
#include "krylov.cuh"
#include "scan.cuh"

namespace cg = cooperative_groups;

namespace hamlss {

namespace {

constexpr double kEps = 2.220446049250313e-16;
constexpr int kIluLptrSmem = 4096;       // level pointers kept in shared memory by the one-block kernels

// ---------------------------------------------------------------- pattern helpers
// dpos[i] = position of a_ii in row i (-1 if absent); lcnt[i] = # columns < i;
// ucnt[i] = # columns > i.
__global__ void k_row_info(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                           int* dpos, int* lcnt, int* ucnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int s = rp[i], e = rp[i + 1], d = -1, lo = 0, hi = 0;
        for (int k = s; k < e; ++k) {
            int c = ci[k];
            if (c < i) ++lo;
            else if (c == i) d = k;
            else ++hi;
        }
        dpos[i] = d;
        lcnt[i] = lo;
        ucnt[i] = hi;
    }
}

// column counts of the pattern (for the transpose)
__global__ void k_col_count(int n, const int* __restrict__ rp, const int* __restrict__ ci, int* cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int k = rp[i]; k < rp[i + 1]; ++k) atomicAdd(&cnt[ci[k]], 1);
}

__global__ void k_col_fill(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                           int* fillpos, int* trow) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int k = rp[i]; k < rp[i + 1]; ++k) trow[atomicAdd(&fillpos[ci[k]], 1)] = i;
}

// Kahn frontier sweep over the dependency DAG of one triangle.
//   LOWER: row i depends on columns j < i of row i; dependents of j are the rows i > j
//          holding column j (transpose entries below the diagonal).
//   UPPER: mirror image.
// indeg must hold the dependency counts; on exit order[] lists the rows level by level,
// lptr[l] is where level l starts, level[i] is the level of row i, *nlev the count.
template <bool LOWER>
__global__ void k_levels(int n, const int* __restrict__ trp, const int* __restrict__ trow,
                         int* indeg, int* order, int* lptr, int* cnt, int* level, int* nlev) {
    cg::grid_group grid = cg::this_grid();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nth = gridDim.x * blockDim.x;
    for (int i = tid; i < n; i += nth)
        if (indeg[i] == 0) order[atomicAdd(&cnt[0], 1)] = i;
    grid.sync();
    int start = 0;
    for (int l = 0;; ++l) {
        const int c = *(volatile int*)&cnt[l];
        if (c == 0) {
            if (tid == 0) { *nlev = l; lptr[l] = start; }
            break;
        }
        if (tid == 0) lptr[l] = start;
        const int next = start + c;
        for (int t = tid; t < c; t += nth) {
            const int i = order[start + t];
            level[i] = l;
            for (int k = trp[i]; k < trp[i + 1]; ++k) {
                const int d = trow[k];
                if (LOWER ? (d > i) : (d < i)) {
                    if (atomicSub(&indeg[d], 1) == 1) order[next + atomicAdd(&cnt[l + 1], 1)] = d;
                }
            }
        }
        start = next;
        grid.sync();
    }
}

// Level sets of a pattern in index order, one block per triangle (block 0 the lower one,
// block 1 the upper one, whose rows are taken backwards).  kChainRows rows are decided at a
// time: a row's dependencies in earlier rows are final and read from a shared-memory ring of
// the last kChainRing levels (older ones from global memory), and its dependence on the row
// just before it -- the west or east neighbour of a grid row -- is a max-plus recurrence
// level[m] = max(level[m-1] + 1, c[m]) solved by a segmented prefix maximum.  Dependencies
// inside the block of rows that are not that neighbour are met by repeating the pass until
// nothing changes (levels only grow, so it ends): a natural-order grid takes a pass for each
// grid row that the block spans.  The next block's pattern is loaded meanwhile.  A pattern
// that needs many passes is given up (nlev[tri] = -1) and left to k_levels.
// 512^2 grid, both triangles at once: 0.99 ms; 13.0 ms one after the other with one grid
// barrier a level.
constexpr int kChainRows = 1024;
constexpr int kChainRing = 16384;
constexpr int kChainPre = 6;             // dependencies of a row held in registers
constexpr int kChainPasses = 24;         // passes a block allowed on average before giving up

__global__ void __launch_bounds__(kChainRows)
k_levels_chain(int n, const int* __restrict__ rp, const int* __restrict__ ci, int* levelL, int* levelU,
               int* nlev) {
    extern __shared__ int chain_ring[];
    __shared__ int w_val[32];
    __shared__ unsigned w_all;           // bit w: every row of warp w continues the chain
    __shared__ int s_max;
    const bool lower = blockIdx.x == 0;
    int* level = lower ? levelL : levelU;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int chunks = (n + kChainRows - 1) / kChainRows;
    if (tid == 0) s_max = 0;
    // row m of the sweep is row i of the matrix
    auto mirror = [&](int i) { return lower ? i : n - 1 - i; };
    int rs1 = 0, re1 = 0;                // row bounds of the next block's row
    int dep[kChainPre];                  // this block's row: its first dependencies (sweep index)
    int rs = 0, re = 0;
    auto bounds = [&](int c, int& s, int& e) {
        const int m = c * kChainRows + tid;
        s = e = 0;
        if (c < chunks && m < n) {
            const int i = mirror(m);
            s = __ldg(&rp[i]);
            e = __ldg(&rp[i + 1]);
        }
    };
    auto deps = [&](int m, int s, int e, int (&d)[kChainPre]) {
        int col[kChainPre];
#pragma unroll
        for (int k = 0; k < kChainPre; ++k) col[k] = s + k < e ? __ldg(&ci[s + k]) : -1;
#pragma unroll
        for (int k = 0; k < kChainPre; ++k) {
            const int dm = s + k < e ? mirror(col[k]) : m;
            d[k] = dm < m ? dm : -1;     // -1: the diagonal or the other triangle
        }
    };
    bounds(0, rs, re);
    deps(tid, rs, re, dep);
    bounds(1, rs1, re1);
    int sweeps = 0, top = -1;
    for (int c = 0; c < chunks; ++c) {
        const int m0 = c * kChainRows, m = m0 + tid;
        int ndep[kChainPre];
        deps(m + kChainRows, rs1, re1, ndep);           // next block, in flight meanwhile
        int rs2, re2;
        bounds(c + 2, rs2, re2);
        // dependencies in earlier blocks: final; the neighbour: a chain link; others: `more`
        int ext = 0;
        bool chain = false, more = false;
        auto take = [&](int dm) {
            if (dm < 0) return;
            if (dm >= m0) {
                if (dm == m - 1) chain = true;
                else more = true;
            } else {
                const int lv = m0 - dm <= kChainRing - kChainRows ? chain_ring[dm & (kChainRing - 1)]
                                                                  : level[mirror(dm)];
                ext = max(ext, lv + 1);
            }
        };
        if (m < n) {
#pragma unroll
            for (int k = 0; k < kChainPre; ++k) take(dep[k]);
            for (int k = rs + kChainPre; k < re; ++k) {
                const int dm = mirror(__ldg(&ci[k]));
                take(dm < m ? dm : -1);
            }
        }
        // first row of a warp's chain ends at the warp boundary: carried across by the warps
        const unsigned cont = __ballot_sync(0xffffffffu, chain);
        int mine = -1;
        bool again = false, first = true;
        do {
            int v = ext;
            if (more && mine >= 0) {
                auto inner = [&](int dm) {
                    if (dm >= m0 && dm != m - 1) v = max(v, chain_ring[dm & (kChainRing - 1)] + 1);
                };
#pragma unroll
                for (int k = 0; k < kChainPre; ++k) inner(dep[k]);
                for (int k = rs + kChainPre; k < re; ++k) {
                    const int dm = mirror(__ldg(&ci[k]));
                    if (dm < m) inner(dm);
                }
            }
            // segmented prefix maximum of v - lane over chain links, inside the warp
            int u = v - lane;
            const unsigned below = ~cont & (0xffffffffu >> (31 - lane));      // segment starts at or before lane
            const int seg = below ? 31 - __clz(below) : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, u, o);
                if (lane - o >= seg) u = max(u, t);
            }
            int lv = u + lane;
            if (lane == 31) w_val[wid] = lv;
            if (wid == 0 && lane == 0) w_all = 0;
            __syncthreads();
            // across warps: warp w's incoming value is the last level of warp w - 1
            if (lane == 0 && cont == 0xffffffffu) atomicOr(&w_all, 1u << wid);
            __syncthreads();
            {
                // value entering this warp: max over warps w' < wid reached through fully
                // linked warps, of w_val[w'] + 32 (wid - 1 - w')
                const unsigned full = w_all;
                int in = -0x40000000;
                if (lane < wid) {
                    // every warp strictly between lane and wid is fully linked
                    const unsigned need = (wid - lane > 1) ? (((1u << (wid - lane - 1)) - 1u) << (lane + 1)) : 0u;
                    if ((full & need) == need) in = w_val[lane] + 32 * (wid - 1 - lane);
                }
                in = __reduce_max_sync(0xffffffffu, in);
                // it reaches the lanes linked to the warp's first one
                const bool linked = wid > 0 && (cont & (0xffffffffu >> (31 - lane))) == (0xffffffffu >> (31 - lane));
                if (linked) lv = max(lv, in + 1 + lane);
            }
            const bool changed = lv != mine;
            mine = lv;
            if (m < n) chain_ring[m & (kChainRing - 1)] = lv;
            // repeated only where some row has other dependencies inside the block
            again = __syncthreads_or(first ? more : changed);
            first = false;
            ++sweeps;
        } while (again && sweeps <= kChainPasses * (c + 16));
        if (sweeps > kChainPasses * (c + 16)) {
            if (tid == 0) nlev[blockIdx.x] = -1;
            return;
        }
        if (m < n) {
            level[mirror(m)] = mine;
            top = max(top, mine);
        }
        rs = rs1; re = re1; rs1 = rs2; re1 = re2;
#pragma unroll
        for (int k = 0; k < kChainPre; ++k) dep[k] = ndep[k];
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) atomicMax(&s_max, top);
    __syncthreads();
    if (tid == 0) nlev[blockIdx.x] = s_max + 1;
}

// (rows of one level in a warp add once: red-black and other coloured orderings have a few
// levels of millions of rows, whose counters every thread would queue at)
__global__ void k_level_hist(int n, const int* __restrict__ level, int* cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int l = level[i];
        const unsigned same = __match_any_sync(__activemask(), l);
        if ((int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&cnt[l], __popc(same));
    }
}

__global__ void k_level_place(int n, const int* __restrict__ level, int* fill, int* order) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int l = level[i], lane = threadIdx.x & 31;
        const unsigned act = __activemask(), same = __match_any_sync(act, l);
        const int first = __ffs(same) - 1;
        int at = 0;
        if (lane == first) at = atomicAdd(&fill[l], __popc(same));
        at = __shfl_sync(act, at, first);
        order[at + __popc(same & ((1u << lane) - 1u))] = i;
    }
}

// Rows of each level by index (a level of at most kSortRows rows; wider ones keep the order
// they were placed in, which no result depends on): neighbouring rows of a level then read
// neighbouring entries.  *maxw receives the widest level.
constexpr int kSortRows = 2048;
__global__ void __launch_bounds__(256)
k_level_sort(int nlev, const int* __restrict__ lptr, int* order, int* maxw) {
    __shared__ int key[kSortRows];
    for (int l = blockIdx.x; l < nlev; l += gridDim.x) {
        const int b = lptr[l], w = lptr[l + 1] - b;
        if (threadIdx.x == 0) atomicMax(maxw, w);
        if (w <= 1 || w > kSortRows) continue;
        int N = 2;
        while (N < w) N <<= 1;
        for (int t = threadIdx.x; t < N; t += blockDim.x) key[t] = t < w ? order[b + t] : INT_MAX;
        __syncthreads();
        for (int kk = 2; kk <= N; kk <<= 1)
            for (int jj = kk >> 1; jj > 0; jj >>= 1) {
                for (int t = threadIdx.x; t < N; t += blockDim.x) {
                    const int p = t ^ jj;
                    if (p > t) {
                        const int x = key[t], y = key[p];
                        if ((x > y) == ((t & kk) == 0)) { key[t] = y; key[p] = x; }
                    }
                }
                __syncthreads();
            }
        for (int t = threadIdx.x; t < w; t += blockDim.x) order[b + t] = key[t];
        __syncthreads();
    }
}

__global__ void k_invert(int n, const int* __restrict__ order, int* pos) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) pos[order[t]] = t;
}

// out[t] = pos[order[t]]
__global__ void k_compose(int n, const int* __restrict__ order, const int* __restrict__ pos, int* out) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) out[t] = pos[order[t]];
}

// Operation lists of the elimination (ilu_row) for rows of at most kOpsRow entries, in
// position order of the lower levels: x = target entry of the row (+ kOpsDiv for the
// division by pivot y), y = factor entry it reads (-1: the pivot is absent).
constexpr int kOpsRow = 8;
constexpr int kOpsDiv = 16;
template <bool FILL>
__global__ void k_ilu_ops(int n, const int* __restrict__ order, const int* __restrict__ rp,
                          const int* __restrict__ ci, const int* __restrict__ dpos, int* optr, int2* ops,
                          int4* info) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = order[t], s = rp[i], e = rp[i + 1];
        int o = FILL ? optr[t] : 0;
        for (int p = s; p < e; ++p) {
            const int k = ci[p];
            if (k >= i) break;
            if (FILL) ops[o] = make_int2(kOpsDiv | (p - s), dpos[k]);
            ++o;
            int pi = p + 1;
            for (int q = rp[k]; q < rp[k + 1]; ++q) {
                const int j = ci[q];
                if (j <= k) continue;
                while (pi < e && ci[pi] < j) ++pi;
                if (pi == e) break;
                if (ci[pi] == j) {
                    if (FILL) ops[o] = make_int2(pi - s, q);
                    ++o;
                }
            }
        }
        if (FILL) info[t] = make_int4(s, e - s, optr[t], o - optr[t]);
        else optr[t] = o;
    }
}

// The elimination from operation lists, one block, a barrier per level.  A row's place and
// lengths (info) are fetched two levels ahead, its values and first operations one level
// ahead, so behind the barrier there is one round of loads -- the factor entries of earlier
// rows that its operations read, all issued together -- and the row's arithmetic.  Walking
// the pattern inside the level (k_ilu_factor_block) costs a chain of dependent loads
// instead: 7.1 us a level on the 512^2 grid, 2.2 us here.
constexpr int kOpsPre = 6;
constexpr int kOpsThreads = 512;
constexpr size_t kOpsSmem = (size_t)kOpsRow * kOpsThreads * sizeof(double);

struct OpsRow {
    int4 info;               // first entry, entries, first operation, operations; y = 0: no row
    int2 op[kOpsPre];
    double own[kOpsRow];
};

__global__ void __launch_bounds__(kOpsThreads, 1)
k_ilu_factor_ops(int nlev, const int* __restrict__ lptr_g, const int4* __restrict__ info,
                 const int* __restrict__ ci, const int2* __restrict__ ops, double* lu, int* status) {
    extern __shared__ double ops_own[];                  // the current row's values, [entry][thread]
    __shared__ int s_lptr[kIluLptrSmem];
    const int tid = threadIdx.x;
    constexpr int NT = kOpsThreads;
    for (int l = tid; l <= nlev && l < kIluLptrSmem; l += NT) s_lptr[l] = lptr_g[l];
    __syncthreads();
    auto lptr = [&](int l) { return l < kIluLptrSmem ? s_lptr[l] : __ldg(&lptr_g[l]); };
    auto own = [&](int k) -> double& { return ops_own[k * NT + tid]; };
    auto where = [&](int l) {
        if (l < nlev) {
            const int t = lptr(l) + tid;
            if (t < lptr(l + 1)) return __ldg(&info[t]);
        }
        return make_int4(0, 0, 0, 0);
    };
    auto fetch = [&](OpsRow& q, int4 in) {
        q.info = in;
#pragma unroll
        for (int k = 0; k < kOpsRow; ++k)
            if (k < in.y) q.own[k] = lu[in.x + k];       // changed only in the row's own level
#pragma unroll
        for (int k = 0; k < kOpsPre; ++k)
            if (k < in.w) q.op[k] = __ldg(&ops[in.z + k]);
    };
    auto run = [&](const OpsRow& q) {
        double val[kOpsPre];
#pragma unroll
        for (int k = 0; k < kOpsPre; ++k)
            if (k < q.info.w) val[k] = q.op[k].y >= 0 ? lu[q.op[k].y] : 0.0;
#pragma unroll
        for (int k = 0; k < kOpsRow; ++k)
            if (k < q.info.y) own(k) = q.own[k];
        double lik = 0.0;
        bool bad = false;
        auto step = [&](int2 op, double x) {
            const int a = op.x & (kOpsDiv - 1);
            if (op.x & kOpsDiv) {
                if (fabs(x) < kEps) {                    // the pivot of this entry's column
                    atomicMin(status, ci[q.info.x + a]);
                    bad = true;
                    return;
                }
                lik = own(a) / x;
                own(a) = lik;
            } else {
                own(a) = __dsub_rn(own(a), __dmul_rn(lik, x));
            }
        };
#pragma unroll
        for (int k = 0; k < kOpsPre; ++k)
            if (k < q.info.w && !bad) step(q.op[k], val[k]);
        for (int k = kOpsPre; k < q.info.w && !bad; ++k) {
            const int2 op = __ldg(&ops[q.info.z + k]);
            step(op, op.y >= 0 ? lu[op.y] : 0.0);
        }
        for (int k = 0; k < q.info.y; ++k) lu[q.info.x + k] = own(k);
    };
    OpsRow cur;
    fetch(cur, where(0));
    int4 in1 = where(1);
    for (int l = 0; l < nlev; ++l) {
        OpsRow nxt;
        fetch(nxt, in1);                                 // level l + 1
        const int4 in2 = where(l + 2);
        if (cur.info.y > 0) {
            run(cur);
            const int e = lptr(l + 1);
            for (int t = lptr(l) + tid + NT; t < e; t += NT) {   // rows beyond the block width
                OpsRow more;
                fetch(more, __ldg(&info[t]));
                run(more);
            }
        }
        __syncthreads();
        cur = nxt;
        in1 = in2;
    }
}

__global__ void k_ilu_factor_block(int nlev, const int* __restrict__ order, const int* __restrict__ lptr,
                                   const int* __restrict__ rp, const int* __restrict__ ci,
                                   const int* __restrict__ dpos, double* lu, int* status) {
    for (int l = 0; l < nlev; ++l) {
        const int b = lptr[l], e = lptr[l + 1];
        for (int t = b + threadIdx.x; t < e; t += blockDim.x) ilu_row(order[t], rp, ci, dpos, lu, status);
        __syncthreads();
    }
}

__global__ void k_ilu_factor_grid(int nlev, const int* __restrict__ order, const int* __restrict__ lptr,
                                  const int* __restrict__ rp, const int* __restrict__ ci,
                                  const int* __restrict__ dpos, double* lu, int* status) {
    cg::grid_group grid = cg::this_grid();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    for (int l = 0; l < nlev; ++l) {
        const int b = lptr[l], e = lptr[l + 1];
        for (int t = b + tid; t < e; t += nth) ilu_row(order[t], rp, ci, dpos, lu, status);
        grid.sync();
    }
}

// facts[0..2] = the longest row's entries below, above the diagonal, and in all;
// facts[5..6] = the entries below and above the diagonal
__global__ void k_max_counts(int n, const int* __restrict__ lcnt, const int* __restrict__ ucnt,
                             const int* __restrict__ rp, int* facts) {
    int a = 0, b = 0, c = 0, nl = 0, nu = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        nl += lcnt[i];
        nu += ucnt[i];
        a = max(a, lcnt[i]);
        b = max(b, ucnt[i]);
        c = max(c, rp[i + 1] - rp[i]);
    }
    a = __reduce_max_sync(0xffffffffu, a);
    b = __reduce_max_sync(0xffffffffu, b);
    c = __reduce_max_sync(0xffffffffu, c);
    nl = __reduce_add_sync(0xffffffffu, nl);
    nu = __reduce_add_sync(0xffffffffu, nu);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&facts[5], nl);
        atomicAdd(&facts[6], nu);
        atomicMax(&facts[0], a);
        atomicMax(&facts[1], b);
        atomicMax(&facts[2], c);
    }
}

__global__ void k_to_float(int n, const double* __restrict__ a, float* __restrict__ b) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = (float)a[i];
}

// Level-ordered L / U copies.  Lrp/Urp are prefix sums of per-slot counts in order.
__global__ void k_perm_counts(int n, const int* __restrict__ order, const int* __restrict__ cnt,
                              int* out) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
        out[t] = cnt[order[t]];
}

__global__ void k_fill_L(int n, const int* __restrict__ order, const int* __restrict__ rp,
                         const int* __restrict__ ci, const double* __restrict__ lu,
                         const int* __restrict__ Lrp, int* Lci, double* Lv) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = order[t];
        int o = Lrp[t];
        for (int p = rp[i]; p < rp[i + 1]; ++p) {
            const int j = ci[p];
            if (j >= i) break;
            Lci[o] = j;
            Lv[o] = lu[p];
            ++o;
        }
    }
}

// U copy: the diagonal (1.0 if absent, as backward_sub assumes, ilu.cpp:251) then the
// upper entries.  bad[0] receives the smallest row with |u_ii| < eps (ilu.cpp:257-259).
__global__ void k_fill_U(int n, const int* __restrict__ order, const int* __restrict__ rp,
                         const int* __restrict__ ci, const double* __restrict__ lu,
                         const int* __restrict__ Urp, int* Uci, double* Uv, double* Ud, int* bad) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = order[t];
        int o = Urp[t];
        double d = 1.0;
        for (int p = rp[i]; p < rp[i + 1]; ++p) {
            const int j = ci[p];
            if (j == i) { d = lu[p]; continue; }
            if (j > i) {
                Uci[o] = j;
                Uv[o] = lu[p];
                ++o;
            }
        }
        Ud[t] = d;
        if (fabs(d) < kEps) atomicMin(bad, i);
    }
}

// ------------------------------------------------------------------------ sweeps
// A triangle in position order with the matrix's own columns and vectors in row order.
template <typename T>
struct TriRows {
    int n = 0, nlev = 0;
    const int* ord = nullptr;
    const int* lptr = nullptr;
    const int* rp = nullptr;
    const int* ci = nullptr;
    const T* v = nullptr;
    const T* dg = nullptr;
};

// One sweep by one block for triangles with long rows (ilu_sweep.cuh's rings hold steps of
// short rows).
//
// One level's critical path is a barrier plus the loads of the vector being solved for; the
// rest of a row's inputs (its index, right-hand side, columns, values, diagonal) do not
// depend on the sweep, so they are fetched ahead in a three-stage pipeline: stage 1 (row
// index, row bounds) two levels ahead, stage 2 (rhs, up to kIluPre columns and values, the
// diagonal) one level ahead, while the current level computes.  The level pointers sit in
// shared memory.  A thread pipelines its first row of each level; rows beyond the block
// width and rows longer than kIluPre take the plain path.  The block's own stores are read
// back with ordinary loads after the barrier (block scope), and every row sums in its
// stored (ascending column) order, so results are bit-identical to the plain loop.
constexpr int kIluPre = 4;

template <typename T>
struct IluStage2 {
    int t, i, o0, cnt;
    T rv, d;
    int c[kIluPre];
    T v[kIluPre];
};

template <typename T, bool DIV, int NT>
__global__ void __launch_bounds__(NT)
k_tri_block(TriRows<T> F, const T* rhs, T* out, const int* gate) {
    __shared__ int s_lptr[kIluLptrSmem];
    if (gate && *(volatile const int*)gate) return;
    const int tid = threadIdx.x;
    for (int l = tid; l <= F.nlev && l < kIluLptrSmem; l += NT) s_lptr[l] = F.lptr[l];
    __syncthreads();
    const int nlev = F.nlev;
    const int* __restrict__ ord = F.ord;
    const int* __restrict__ rp = F.rp;
    const int* __restrict__ ci = F.ci;
    const T* __restrict__ v = F.v;
    const T* __restrict__ dg = F.dg;
    auto lptr = [&](int l) { return l < kIluLptrSmem ? s_lptr[l] : __ldg(&F.lptr[l]); };
    // stage 1 of a level: (t, i, o0, cnt) of this thread's first row, t = -1 if none
    auto stage1 = [&](int l, int& t, int& i, int& o0, int& cnt) {
        t = -1;
        if (l < nlev) {
            const int b = lptr(l), e = lptr(l + 1);
            if (b + tid < e) {
                t = b + tid;
                i = ord[t];
                o0 = rp[t];
                cnt = rp[t + 1] - o0;
            }
        }
    };
    auto stage2 = [&](IluStage2<T>& q, int t, int i, int o0, int cnt) {
        q.t = t;
        if (t < 0) return;
        q.i = i;
        q.o0 = o0;
        q.cnt = cnt;
        q.rv = rhs[i];
        if (DIV) q.d = dg[t];
#pragma unroll
        for (int k = 0; k < kIluPre; ++k)
            if (k < cnt) {
                q.c[k] = ci[o0 + k];
                q.v[k] = v[o0 + k];
            }
    };
    int t1, i1, o1, c1;                  // stage 1 of level l + 1
    IluStage2<T> cur;
    {
        int t0, i0, o0, c0;
        stage1(0, t0, i0, o0, c0);
        stage2(cur, t0, i0, o0, c0);
        stage1(1, t1, i1, o1, c1);
    }
    for (int l = 0; l < nlev; ++l) {
        IluStage2<T> nxt;
        stage2(nxt, t1, i1, o1, c1);     // level l + 1, in flight while level l computes
        int t2, i2, o2, c2;
        stage1(l + 2, t2, i2, o2, c2);   // level l + 2
        if (cur.t >= 0) {
            T s = cur.rv;
            if (cur.cnt <= kIluPre) {
#pragma unroll
                for (int k = 0; k < kIluPre; ++k)
                    if (k < cur.cnt) s = sub_mul<T>(s, cur.v[k], out[cur.c[k]]);
            } else {
                for (int o = cur.o0; o < cur.o0 + cur.cnt; ++o) s = sub_mul<T>(s, v[o], out[ci[o]]);
            }
            out[cur.i] = DIV ? s / cur.d : s;
            // rows of this level beyond the block width
            const int e = lptr(l + 1);
            for (int t = cur.t + NT; t < e; t += NT) {
                const int i = ord[t];
                T s2 = rhs[i];
                for (int o = rp[t]; o < rp[t + 1]; ++o) s2 = sub_mul<T>(s2, v[o], out[ci[o]]);
                out[i] = DIV ? s2 / dg[t] : s2;
            }
        }
        __syncthreads();
        cur = nxt;
        t1 = t2; i1 = i2; o1 = o2; c1 = c2;
    }
}

// The same sweep with the whole grid (cooperative launch) for triangles with wide levels: the
// lower triangle's, the upper one's (nlev = 0: not this one), or one after the other.  (The
// factor through the read-only path, so that a long row's loads go out several at a time: one row
// of 100,000 entries 32 -> 16 ms.)
template <typename T, bool DIV>
__device__ __forceinline__ void grid_sweep(const TriRows<T>& F, const T* rhs, T* out) {
    cg::grid_group grid = cg::this_grid();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    for (int l = 0; l < F.nlev; ++l) {
        const int b = F.lptr[l], e = F.lptr[l + 1];
        for (int t = b + tid; t < e; t += nth) {
            const int i = __ldg(&F.ord[t]), o1 = __ldg(&F.rp[t + 1]);
            T s = __ldcg(&rhs[i]);
#pragma unroll 4
            for (int o = __ldg(&F.rp[t]); o < o1; ++o)
                s = sub_mul<T>(s, __ldg(&F.v[o]), __ldcg(&out[__ldg(&F.ci[o])]));
            out[i] = DIV ? s / F.dg[t] : s;
        }
        if (l + 1 < F.nlev) grid.sync();
    }
}

template <typename T>
__global__ void k_tri_grid(TriRows<T> L, TriRows<T> U, const T* rhs, T* y, T* z, const int* gate) {
    if (gate && *(volatile const int*)gate) return;
    grid_sweep<T, false>(L, rhs, y);
    if (L.nlev && U.nlev) cg::this_grid().sync();
    grid_sweep<T, true>(U, y, z);
}

// ------------------------------------------------------------------------- ILUT
// ILUT(tau, p) (ilu.cpp:94-220) on the device.  The reference eliminates row by row with
// a dense work row; row i needs the finished U rows of the pivots k < i it eliminates.
// Here one warp takes one row at a time, rows claimed in increasing order (atomic ticket,
// cooperative launch: every claimed row belongs to a running warp, so a row only waits on
// rows that can finish); the work row's touched columns live in the warp's shared memory
// (column, value, active flag) and the pending pivots in a min-heap, so the columns are
// visited in the reference's ascending order and every value gets the reference's
// operations (separate multiply and subtract, the same division, the same drops).  The
// keep-largest selection is the reference's heap select (make_heap / pop_heap over the
// row in column order).  Each finished row is published (entries, counts, then a done
// flag after a fence, then a count of finished rows); a wait on a done flag gives up when
// no row at all has finished for about a second (the kernel records *err, every warp
// stops, and the host fails with HAMLSS_ERR_TIMEOUT).
constexpr int kIlutWarps = 4;
constexpr int kIlutCap = 512;            // touched columns a work row may hold
// per warp: columns, values, flags, pending heap, and a row buffer of kIlutCap + 1 entries
constexpr size_t kIlutWarpBytes = (size_t)kIlutCap * (4 + 8 + 1 + 4) + 16 * ((size_t)kIlutCap + 1);
constexpr long long kIlutWaitCycles = 2000000000LL;

struct IlutArgs {
    int n, fill_p;
    double drop_tol;
    const int* rp;
    const int* ci;
    const double* v;
    const int* off;                      // capacity offsets: row i's L at off[i], U at off[i] + max(keep, 1)
    int* ecol;
    double* eval;
    int* lcnt;
    int* ucnt;
    unsigned long long* done;            // of a finished row: U's first slot, its entries << 32; else 0
    int* ticket;
    int* err;                            // 1 bounded wait ran out, 2 work row overflow
    int* finished;                       // rows published so far
};

struct IlutEntry {
    int col;
    double val;
};

__device__ __forceinline__ bool ilut_first(const IlutEntry& a, const IlutEntry& b) {
    return fabs(a.val) > fabs(b.val);
}

__device__ void ilut_adjust(IlutEntry* h, int hole, int len, IlutEntry value) {
    const int top = hole;
    int child = hole;
    while (child < (len - 1) / 2) {
        child = 2 * (child + 1);
        if (ilut_first(h[child], h[child - 1])) --child;
        h[hole] = h[child];
        hole = child;
    }
    if ((len & 1) == 0 && child == (len - 2) / 2) {
        child = 2 * (child + 1);
        h[hole] = h[child - 1];
        hole = child - 1;
    }
    int parent = (hole - 1) / 2;
    while (hole > top && ilut_first(h[parent], value)) {
        h[hole] = h[parent];
        hole = parent;
        parent = (hole - 1) / 2;
    }
    h[hole] = value;
}

// keep_largest (ilu.cpp:186-197) on a row in column order: heap select, then column order.
__device__ void ilut_keep(IlutEntry* row, int* len, int keep) {
    if (keep <= 0 || *len <= keep) return;
    for (int parent = (keep - 2) / 2; keep >= 2; --parent) {
        ilut_adjust(row, parent, keep, row[parent]);
        if (parent == 0) break;
    }
    for (int t = keep; t < *len; ++t)
        if (ilut_first(row[t], row[0])) {
            IlutEntry v = row[t];
            row[t] = row[0];
            ilut_adjust(row, 0, keep, v);
        }
    *len = keep;
    for (int a = 1; a < keep; ++a) {                 // insertion sort by column
        IlutEntry x = row[a];
        int b = a - 1;
        while (b >= 0 && row[b].col > x.col) { row[b + 1] = row[b]; --b; }
        row[b + 1] = x;
    }
}

__device__ __forceinline__ void heap_push(int* h, int& nh, int x) {
    int c = nh++;
    h[c] = x;
    while (c > 0 && h[(c - 1) / 2] > h[c]) {
        const int t = h[c];
        h[c] = h[(c - 1) / 2];
        h[(c - 1) / 2] = t;
        c = (c - 1) / 2;
    }
}

__device__ __forceinline__ int heap_pop(int* h, int& nh) {
    const int top = h[0];
    h[0] = h[--nh];
    for (int c = 0;;) {
        const int l = 2 * c + 1, r = l + 1;
        int m = c;
        if (l < nh && h[l] < h[m]) m = l;
        if (r < nh && h[r] < h[m]) m = r;
        if (m == c) break;
        const int t = h[c];
        h[c] = h[m];
        h[m] = t;
        c = m;
    }
    return top;
}

// The work-row slots that are active, at least tau in magnitude and below (lower) or above
// column i, gathered by the warp into dst[0..count) and sorted by column (warp bitonic sort;
// columns are distinct).  dst must hold the next power of two >= count entries.
__device__ int ilut_gather_sorted(const int* scol, const double* sval, const unsigned char* sact, int nt,
                                  int i, double tau, bool lower, IlutEntry* dst, int lane) {
    int cnt = 0;
    for (int b0 = 0; b0 < nt; b0 += 32) {
        const int t = b0 + lane;
        bool take = false;
        int c = 0;
        double v = 0.0;
        if (t < nt) {
            c = scol[t];
            v = sval[t];
            take = sact[t] && fabs(v) >= tau && (lower ? c < i : c > i);
        }
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (take) {
            const int q = cnt + __popc(m & ((1u << lane) - 1u));
            dst[q].col = c;
            dst[q].val = v;
        }
        cnt += __popc(m);
    }
    int N = 1;
    while (N < cnt) N <<= 1;
    for (int t = cnt + lane; t < N; t += 32) {
        dst[t].col = INT_MAX;
        dst[t].val = 0.0;
    }
    __syncwarp();
    for (int kk = 2; kk <= N; kk <<= 1)
        for (int jj = kk >> 1; jj > 0; jj >>= 1) {
            for (int t = lane; t < N; t += 32) {
                const int p = t ^ jj;
                if (p > t) {
                    const IlutEntry x = dst[t], y = dst[p];
                    if ((x.col > y.col) == ((t & kk) == 0)) {
                        dst[t] = y;
                        dst[p] = x;
                    }
                }
            }
            __syncwarp();
        }
    return cnt;
}

__global__ void __launch_bounds__(32 * kIlutWarps) k_ilut_rows(IlutArgs a) {
    extern __shared__ unsigned char ilut_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char* base = ilut_smem + (size_t)wid * kIlutWarpBytes;
    int* scol = reinterpret_cast<int*>(base);
    double* sval = reinterpret_cast<double*>(base + 4 * kIlutCap);
    unsigned char* sact = base + 12 * kIlutCap;
    int* heap = reinterpret_cast<int*>(base + 13 * kIlutCap);
    IlutEntry* row = reinterpret_cast<IlutEntry*>(base + 17 * kIlutCap);
    for (;;) {
        int i = 0;
        if (lane == 0) i = *(volatile int*)a.err ? a.n : atomicAdd(a.ticket, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= a.n) break;
        const int rs = a.rp[i], re = a.rp[i + 1], orig = re - rs;
        const int keep = orig + a.fill_p;
        const int half = keep > 1 ? keep : 1;        // capacity of each half of the row
        int nt = min(orig, kIlutCap);
        bool overflow = orig > kIlutCap;
        for (int t = lane; t < nt; t += 32) {
            scol[t] = a.ci[rs + t];
            sval[t] = a.v[rs + t];
            sact[t] = 1;
        }
        __syncwarp();
        double tau = 0.0;
        int nh = 0;
        if (lane == 0) {
            double norm = 0.0;
            for (int t = 0; t < nt; ++t) norm = __dadd_rn(norm, __dmul_rn(sval[t], sval[t]));
            tau = a.drop_tol * sqrt(norm);
            for (int t = 0; t < nt; ++t)
                if (scol[t] < i) heap_push(heap, nh, scol[t]);
        }
        tau = __shfl_sync(0xffffffffu, tau, 0);
        nh = __shfl_sync(0xffffffffu, nh, 0);
        while (nh > 0) {
            int k = 0;
            if (lane == 0) k = heap_pop(heap, nh);
            k = __shfl_sync(0xffffffffu, k, 0);
            nh = __shfl_sync(0xffffffffu, nh, 0);
            // slot of column k
            int sk = -1;
            for (int b0 = 0; b0 < nt && sk < 0; b0 += 32) {
                const int t = b0 + lane;
                const unsigned m = __ballot_sync(0xffffffffu, t < nt && scol[t] == k);
                if (m) sk = b0 + __ffs(m) - 1;
            }
            if (sk < 0 || !sact[sk]) continue;
            const double wk = sval[sk];
            if (fabs(wk) < tau) {
                __syncwarp();
                if (lane == 0) { sval[sk] = 0.0; sact[sk] = 0; }
                __syncwarp();
                continue;
            }
            // row k must be finished: its published word says where its U entries are.  Row i
            // usually waits for row i - 1, so this wait, and what follows it, is the chain that
            // bounds the factorisation: one load a poll (progress and errors are looked at
            // every 32nd), and the pivot comes with the first 32 entries instead of before them
            unsigned long long at = 0;
            if (lane == 0) {
                const volatile unsigned long long* d = a.done + k;
                at = *d;
                if (at == 0) {
                    int seen = *(volatile int*)a.finished;
                    long long t0 = clock64();
                    for (int poll = 1; (at = *d) == 0; ++poll) {
                        if ((poll & 31) == 0) {
                            if (*(volatile int*)a.err) break;
                            const int now = *(volatile int*)a.finished;
                            if (now != seen) {
                                seen = now;
                                t0 = clock64();
                            } else if (clock64() - t0 > kIlutWaitCycles) {
                                atomicExch(a.err, 1);
                                break;
                            }
                        }
                        __nanosleep(20);
                    }
                }
                __threadfence();
            }
            at = __shfl_sync(0xffffffffu, at, 0);
            const int us = (int)(unsigned)at, ul = (int)(at >> 32);       // (a wait that ran out: no entries)
            int j0 = -1;
            double u0 = 0.0;
            if (lane < ul) {
                j0 = __ldcg(&a.ecol[us + lane]);
                u0 = __ldcg(&a.eval[us + lane]);
            }
            const int jd = __shfl_sync(0xffffffffu, j0, 0);
            const double ud = __shfl_sync(0xffffffffu, u0, 0);
            const double ukk = jd == k ? ud : 0.0;
            if (fabs(ukk) < 2.220446049250313e-16) {
                __syncwarp();
                if (lane == 0) sact[sk] = 0;
                __syncwarp();
                continue;
            }
            const double lik = wk / ukk;
            __syncwarp();
            if (lane == 0) sval[sk] = lik;
            __syncwarp();
            for (int q0 = 0; q0 < ul; q0 += 32) {
                const int q = q0 + lane;
                int j = -1;
                double prod = 0.0;
                if (q < ul) {
                    j = q0 ? __ldcg(&a.ecol[us + q]) : j0;
                    if (j <= k) j = -1;
                    else prod = __dmul_rn(lik, q0 ? __ldcg(&a.eval[us + q]) : u0);
                }
                int slot = -1;
                if (j >= 0)
                    for (int t = 0; t < nt; ++t)
                        if (scol[t] == j) { slot = t; break; }
                const unsigned need = __ballot_sync(0xffffffffu, j >= 0 && slot < 0);
                if (j >= 0 && slot < 0) {
                    slot = nt + __popc(need & ((1u << lane) - 1u));
                    if (slot < kIlutCap) {
                        scol[slot] = j;
                        sval[slot] = 0.0;
                        sact[slot] = 0;
                    }
                }
                nt += __popc(need);
                if (nt > kIlutCap) { overflow = true; nt = kIlutCap; }
                bool push = false;
                if (j >= 0 && slot < kIlutCap) {
                    if (!sact[slot] && fabs(prod) >= tau) {
                        sact[slot] = 1;
                        push = j < i;
                    }
                    sval[slot] = __dsub_rn(sval[slot], prod);
                }
                __syncwarp();
                unsigned pm = __ballot_sync(0xffffffffu, push);
                while (pm) {
                    const int l = __ffs(pm) - 1;
                    const int jj = __shfl_sync(0xffffffffu, j, l);
                    if (lane == 0) heap_push(heap, nh, jj);
                    pm &= pm - 1;
                }
                nh = __shfl_sync(0xffffffffu, nh, 0);
                __syncwarp();
            }
        }
        // collect U and L (the warp gathers and sorts by column; lane 0 applies the fill
        // limit, a sequential heap select): U first, since later rows wait for it alone
        const int o = a.off[i];
        double diag = 0.0;
        for (int b0 = 0; b0 < nt; b0 += 32) {
            const int t = b0 + lane;
            const unsigned m = __ballot_sync(0xffffffffu, t < nt && scol[t] == i);
            if (m) {
                diag = __shfl_sync(0xffffffffu, t < nt ? sval[t] : 0.0, __ffs(m) - 1);
                break;
            }
        }
        if (fabs(diag) < 2.220446049250313e-16) diag = (diag >= 0 ? 1.0 : -1.0) * 2.220446049250313e-16 * 1e6;
        int nu = 1 + ilut_gather_sorted(scol, sval, sact, nt, i, tau, false, row + 1, lane);
        if (lane == 0) {
            row[0].col = i;
            row[0].val = diag;
            ilut_keep(row, &nu, keep);
        }
        nu = __shfl_sync(0xffffffffu, nu, 0);
        __syncwarp();
        for (int t = lane; t < nu; t += 32) {
            a.ecol[o + half + t] = row[t].col;
            a.eval[o + half + t] = row[t].val;
        }
        __threadfence();                               // every lane's entries, then the word
        __syncwarp();
        if (lane == 0) {
            *(volatile unsigned long long*)(a.done + i) = (unsigned long long)nu << 32 | (unsigned)(o + half);
            atomicAdd(a.finished, 1);
        }
        __syncwarp();                                  // row[] is reused for L
        int nl = ilut_gather_sorted(scol, sval, sact, nt, i, tau, true, row, lane);
        if (lane == 0) ilut_keep(row, &nl, keep);
        nl = __shfl_sync(0xffffffffu, nl, 0);
        __syncwarp();
        for (int t = lane; t < nl; t += 32) {
            a.ecol[o + t] = row[t].col;
            a.eval[o + t] = row[t].val;
        }
        if (lane == 0) {
            a.lcnt[i] = nl;
            a.ucnt[i] = nu;
            if (overflow) atomicExch(a.err, 2);
        }
        __syncwarp();
    }
}

// Capacity per row (2 * (row length + fill_p)): L in the first half, U in the second.
__global__ void k_ilut_caps(int n, const int* __restrict__ rp, int fill_p, int* cap) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int keep = rp[i + 1] - rp[i] + fill_p;
        cap[i] = 2 * (keep > 1 ? keep : 1);
    }
}

__global__ void k_ilut_counts(int n, const int* __restrict__ lcnt, const int* __restrict__ ucnt, int* cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        cnt[i] = lcnt[i] + ucnt[i];
}

// Compact the capacity layout into the L\U CSR (row: L entries, then U entries).
__global__ void k_ilut_compact(int n, const int* __restrict__ rp, int fill_p, const int* __restrict__ off,
                               const int* __restrict__ lcnt, const int* __restrict__ ucnt,
                               const int* __restrict__ ecol, const double* __restrict__ eval,
                               const int* __restrict__ frp, int* fci, double* flu) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int keep = rp[i + 1] - rp[i] + fill_p;
        const int half = keep > 1 ? keep : 1;
        int o = frp[i];
        for (int t = 0; t < lcnt[i]; ++t, ++o) { fci[o] = ecol[off[i] + t]; flu[o] = eval[off[i] + t]; }
        for (int t = 0; t < ucnt[i]; ++t, ++o) { fci[o] = ecol[off[i] + half + t]; flu[o] = eval[off[i] + half + t]; }
    }
}

template <typename K>
int coop_blocks(Ctx& ctx, K kernel, int threads) {
    int per = occupancy_blocks(kernel, threads);
    return std::max(1, std::min(per, 4) * ctx.sm_count);
}

template <typename K, typename... Args>
void coop_launch(cudaStream_t s, K kernel, int blocks, int threads, Args... args) {
    void* ptrs[] = {(void*)&args...};
    HAMLSS_CUDA(cudaLaunchCooperativeKernel((const void*)kernel, dim3(blocks), dim3(threads), ptrs, 0, s));
}

}  // namespace

// ---------------------------------------------------------------------- the object
// (the kernel of a triangle's sweep: tri_mode, rules.hpp)
struct Triangle {
    int nlev = 0, nnz = 0, max_row = 0, max_width = 0;
    TriMode mode = TriMode::GRID;
    DBuf<int> ord, lptr, level;
    DBuf<int> code, code32, sptr;        // RING: entry codes, step bounds (ilu_sweep.cuh)
    int nsteps = 0, step_rows = 0;
    bool far = false;                    // RING: entries beyond the ring
    DBuf<int> rp, ci;                    // the other modes: row bounds and columns
    DBuf<double> v, dg;                  // in position order (RING: [row][place], with reciprocals)
    DBuf<float> v32, dg32;
};

// (values, diagonals, codes) of a triangle by value type
inline std::tuple<DBuf<double>&, DBuf<double>&, DBuf<int>&> tri_bufs(Triangle& t, double) { return {t.v, t.dg, t.code}; }
inline std::tuple<DBuf<float>&, DBuf<float>&, DBuf<int>&> tri_bufs(Triangle& t, float) { return {t.v32, t.dg32, t.code32}; }

// Calls f(std::integral_constant<int, K>) with the entry places a RING triangle's rows get.
template <typename F>
void with_places(const Triangle& t, F&& f) {
    switch (tri_places(t.max_row)) {
        case 2: return f(std::integral_constant<int, 2>{});
        case 4: return f(std::integral_constant<int, 4>{});
        case 8: return f(std::integral_constant<int, 8>{});
        default: return f(std::integral_constant<int, 16>{});
    }
}

template <typename T, int K, TriOp OP>
void launch_tri(Ctx& ctx, const Lane& ln, bool far, int rows, const TriView<T>& F, const T* rhs, T* out,
                const int* gate) {
    using S = TriShape<T, K, OP>;
    static DeviceOnce raised;
    raised(ctx.device, [] {
        for (auto f : {k_tri_sweep<T, K, OP, true>, k_tri_sweep<T, K, OP, false>})
            HAMLSS_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem_bytes));
    });
    auto kern = far ? k_tri_sweep<T, K, OP, true> : k_tri_sweep<T, K, OP, false>;
    kern<<<1, rows + 32, S::smem_bytes, ln.stream>>>(F, rhs, out, gate, ln.err.p);
}

struct IluPrec : Prec {
    hamlss_mat* A = nullptr;
    // pattern of the factor: A's for ILU(0); the factor's own (frp, fci) for ILUT
    const int* prp = nullptr;
    const int* pci = nullptr;
    int pnnz = 0;
    DBuf<int> frp, fci;
    DBuf<int> dpos;
    DBuf<double> lu;
    Triangle L, U;
    DBuf<int> u_from_l;          // position in L of the row at each position of U (both RING)
    DBuf<double> y, s1, s2;      // y between the sweeps in row order; vectors in position order
    DBuf<float> y32, s132, s232;
    int bad_diag_row = -1;       // backward_sub would throw on this row
    bool f32_ready = false;

    void check_apply() const {
        if (bad_diag_row >= 0)
            fail(HAMLSS_ERR_ZERO_PIVOT,
                 "ILU backward sub: near-zero U diagonal at row " + std::to_string(bad_diag_row));
    }

    template <typename T, bool GATHER>
    void permute(Ctx& ctx, const Lane& ln, const int* idx, const T* in, T* out, const int* gate) {
        k_permute<T, GATHER><<<std::max(1, std::min(ceil_div(n, 256), ctx.sm_count * 8)), 256, 0, ln.stream>>>(
            n, idx, in, out, gate);
        HAMLSS_LAUNCH_CHECK();
    }

    // a RING triangle's rows; `pos`: position of each row; `bad`: see k_fill_U
    template <typename T, bool DIV>
    void pack(Ctx& ctx, Triangle& t, const int* pos, int* far, int* bad) {
        constexpr TriOp op = DIV ? TriOp::BACKWARD : TriOp::FORWARD;
        with_places(t, [&](auto k) {
            constexpr int K = decltype(k)::value;
            constexpr int RB = TriShape<T, K, op>::RB;
            const int rows = ceil_div(n, RB) * RB;
            auto [tv, tdg, tcode] = tri_bufs(t, T(0));
            tv.ensure((size_t)rows * K);
            tcode.ensure((size_t)rows * K);
            if (DIV) tdg.ensure((size_t)rows * 2);
            k_tri_pack<T, K, op><<<std::min(ceil_div(rows, 256), ctx.sm_count * 8), 256, 0, ctx.lane.stream>>>(
                n, t.ord.p, t.level.p, t.lptr.p, pos, prp, pci, lu.p, tv.p, tcode.p, tdg.p, far, bad);
        });
        HAMLSS_LAUNCH_CHECK();
    }

    // a RING triangle's steps, which fit the kernels of both value types
    template <bool DIV>
    void make_steps(Ctx& ctx, Triangle& t) {
        constexpr TriOp op = DIV ? TriOp::BACKWARD : TriOp::FORWARD;
        with_places(t, [&](auto k) {
            constexpr int K = decltype(k)::value;
            t.step_rows = std::min(TriShape<double, K, op>::max_rows, TriShape<float, K, op>::max_rows);
        });
        t.step_rows = std::max(32, std::min((t.max_width + 31) / 32 * 32, t.step_rows));
        cudaStream_t s = ctx.lane.stream;
        const int g = std::max(1, std::min(ceil_div(t.nlev + 1, 256), ctx.sm_count * 8));
        DBuf<int> first(t.nlev + 1);
        HAMLSS_CUDA(cudaMemsetAsync(first.p + t.nlev, 0, sizeof(int), s));
        k_step_count<<<g, 256, 0, s>>>(t.nlev, t.lptr.p, t.step_rows, first.p);
        HAMLSS_LAUNCH_CHECK();
        t.nsteps = (int)exclusive_scan(ctx, first.p, t.nlev + 1);
        t.sptr.ensure(t.nsteps + 1);
        k_step_fill<<<g, 256, 0, s>>>(t.nlev, t.lptr.p, t.step_rows, first.p, t.sptr.p);
        HAMLSS_LAUNCH_CHECK();
    }

    // rhs -> out: in position order for RING, in row order for the others
    template <typename T, bool DIV>
    void sweep(Ctx& ctx, const Lane& ln, Triangle& t, const T* rhs, T* out, const int* gate) {
        auto [tv, tdg, tcode] = tri_bufs(t, T(0));
        if (t.mode == TriMode::RING) {
            constexpr TriOp op = DIV ? TriOp::BACKWARD : TriOp::FORWARD;
            const TriView<T> F{n, t.nsteps, t.sptr.p, tv.p, tcode.p, tdg.p, nullptr, nullptr, nullptr};
            with_places(t, [&](auto k) {
                constexpr int K = decltype(k)::value;
                launch_tri<T, K, op>(ctx, ln, t.far, t.step_rows, F, rhs, out, gate);
            });
            HAMLSS_LAUNCH_CHECK();
            return;
        }
        const TriRows<T> F = rows_of<T>(t);
        if (t.mode == TriMode::BLOCK) {
            k_tri_block<T, DIV, 1024><<<1, 1024, 0, ln.stream>>>(F, rhs, out, gate);
            HAMLSS_LAUNCH_CHECK();
        } else if (DIV) {
            grid_launch<T>(ctx, ln, TriRows<T>{}, F, nullptr, const_cast<T*>(rhs), out, gate);
        } else {
            grid_launch<T>(ctx, ln, F, TriRows<T>{}, rhs, out, nullptr, gate);
        }
    }

    template <typename T>
    TriRows<T> rows_of(Triangle& t) const {
        auto [tv, tdg, tcode] = tri_bufs(t, T(0));
        return TriRows<T>{n, t.nlev, t.ord.p, t.lptr.p, t.rp.p, t.ci.p, tv.p, tdg.p};
    }
    template <typename T>
    void grid_launch(Ctx& ctx, const Lane& ln, TriRows<T> FL, TriRows<T> FU, const T* rhs, T* y, T* z, const int* gate) {
        static const int blocks = coop_blocks(ctx, k_tri_grid<T>, 256);
        coop_launch(ln.stream, k_tri_grid<T>, blocks, 256, FL, FU, rhs, y, z, gate);
    }

    template <typename T>
    void run(Ctx& ctx, const Lane& ln, const T* r, T* yb, T* a, T* c, T* z, const int* gate) {
        check_apply();
        if (!n) return;
        ProfScope ps(ln, "ilu_sweep", (double)sizeof(T) * (L.nnz + U.nnz + 4.0 * n) + 4.0 * (L.nnz + U.nnz + 4.0 * n));
        const bool lring = L.mode == TriMode::RING, uring = U.mode == TriMode::RING;
        if (L.mode == TriMode::GRID && U.mode == TriMode::GRID)
            return grid_launch<T>(ctx, ln, rows_of<T>(L), rows_of<T>(U), r, yb, z, gate);
        if (lring) {
            permute<T, true>(ctx, ln, L.ord.p, r, a, gate);
            sweep<T, false>(ctx, ln, L, a, c, gate);
            if (!uring) permute<T, false>(ctx, ln, L.ord.p, c, yb, gate);
        } else {
            sweep<T, false>(ctx, ln, L, r, yb, gate);
        }
        if (uring) {
            permute<T, true>(ctx, ln, lring ? u_from_l.p : U.ord.p, lring ? c : yb, a, gate);
            sweep<T, true>(ctx, ln, U, a, c, gate);
            permute<T, false>(ctx, ln, U.ord.p, c, z, gate);
        } else {
            sweep<T, true>(ctx, ln, U, yb, z, gate);
        }
    }

    void apply(Ctx& ctx, const Lane& ln, const double* r, double* z, const int* gate) override {
        run<double>(ctx, ln, r, y.p, s1.p, s2.p, z, gate);
    }
    void prepare32(Ctx& ctx) override {
        if (f32_ready) return;
        cudaStream_t s = ctx.lane.stream;
        if (n) {
            const int g = std::max(1, std::min(ceil_div(n, 256), ctx.sm_count * 8));
            for (Triangle* t : {&L, &U}) {
                if (t->mode == TriMode::RING) {
                    DBuf<int> pos(n), far(1);          // (t->far is known)
                    k_invert<<<g, 256, 0, s>>>(n, t->ord.p, pos.p);
                    if (t == &L) pack<float, false>(ctx, L, pos.p, far.p, nullptr);
                    else pack<float, true>(ctx, U, pos.p, far.p, nullptr);
                    continue;
                }
                t->v32.ensure(std::max(t->nnz, 1));
                if (t->nnz) k_to_float<<<std::min(ceil_div(t->nnz, 256), ctx.sm_count * 8), 256, 0, s>>>(t->nnz, t->v.p, t->v32.p);
                if (t == &U) {
                    t->dg32.ensure(n);
                    k_to_float<<<g, 256, 0, s>>>(n, t->dg.p, t->dg32.p);
                }
                HAMLSS_LAUNCH_CHECK();
            }
        }
        y32.ensure(std::max(n, 1));
        s132.ensure(std::max(n, 1));
        s232.ensure(std::max(n, 1));
        f32_ready = true;
    }
    void apply32(Ctx& ctx, const Lane& ln, const float* r, float* z, const int* gate) override {
        prepare32(ctx);
        run<float>(ctx, ln, r, y32.p, s132.p, s232.p, z, gate);
    }
    bool has32() const override { return true; }
};

namespace {
void finish_ilu(Ctx& ctx, IluPrec* P, bool factorise);
}  // namespace

std::unique_ptr<Prec> make_ilu0(Ctx& ctx, hamlss_mat* A) {
    auto P = std::make_unique<IluPrec>();
    P->kind = HAMLSS_PREC_ILU;
    P->A = A;
    const int n = A->A.n;
    const int nnz = A->A.nnz;
    P->n = n;
    if (A->A.n != A->A.m) fail(HAMLSS_ERR_SIZE, "ILU needs a square matrix");
    cudaStream_t s = ctx.lane.stream;
    AllocScope scope(s);                 // setup buffers from the stream-ordered pool
    P->prp = A->A.rp.p;
    P->pci = A->A.ci.p;
    P->pnnz = nnz;
    P->lu.ensure(nnz);
    if (nnz) HAMLSS_CUDA(cudaMemcpyAsync(P->lu.p, A->A.v.p, sizeof(double) * nnz, cudaMemcpyDeviceToDevice, s));
    finish_ilu(ctx, P.get(), true);
    return P;
}

std::unique_ptr<Prec> make_ilut(Ctx& ctx, hamlss_mat* A, double drop_tol, int fill_p) {
    auto P = std::make_unique<IluPrec>();
    P->kind = HAMLSS_PREC_ILU;
    P->A = A;
    const int n = A->A.n;
    P->n = n;
    if (A->A.n != A->A.m) fail(HAMLSS_ERR_SIZE, "ILU needs a square matrix");
    if (fill_p < 0) fail(HAMLSS_ERR_INVALID, "ILUT: fill_per_row must be >= 0");
    cudaStream_t s = ctx.lane.stream;
    AllocScope scope(s);
    const int g = std::max(1, std::min(ceil_div(n, 256), ctx.sm_count * 8));
    // capacity layout: row i owns 2 * max(row length + fill_p, 1) slots
    DBuf<int> off(n + 1), lcnt(std::max(n, 1)), ucnt(std::max(n, 1)), flags(3);
    DBuf<unsigned long long> done(std::max(n, 1));
    HAMLSS_CUDA(cudaMemsetAsync(off.p + n, 0, sizeof(int), s));
    if (n) k_ilut_caps<<<g, 256, 0, s>>>(n, A->A.rp.p, fill_p, off.p);
    HAMLSS_LAUNCH_CHECK();
    const long long total = exclusive_scan(ctx, off.p, n + 1);
    if (total > INT_MAX) fail(HAMLSS_ERR_NOMEM, "ILUT: factor capacity exceeds 2^31 entries");
    DBuf<int> ecol(std::max<long long>(total, 1));
    DBuf<double> eval(std::max<long long>(total, 1));
    lcnt.zero(s);
    ucnt.zero(s);
    done.zero(s);
    flags.zero(s);
    if (n) {
        static DeviceOnce raised;
        raised(ctx.device, [] {
            HAMLSS_CUDA(cudaFuncSetAttribute(k_ilut_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)(kIlutWarpBytes * kIlutWarps)));
        });
        const size_t smem = kIlutWarpBytes * kIlutWarps;
        int per = 0;
        HAMLSS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_ilut_rows, 32 * kIlutWarps, smem));
        const int blocks = std::max(1, std::min(std::max(per, 1) * ctx.sm_count, ceil_div(n, kIlutWarps)));
        IlutArgs a;
        a.n = n;
        a.fill_p = fill_p;
        a.drop_tol = drop_tol;
        a.rp = A->A.rp.p;
        a.ci = A->A.ci.p;
        a.v = A->A.v.p;
        a.off = off.p;
        a.ecol = ecol.p;
        a.eval = eval.p;
        a.lcnt = lcnt.p;
        a.ucnt = ucnt.p;
        a.done = done.p;
        a.ticket = flags.p;
        a.err = flags.p + 1;
        a.finished = flags.p + 2;
        void* args[] = {&a};
        HAMLSS_CUDA(cudaLaunchCooperativeKernel((const void*)k_ilut_rows, dim3(blocks), dim3(32 * kIlutWarps),
                                                args, smem, s));
        int h[2] = {0, 0};
        flags.download(h, 2, s);
        HAMLSS_CUDA(cudaStreamSynchronize(s));
        if (h[1] == 1) fail(HAMLSS_ERR_TIMEOUT, "ILUT: a bounded wait for an earlier row ran out");
        if (h[1] == 2) fail(HAMLSS_ERR_NOMEM, "ILUT: a work row touched more than 512 columns");
    }
    // compact into the L\U CSR
    P->frp.ensure(n + 1);
    HAMLSS_CUDA(cudaMemsetAsync(P->frp.p + n, 0, sizeof(int), s));
    if (n) k_ilut_counts<<<g, 256, 0, s>>>(n, lcnt.p, ucnt.p, P->frp.p);
    HAMLSS_LAUNCH_CHECK();
    const long long fnnz = exclusive_scan(ctx, P->frp.p, n + 1);
    P->fci.ensure(std::max<long long>(fnnz, 1));
    P->lu.ensure(std::max<long long>(fnnz, 1));
    if (n)
        k_ilut_compact<<<g, 256, 0, s>>>(n, A->A.rp.p, fill_p, off.p, lcnt.p, ucnt.p, ecol.p, eval.p,
                                          P->frp.p, P->fci.p, P->lu.p);
    HAMLSS_LAUNCH_CHECK();
    P->prp = P->frp.p;
    P->pci = P->fci.p;
    P->pnnz = (int)fnnz;
    finish_ilu(ctx, P.get(), false);
    return P;
}

std::unique_ptr<Prec> make_ilu(Ctx& ctx, hamlss_mat* A, const hamlss_params& p) {
    if (p.drop_tol > 0.0 || p.fill_per_row > 0) return make_ilut(ctx, A, p.drop_tol, p.fill_per_row);
    return make_ilu0(ctx, A);
}

namespace {
// ILU(0) by the triangular sweep's kernel, where every elimination touches only the row's
// diagonal: 0.58 us a level on the 512^2 grid, against 2.2 (k_ilu_factor_ops).  false: another pattern.
template <int K>
bool factor_by_sweep_k(Ctx& ctx, IluPrec* P, const int* pos, int* status) {
    const int n = P->n;
    cudaStream_t s = ctx.lane.stream;
    constexpr int RB = TriShape<double, K, TriOp::FACTOR>::RB;
    if (P->L.step_rows > TriShape<double, K, TriOp::FACTOR>::max_rows) return false;
    const size_t rows = (size_t)ceil_div(n, RB) * RB;
    const int g = std::max(1, std::min(ceil_div((long long)rows, 256), ctx.sm_count * 8));
    DBuf<double> val(rows * K), up(rows * K), low(rows * K), diag(rows), d(rows);
    DBuf<int> code(rows * K), flags(2);                       // entries beyond the ring, another pattern
    flags.zero(s);
    k_factor_pack<K><<<g, 256, 0, s>>>(n, P->L.ord.p, P->L.level.p, P->L.lptr.p, pos, P->prp, P->pci, P->dpos.p,
                                       P->lu.p, val.p, code.p, up.p, diag.p, flags.p, flags.p + 1);
    HAMLSS_LAUNCH_CHECK();
    int h[2];
    flags.download(h, 2, s);
    HAMLSS_CUDA(cudaStreamSynchronize(s));
    if (h[1]) return false;
    const TriView<double> F{n, P->L.nsteps, P->L.sptr.p, val.p, code.p, up.p, low.p, P->L.ord.p, status};
    launch_tri<double, K, TriOp::FACTOR>(ctx, ctx.lane, h[0] != 0, P->L.step_rows, F, diag.p, d.p, nullptr);
    k_factor_unpack<K><<<g, 256, 0, s>>>(n, P->L.ord.p, P->prp, P->pci, P->dpos.p, low.p, d.p, P->lu.p);
    HAMLSS_LAUNCH_CHECK();
    return true;
}

bool factor_by_sweep(Ctx& ctx, IluPrec* P, const int* pos, int* status) {
    return P->L.max_row <= 2 ? factor_by_sweep_k<2>(ctx, P, pos, status) : factor_by_sweep_k<4>(ctx, P, pos, status);
}

// Pattern information, level sets, (for ILU(0)) the factorisation, and the level-ordered
// L / U copies of an ILU preconditioner whose pattern (prp, pci, pnnz) and values (lu)
// are set.
void finish_ilu(Ctx& ctx, IluPrec* P, bool factorise) {
    const int n = P->n;
    const int nnz = P->pnnz;
    cudaStream_t s = ctx.lane.stream;
    const int g = std::max(1, std::min(ceil_div(n, 256), ctx.sm_count * 8));
    const int* rp = P->prp;
    const int* ci = P->pci;
    if (n == 0) return;
    P->y.ensure(n); P->s1.ensure(n); P->s2.ensure(n);
    Triangle* tri[2] = {&P->L, &P->U};
    DBuf<int> lcnt(n), ucnt(n);
    // longest rows (L, U, whole), level counts (2), entries (2), widest levels (2),
    // entries beyond the ring (2)
    DBuf<int> facts(11);
    facts.zero(s);
    P->dpos.ensure(n);
    k_row_info<<<g, 256, 0, s>>>(n, rp, ci, P->dpos.p, lcnt.p, ucnt.p);
    k_max_counts<<<g, 256, 0, s>>>(n, lcnt.p, ucnt.p, rp, facts.p);
    HAMLSS_LAUNCH_CHECK();
    // level sets
    P->L.level.ensure(n);
    P->U.level.ensure(n);
    {
        static DeviceOnce raised;
        raised(ctx.device, [] {
            HAMLSS_CUDA(cudaFuncSetAttribute(k_levels_chain, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            kChainRing * (int)sizeof(int)));
        });
        k_levels_chain<<<2, kChainRows, kChainRing * sizeof(int), s>>>(n, rp, ci, P->L.level.p, P->U.level.p,
                                                                      facts.p + 3);
        HAMLSS_LAUNCH_CHECK();
    }
    int hf[7];
    facts.download(hf, 7, s);
    HAMLSS_CUDA(cudaStreamSynchronize(s));
    const int max_row = hf[2];
    P->L.max_row = hf[0];
    P->U.max_row = hf[1];
    if (hf[3] < 0 || hf[4] < 0) {
        DBuf<int> dpos;
        pattern_levels(ctx, n, nnz, rp, ci, dpos, P->L.level, P->U.level, &hf[3], &hf[4]);
    }
    P->L.nlev = hf[3];
    P->U.nlev = hf[4];
    // rows grouped by level, in index order inside a level
    DBuf<int> pos[2];
    for (int k = 0; k < 2; ++k) {
        Triangle& t = *tri[k];
        t.lptr.ensure(t.nlev + 1);
        HAMLSS_CUDA(cudaMemsetAsync(t.lptr.p, 0, sizeof(int) * (t.nlev + 1), s));
        k_level_hist<<<g, 256, 0, s>>>(n, t.level.p, t.lptr.p);
        HAMLSS_LAUNCH_CHECK();
        scan_in_place(ctx, t.lptr.p, t.nlev + 1);
        DBuf<int> fill(t.nlev + 1);
        HAMLSS_CUDA(cudaMemcpyAsync(fill.p, t.lptr.p, sizeof(int) * (t.nlev + 1), cudaMemcpyDeviceToDevice, s));
        t.ord.ensure(n);
        pos[k].ensure(n);
        k_level_place<<<g, 256, 0, s>>>(n, t.level.p, fill.p, t.ord.p);
        k_level_sort<<<std::min(t.nlev, ctx.sm_count * 8), 256, 0, s>>>(t.nlev, t.lptr.p, t.ord.p, facts.p + 7 + k);
        k_invert<<<g, 256, 0, s>>>(n, t.ord.p, pos[k].p);
        HAMLSS_LAUNCH_CHECK();
        t.mode = tri_mode(n, t.nlev, hf[5 + k], t.max_row);
    }
    if (P->L.mode == TriMode::RING || P->U.mode == TriMode::RING) {
        int hw[2];
        HAMLSS_CUDA(cudaMemcpyAsync(hw, facts.p + 7, sizeof(hw), cudaMemcpyDeviceToHost, s));
        HAMLSS_CUDA(cudaStreamSynchronize(s));
        P->L.max_width = hw[0];
        P->U.max_width = hw[1];
    }
    if (P->L.mode == TriMode::RING) P->make_steps<false>(ctx, P->L);
    if (P->U.mode == TriMode::RING) P->make_steps<true>(ctx, P->U);
    // factorisation (ILU(0); ILUT arrives factored)
    if (factorise) {
        DBuf<int> status(1);
        int init = 0x7fffffff;
        status.upload(&init, 1, s);
        if (P->L.mode == TriMode::GRID) {
            int fb = coop_blocks(ctx, k_ilu_factor_grid, 256);
            coop_launch(s, k_ilu_factor_grid, fb, 256, P->L.nlev, (const int*)P->L.ord.p,
                        (const int*)P->L.lptr.p, rp, ci, (const int*)P->dpos.p, P->lu.p, status.p);
        } else if (P->L.mode == TriMode::RING && P->L.max_row <= 4 && factor_by_sweep(ctx, P, pos[0].p, status.p)) {
            // (done)
        } else if (max_row <= kOpsRow) {
            DBuf<int> optr(n + 1);
            HAMLSS_CUDA(cudaMemsetAsync(optr.p + n, 0, sizeof(int), s));
            k_ilu_ops<false><<<g, 256, 0, s>>>(n, P->L.ord.p, rp, ci, P->dpos.p, optr.p, nullptr, nullptr);
            HAMLSS_LAUNCH_CHECK();
            const long long total = exclusive_scan(ctx, optr.p, n + 1);
            if (total > INT_MAX) fail(HAMLSS_ERR_NOMEM, "ILU(0): elimination list exceeds 2^31 operations");
            DBuf<int2> ops(std::max<long long>(total, 1));
            DBuf<int4> info(n);
            k_ilu_ops<true><<<g, 256, 0, s>>>(n, P->L.ord.p, rp, ci, P->dpos.p, optr.p, ops.p, info.p);
            k_ilu_factor_ops<<<1, kOpsThreads, kOpsSmem, s>>>(P->L.nlev, P->L.lptr.p, info.p, ci, ops.p, P->lu.p,
                                                             status.p);
            HAMLSS_LAUNCH_CHECK();
        } else {
            k_ilu_factor_block<<<1, 1024, 0, s>>>(P->L.nlev, P->L.ord.p, P->L.lptr.p, rp, ci, P->dpos.p,
                                                 P->lu.p, status.p);
            HAMLSS_LAUNCH_CHECK();
        }
        int h = 0;
        status.download(&h, 1, s);
        HAMLSS_CUDA(cudaStreamSynchronize(s));
        if (lane_take_timeout(ctx.lane))
            fail(HAMLSS_ERR_TIMEOUT, "ILU(0): the elimination gave up waiting for its bulk copies");
        if (h != 0x7fffffff)
            fail(HAMLSS_ERR_ZERO_PIVOT, "ILU(0): near-zero pivot at row " + std::to_string(h));
    }
    // level-ordered factor copies
    DBuf<int> bad(1);
    int init = 0x7fffffff;
    bad.upload(&init, 1, s);
    for (int k = 0; k < 2; ++k) {
        Triangle& t = *tri[k];
        t.nnz = hf[5 + k];
        if (t.mode == TriMode::RING) {
            if (k == 0) P->pack<double, false>(ctx, t, pos[0].p, facts.p + 9, nullptr);
            else P->pack<double, true>(ctx, t, pos[1].p, facts.p + 10, bad.p);
            continue;
        }
        t.rp.ensure(n + 1);
        HAMLSS_CUDA(cudaMemsetAsync(t.rp.p + n, 0, sizeof(int), s));
        k_perm_counts<<<g, 256, 0, s>>>(n, t.ord.p, k == 0 ? lcnt.p : ucnt.p, t.rp.p);
        HAMLSS_LAUNCH_CHECK();
        scan_in_place(ctx, t.rp.p, n + 1);
        t.ci.ensure(std::max(t.nnz, 1));
        t.v.ensure(std::max(t.nnz, 1));
        if (k == 0) {
            k_fill_L<<<g, 256, 0, s>>>(n, t.ord.p, rp, ci, P->lu.p, t.rp.p, t.ci.p, t.v.p);
        } else {
            t.dg.ensure(n);
            k_fill_U<<<g, 256, 0, s>>>(n, t.ord.p, rp, ci, P->lu.p, t.rp.p, t.ci.p, t.v.p, t.dg.p, bad.p);
        }
        HAMLSS_LAUNCH_CHECK();
    }
    if (P->L.mode == TriMode::RING && P->U.mode == TriMode::RING) {
        P->u_from_l.ensure(n);
        k_compose<<<g, 256, 0, s>>>(n, P->U.ord.p, pos[0].p, P->u_from_l.p);
        HAMLSS_LAUNCH_CHECK();
    }
    int hb = 0, hfar[2];
    bad.download(&hb, 1, s);
    HAMLSS_CUDA(cudaMemcpyAsync(hfar, facts.p + 9, sizeof(hfar), cudaMemcpyDeviceToHost, s));
    HAMLSS_CUDA(cudaStreamSynchronize(s));
    P->bad_diag_row = hb != 0x7fffffff ? hb : -1;
    P->L.far = hfar[0] != 0;
    P->U.far = hfar[1] != 0;
}
}  // namespace

// Level sets of the strictly lower and strictly upper dependency DAGs of a square CSR
// pattern (the definitions make_ilu0 uses), without factorising.  The batched solver
// calls this on its block-diagonal matrix: blocks never depend on one another, so every
// row's level is its level inside its own system.
void pattern_levels(Ctx& ctx, int n, int nnz, const int* rp, const int* ci, DBuf<int>& dpos,
                    DBuf<int>& levelL, DBuf<int>& levelU, int* nlevL, int* nlevU) {
    cudaStream_t s = ctx.lane.stream;
    dpos.ensure(std::max(n, 1));
    levelL.ensure(std::max(n, 1));
    levelU.ensure(std::max(n, 1));
    *nlevL = *nlevU = 0;
    if (n == 0) return;
    const int g = std::max(1, std::min(ceil_div(n, 256), ctx.sm_count * 8));
    DBuf<int> lcnt(n), ucnt(n), trp(n + 1), trow(std::max(nnz, 1)), fill(n), indeg(n), cnt(n + 2),
        order(n), lptr(n + 1), nl(2);
    k_row_info<<<g, 256, 0, s>>>(n, rp, ci, dpos.p, lcnt.p, ucnt.p);
    HAMLSS_CUDA(cudaMemsetAsync(trp.p, 0, sizeof(int) * (n + 1), s));
    k_col_count<<<g, 256, 0, s>>>(n, rp, ci, trp.p);
    HAMLSS_LAUNCH_CHECK();
    scan_in_place(ctx, trp.p, n + 1);
    HAMLSS_CUDA(cudaMemcpyAsync(fill.p, trp.p, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
    k_col_fill<<<g, 256, 0, s>>>(n, rp, ci, fill.p, trow.p);
    HAMLSS_LAUNCH_CHECK();
    const int lb = coop_blocks(ctx, k_levels<true>, 256);
    HAMLSS_CUDA(cudaMemcpyAsync(indeg.p, lcnt.p, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
    HAMLSS_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(int) * (n + 2), s));
    coop_launch(s, k_levels<true>, lb, 256, n, (const int*)trp.p, (const int*)trow.p, indeg.p,
                order.p, lptr.p, cnt.p, levelL.p, nl.p);
    HAMLSS_CUDA(cudaMemcpyAsync(indeg.p, ucnt.p, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
    HAMLSS_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(int) * (n + 2), s));
    coop_launch(s, k_levels<false>, lb, 256, n, (const int*)trp.p, (const int*)trow.p, indeg.p,
                order.p, lptr.p, cnt.p, levelU.p, nl.p + 1);
    int h[2];
    HAMLSS_CUDA(cudaMemcpyAsync(h, nl.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    HAMLSS_CUDA(cudaStreamSynchronize(s));
    *nlevL = h[0];
    *nlevU = h[1];
}

// Inspection entry points (hamlss.h).
int ilu_copy_factors(const Prec* M, double* out, cudaStream_t s) {
    auto* P = dynamic_cast<const IluPrec*>(M);
    if (!P) return HAMLSS_ERR_INVALID;
    if (P->pnnz) P->lu.download(out, P->pnnz, s);
    HAMLSS_CUDA(cudaStreamSynchronize(s));
    return HAMLSS_OK;
}

int ilu_factor_csr(const Prec* M, int* nnz, int* rp, int* ci, double* v, cudaStream_t s) {
    auto* P = dynamic_cast<const IluPrec*>(M);
    if (!P) return HAMLSS_ERR_INVALID;
    *nnz = P->pnnz;
    if (rp) HAMLSS_CUDA(cudaMemcpyAsync(rp, P->prp, sizeof(int) * (P->n + 1), cudaMemcpyDeviceToHost, s));
    if (ci && P->pnnz) HAMLSS_CUDA(cudaMemcpyAsync(ci, P->pci, sizeof(int) * P->pnnz, cudaMemcpyDeviceToHost, s));
    if (v && P->pnnz) P->lu.download(v, P->pnnz, s);
    HAMLSS_CUDA(cudaStreamSynchronize(s));
    return HAMLSS_OK;
}

int ilu_copy_levels(const Prec* M, int which, int* level, int* nlev, cudaStream_t s) {
    auto* P = dynamic_cast<const IluPrec*>(M);
    if (!P) return HAMLSS_ERR_INVALID;
    if (P->n) (which == 0 ? P->L : P->U).level.download(level, P->n, s);
    HAMLSS_CUDA(cudaStreamSynchronize(s));
    *nlev = which == 0 ? P->L.nlev : P->U.nlev;
    return HAMLSS_OK;
}

}  // namespace hamlss
