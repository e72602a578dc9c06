// ilu_sweep.cuh -- triangular sweeps of the ILU preconditioners by one thread block whose
// working set stays in shared memory.
//
// What bounds a level-scheduled sweep with narrow levels (the 5-point grids have at most
// n_side rows a level and 2 n_side levels) is the latency of one level: a barrier plus the
// loads of the values solved for one level earlier.  Through L1/L2 that was ~1.1 us a level
// (2.28 ms per apply of ILU(0) on a 512^2 grid, 1,023 levels a sweep).  Here
//   - rows are stored level by level ("positions"), and the solution of the last kTriRing
//     positions is kept in a shared-memory ring, so a level reads its operands with
//     shared-memory loads; an entry's ring slot is worked out at setup (code >= 0), and an
//     entry further back than the ring reads the solution in global memory (code = ~position);
//   - rows have K entry places (K = 2, 4, 8 or 16), kept together a row, so a row is a few
//     wide shared-memory loads at fixed strides; an unused place has value 0 and reads a ring
//     slot that holds 0 (s - 0 * 0 leaves every s as it is).  A step is bound by the
//     instructions a warp issues one after another (~8 cycles each): with row pointers it took
//     ~180, 1.0 us a level at 512 rows, with a ring of whole blocks and checks inside ~100,
//     0.37 us;
//   - a producer warp keeps a ring of such blocks, and of the right-hand side, filled by bulk
//     copies (cp.async.bulk) several levels ahead, each block completing on its own mbarrier,
//     which the row threads wait for only when a step enters a new block; step bounds come
//     from a table made at setup, so neither side computes anything between barriers (a
//     producer that worked each step out kept a level at 0.25 us);
//   - a thread moves its row of the next step into registers before the barrier, so behind
//     the barrier there are only the ring loads and the row's arithmetic.
// Measured on a 512^2 grid (1,023 levels, 256 rows on average): 275 us forward and 377 us
// backward in FP64 (2.28 ms together through L1/L2); 256^2 in FP32 75 and 93 us (580 us);
// an ILUT factor with 720 levels of 45 rows 153 us (2.0 ms with a grid barrier a level);
// the ILU(0) elimination of the 512^2 grid 590 us (2.28 ms from the operation list).
// The right-hand side is gathered into position order, and the solution scattered back, by
// small full-grid kernels beside the sweep (k_permute).  Every row subtracts its products in
// column order with separate multiply and subtract, so the results are those of the plain
// loop bit for bit (ilu.cpp:230-237, :249-260).
//
// A level of more rows than threads takes several steps.  A block is refilled once all its
// rows lie before the current step (the step's barrier tells the producer).  Waits on the
// copies are bounded (~1 s): a thread whose wait ran out sets the lane's error word and only
// keeps to the barriers from then on; the producer issues no more copies and lets those in
// flight land, and the host reports HAMLSS_ERR_TIMEOUT from the call (setup, apply or solve).
#pragma once

#include <climits>

#include "engine.cuh"
#include "exact_div.hpp"

namespace hamlss {

constexpr int kTriRing = 4096;            // solution values kept (positions); slot kTriRing holds 0
constexpr int kTriSteps = 512;            // step bounds kept in shared memory at a time (even)

// What a step does with a row: FORWARD s = rhs - sum v y, BACKWARD the same divided by the
// diagonal, FACTOR the ILU(0) elimination of a row whose lower entries each update only its
// diagonal (five-point grids): l_k = v_k / d_k, d = a_ii - sum l_k u_k, with d_k the earlier
// rows' diagonals (the ring) and u_k the matrix's own upper entries.
enum class TriOp { FORWARD, BACKWARD, FACTOR };

template <typename T, int K, TriOp OP>
struct TriShape {
    // rows in the ring, and a refill of it
    static constexpr int RR = K <= 2 ? 4096 : K <= 4 ? 2048 : K <= 8 ? 1024 : 512;
    static constexpr int RB = RR / 8, NB = 8;
    // the current and the next step and a misaligned end fit the ring
    static constexpr int cap = (RR - RB) / 2 / 32 * 32;
    static constexpr int most = K <= 2 ? 864 : 416;                    // leaves 72 or 144 registers a thread
    static constexpr int max_rows = cap < most ? cap : most;           // rows a step
    // T's a row beside its entries' values: diagonal and reciprocal, or the upper entries
    static constexpr int extra = OP == TriOp::BACKWARD ? 2 : OP == TriOp::FACTOR ? K : 0;
    static constexpr size_t row_bytes = K * (sizeof(T) + 4) + (extra + 1) * sizeof(T);
    static constexpr size_t ring_bytes = (kTriRing + 16) * sizeof(T);
    static constexpr size_t smem_bytes = ring_bytes + RR * row_bytes + 4 * (kTriSteps + 4);
    static_assert(max_rows >= 32 && smem_bytes <= 227 * 1024 - 256, "ring shape");
};

// One triangle in position order; the arrays reach to a multiple of RB rows.
template <typename T>
struct TriView {
    int n, nsteps;
    const int* sptr;                      // nsteps + 1: step s holds rows [sptr[s], sptr[s + 1])
    const T* val;                         // [row][place]
    const int* code;                      // [row][place]
    const T* dg;                          // [row]: diagonal, its reciprocal (BACKWARD), or
                                          // [row][place] upper entries (FACTOR)
    T* low;                               // FACTOR: [row][place] eliminated entries
    const int* order;                     // FACTOR: the row at each position
    int* status;                          // FACTOR: the smallest row with a vanishing pivot
};

template <typename T>
__device__ __forceinline__ T sub_mul(T s, T a, T b);
template <>
__device__ __forceinline__ double sub_mul<double>(double s, double a, double b) {
    return __dsub_rn(s, __dmul_rn(a, b));
}
template <>
__device__ __forceinline__ float sub_mul<float>(float s, float a, float b) {
    return __fsub_rn(s, __fmul_rn(a, b));
}

template <typename T, int K, int EXTRA>
struct TriRow {
    T rv;
    alignas(16) T d[EXTRA > 0 ? EXTRA : 1];
    alignas(16) int c[K];                 // byte offset of the value in the ring, or ~position
    alignas(16) T v[K];
};

// COUNT consecutive 4- or 8-byte items, aligned to their total size up to 16 bytes
template <int COUNT, typename X>
__device__ __forceinline__ void load_packed(X (&dst)[COUNT], const X* src) {
    constexpr int bytes = COUNT * (int)sizeof(X);
    if constexpr (bytes == 8) {
        *reinterpret_cast<int2*>(dst) = *reinterpret_cast<const int2*>(src);
    } else {
#pragma unroll
        for (int k = 0; k < bytes / 16; ++k) reinterpret_cast<int4*>(dst)[k] = reinterpret_cast<const int4*>(src)[k];
    }
}

// FAR: the triangle has entries beyond the ring.
template <typename T, int K, TriOp OP, bool FAR>
__global__ void __launch_bounds__(TriShape<T, K, OP>::max_rows + 32, 1)
k_tri_sweep(TriView<T> F, const T* __restrict__ rhs, T* out, const int* gate, int* err) {
    using S = TriShape<T, K, OP>;
    constexpr int RR = S::RR, RB = S::RB, NB = S::NB, EX = S::extra;
    using Row = TriRow<T, K, EX>;
    extern __shared__ __align__(128) unsigned char tri_smem[];
    __shared__ uint64_t full[NB];
    __shared__ int s_stop;
    if (gate && *(volatile const int*)gate) return;
    unsigned char* ring = tri_smem;
    T* s_val = reinterpret_cast<T*>(tri_smem + S::ring_bytes);
    T* s_rhs = s_val + RR * K;
    T* s_dg = s_rhs + RR;
    int* s_code = reinterpret_cast<int*>(s_dg + EX * RR);
    int* s_ptr = s_code + RR * K;                                      // bounds of steps sbase ..
    const int NT = (int)blockDim.x - 32;                               // rows a step
    const bool rows = (int)threadIdx.x < NT;
    const bool producer = (int)threadIdx.x == NT;
    const int nblk = (F.n + RB - 1) / RB;
    int issued = 0;                                                    // producer
    // blocks up to the one that replaces a block whose rows all lie before `row0`
    auto refill = [&](int row0) {
        for (; issued < nblk && (issued - NB + 1) * RB <= row0; ++issued) {
            const int slot = issued % NB, r0 = issued * RB, q0 = slot * RB;
            const unsigned nr = (unsigned)((min(RB, F.n - r0) + 3) & ~3);
            mbar_arrive_tx(&full[slot], nr * (unsigned)sizeof(T) + (unsigned)(RB * (K * (sizeof(T) + 4) + EX * sizeof(T))));
            bulk_load(s_val + q0 * K, F.val + (size_t)r0 * K, RB * K * sizeof(T), &full[slot]);
            bulk_load(s_code + q0 * K, F.code + (size_t)r0 * K, RB * K * 4, &full[slot]);
            if (EX) bulk_load(s_dg + q0 * EX, F.dg + (size_t)r0 * EX, RB * EX * sizeof(T), &full[slot]);
            bulk_load(s_rhs + q0, rhs + r0, nr * (unsigned)sizeof(T), &full[slot]);
        }
    };
    if (producer) {
        for (int k = 0; k < NB; ++k) mbar_init(&full[k], 1);
        mbar_fence_init();
        s_stop = 0;
        *reinterpret_cast<T*>(ring + kTriRing * sizeof(T)) = T(OP == TriOp::FACTOR ? 1 : 0);
    }
    __syncthreads();
    if (producer) refill(0);

    int tid = threadIdx.x;
    int landed = 0;                       // rows known to have landed (row threads)
    auto wait_rows = [&](int end) {
        while (landed < end && tid < RR) {
            const int blk = landed / RB;
            const unsigned phase = (unsigned)((blk / NB) & 1);
            if (!mbar_try_wait(&full[blk % NB], phase) && !mbar_wait_bounded(&full[blk % NB], phase)) {
                tid = 1 << 30;            // no rows for this thread from here on
                s_stop = 1;
                raise_word(err);
            }
            landed += RB;
        }
    };
    auto load_row = [&](Row& q, int t) {
        const int r = t & (RR - 1);
        load_packed<K>(q.c, s_code + r * K);
        load_packed<K>(q.v, s_val + r * K);
        q.rv = s_rhs[r];
        if constexpr (EX > 0) load_packed<EX>(q.d, s_dg + r * EX);
    };
    // entry `place` of the row at position t met a pivot below eps: note the pivot's row
    auto vanishing = [&](int t, int place) {
        const int c = F.code[(size_t)t * K + place];
        int p;                                                         // its position, from the ring slot
        if (c < 0) p = ~c;
        else {
            // the latest position before t in that slot
            const int slot = c / (int)sizeof(T);
            p = (t & ~(kTriRing - 1)) + slot;
            if (p >= t) p -= kTriRing;
        }
        atomicMin(F.status, F.order[p]);
    };
    // one step: this thread's row of [b, e) (in q) is solved while its row of the next step,
    // [e, ne), is loaded
    auto step = [&](const Row& q, Row& nq, int b, int e, int ne) {
        const int t = b + tid, nt = e + tid;
        const bool has = t < e;
        T y[K];
        if (has) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int c = q.c[k];
                if (!FAR || c >= 0) y[k] = *reinterpret_cast<const T*>(ring + c);
                else y[k] = out[~c];
            }
        }
        if (landed < ne) wait_rows(ne);
        if (nt < ne) load_row(nq, nt);
        if (has) {
            T sum = q.rv;
            if constexpr (OP == TriOp::FACTOR) {
                // (an unused place divides 0 by the slot that holds 1 here)
                T l[K];
#pragma unroll
                for (int k = 0; k < K; ++k) l[k] = q.v[k] / y[k];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    if (fabs(y[k]) < T(2.220446049250313e-16)) vanishing(t, k);
                    F.low[(size_t)t * K + k] = l[k];
                    sum = sub_mul<T>(sum, l[k], q.d[k]);
                }
            } else {
#pragma unroll
                for (int k = 0; k < K; ++k) sum = sub_mul<T>(sum, q.v[k], y[k]);
                if (OP == TriOp::BACKWARD) sum = div_by<T>(sum, q.d[0], q.d[1]);
            }
            *reinterpret_cast<T*>(ring + (t & (kTriRing - 1)) * sizeof(T)) = sum;
            out[t] = sum;
        }
    };
    Row qa, qb;
    for (int sbase = 0; sbase < F.nsteps; sbase += kTriSteps) {
        // the window's bounds and two more (past the last step: n)
        const int steps = min(kTriSteps, F.nsteps - sbase);
        for (int k = threadIdx.x; k <= steps + 1; k += blockDim.x) s_ptr[k] = F.sptr[min(sbase + k, F.nsteps)];
        __syncthreads();
        int b = s_ptr[0], e = s_ptr[1], ne = s_ptr[2];
        if (rows) {
            if (sbase == 0) {
                wait_rows(e);
                if (b + tid < e) load_row(qa, b + tid);
            }
            for (int s = 0;;) {
                int nne = s_ptr[s + 3];   // read past steps + 1 only where it is not used
                step(qa, qb, b, e, ne);
                __syncthreads();
                if (++s == steps) break;
                b = e; e = ne; ne = nne;
                nne = s_ptr[s + 3];
                step(qb, qa, b, e, ne);
                __syncthreads();
                if (++s == steps) break;
                b = e; e = ne; ne = nne;
            }
        } else {
            for (int s = 0; s < steps; ++s) {
                if (producer && !*(volatile int*)&s_stop) refill(s_ptr[s]);
                __syncthreads();
            }
        }
    }
    if (producer && s_stop)                                            // copies still in flight
        for (int k = max(0, issued - NB); k < issued; ++k) mbar_wait_bounded(&full[k % NB], (unsigned)((k / NB) & 1));
}

// Steps of each level (count) and their bounds (fill): a level's rows in steps of `rows`.
__global__ void k_step_count(int nlev, const int* __restrict__ lptr, int rows, int* cnt) {
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < nlev; l += gridDim.x * blockDim.x)
        cnt[l] = (lptr[l + 1] - lptr[l] + rows - 1) / rows;
}

__global__ void k_step_fill(int nlev, const int* __restrict__ lptr, int rows, const int* __restrict__ first, int* sptr) {
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l <= nlev; l += gridDim.x * blockDim.x) {
        int s = first[l];
        if (l == nlev) sptr[s] = lptr[nlev];
        else
            for (int r = lptr[l]; r < lptr[l + 1]; r += rows) sptr[s++] = r;
    }
}

// A triangle's rows from the factor's pattern and values into position order; `end - q` is
// how far position q lies behind the end of the row's level (*far is set when that is beyond
// the ring).  Places of rows from n up to a multiple of RB are padded.
template <typename T, int K, TriOp OP>
__global__ void __launch_bounds__(256)
k_tri_pack(int n, const int* __restrict__ order, const int* __restrict__ level, const int* __restrict__ lptr,
           const int* __restrict__ pos, const int* __restrict__ rp, const int* __restrict__ ci,
           const double* __restrict__ lu, T* val, int* code, T* dg, int* far, int* bad) {
    constexpr int RB = TriShape<T, K, OP>::RB;
    constexpr bool DIV = OP == TriOp::BACKWARD;
    const int total = (n + RB - 1) / RB * RB;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        T* v = val + (size_t)t * K;
        int* c = code + (size_t)t * K;
        int k = 0;
        double d = 1.0;                       // absent diagonal (ilu.cpp:251)
        if (t < n) {
            const int i = order[t], end = lptr[level[i] + 1];
            for (int p = rp[i]; p < rp[i + 1]; ++p) {
                const int j = ci[p];
                if (DIV && j == i) d = lu[p];
                if (DIV ? j > i : j < i) {
                    const int q = pos[j];
                    if (end - q <= kTriRing) {
                        c[k] = (q & (kTriRing - 1)) * (int)sizeof(T);
                    } else {
                        c[k] = ~q;
                        *far = 1;
                    }
                    v[k] = (T)lu[p];
                    ++k;
                }
            }
            if (DIV && bad && fabs(d) < 2.220446049250313e-16) atomicMin(bad, i);
        }
        if (DIV) {
            dg[(size_t)t * 2] = (T)d;
            dg[(size_t)t * 2 + 1] = recip_of<T>((T)d);
        }
        for (; k < K; ++k) {
            c[k] = kTriRing * (int)sizeof(T);
            v[k] = T(0);
        }
    }
}

// The FACTOR form of a matrix's rows: lower entries, their codes, the upper entries (k, i)
// they meet, and the diagonals.  *no is set when a row does not have that form: a lower entry
// (i, k) whose elimination touches anything but a_ii, or a row without a diagonal.
template <int K>
__global__ void __launch_bounds__(256)
k_factor_pack(int n, const int* __restrict__ order, const int* __restrict__ level, const int* __restrict__ lptr,
              const int* __restrict__ pos, const int* __restrict__ rp, const int* __restrict__ ci,
              const int* __restrict__ dpos, const double* __restrict__ a, double* val, int* code, double* up,
              double* diag, int* far, int* no) {
    constexpr int RB = TriShape<double, K, TriOp::FACTOR>::RB;
    const int total = (n + RB - 1) / RB * RB;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        int k = 0;
        double d = 1.0;
        if (t < n) {
            const int i = order[t], end = lptr[level[i] + 1], e = rp[i + 1], di = dpos[i];
            if (di < 0) *no = 1;
            else d = a[di];
            for (int p = rp[i]; p < e; ++p) {
                const int j = ci[p];
                if (j >= i) break;
                // entries of row j right of its diagonal that row i has too: only column i
                double u = 0.0;
                bool hit = false, other = false;
                int pi = p + 1;
                for (int q = rp[j]; q < rp[j + 1]; ++q) {
                    const int c = ci[q];
                    if (c <= j) continue;
                    while (pi < e && ci[pi] < c) ++pi;
                    if (pi < e && ci[pi] == c) {
                        if (c == i) { hit = true; u = a[q]; }
                        else other = true;
                    }
                }
                if (!hit || other) *no = 1;
                const int q = pos[j];
                if (end - q <= kTriRing) {
                    code[(size_t)t * K + k] = (q & (kTriRing - 1)) * (int)sizeof(double);
                } else {
                    code[(size_t)t * K + k] = ~q;
                    *far = 1;
                }
                val[(size_t)t * K + k] = a[p];
                up[(size_t)t * K + k] = u;
                ++k;
            }
        }
        diag[t] = d;
        for (; k < K; ++k) {
            code[(size_t)t * K + k] = kTriRing * (int)sizeof(double);
            val[(size_t)t * K + k] = 0.0;
            up[(size_t)t * K + k] = 0.0;
        }
    }
}

template <int K>
__global__ void __launch_bounds__(256)
k_factor_unpack(int n, const int* __restrict__ order, const int* __restrict__ rp, const int* __restrict__ ci,
                const int* __restrict__ dpos, const double* __restrict__ low, const double* __restrict__ diag,
                double* lu) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = order[t];
        for (int p = rp[i], k = 0; p < rp[i + 1] && ci[p] < i; ++p, ++k) lu[p] = low[(size_t)t * K + k];
        lu[dpos[i]] = diag[t];
    }
}

// out[k] = in[idx[k]] (GATHER) or out[idx[k]] = in[k]
template <typename T, bool GATHER>
__global__ void __launch_bounds__(256)
k_permute(int n, const int* __restrict__ idx, const T* __restrict__ in, T* __restrict__ out, const int* gate) {
    if (gate && *(volatile const int*)gate) return;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        if (GATHER) out[k] = in[idx[k]];
        else out[idx[k]] = in[k];
    }
}

}  // namespace hamlss
