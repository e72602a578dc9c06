// cg_persist.cuh -- the CG iteration as one persistent kernel for systems whose matrix
// fits the chip's shared memory.
//
// What bounds CG on such systems is launches and their grid-wide reductions, then L2: two
// launches a trip took 11.5 us at 4,096 rows (nothing to do with the arithmetic) and 26.5 us
// at 491,401 (77 MB a trip through L2).  Here one launch runs many trips: each block owns a
// range of rows, with its matrix entries in shared memory (values and 16-bit column offsets),
// its x, r, p, q in registers, and the part of p its rows multiply -- its own rows and the
// columns around them -- in shared memory.  Per trip only z = M^-1 r of the neighbouring rows
// and the sums of the two reductions cross the chip.
//
// What is left is the latency of those two all-block sums, so there are two forms:
//   CLUSTER  one thread-block cluster of up to 16 blocks: sums stored into every block's
//            shared memory, one cluster barrier.  A cluster sits in one GPC, so nothing
//            crosses between the two dies (~1,700 cycles a sum at 16 blocks, against 1,800
//            to 4,300 for the same blocks exchanging through L2, depending on where they sit)
//   grid     a cooperative launch of a block per SM: sums through L2 behind a barrier on one
//            counter (~4,400 cycles; every block polling every other's word took ~8,600)
// Every block gets all blocks' sums, adds them in block order, and works out alpha, beta and
// the stop tests for itself.
//
// Measured, Jacobi, FP64, us a trip: 64^2 11.5 -> 2.9, 256^2 15 -> 6.5, 701^2 26.5 -> 11.8 (of
// which 5.5 are the two sums, the rest instructions of the 7 rows a thread); the limit is
// the shared memory, 3,584 rows of 5 entries a block.
//
// With one tile of 256 rows a block the sums are formed in the order of the launch-by-launch
// kernels (k_spmv / k_vec of 256-row blocks, block sums added in block order), so the
// iterates agree with them bit for bit; larger systems add a thread's rows first.
//
// The grid's waits are bounded (~1 s): a wait that runs out ends the loop in every block (the
// others' waits run out in turn), sets the lane's error word, and the host reports
// HAMLSS_ERR_TIMEOUT.
#pragma once

#include <cooperative_groups.h>

#include "engine.cuh"

namespace hamlss {

constexpr int kPersistMaxSlots = 7;       // rows a thread

// Sum of eight values in the order of a 32-lane xor tree over them (the rest zeros).
__device__ __forceinline__ double tree8(const double* s, int stride) {
    return ((s[0] + s[4 * stride]) + (s[2 * stride] + s[6 * stride])) +
           ((s[stride] + s[5 * stride]) + (s[3 * stride] + s[7 * stride]));
}

constexpr int kClusterBlocks = kPersistClusterBlocks;

// Shared memory and global words of the all-block sums.
struct SumSpace {
    double warp[16 * 2];                  // this block's warps
    double grp1[8], grp2[8 * 2];          // grid: sums of 32 blocks each (beyond the grid 0)
    double part[2][kClusterBlocks * 2];   // cluster: every block's sums, two sets
    int fail;
};

// Sums of v over all blocks, the same in every thread of every block, also ordering every
// block's global writes before them.  `k`: number of this reduction in the launch, from 0.
// `words`: grid only, two sets of kPersistMaxBlocks * 2 partial sums; `count`: zero at launch.
// false: a wait ran out.
template <int NV, bool CLUSTER>
__device__ __forceinline__ bool all_sums(double (&v)[NV], SumSpace& sp, int k, double* words, unsigned* count) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nb = gridDim.x;
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int c = 0; c < NV; ++c) v[c] = warp_sum(v[c]);
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < NV; ++c) sp.warp[wid * NV + c] = v[c];
    }
    __syncthreads();
    auto block_total = [&](int c) {
        if (nw == 8) return tree8(sp.warp + c, NV);
        double h[8];
#pragma unroll
        for (int w = 0; w < 8; ++w) h[w] = sp.warp[w * NV + c] + sp.warp[(w + 8) * NV + c];
        return tree8(h, 1);
    };
    if constexpr (CLUSTER) {
        auto cluster = cooperative_groups::this_cluster();
        double* set = sp.part[k & 1];
        if (tid < nb * NV) {
            const int to = tid / NV, c = tid - to * NV;
            *cluster.map_shared_rank(&set[blockIdx.x * NV + c], to) = block_total(c);
        }
        cluster.sync();
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            double h[8];                  // blocks i and i + 8 (blocks beyond the cluster are 0)
#pragma unroll
            for (int i = 0; i < 8; ++i) h[i] = set[i * NV + c] + set[(i + 8) * NV + c];
            v[c] = tree8(h, 1);
        }
        return true;
    } else {
        double* set = words + (size_t)(k & 1) * kPersistMaxBlocks * 2;
        double* grp = NV == 1 ? sp.grp1 : sp.grp2;
        if (tid == 0) {
#pragma unroll
            for (int c = 0; c < NV; ++c) set[blockIdx.x * NV + c] = block_total(c);
            __threadfence();
            atomicAdd(count, 1u);
            const unsigned want = (unsigned)(k + 1) * (unsigned)nb;
            const long long t0 = clock64();
            while (*(volatile unsigned*)count < want)
                if (clock64() - t0 > (1ll << 31)) {
                    sp.fail = 1;
                    break;
                }
            __threadfence();
        }
        __syncthreads();
        if (wid < (nb + 31) >> 5) {
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                const double t = warp_sum(tid < nb ? __ldcg(&set[tid * NV + c]) : 0.0);
                if (lane == 0) grp[wid * NV + c] = t;
            }
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < NV; ++c) v[c] = tree8(grp + c, NV);
        return *(volatile int*)&sp.fail == 0;
    }
}

template <typename T>
struct PersistArgs {
    int n, rows, max_trips;               // rows a block (a multiple of 32)
    const int* rp;
    const int* ci;
    const T* v;
    T* x;
    T* r;
    T* p;
    T* z;
    const T* dinv;
    double* words;                        // grid: partial sums and the barrier's counter
    unsigned* count;
    int* err;
    int window, entries;                  // shared-memory capacities
};

// `Fin`: fin.pq(s, tot) after p.q, fin.upd(s, tot) after ||r||^2 and r.z; both run in one
// thread of each block on its copy of the state and may set s->halt.  fin.leave(s): leave
// the loop after a trip (state saved, not halted).
template <typename T, bool JAC, int SLOTS, bool CLUSTER, typename State, typename Fin>
__global__ void __launch_bounds__(512, 1)
k_cg_persist(PersistArgs<T> a, State* gs, Fin fin) {
    extern __shared__ __align__(16) unsigned char persist_smem_raw[];
    __shared__ State S;
    __shared__ SumSpace sp;
    __shared__ int s_lo, s_hi;
    const int tid = threadIdx.x, NT = blockDim.x;
    const int r0 = blockIdx.x * a.rows, r1 = min(a.n, r0 + a.rows);
    if (*(volatile const int*)&gs->halt) return;
    if (tid == 0) {
        S = *gs;
        s_lo = r0;
        s_hi = r1;
    }
    for (int k = tid; k < (int)(sizeof(SumSpace) / sizeof(int)); k += NT) reinterpret_cast<int*>(&sp)[k] = 0;
    __syncthreads();
    // columns the block's rows reach (sorted rows: the first and the last entry)
    for (int row = r0 + tid; row < r1; row += NT) {
        const int b = a.rp[row], e = a.rp[row + 1];
        if (b < e) {
            atomicMin(&s_lo, a.ci[b]);
            atomicMax(&s_hi, a.ci[e - 1] + 1);
        }
    }
    __syncthreads();
    const int w0 = s_lo, w1 = s_hi, e0 = a.rp[r0], ne = a.rp[r1] - e0;
    T* pw = reinterpret_cast<T*>(persist_smem_raw);
    T* sv = pw + ((a.window + 1) & ~1);
    unsigned short* si = reinterpret_cast<unsigned short*>(sv + ((a.entries + 3) & ~3));
    for (int k = tid; k < ne; k += NT) {
        sv[k] = a.v[e0 + k];
        si[k] = (unsigned short)(a.ci[e0 + k] - w0);
    }
    for (int j = w0 + tid; j < w1; j += NT) pw[j - w0] = a.p[j];
    T x[SLOTS], r[SLOTS], q[SLOTS], di[SLOTS];
    int ent[SLOTS];                       // first entry, length << 16
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
        const int row = r0 + s * NT + tid;
        x[s] = r[s] = q[s] = di[s] = T(0);
        ent[s] = 0;
        if (row < r1) {
            x[s] = a.x[row];
            r[s] = a.r[row];
            if (JAC) di[s] = a.dinv[row];
            const int b = a.rp[row] - e0;
            ent[s] = b | (a.rp[row + 1] - e0 - b) << 16;
        }
    }
    auto precond = [&](T ri, T d) { return JAC ? (T)__dmul_rn((double)d, (double)ri) : ri; };
    const int below = r0 - w0, outside = below + (w1 - r1);
    bool ok = true;
    __syncthreads();
    if (CLUSTER) cooperative_groups::this_cluster().sync();   // every block's sums space is clear
    for (int trip = 0; trip < a.max_trips; ++trip) {
        // p = z + beta p over the window: the outside part from the neighbours' z
        const double beta = S.beta;
        for (int k0 = 0; k0 < outside; k0 += 4 * NT) {
            T zo[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int o = k0 + k * NT + tid;
                if (o < outside) {
                    const int j = o < below ? w0 + o : r1 + (o - below);
                    zo[k] = trip ? __ldcg(&a.z[j]) : precond(a.r[j], JAC ? a.dinv[j] : T(0));
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int o = k0 + k * NT + tid;
                if (o < outside) {
                    const int c = o < below ? o : r1 - w0 + (o - below);
                    pw[c] = (T)__dadd_rn((double)zo[k], __dmul_rn(beta, (double)pw[c]));
                }
            }
        }
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
            const int row = r0 + s * NT + tid;
            if (row < r1)
                pw[row - w0] = (T)__dadd_rn((double)precond(r[s], di[s]), __dmul_rn(beta, (double)pw[row - w0]));
        }
        __syncthreads();
        double pq[1] = {0.0};
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
            const int row = r0 + s * NT + tid;
            if (row < r1) {
                // in column order, four entries' loads in flight at a time
                double sum = 0.0;
                const int b = ent[s] & 0xffff, e = b + (int)((unsigned)ent[s] >> 16);
                int k = b;
                for (; k + 4 <= e; k += 4) {
                    const T a0 = sv[k], a1 = sv[k + 1], a2 = sv[k + 2], a3 = sv[k + 3];
                    const T p0 = pw[si[k]], p1 = pw[si[k + 1]], p2 = pw[si[k + 2]], p3 = pw[si[k + 3]];
                    sum = mul_add<T>(sum, a0, (double)p0);
                    sum = mul_add<T>(sum, a1, (double)p1);
                    sum = mul_add<T>(sum, a2, (double)p2);
                    sum = mul_add<T>(sum, a3, (double)p3);
                }
                for (; k < e; ++k) sum = mul_add<T>(sum, sv[k], (double)pw[si[k]]);
                q[s] = (T)sum;
                pq[0] += (double)pw[row - w0] * (double)q[s];
            }
        }
        ok = all_sums<1, CLUSTER>(pq, sp, 2 * trip, a.words, a.count);
        if (!ok) break;
        if (tid == 0) fin.pq(&S, pq);
        __syncthreads();
        if (S.halt) break;
        const double alpha = S.alpha;
        double rr[2] = {0.0, 0.0};
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
            const int row = r0 + s * NT + tid;
            if (row < r1) {
                x[s] = (T)__dadd_rn((double)x[s], __dmul_rn(alpha, (double)pw[row - w0]));
                r[s] = (T)__dadd_rn((double)r[s], __dmul_rn(-alpha, (double)q[s]));
                const T z = precond(r[s], di[s]);
                a.z[row] = z;
                const double rd = (double)r[s];
                rr[0] += rd * rd;
                rr[1] += rd * (double)z;
            }
        }
        ok = all_sums<2, CLUSTER>(rr, sp, 2 * trip + 1, a.words, a.count);
        if (!ok) break;
        if (tid == 0) fin.upd(&S, rr);
        __syncthreads();
        if (S.halt || fin.leave(&S)) break;
    }
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
        const int row = r0 + s * NT + tid;
        if (row < r1) {
            a.x[row] = x[s];
            a.r[row] = r[s];
            a.p[row] = pw[row - w0];
        }
    }
    if (CLUSTER) cooperative_groups::this_cluster().sync();   // no block leaves while sums are stored into it
    if (tid == 0) {
        if (!ok) raise_word(a.err);
        if (blockIdx.x == 0) {
            if (!ok) fin.timeout(&S);
            *gs = S;
        }
    }
}

}  // namespace hamlss
