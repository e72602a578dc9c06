// engine.cu -- context / lane setup, device CSR helpers, Jacobi, residual check.
#include <mutex>
#include <cmath>
#include <cstring>

#include "krylov.cuh"

namespace hamlss {

void pool_keep_memory(int device) {
    static std::mutex mu;
    static bool done[64] = {};
    std::lock_guard<std::mutex> g(mu);
    if (device < 0 || device >= 64 || done[device]) return;
    cudaMemPool_t pool;
    HAMLSS_CUDA(cudaDeviceGetDefaultMemPool(&pool, device));
    uint64_t keep = UINT64_MAX;
    HAMLSS_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    done[device] = true;
}

void lane_init(Lane& L, int sm_count) {
    HAMLSS_CUDA(cudaStreamCreateWithFlags(&L.stream, cudaStreamNonBlocking));
    // every reducing launch has at most sm_count * kMaxBlocksPerSm blocks of at most
    // kMaxRed sums each (red_check enforces it before the launch)
    L.red_cap = (size_t)std::max(sm_count, 1) * kMaxBlocksPerSm * kMaxRed;
    L.partials.alloc(L.red_cap);
    L.err.alloc(1);
    *L.err.p = 0;
    L.ticket.alloc(1);
    L.ticket.zero(L.stream);
}

bool lane_take_timeout(const Lane& L) {
    volatile int* e = L.err.p;
    const bool out = *e != 0;
    if (out) *e = 0;
    return out;
}

void lane_destroy(Lane& L) {
    if (L.stream) {
        cudaStreamSynchronize(L.stream);
        cudaStreamDestroy(L.stream);
        L.stream = nullptr;
    }
    L.partials.release();
    L.ticket.release();
    L.sums.release();
}

namespace {

__global__ void k_to_f32(const double* __restrict__ a, float* __restrict__ b, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

// flags[0]: bad row_ptr, flags[1]: column out of range, flags[2]: unsorted/duplicate row
__global__ void k_validate(int n, int m, int nnz, const int* __restrict__ rp,
                           const int* __restrict__ ci, int* flags) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int s = rp[i], e = rp[i + 1];
        if (i == 0 && s != 0) flags[0] = 1;
        if (i == n - 1 && e != nnz) flags[0] = 1;
        if (e < s || s < 0 || e > nnz) { flags[0] = 1; continue; }
        int prev = -1;
        for (int k = s; k < e; ++k) {
            int c = ci[k];
            if (c < 0 || c >= m) flags[1] = 1;
            if (c <= prev) flags[2] = 1;
            prev = c;
        }
    }
}

__global__ void k_diag(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                       const double* __restrict__ v, double* __restrict__ d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double di = 0.0;
        for (int k = rp[i]; k < rp[i + 1]; ++k)
            if (ci[k] == i) { di = v[k]; break; }
        d[i] = di;
    }
}

// JacobiPreconditioner::setup (jacobi.cpp:23-31): first zero diagonal row -> error.
__global__ void k_jacobi_setup(int n, const double* __restrict__ d, double omega,
                               double* __restrict__ inv, int* bad_row) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double di = d[i];
        if (fabs(di) < 2.220446049250313e-16) { atomicMin(bad_row, i); inv[i] = 0.0; }
        else inv[i] = omega / di;
    }
}

template <typename T>
__global__ void k_jacobi_apply(int n, const T* __restrict__ inv, const T* __restrict__ r,
                               T* __restrict__ z, const int* gate) {
    if (gate && *(volatile const int*)gate) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        z[i] = (T)__dmul_rn((double)inv[i], (double)r[i]);
}

// mx[0]: the longest row; mx[1]: the most entries of `group` rows from a multiple of it (group > 0)
__global__ void k_row_len_max(int n, const int* __restrict__ rp, int group, int* mx) {
    int m = 0, g = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        m = max(m, rp[i + 1] - rp[i]);
        if (group > 0 && i % group == 0) g = max(g, rp[min(n, i + group)] - rp[i]);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    g = __reduce_max_sync(0xffffffffu, g);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&mx[0], m);
        atomicMax(&mx[1], g);
    }
}

// near[0] += places k that rows i and i + 1 both have, near[1] += those whose columns lie at
// most kNearColumns apart; every `stride`-th row, the first eight places
__global__ void k_row_neighbours(int n, int stride, const int* __restrict__ rp, const int* __restrict__ ci, int* near) {
    int pairs = 0, close = 0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; (long long)t * stride < n - 1; t += gridDim.x * blockDim.x) {
        const int i = t * stride, a = rp[i], b = rp[i + 1], len = min(8, min(b - a, rp[i + 2] - b));
        pairs += max(len, 0);
        for (int k = 0; k < len; ++k) close += abs(ci[a + k] - ci[b + k]) <= kNearColumns;
    }
    pairs = __reduce_add_sync(0xffffffffu, pairs);
    close = __reduce_add_sync(0xffffffffu, close);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&near[0], pairs);
        atomicAdd(&near[1], close);
    }
}

__global__ void k_rows_longer(int n, const int* __restrict__ rp, int len, int* list, int* count) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (rp[i + 1] - rp[i] > len) list[atomicAdd(count, 1)] = i;
}

// most[0], most[1] = the most entries, and columns spanned, of `rows` consecutive rows
// (block b: rows [b * rows, ...)) of a matrix with sorted rows; the block's own rows count
// as columns.
__global__ void __launch_bounds__(256)
k_persist_plan(int n, int rows, const int* __restrict__ rp, const int* __restrict__ ci, int* most) {
    __shared__ int lo, hi;
    const int r0 = blockIdx.x * rows, r1 = min(n, r0 + rows);
    if (threadIdx.x == 0) { lo = r0; hi = r1; }
    __syncthreads();
    for (int row = r0 + threadIdx.x; row < r1; row += blockDim.x) {
        const int b = rp[row], e = rp[row + 1];
        if (b < e) {
            atomicMin(&lo, ci[b]);
            atomicMax(&hi, ci[e - 1] + 1);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(&most[0], rp[r1] - rp[r0]);
        atomicMax(&most[1], hi - lo);
    }
}

}  // namespace

void ensure_persist_plan(Ctx& ctx, hamlss_mat* M) {
    if (M->persist_rows >= 0) return;
    M->persist_rows = 0;
    const int n = M->A.n;
    if (n == 0 || ctx.sm_count < 1) return;
    // equal shares of whole warps, one 256-row tile at least: of a cluster's blocks up to
    // kPersistClusterRows rows where a block's memory holds them, else of a block per SM
    for (const bool cluster : {true, false}) {
        if (cluster && n > kPersistClusterRows) continue;
        const int blocks = cluster ? kPersistClusterBlocks : ctx.sm_count;
        const int rows = std::max(256, ceil_div(ceil_div(n, blocks), 32) * 32);
        if (rows > kPersistMaxRows) return;
        cudaStream_t s = ctx.lane.stream;
        DBuf<int> most(2);
        most.zero(s);
        k_persist_plan<<<ceil_div(n, rows), 256, 0, s>>>(n, rows, M->A.rp.p, M->A.ci.p, most.p);
        HAMLSS_LAUNCH_CHECK();
        int h[2];
        most.download(h, 2, s);
        HAMLSS_CUDA(cudaStreamSynchronize(s));
        M->persist_entries = h[0];
        M->persist_window = h[1];
        M->persist_rows = rows;
        M->persist_cluster = cluster;
        if (persist_smem<double>(h[0], h[1]) <= kPersistSmem) return;
    }
}

Csr<float> DevMat::f32(cudaStream_t s) {
    if (!v32_valid) {
        v32.ensure(nnz);
        if (nnz) {
            k_to_f32<<<std::min(ceil_div(nnz, 256), 148 * 16), 256, 0, s>>>(v.p, v32.p, nnz);
            HAMLSS_LAUNCH_CHECK();
        }
        v32_valid = true;
    }
    return Csr<float>{n, m, nnz, rp.p, ci.p, v32.p};
}

int validate_csr(Ctx& ctx, const Csr<double>& A) {
    if (A.n == 0) return HAMLSS_OK;
    DBuf<int> flags(3);
    flags.zero(ctx.lane.stream);
    k_validate<<<std::min(ceil_div(A.n, 256), ctx.sm_count * 8), 256, 0, ctx.lane.stream>>>(
        A.n, A.m, A.nnz, A.rp, A.ci, flags.p);
    HAMLSS_LAUNCH_CHECK();
    int h[3];
    flags.download(h, 3, ctx.lane.stream);
    HAMLSS_CUDA(cudaStreamSynchronize(ctx.lane.stream));
    return (h[0] || h[1] || h[2]) ? HAMLSS_ERR_MALFORMED : HAMLSS_OK;
}

void ensure_row_profile(Ctx& ctx, hamlss_mat* M) {
    if (M->n_long >= 0) return;
    const int n = M->A.n;
    M->n_long = 0;
    M->long_len = INT_MAX;
    if (n == 0) return;
    cudaStream_t s = ctx.lane.stream;
    DBuf<int> cnt(4);
    cnt.zero(s);
    const int g = std::min(ceil_div(n, 256), ctx.sm_count * 8);
    const int R = prod_rows(ctx.sm_count, M->A.f64());
    k_row_len_max<<<g, 256, 0, s>>>(n, M->A.rp.p, R, cnt.p);
    HAMLSS_LAUNCH_CHECK();
    if (stream_group(M->A.f64()) == 1) {
        const int stride = std::max(1, n / kNeighbourRows);
        k_row_neighbours<<<std::min(ceil_div(n / stride, 256), ctx.sm_count * 8), 256, 0, s>>>(
            n, stride, M->A.rp.p, M->A.ci.p, cnt.p + 2);
        HAMLSS_LAUNCH_CHECK();
    }
    int hm[4];
    cnt.download(hm, 4, s);
    HAMLSS_CUDA(cudaStreamSynchronize(s));
    int h = hm[0];
    M->A.scattered = gathers_scattered(hm[2], hm[3]);
    M->A.uneven = R > 0 && prod_uneven(h, hm[1], M->A.nnz);
    const double avg = (double)M->A.nnz / n;
    if (h <= kSkewRow || h <= kSkewRatio * avg) return;
    const int len = std::max(kSkewRow, (int)std::ceil(kSkewRatio * avg));
    M->long_rows.ensure(n);
    cnt.zero(s);
    k_rows_longer<<<g, 256, 0, s>>>(n, M->A.rp.p, len, M->long_rows.p, cnt.p);
    HAMLSS_LAUNCH_CHECK();
    cnt.download(&h, 1, s);
    HAMLSS_CUDA(cudaStreamSynchronize(s));
    M->n_long = h;
    M->long_len = len;
}

void ensure_diag(Ctx& ctx, hamlss_mat* M) {
    if (M->diag_valid) return;
    M->diag.ensure(M->A.n);
    if (M->A.n) {
        ProfScope ps(ctx.lane, "setup", 16.0 * M->A.n + 12.0 * M->A.nnz);
        k_diag<<<std::min(ceil_div(M->A.n, 256), ctx.sm_count * 8), 256, 0, ctx.lane.stream>>>(
            M->A.n, M->A.rp.p, M->A.ci.p, M->A.v.p, M->diag.p);
        HAMLSS_LAUNCH_CHECK();
    }
    M->diag_valid = true;
}

// ---------------------------------------------------------------------------- Jacobi
void JacobiPrec::apply(Ctx& ctx, const Lane& L, const double* r, double* z, const int* gate) {
    if (!n) return;
    ProfScope ps(L, "jacobi", 24.0 * n);
    k_jacobi_apply<double><<<std::min(ceil_div(n, 256), ctx.sm_count * 8), 256, 0, L.stream>>>(
        n, inv.p, r, z, gate);
    HAMLSS_LAUNCH_CHECK();
}

void JacobiPrec::prepare32(Ctx& ctx) {
    if (inv32_valid) return;
    inv32.ensure(n);
    if (n) {
        k_to_f32<<<std::min(ceil_div(n, 256), 148 * 16), 256, 0, ctx.lane.stream>>>(inv.p, inv32.p, n);
        HAMLSS_LAUNCH_CHECK();
    }
    inv32_valid = true;
}

void JacobiPrec::apply32(Ctx& ctx, const Lane& L, const float* r, float* z, const int* gate) {
    prepare32(ctx);
    if (!n) return;
    ProfScope ps(L, "jacobi", 12.0 * n);
    k_jacobi_apply<float><<<std::min(ceil_div(n, 256), ctx.sm_count * 8), 256, 0, L.stream>>>(
        n, inv32.p, r, z, gate);
    HAMLSS_LAUNCH_CHECK();
}

std::unique_ptr<Prec> make_jacobi(Ctx& ctx, hamlss_mat* A, double omega) {
    ensure_diag(ctx, A);
    auto J = std::make_unique<JacobiPrec>();
    J->kind = HAMLSS_PREC_JACOBI;
    J->n = A->A.n;
    J->inv.ensure(J->n);
    DBuf<int> bad(1);
    int init = 0x7fffffff;
    bad.upload(&init, 1, ctx.lane.stream);
    if (J->n) {
        ProfScope ps(ctx.lane, "setup", 16.0 * J->n);
        k_jacobi_setup<<<std::min(ceil_div(J->n, 256), ctx.sm_count * 8), 256, 0, ctx.lane.stream>>>(
            J->n, A->diag.p, omega, J->inv.p, bad.p);
        HAMLSS_LAUNCH_CHECK();
    }
    int h = 0;
    bad.download(&h, 1, ctx.lane.stream);
    HAMLSS_CUDA(cudaStreamSynchronize(ctx.lane.stream));
    if (h != 0x7fffffff)
        fail(HAMLSS_ERR_ZERO_DIAG, "JacobiPreconditioner: zero diagonal at row " + std::to_string(h));
    return J;
}

// ------------------------------------------------------------------ true residual
namespace {
struct EpiRes2 {
    const double* b;
    HAMLSS_NO_LOAD
    template <int NV>
    __device__ __forceinline__ void operator()(int i, double ax, double (&acc)[NV]) const {
        double bi = b[i];
        double ri = __dsub_rn(bi, ax);
        acc[0] += bi * bi;
        acc[1] += ri * ri;
    }
};
struct FinStore2 {
    double* out;
    template <int NV>
    __device__ void operator()(const double (&t)[NV]) const { out[0] = t[0]; out[1] = t[1]; }
};
}  // namespace

double true_relative_residual(Ctx& ctx, hamlss_mat* A, const double* b, const double* x,
                              Workspace& ws) {
    ws.small.ensure(4096);
    double* out = ws.small.p + 4000;
    launch_spmv<double, 2>(ctx.sm_count, ctx.lane, A->A.f64(), XVec<double>{x}, EpiRes2{b},
                           FinStore2{out});
    double h[2];
    HAMLSS_CUDA(cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, ctx.lane.stream));
    HAMLSS_CUDA(cudaStreamSynchronize(ctx.lane.stream));
    double bn = std::sqrt(h[0]), rn = std::sqrt(h[1]);
    return bn > 2.220446049250313e-16 ? rn / bn : rn;
}

}  // namespace hamlss
