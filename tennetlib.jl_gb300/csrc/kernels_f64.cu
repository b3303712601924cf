// FP64 kernels of the sweep engine:
//  * grouped block-sparse GEMM (CUDA-core DFMA) -- the FP64 GPU path of every contraction
//    of the two-site effective Hamiltonian and of the environment updates;
//  * block linear combination -- the MPO step between the two GEMM stages;
//  * Krylov vector kernels (multi-dot, multi-axpy, scaling, linear combination) with
//    warp-shuffle reductions and a deterministic two-stage finalisation.
#include <cuda_runtime.h>

#include "tn_internal.h"

namespace tn {

// ------------------------------------------------------------------------------------
// grouped GEMM: 128 threads per TM x TN output tile, one thread adds its outputs along the
// whole k range of the task
//
// Bound by the FP64 pipe: a warp-wide DFMA holds its SM sub-partition for 64 clocks (measured:
// 1.7 FMA per clock and SM with one warp per sub-partition, 2.0 at most; DMMA the same), so a
// multiplication by padding costs as much as a real one, while loads, shared memory and issue
// slots are nearly free.  Hence small tiles of 8 x 4 warp patches (patches outside the block
// are skipped), k taken to its exact end, the segments of a task run together into one k range
// (four 4-long segments fill a 16-deep chunk), four warps so that every sub-partition works,
// and the next chunk's loads in flight during the products.  Each output is one chain of fused
// multiply-adds in segment order.  On the 64 x 64 x 16 tiles of 256 threads that this replaced
// a 4 x 4 x 4 block took 16 us of multiplications by zeros.
// The tile is GemmPlan::finalize's choice.  Measured, whole calls in FP64: DMRG run of a
// 12-site chain 118 -> 71 ms, sweep of a 20-site cylinder at chi = 160 236 -> 95 ms, TDVP of
// a 12-site chain (complex) 209 -> 91 ms, sweep of a 16-site tree at chi = 16 75 -> 41 ms.
// ------------------------------------------------------------------------------------
namespace {
constexpr int BK = 16;
constexpr int GEMM_THREADS = 128;

template <int TM, int TN>
__global__ void __launch_bounds__(GEMM_THREADS)
gemm_f64_kernel(const Seg* __restrict__ segs, const Task* __restrict__ tasks,
                const Tile* __restrict__ tiles, const __grid_constant__ Bases b) {
    constexpr int RP = TM / 16, CP = TN / 8;          // 8-row and 4-column patches of a warp
    constexpr int NA = TM * BK / GEMM_THREADS, NB = TN * BK / GEMM_THREADS;  // loads per thread
    __shared__ double As[BK][TM + 1];
    __shared__ double Bs[BK][TN + 1];
    const Tile t = tiles[blockIdx.x];
    const Task tk = tasks[t.task];
    const Seg* const seg0 = segs + tk.seg0;
    const int K = tk.nseg ? seg0[tk.nseg - 1].kpre + seg0[tk.nseg - 1].k : 0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = (warp & 1) * (TM / 2) + (lane & 7);
    const int col0 = (warp >> 1) * (TN / 2) + (lane >> 3);
    // rows and columns of the block from this warp's first patch on
    const int mrem = tk.m - t.m0 - (warp & 1) * (TM / 2);
    const int nrem = tk.n - t.n0 - (warp >> 1) * (TN / 2);
    double acc[RP][CP];
#pragma unroll
    for (int i = 0; i < RP; ++i)
#pragma unroll
        for (int j = 0; j < CP; ++j) acc[i][j] = 0.0;

    if (K > 0) {
        // element order of the loads: along the operand's contiguous index (as the first
        // segment has it; the others of a task are alike)
        const bool ka = seg0->ta != 0, kb = seg0->tb == 0;  // k is the contiguous index
        const Seg *wa = seg0, *wb = seg0;  // segments of this thread's last loads
        double ra[NA], rb[NB];
        auto load = [&](int k0) {
#pragma unroll
            for (int r = 0; r < NA; ++r) {
                const int e = tid + GEMM_THREADS * r;
                const int i = t.m0 + (ka ? e / BK : e % TM);
                const int kf = k0 + (ka ? e % BK : e / TM);
                double v = 0.0;
                if (kf < K && i < tk.m) {
                    while (kf >= wa->kpre + wa->k) ++wa;
                    const double* A = b.p[wa->abuf] + wa->aoff;
                    const int64_t k = kf - wa->kpre;
                    v = wa->ta ? A[k + int64_t(i) * wa->lda] : A[i + k * wa->lda];
                    v = wa->sgn < 0 ? -v : v;
                }
                ra[r] = v;
            }
#pragma unroll
            for (int r = 0; r < NB; ++r) {
                const int e = tid + GEMM_THREADS * r;
                const int j = t.n0 + (kb ? e / BK : e % TN);
                const int kf = k0 + (kb ? e % BK : e / TN);
                double v = 0.0;
                if (kf < K && j < tk.n) {
                    while (kf >= wb->kpre + wb->k) ++wb;
                    const double* B = b.p[wb->bbuf] + wb->boff;
                    const int64_t k = kf - wb->kpre;
                    v = wb->tb ? B[j + k * wb->ldb] : B[k + int64_t(j) * wb->ldb];
                }
                rb[r] = v;
            }
        };
        load(0);
        for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
            for (int r = 0; r < NA; ++r) {
                const int e = tid + GEMM_THREADS * r;
                As[ka ? e % BK : e / TM][ka ? e / BK : e % TM] = ra[r];
            }
#pragma unroll
            for (int r = 0; r < NB; ++r) {
                const int e = tid + GEMM_THREADS * r;
                Bs[kb ? e % BK : e / TN][kb ? e / BK : e % TN] = rb[r];
            }
            __syncthreads();
            if (k0 + BK < K) load(k0 + BK);
            const int kv = min(BK, K - k0);
#pragma unroll 4
            for (int kk = 0; kk < kv; ++kk) {
                double a[RP], q[CP];
#pragma unroll
                for (int i = 0; i < RP; ++i) a[i] = As[kk][row0 + 8 * i];
#pragma unroll
                for (int j = 0; j < CP; ++j) q[j] = Bs[kk][col0 + 4 * j];
#pragma unroll
                for (int i = 0; i < RP; ++i)
#pragma unroll
                    for (int j = 0; j < CP; ++j)
                        if (8 * i < mrem && 4 * j < nrem) acc[i][j] = fma(a[i], q[j], acc[i][j]);
            }
            __syncthreads();
        }
    }
    double* __restrict__ C = b.p[tk.cbuf] + tk.coff;
#pragma unroll
    for (int j = 0; j < CP; ++j) {
        const int gj = t.n0 + col0 + 4 * j;
        if (gj >= tk.n) continue;
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            const int gi = t.m0 + row0 + 8 * i;
            if (gi < tk.m) {
                double* c = C + gi + int64_t(gj) * tk.ldc;
                *c = tk.accum ? *c + acc[i][j] : acc[i][j];
            }
        }
    }
}

__global__ void __launch_bounds__(256)
combine_kernel(const CombOut* __restrict__ outs, const CombTerm* __restrict__ terms,
               const CombTile* __restrict__ tiles, Bases b) {
    const CombTile t = tiles[blockIdx.x];
    const CombOut o = outs[t.out];
    const int r = t.r0 + (threadIdx.x & 31);
    const int cb = t.c0 + (threadIdx.x >> 5);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const bool rok = r < o.rows;
    for (int ti = 0; ti < o.nt; ++ti) {
        const CombTerm tm = terms[o.t0 + ti];
        const double* __restrict__ src = b.p[tm.sbuf] + tm.soff;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = cb + 8 * j;
            if (rok && c < o.cols) acc[j] = fma(tm.coef, src[r + int64_t(c) * tm.lds], acc[j]);
        }
    }
    double* __restrict__ dst = b.p[o.dbuf] + o.doff;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = cb + 8 * j;
        if (rok && c < o.cols) dst[r + int64_t(c) * o.ldd] = acc[j];
    }
}

// ------------------------------------------------------------------------------------
// Krylov vector kernels
// ------------------------------------------------------------------------------------
constexpr int KMAX = 32;
struct VecPtrs {
    const double* p[KMAX];
};
constexpr int BLAS_THREADS = 256;
constexpr int BLAS_PARTS = 2 * 152;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int K>
__global__ void __launch_bounds__(BLAS_THREADS)
multi_dot_kernel(VecPtrs V, int kk, const double* __restrict__ w, int64_t n,
                 double* __restrict__ part) {
    double acc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = 0.0;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        const double x = w[i];
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (k < kk) acc[k] = fma(V.p[k][i], x, acc[k]);
    }
    __shared__ double red[BLAS_THREADS / 32][K];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double v = warp_sum(acc[k]);
        if (lane == 0) red[wid][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < kk) {
        double s = 0.0;
        for (int j = 0; j < BLAS_THREADS / 32; ++j) s += red[j][threadIdx.x];
        part[int64_t(threadIdx.x) * gridDim.x + blockIdx.x] = s;
    }
}

__global__ void finalize_dot_kernel(const double* __restrict__ part, int nparts, int kk,
                                    double* __restrict__ out) {
    // one warp per result, fixed summation order
    const int k = blockIdx.x;
    if (k >= kk) return;
    double s = 0.0;
    for (int j = threadIdx.x; j < nparts; j += 32) s += part[int64_t(k) * nparts + j];
    s = warp_sum(s);
    if (threadIdx.x == 0) out[k] = s;
}

__global__ void __launch_bounds__(BLAS_THREADS)
multi_axpy_kernel(double* __restrict__ w, VecPtrs V, int kk, const double* __restrict__ h,
                  double sign, int64_t n) {
    __shared__ double hs[KMAX];
    if (threadIdx.x < kk) hs[threadIdx.x] = sign * h[threadIdx.x];
    __syncthreads();
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        double x = w[i];
        for (int k = 0; k < kk; ++k) x = fma(hs[k], V.p[k][i], x);
        w[i] = x;
    }
}

__global__ void __launch_bounds__(BLAS_THREADS)
scale_into_kernel(double* __restrict__ dst, const double* __restrict__ src,
                  const double* __restrict__ denom_sq, double hscale, int64_t n) {
    double s = hscale;
    if (denom_sq) s = hscale / sqrt(*denom_sq);
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        dst[i] = src[i] * s;
}

__global__ void __launch_bounds__(BLAS_THREADS)
lincomb_kernel(double* __restrict__ dst, VecPtrs V, int kk, const double* __restrict__ coef,
               int64_t n) {
    __shared__ double cs[KMAX];
    if (threadIdx.x < kk) cs[threadIdx.x] = coef[threadIdx.x];
    __syncthreads();
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        double x = 0.0;
        for (int k = 0; k < kk; ++k) x = fma(cs[k], V.p[k][i], x);
        dst[i] = x;
    }
}

// One fused Gram-Schmidt pass over a Krylov residual w:
//   (optional)  w += sign * sum_k hin[k] V_k
//   (optional)  out[k] = V_k . w   for k < kk          (with the updated w)
//   (optional)  out[kk or 0] = w . w
// Partial sums of every block go to `part`; the last block to finish (atomic ticket)
// adds them in block order, so results are deterministic, and resets the ticket.
template <int K>
__global__ void __launch_bounds__(BLAS_THREADS)
gs_pass_kernel(VecPtrs V, int kk, double* __restrict__ w, const double* __restrict__ hin,
               double sign, int64_t n, int dots, int norm, double* __restrict__ part,
               double* __restrict__ out, unsigned* __restrict__ ticket) {
    __shared__ double hs[KMAX];
    __shared__ double red[BLAS_THREADS / 32][K + 1];
    __shared__ int last;
    if (hin && threadIdx.x < kk) hs[threadIdx.x] = sign * hin[threadIdx.x];
    __syncthreads();
    double acc[K + 1];
#pragma unroll
    for (int k = 0; k <= K; ++k) acc[k] = 0.0;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        double x = w[i];
        if (hin) {
            for (int k = 0; k < kk; ++k) x = fma(hs[k], V.p[k][i], x);
            w[i] = x;
        }
        if (dots) {
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (k < kk) acc[k] = fma(V.p[k][i], x, acc[k]);
        }
        if (norm) acc[K] = fma(x, x, acc[K]);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nres = (dots ? kk : 0) + (norm ? 1 : 0);
#pragma unroll
    for (int k = 0; k <= K; ++k) {
        const double v = warp_sum(acc[k]);
        if (lane == 0) red[wid][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < nres) {
        const int src = (dots && threadIdx.x < kk) ? threadIdx.x : K;
        double sum = 0.0;
        for (int j = 0; j < BLAS_THREADS / 32; ++j) sum += red[j][src];
        part[int64_t(threadIdx.x) * gridDim.x + blockIdx.x] = sum;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int j = wid; j < nres; j += BLAS_THREADS / 32) {
        double sum = 0.0;
        for (int bb = lane; bb < (int)gridDim.x; bb += 32)
            sum += reinterpret_cast<volatile double*>(part)[int64_t(j) * gridDim.x + bb];
        sum = warp_sum(sum);
        if (lane == 0) out[j] = sum;
    }
    if (threadIdx.x == 0) *ticket = 0u;
}

__global__ void __launch_bounds__(BLAS_THREADS)
block_dot_kernel(const BlockDot* __restrict__ descs, double* __restrict__ out) {
    __shared__ double red[BLAS_THREADS / 32];
    const BlockDot D = descs[blockIdx.x];
    const int64_t n = int64_t(D.rows) * D.cols;
    double acc = 0.0;
    for (int64_t e = threadIdx.x; e < n; e += blockDim.x) {
        const int r = int(e % D.rows), c = int(e / D.rows);
        acc = fma(D.x[r + int64_t(c) * D.ldx], D.y[r + int64_t(c) * D.ldy], acc);
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < BLAS_THREADS / 32; ++w) s += red[w];
        out[blockIdx.x] = s;
    }
}

int grid_for(int64_t n) {
    int64_t g = (n + BLAS_THREADS - 1) / BLAS_THREADS;
    if (g > BLAS_PARTS) g = BLAS_PARTS;
    if (g < 1) g = 1;
    return int(g);
}

VecPtrs make_ptrs(const double* const* V, int K) {
    VecPtrs p{};
    TN_REQUIRE(K <= KMAX, "too many Krylov vectors for one kernel (max 32)");
    for (int k = 0; k < K; ++k) p.p[k] = V[k];
    return p;
}
}  // namespace

void launch_gemm_f64(const GemmPlan& p, const Bases& b, cudaStream_t s) {
    if (p.tiles.empty()) return;
    auto* kernel = p.tile_n == 32   ? gemm_f64_kernel<32, 32>
                   : p.tile_n == 16 ? gemm_f64_kernel<16, 16>
                                    : gemm_f64_kernel<16, 8>;
    kernel<<<unsigned(p.tiles.size()), GEMM_THREADS, 0, s>>>(
        p.dsegs.as<Seg>(), p.dtasks.as<Task>(), p.dtiles.as<Tile>(), b);
    TN_CUDA(cudaGetLastError());
    count_launch();
}

void launch_combine(const CombPlan& p, const Bases& b, cudaStream_t s) {
    if (p.tiles.empty()) return;
    combine_kernel<<<unsigned(p.tiles.size()), 256, 0, s>>>(
        p.douts.as<CombOut>(), p.dterms.as<CombTerm>(), p.dtiles.as<CombTile>(), b);
    TN_CUDA(cudaGetLastError());
    count_launch();
}

int blas_nparts() { return BLAS_PARTS; }

void launch_block_dots(const BlockDot* d, int n, double* out, cudaStream_t s) {
    if (n <= 0) return;
    block_dot_kernel<<<n, BLAS_THREADS, 0, s>>>(d, out);
    TN_CUDA(cudaGetLastError());
    count_launch();
}

void launch_multi_dot(const double* const* V, int K, const double* w, int64_t n,
                      double* part, double* out, cudaStream_t s) {
    if (K <= 0) return;
    VecPtrs P = make_ptrs(V, K);
    const int g = BLAS_PARTS;  // fixed part count: deterministic, finalize reads g parts
    if (K <= 4)
        multi_dot_kernel<4><<<g, BLAS_THREADS, 0, s>>>(P, K, w, n, part);
    else if (K <= 8)
        multi_dot_kernel<8><<<g, BLAS_THREADS, 0, s>>>(P, K, w, n, part);
    else if (K <= 16)
        multi_dot_kernel<16><<<g, BLAS_THREADS, 0, s>>>(P, K, w, n, part);
    else
        multi_dot_kernel<32><<<g, BLAS_THREADS, 0, s>>>(P, K, w, n, part);
    TN_CUDA(cudaGetLastError());
    count_launch();
    finalize_dot_kernel<<<K, 32, 0, s>>>(part, g, K, out);
    TN_CUDA(cudaGetLastError());
    count_launch();
    count_krylov_bytes(int64_t(K + 1) * n * 8);
}

void launch_multi_axpy(double* w, const double* const* V, int K, const double* h, double sign,
                       int64_t n, cudaStream_t s) {
    if (K <= 0 || n <= 0) return;
    multi_axpy_kernel<<<grid_for(n), BLAS_THREADS, 0, s>>>(w, make_ptrs(V, K), K, h, sign, n);
    TN_CUDA(cudaGetLastError());
    count_launch();
    count_krylov_bytes(int64_t(K + 2) * n * 8);
}

void launch_gs_pass(const double* const* V, int K, double* w, const double* hin, double sign,
                    int64_t n, bool dots, bool norm, double* part, double* out, unsigned* ticket,
                    cudaStream_t s) {
    VecPtrs P = K > 0 ? make_ptrs(V, K) : VecPtrs{};
    const int g = BLAS_PARTS;
    const int d = dots ? 1 : 0, nm = norm ? 1 : 0;
    if (K <= 4)
        gs_pass_kernel<4><<<g, BLAS_THREADS, 0, s>>>(P, K, w, hin, sign, n, d, nm, part, out, ticket);
    else if (K <= 8)
        gs_pass_kernel<8><<<g, BLAS_THREADS, 0, s>>>(P, K, w, hin, sign, n, d, nm, part, out, ticket);
    else if (K <= 16)
        gs_pass_kernel<16><<<g, BLAS_THREADS, 0, s>>>(P, K, w, hin, sign, n, d, nm, part, out, ticket);
    else
        gs_pass_kernel<32><<<g, BLAS_THREADS, 0, s>>>(P, K, w, hin, sign, n, d, nm, part, out, ticket);
    TN_CUDA(cudaGetLastError());
    count_launch();
    count_krylov_bytes(int64_t(1 + ((hin || dots) ? K : 0) + (hin ? 1 : 0)) * n * 8);
}

void launch_scale_into(double* dst, const double* src, const double* denom_sq,
                       double host_scale, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    scale_into_kernel<<<grid_for(n), BLAS_THREADS, 0, s>>>(dst, src, denom_sq, host_scale, n);
    TN_CUDA(cudaGetLastError());
    count_launch();
    count_krylov_bytes(2 * n * 8);
}

void launch_lincomb(double* dst, const double* const* V, int K, const double* coef, int64_t n,
                    cudaStream_t s) {
    if (n <= 0) return;
    lincomb_kernel<<<grid_for(n), BLAS_THREADS, 0, s>>>(dst, make_ptrs(V, K), K, coef, n);
    TN_CUDA(cudaGetLastError());
    count_launch();
    count_krylov_bytes(int64_t(K + 1) * n * 8);
}

}  // namespace tn
