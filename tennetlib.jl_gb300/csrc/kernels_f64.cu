// FP64 kernels of the sweep engine:
//  * grouped block-sparse GEMM (CUDA-core DFMA) -- the FP64 GPU path of every contraction
//    of the two-site effective Hamiltonian and of the environment updates;
//  * block linear combination -- the MPO step between the two GEMM stages;
//  * Krylov vector kernels (Gram-Schmidt passes, multi-axpy, scaling, linear combinations) with
//    warp-shuffle reductions and a deterministic two-stage finalisation.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "reduce.cuh"
#include "tn_internal.h"

namespace tn {

// ------------------------------------------------------------------------------------
// grouped GEMM: 128 threads per TM x TN output tile, one thread adds its outputs along the
// whole k range of the task
//
// Bound by the FP64 pipe: a warp-wide DFMA holds its SM sub-partition for 64 clocks (measured:
// 1.7 FMA per clock and SM with one warp per sub-partition, 2.0 at most; DMMA the same), so a
// multiplication by padding costs as much as a real one, while loads, shared memory and issue
// slots are nearly free (launches of a few us are bound by the latency of their loads: a 20-site
// cylinder's 6 to 17 us launches have the pipe 8 to 17% active).  Hence small tiles of 8 x 4 warp patches (patches outside the block
// are skipped), k taken to its exact end, the segments of a task run together into one k range
// (four 4-long segments fill a 16-deep chunk), four warps so that every sub-partition works,
// and the next chunk's loads in flight during the products.  Each output is one chain of fused
// multiply-adds in segment order.  On the 64 x 64 x 16 tiles of 256 threads that this replaced
// a 4 x 4 x 4 block took 16 us of multiplications by zeros.
// The tile is GemmPlan::prepare's choice.  Measured, whole calls in FP64: DMRG run of a
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
               const CombTile* __restrict__ tiles, const __grid_constant__ Bases b) {
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

__global__ void __launch_bounds__(BLAS_THREADS)
multi_axpy_kernel(double* __restrict__ w, const __grid_constant__ VecPtrs V, int kk, const double* __restrict__ h,
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

// dst_j = sum_k c[j][k] V_k for several outputs in one launch, the coefficients as kernel
// arguments (a Ritz restart of Lanczos: one upload, launch and host wait per vector before)
struct LinArgs {
    double* dst[KMAX];
    double c[KMAX][KMAX];
};
__global__ void __launch_bounds__(BLAS_THREADS)
lincomb_multi_kernel(const __grid_constant__ LinArgs a, const __grid_constant__ VecPtrs V, int nd,
                     int kk, int64_t n) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        for (int j = 0; j < nd; ++j) {
            double x = 0.0;
            for (int k = 0; k < kk; ++k) x = fma(a.c[j][k], V.p[k][i], x);
            a.dst[j][i] = x;
        }
}

// dst = sum_k (re_k + i im_k) V_k on planar complex vectors of nc values per plane, real c:
// the products of the imaginary parts enter as dst_re -= sum im V_im, dst_im += sum im V_re
struct CLinArgs {
    double re[KMAX], im[KMAX];
};
__global__ void __launch_bounds__(BLAS_THREADS)
lincomb_complex_kernel(double* __restrict__ dst, const __grid_constant__ CLinArgs a,
                       const __grid_constant__ VecPtrs V, int kk, int64_t nc) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nc; i += stride) {
        double xr = 0.0, xi = 0.0, wr = 0.0, wi = 0.0;
        for (int k = 0; k < kk; ++k) {
            const double vr = V.p[k][i], vi = V.p[k][i + nc];
            xr = fma(a.re[k], vr, xr);
            xi = fma(a.re[k], vi, xi);
            wr = fma(a.im[k], vr, wr);
            wi = fma(a.im[k], vi, wi);
        }
        dst[i] = xr - wi;
        dst[i + nc] = xi + wr;
    }
}

// results for the host: `values` in mapped pinned memory, then the sequence number
__device__ __forceinline__ void host_post(const HostPost& p) {
    __threadfence_system();
    if (threadIdx.x == 0) *reinterpret_cast<volatile unsigned long long*>(p.flag) = p.seq;
}

// One Gram-Schmidt pass over a Krylov residual w:
//   (optional)  w += sign * sum_k hin[k] V_k
//   out[k] = V_k . w for k < kk (with the updated w), or with `norm` out[0] = w . w
// A block sums 256 elements (and those a whole grid of BLAS_PARTS blocks further on) over warps
// and then over its warps; the last block to finish (atomic ticket) adds the blocks' sums in
// block order, so results are deterministic and independent of the grid, which covers n only.
// With a host post the last block also hands over h1 = post_h1[0..kk), hin and its results.
//
// Bound by the FP64 pipe and latency at the sizes of small and middle bonds.  Before, 304
// blocks of any n and plain butterflies took 10.2 (4 vectors) and 13.5 us (8 vectors) a pass.
template <int C>
__global__ void __launch_bounds__(BLAS_THREADS)
gs_pass_kernel(const __grid_constant__ VecPtrs V, int kk, double* __restrict__ w,
               const double* __restrict__ hin, double sign, int64_t n, int norm,
               double* __restrict__ part, double* __restrict__ out,
               unsigned* __restrict__ ticket, const double* __restrict__ post_h1,
               HostPost post) {
    __shared__ double hs[KMAX];
    __shared__ double red[BLAS_THREADS / 32][C];
    __shared__ int last;
    if (hin && threadIdx.x < kk) hs[threadIdx.x] = sign * hin[threadIdx.x];
    __syncthreads();
    double acc[C];
#pragma unroll
    for (int k = 0; k < C; ++k) acc[k] = 0.0;
    const int64_t stride = int64_t(BLAS_PARTS) * BLAS_THREADS;
    for (int64_t i = int64_t(blockIdx.x) * BLAS_THREADS + threadIdx.x; i < n; i += stride) {
        double x = w[i];
        if (hin) {
            for (int k = 0; k < kk; ++k) x = fma(hs[k], V.p[k][i], x);
            w[i] = x;
        }
        if (norm) {
            acc[0] = fma(x, x, acc[0]);
        } else {
#pragma unroll
            for (int k = 0; k < C; ++k)
                if (k < kk) acc[k] = fma(V.p[k][i], x, acc[k]);
        }
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nres = norm ? 1 : kk;
    const double v = warp_sum_multi<C>(acc, lane);
    if (warp_sum_owner<C>(lane)) red[wid][warp_sum_index<C>(lane)] = v;
    __syncthreads();
    if (threadIdx.x < nres) {
        double sum = 0.0;
#pragma unroll
        for (int j = 0; j < BLAS_THREADS / 32; ++j) sum += red[j][threadIdx.x];
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
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)  // the butterfly's steps that add no zeros
            if (o < (int)gridDim.x) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) {
            out[j] = sum;
            if (post.values) post.values[GS_NORM + j] = sum;
        }
    }
    if (threadIdx.x == 0) *ticket = 0u;
    if (post.values) {
        if (threadIdx.x < kk && post_h1) {
            post.values[threadIdx.x] = post_h1[threadIdx.x];
            post.values[GS_H2 + threadIdx.x] = hin[threadIdx.x];
        }
        if (threadIdx.x == 0 && post.start) post.values[GS_START] = *post.start;
        __syncthreads();
        host_post(post);
    }
}

// The whole double Gram-Schmidt step of a short residual in one launch:
//   h1 = V^T w, w -= V h1, h2 = V^T w, w -= V h2, |w|^2, next = w / |w|
// A cluster of CL CTAs keeps w and the basis in registers, each thread one element of up to
// gs2_parts(C) parts of 256 elements; the parts' sums meet through distributed shared memory.  A
// ninth warp posts the results to the host while the others form the next vector.  The sums are
// formed in gs_pass_kernel's order (element, warp, the part's eight warps, parts by lane; adds
// of zeros left out), so the results are the same bits as its three passes.
// Bound by chains of FP64 operations (65 clocks each, the reciprocal root 2000) and the barriers.
// Three passes and the scaling of the next vector were four launches and at least 34 us for any
// n; this is one of 9 (n = 250, K = 1) to 25 us (n = 8000, K = 4; 12-site DMRG run 71 -> 47 ms, 64-site run in split precision
// 565 -> 440 ms, both with the results posted to the host).  Vectors too long for it (gs2_cluster)
// take the passes, which spread the parts over all SMs.
constexpr int GS2_THREADS = BLAS_THREADS + 32;
constexpr int gs2_parts(int C) { return C <= 4 ? 4 : C == 8 ? 3 : C == 16 ? 2 : 1; }
template <int C>
__global__ void __launch_bounds__(GS2_THREADS, 1)
gs2_kernel(const __grid_constant__ VecPtrs V, int kk, double* __restrict__ w,
           double* __restrict__ next, int n, double* __restrict__ out, HostPost post) {
    namespace cg = cooperative_groups;
    constexpr int PARTS = gs2_parts(C), WARPS = BLAS_THREADS / 32;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ double red[WARPS][C];
    __shared__ double sums[3][PARTS][C];  // this CTA's parts, one array per phase
    __shared__ double hs[3][C];           // h1, h2, |w|^2
    const int CL = int(cl.num_blocks()), rank = int(cl.block_rank());
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int P = (n + BLAS_THREADS - 1) / BLAS_THREADS;  // part p: CTA p % CL, slot p / CL
    double x[PARTS], v[PARTS][C];
#pragma unroll
    for (int s = 0; s < PARTS; ++s) {
        const int i = (s * CL + rank) * BLAS_THREADS + int(threadIdx.x);
        const bool in = wid < WARPS && i < n;
        x[s] = in ? w[i] : 0.0;
#pragma unroll
        for (int k = 0; k < C; ++k) v[s][k] = in && k < kk ? V.p[k][i] : 0.0;
    }
    // sum of the part's warps for every result (a barrier before and after)
    auto part_sum = [&](int f, int s, double r, int nres, bool owner, int idx) {
        if (wid < WARPS && owner) red[wid][idx] = r;
        __syncthreads();
        if (threadIdx.x < nres) {
            const int live = (n - (s * CL + rank) * BLAS_THREADS + 31) / 32;  // warps with elements
            double sum = red[0][threadIdx.x];
#pragma unroll
            for (int j = 1; j < WARPS; ++j)
                if (j < live) sum += red[j][threadIdx.x];
            sums[f][s][threadIdx.x] = sum;
        }
        __syncthreads();
    };
    // sums over the parts of phase f for every result, into hs[f] (all CTAs alike)
    auto finish = [&](int f, int nres) {
        if (P == 1) {
            if (threadIdx.x < nres) hs[f][threadIdx.x] = sums[f][0][threadIdx.x];
            __syncthreads();
            return;
        }
        cl.sync();
        if (wid < WARPS)
            for (int j = wid; j < nres; j += WARPS) {
                double s = 0.0;
                if (lane < P) s = cl.map_shared_rank(&sums[f][lane / CL][j], lane % CL)[0];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)  // the butterfly's steps that add no zeros
                    if (o < P) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) hs[f][j] = s;
            }
        __syncthreads();
    };
#pragma unroll
    for (int f = 0; f < 2; ++f) {
#pragma unroll
        for (int s = 0; s < PARTS; ++s) {
            if (s * CL + rank >= P) continue;
            double acc[C];
#pragma unroll
            for (int k = 0; k < C; ++k) acc[k] = k < kk ? v[s][k] * x[s] : 0.0;
            const double r = warp_sum_multi<C>(acc, lane);
            part_sum(f, s, r, kk, warp_sum_owner<C>(lane), warp_sum_index<C>(lane));
        }
        finish(f, kk);
#pragma unroll
        for (int s = 0; s < PARTS; ++s) {
            if (s * CL + rank >= P) continue;
#pragma unroll
            for (int k = 0; k < C; ++k)
                if (k < kk) x[s] = fma(-hs[f][k], v[s][k], x[s]);
        }
    }
#pragma unroll
    for (int s = 0; s < PARTS; ++s) {
        if (s * CL + rank >= P) continue;
        part_sum(2, s, warp_sum(x[s] * x[s]), 1, lane == 0, 0);
    }
    finish(2, 1);
    if (wid < WARPS) {
        const double scale = next ? 1.0 / sqrt(hs[2][0]) : 0.0;
#pragma unroll
        for (int s = 0; s < PARTS; ++s) {
            const int i = (s * CL + rank) * BLAS_THREADS + int(threadIdx.x);
            if (s * CL + rank < P && i < n) {
                w[i] = x[s];
                if (next) next[i] = x[s] * scale;
            }
        }
        if (rank == 0 && threadIdx.x < kk) {
            out[threadIdx.x] = hs[0][threadIdx.x];
            out[GS_H2 + threadIdx.x] = hs[1][threadIdx.x];
            if (threadIdx.x == 0) out[GS_NORM] = hs[2][0];
        }
    } else if (rank == 0) {
        if (lane < kk) {
            post.values[lane] = hs[0][lane];
            post.values[GS_H2 + lane] = hs[1][lane];
        }
        if (lane == 0) {
            post.values[GS_NORM] = hs[2][0];
            if (post.start) post.values[GS_START] = *post.start;
        }
        __syncwarp();
        __threadfence_system();
        if (lane == 0) *reinterpret_cast<volatile unsigned long long*>(post.flag) = post.seq;
    }
    if (P > 1) cl.sync();  // the other CTAs read this one's sums until here
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
    if (p.tasks.empty()) return;
    p.prepare(s);
    if (p.ntiles == 0) return;
    auto* kernel = p.tile_n == 32   ? gemm_f64_kernel<32, 32>
                   : p.tile_n == 16 ? gemm_f64_kernel<16, 16>
                                    : gemm_f64_kernel<16, 8>;
    kernel<<<unsigned(p.ntiles), GEMM_THREADS, 0, s>>>(
        p.tab.at<Seg>(p.osegs), p.tab.at<Task>(p.otasks), p.tab.at<Tile>(p.otiles), b);
    TN_CUDA(cudaGetLastError());
    count_launch();
}

void launch_combine(const CombPlan& p, const Bases& b, cudaStream_t s) {
    if (p.tiles.empty()) return;
    combine_kernel<<<unsigned(p.tiles.size()), 256, 0, s>>>(
        p.tab.at<CombOut>(p.oouts), p.tab.at<CombTerm>(p.oterms), p.tab.at<CombTile>(p.otiles), b);
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
                      double* part, double* out, unsigned* ticket, cudaStream_t s) {
    if (K <= 0) return;
    launch_gs_pass(V, K, const_cast<double*>(w), nullptr, 0.0, n, false, part, out, ticket, s);
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
                    int64_t n, bool norm, double* part, double* out, unsigned* ticket,
                    cudaStream_t s, const double* post_h1, const HostPost& post) {
    VecPtrs P = K > 0 ? make_ptrs(V, K) : VecPtrs{};
    const int g = grid_for(n);
    const int nm = norm ? 1 : 0, nres = norm ? 1 : K;
    auto* kernel = nres <= 1    ? gs_pass_kernel<1>
                   : nres <= 2  ? gs_pass_kernel<2>
                   : nres <= 4  ? gs_pass_kernel<4>
                   : nres <= 8  ? gs_pass_kernel<8>
                   : nres <= 16 ? gs_pass_kernel<16>
                                : gs_pass_kernel<32>;
    kernel<<<g, BLAS_THREADS, 0, s>>>(P, K, w, hin, sign, n, nm, part, out, ticket, post_h1, post);
    TN_CUDA(cudaGetLastError());
    count_launch();
    count_krylov_bytes(int64_t(1 + ((hin || !norm) ? K : 0) + (hin ? 1 : 0)) * n * 8);
}

// CTAs of gs2_kernel's cluster for n elements and K vectors, 0: too long for it.  A CTA's parts
// come one after the other, so the line is where they take as long as the passes (back-to-back
// launches): K = 4: 24.6 against 25.6 us at four parts per CTA (n = 8000) and 33 against 27 at
// six; K = 8: 21.5 against 27.7 at two and 33 against 29 at four; K = 16: 29 against 34 at two
// and 49 against 35 at four; K = 24: 27 against 43 at one and 45 against 45 at two.
static int gs2_cluster(int64_t n, int K) {
    const int64_t P = (n + BLAS_THREADS - 1) / BLAS_THREADS;
    const int parts = gs2_parts(K <= 4 ? 4 : K <= 8 ? 8 : K <= 16 ? 16 : 32);
    if (P < 1 || P > 8 * parts) return 0;
    int c = 1;
    while (c < 8 && c < P) c *= 2;
    return c;
}

void launch_gs2(const double* const* V, int K, double* w, double* next, int64_t n, double* part,
                double* out, unsigned* ticket, const HostPost& post, cudaStream_t s) {
    const int c = gs2_cluster(n, K);
    if (c == 0) {
        launch_gs_pass(V, K, w, nullptr, 0.0, n, false, part, out, ticket, s);
        launch_gs_pass(V, K, w, out, -1.0, n, false, part, out + GS_H2, ticket, s);
        launch_gs_pass(V, K, w, out + GS_H2, -1.0, n, true, part, out + GS_NORM, ticket, s, out, post);
        if (next) launch_scale_into(next, w, out + GS_NORM, 1.0, n, s);
        return;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(c));
    cfg.blockDim = dim3(GS2_THREADS);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = unsigned(c);
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    auto* kernel = K <= 1    ? gs2_kernel<1>
                   : K <= 2  ? gs2_kernel<2>
                   : K <= 4  ? gs2_kernel<4>
                   : K <= 8  ? gs2_kernel<8>
                   : K <= 16 ? gs2_kernel<16>
                             : gs2_kernel<32>;
    TN_CUDA(cudaLaunchKernelEx(&cfg, kernel, make_ptrs(V, K), K, w, next, int(n), out, post));
    count_launch();
    count_krylov_bytes(int64_t(2 * K + 2 + (next ? 1 : 0)) * n * 8);
}

void launch_scale_into(double* dst, const double* src, const double* denom_sq,
                       double host_scale, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    scale_into_kernel<<<grid_for(n), BLAS_THREADS, 0, s>>>(dst, src, denom_sq, host_scale, n);
    TN_CUDA(cudaGetLastError());
    count_launch();
    count_krylov_bytes(2 * n * 8);
}

void launch_lincomb(double* const* dst, int nd, const double* const* V, int K,
                    const double* coef, int64_t n, cudaStream_t s) {
    if (n <= 0 || nd <= 0) return;
    TN_REQUIRE(nd <= KMAX, "too many linear combinations for one kernel");
    LinArgs a;
    for (int j = 0; j < nd; ++j) {
        a.dst[j] = dst[j];
        for (int k = 0; k < K; ++k) a.c[j][k] = coef[j * K + k];
    }
    lincomb_multi_kernel<<<grid_for(n), BLAS_THREADS, 0, s>>>(a, make_ptrs(V, K), nd, K, n);
    TN_CUDA(cudaGetLastError());
    count_launch();
    count_krylov_bytes(int64_t(K + 1) * nd * n * 8);
}

void launch_lincomb_complex(double* dst, const double* const* V, int K, const double* re,
                            const double* im, int64_t nc, cudaStream_t s) {
    if (nc <= 0) return;
    CLinArgs a;
    VecPtrs P = make_ptrs(V, K);
    for (int k = 0; k < K; ++k) {
        a.re[k] = re[k];
        a.im[k] = im[k];
    }
    lincomb_complex_kernel<<<grid_for(nc), BLAS_THREADS, 0, s>>>(dst, a, P, K, nc);
    TN_CUDA(cudaGetLastError());
    count_launch();
    count_krylov_bytes(int64_t(K + 1) * 2 * nc * 8);
}

}  // namespace tn
