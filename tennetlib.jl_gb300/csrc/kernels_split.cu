// Split-precision grouped GEMM on the 5th-generation tensor cores (tcgen05, sm_103a):
// FP64 operands are cut into bf16 slices (Ozaki scheme I: Ozaki, Ogita, Oishi & Rump,
// Numer. Algorithms 59, 2012) whose pairwise products are exact in the FP32 tensor-core
// accumulator; the partial sums are combined in double-float registers and rescaled to
// FP64, so the result carries ~8*s+1 significant bits per operand element.
//
//  * pack kernel: for every row of op(A) (every column of op(B)) a power-of-two exponent
//    E with max|x| < 2^E; x * 2^(8s-E) rounded to an integer X (|X| <= 2^(8s)) is written
//    as balanced base-256 digits d_1..d_s (|d_1| <= 256, |d_i| <= 128), stored as the
//    bf16 values d_i * 2^(-8(i-1)) in the canonical UMMA K-major SWIZZLE_128B tile layout
//    (8-row x 128-byte atoms, 16-byte chunks XOR-ed with the row index), one contiguous
//    tile per (row tile, k tile, slice), so that a 1D bulk copy moves it to shared memory;
//  * MMA kernel: persistent, one CTA per SM, warp-specialised (warp 0 producer, warp 1
//    MMA issuer + TMEM owner, warps 2-9 epilogue: lane quadrant warp % 4, column half
//    (warp - 2) / 4).  For each 128 x 64 output tile and each
//    k tile the slice pairs (i, j) with i + j <= s + 1 are multiplied into four TMEM
//    accumulators: level 2, 3, 4 (exact: integer multiples of 2^-8(l-2) below 2^24 for a
//    chunk of 128 k) and levels >= 5 (scaled, rounded far below the result's precision).
//    Every chunk of two k tiles the epilogue drains the accumulators (double-buffered in
//    TMEM) into (hi, lo) FP32 pairs with error-free additions; at the end of the tile the
//    pair is rescaled by 2^(E_row + E_col - 16) in FP64 and stored.
// Small blocks (a chi = 50 bond has blocks of 15 to 30 rows) use a corner of their 128 x 64 tile
// and 64-deep k tiles: only the 8-row atoms that hold rows are copied, only the 16-deep steps
// with valid k and the columns of the block are multiplied, only its columns and row quadrants
// are drained and converted, each as before to the bit (22.9 -> 15.6 us per launch there, with
// the packs 69 -> 44 us per H_eff product; 64-site DMRG run 440 -> 360 ms).
// Every mbarrier wait is bounded (about one second); a wait that gives up sets the error
// word, and all roles then drain with bounded waits, free TMEM and return.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "tn_internal.h"

namespace tn {
namespace {

constexpr int BM = 128;            // rows of an output tile (UMMA M)
constexpr int BN = 64;             // columns of an output tile (UMMA N)
constexpr int BKT = 64;            // k elements per tile (one 128-byte swizzle row of bf16)
constexpr int A_TILE = BM * BKT * 2;   // 16 KB
constexpr int B_TILE = BN * BKT * 2;   // 8 KB
constexpr int STAGE = A_TILE + B_TILE; // 24 KB
constexpr int NST = 8;             // ring stages (192 KB)
constexpr int KC = 2;              // k tiles per exact accumulation chunk
constexpr int NACC = 4;            // accumulators: level 2, 3, 4, >= 5
constexpr int TMEM_COLS = 512;     // 2 buffers x 4 accumulators x 64 columns
constexpr int THREADS = 320;       // 10 warps: producer, MMA, 8 epilogue
constexpr long long WAIT_LIMIT = 2000000000LL;  // clock cycles (about one second)

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait.  Returns false (and sets *err) when the limit passes or an error is
// already flagged.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err,
                                          volatile int* shared_err) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_try(bar, parity)) return true;
        if (*shared_err) return false;
        if (clock64() - t0 > WAIT_LIMIT) {
            *shared_err = 1;
            atomicExch(err, 1);
            return false;
        }
    }
}

// the error flag as the whole warp sees it (lanes may read it at different times)
__device__ __forceinline__ bool warp_err(volatile int* shared_err) {
    return __any_sync(0xffffffffu, *shared_err != 0);
}

// Bounded wait used only to drain before exit (no error bookkeeping).
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try(bar, parity))
        if (clock64() - t0 > WAIT_LIMIT) return;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The whole warp runs the issuing code on values that are uniform to the compiler, with one
// lane's predicate on the instructions: descriptors then live in uniform registers.  Issued from a
// one-lane branch with per-thread values, each product took 230 clocks whatever its width
// (measured alone: 71 from a branch, 39 for 16 columns, 48 for 64 and 64 for 128 this way), and a
// k tile of one 16-deep step 5700 clocks instead of 2100.
__device__ __forceinline__ uint32_t elect_lane() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(r));
    return r;
}

// (the copies of a stage, like the products, are issued by a whole warp with one lane's predicate)
// a value that all lanes have alike, known as such to the compiler
__device__ __forceinline__ uint32_t uniform(uint32_t x) { return __shfl_sync(0xffffffffu, x, 0); }

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes, uint32_t lead) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n"
        " @q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}\n" ::"r"(smem_u32(bar)),
        "r"(bytes), "r"(lead)
        : "memory");
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes,
                                         uint64_t* bar, uint32_t lead) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %4, 0;\n"
        " @q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
        "}\n" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar)), "r"(lead)
        : "memory");
}

// K-major SWIZZLE_128B shared-memory matrix descriptor (start address, LBO = 16 B,
// SBO = 1024 B between 8-row groups, descriptor version 1, layout type 2 = 128B swizzle):
// low and high 32 bits; the start address, in 16-byte units, is the low word's lower half
__device__ __forceinline__ uint32_t sdesc_lo(uint32_t saddr) {
    return ((saddr & 0x3FFFF) >> 4) | (1u << 16);
}
constexpr uint32_t SDESC_HI = (1024 >> 4) | (1u << 14) | (2u << 29);

// Instruction descriptor of kind::f16: D = F32, A = B = BF16, both K-major, N = 64, M = 128.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo,
                                         uint32_t idesc, bool accumulate, uint32_t lead) {
    asm volatile(
        "{\n .reg .pred p, q;\n .reg .b64 a, b;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %6, 0;\n"
        " mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(uint32_t(accumulate)), "r"(SDESC_HI), "r"(lead));
}

__device__ __forceinline__ void mma_commit(uint64_t* bar, uint32_t lead) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(
            smem_u32(bar)),
        "r"(lead)
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
          "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]),
          "=f"(v[14]), "=f"(v[15])
        : "r"(taddr));
}

// waits for the loads above; the values pass through it, so that none is read before
__device__ __forceinline__ void tmem_wait(float (&v)[NACC][16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int l = 0; l < NACC; ++l)
#pragma unroll
        for (int c = 0; c < 16; ++c) asm volatile("" : "+f"(v[l][c]));
}

// error-free addition of a into (hi, lo) (Knuth's TwoSum, lo collects the rounding errors)
__device__ __forceinline__ void df_add(float& hi, float& lo, float a) {
    const float s = hi + a;
    const float bp = s - hi;
    const float e = (hi - (s - bp)) + (a - bp);
    hi = s;
    lo += e;
}

__device__ __forceinline__ double pow2(int e) {
    return __longlong_as_double(static_cast<long long>(1023 + e) << 52);
}

// x, for arithmetic that has to stay in its branch: the compiler else takes it out and selects
// between the results, and an FP64 operation holds the pipe for 64 clocks whether used or not
__device__ __forceinline__ float branch_only(float x) {
    asm volatile("" : "+f"(x));
    return x;
}
__device__ __forceinline__ double branch_only(double x) {
    asm volatile("" : "+d"(x));
    return x;
}

// double(x) of a zero or normal number, exactly, on the integer pipe (a conversion holds the FP64
// pipe as long as an add does)
__device__ __forceinline__ bool plain(float x) {
    const unsigned a = __float_as_uint(x) & 0x7fffffffu;
    return a == 0u || a - 0x00800000u < 0x7f000000u;
}
__device__ __forceinline__ double widen(float x) {
    const unsigned u = __float_as_uint(x), a = u & 0x7fffffffu;
    const unsigned hi = a ? (a >> 3) + 0x38000000u : 0u;
    return __hiloint2double(int(hi | (u & 0x80000000u)), int(u << 29));
}

// v * 2^e, exactly the product, on the exponent field: v zero, or v and the result normal
__device__ __forceinline__ double scale2(double v, int e) {
    const int hi = __double2hiint(v), lo = __double2loint(v);
    return __hiloint2double(((hi & 0x7fffffff) | lo) == 0 ? hi : hi + (e << 20), lo);
}

// ------------------------------------------------------------------------------------
// pack kernels.  Only what the MMA kernel copies and multiplies is written: rows up to the
// next multiple of 8 (one swizzle atom), and of a k tile the 16-deep MMA steps that hold valid
// k (split_ksteps; a charge block of 14 x 14 fills 16 rows and one step of four, a sixteenth of
// its A tile).
// ------------------------------------------------------------------------------------
constexpr int PACK_THREADS = 256, PACK_MAXTHREADS = 1024;
constexpr int PACK_ROWS = 8;

// 8-wide chunks of k tile t that are packed
__device__ __forceinline__ int pack_chunks(int t, int kvalid) {
    return t < SPLIT_KMASK ? 2 * ((kvalid + 15) / 16) : BKT / 8;
}

// EL elements of row r (k = EL pr ... of a k tile at tile0): balanced base-256 digits.
// x * 2^(8s - E) = sig * 2^(ex - 1075 + 8s - E), sig the 53-bit significand: the rounded
// integer is sig shifted right by sh = 1075 + E - 8s - ex (round half away from zero), integer
// pipe only.  mxb is the row's largest |x| as a bit pattern, 0 for an empty row.
template <int SL, int EL>
__device__ __forceinline__ void pack_digits(const long long (&v)[EL], unsigned long long mxb,
                                            int r, int pr, uint8_t* tile0, int tile_bytes) {
    const int E = mxb ? int((mxb >> 52) & 0x7ff) - 1022 : 0;
    const int base_sh = 1075 + E - 8 * SL;
    __nv_bfloat16 dig[SL][EL];
#pragma unroll
    for (int q = 0; q < EL; ++q) {
        long long X = 0;
        const int ex = int((v[q] >> 52) & 0x7ff);
        if (mxb && ex) {  // subnormals are far below the row scale: they round to 0
            const long long m = (v[q] & 0xfffffffffffffLL) | (1LL << 52);
            const int sh = base_sh - ex;
            long long a = 0;
            if (sh <= 0) a = m << (-sh);
            else if (sh < 63) a = (m + (1LL << (sh - 1))) >> sh;
            X = v[q] < 0 ? -a : a;
        }
#pragma unroll
        for (int i = SL - 1; i >= 1; --i) {
            int d = int(X & 255);
            if (d > 128) d -= 256;
            X = (X - d) >> 8;
            dig[i][q] = __float2bfloat16_rn(ldexpf(float(d), -8 * i));
        }
        dig[0][q] = __float2bfloat16_rn(float(X));
    }
    // swizzled position: 8-row atoms of 1024 bytes, 16-byte chunks XOR-ed with the row
    const int ch = pr * EL / 8;
    const int off = (r >> 3) * 1024 + (r & 7) * 128 + ((ch ^ (r & 7)) << 4) + pr * EL % 8 * 2;
    using W = typename std::conditional<EL == 8, uint4, unsigned>::type;
    static_assert(sizeof(W) == 2 * EL, "two or eight elements");
#pragma unroll
    for (int i = 0; i < SL; ++i) {
        W w;
        __builtin_memcpy(&w, dig[i], sizeof(W));
        *reinterpret_cast<W*>(tile0 + int64_t(i) * tile_bytes + off) = w;
    }
}

// EL elements from k = EL ch on (zeros beyond the rows and valid k) and their largest |x|
template <int EL>
__device__ __forceinline__ unsigned long long pack_load(long long (&v)[EL], const KTileSrc& ks,
                                                        const Bases& b, int row, bool live, int ch) {
    const long long* x = reinterpret_cast<const long long*>(b.p[ks.buf] + ks.off) +
                         int64_t(row) * ks.sr;
    unsigned long long mx = 0ull;
#pragma unroll
    for (int q = 0; q < EL; ++q) {
        const int k = ch * EL + q;
        v[q] = live && k < ks.kvalid ? x[int64_t(k) * ks.sk] : 0ll;
        const unsigned long long a = (unsigned long long)v[q] & 0x7fffffffffffffffull;
        mx = a > mx ? a : mx;
    }
    return mx;
}

// A row tile is shared by CTAs of PACK_ROWS rows (gridDim.y), each packing all k tiles of its
// rows: the row maxima stay within a CTA.  Work item: one row and two k, so that a k tile of 8
// rows is one item for each of 256 threads; the block has the threads that the longest job has
// items for (1024 at most), and the elements stay in registers between the maximum and the digits
// while the k tiles do.  Consecutive threads take consecutive rows so that the loads of a
// column-major operand come in 64-byte pieces.  Bound by latency, of the loads and of the
// instructions: with eight elements a thread the straight code was four times as long and 64
// threads of a CTA of 256 worked (one k tile; 31 us for the 4096 x 64 operands of four
// instances; the blocks of a chi = 50 bond took 6.2 us, before that, with 32 rows per CTA and
// whole tiles written, 12.4 us).
template <int SL>
__global__ void __launch_bounds__(PACK_MAXTHREADS)
split_pack_kernel(const PackJob* __restrict__ jobs, const KTileSrc* __restrict__ ksrc,
                  const __grid_constant__ Bases b, uint8_t* __restrict__ out,
                  int* __restrict__ expo, int tile_rows) {
    __shared__ unsigned long long rowmax[PACK_ROWS];
    const PackJob jb = jobs[blockIdx.x];
    const int r0 = blockIdx.y * PACK_ROWS;
    if (r0 >= jb.rows) return;
    const int tile_bytes = tile_rows * BKT * 2;
    constexpr int PER_TILE = PACK_ROWS * BKT / 2;  // (row, pair of k) items per k tile
    const int nitems = PER_TILE * jb.nkt, nthr = blockDim.x;
    if (threadIdx.x < PACK_ROWS) rowmax[threadIdx.x] = 0ull;
    __syncthreads();
    const int rl = threadIdx.x % PACK_ROWS, r = r0 + rl;
    const bool live = r < jb.rows;
    long long v[2];
    // row maxima of |x| as IEEE bit patterns (integer compare, no FP64 pipe): over the four lanes
    // of a row, then over the warps
    for (int it = threadIdx.x; it < nitems; it += nthr) {
        const KTileSrc ks = ksrc[jb.kt0 + it / PER_TILE];
        unsigned long long mx =
            pack_load(v, ks, b, jb.row0 + r, live, (it % PER_TILE) / PACK_ROWS);
#pragma unroll
        for (int d = PACK_ROWS; d < 32; d *= 2) {
            const unsigned long long o = __shfl_xor_sync(0xffffffffu, mx, d);
            mx = o > mx ? o : mx;
        }
        if (mx && (threadIdx.x & 31) < PACK_ROWS) atomicMax(&rowmax[rl], mx);
    }
    __syncthreads();
    const unsigned long long mxb = rowmax[rl];
    if (threadIdx.x < PACK_ROWS && live)
        expo[jb.eoff + r] = mxb ? int((mxb >> 52) & 0x7ff) - 1022 : 0;
    for (int it = threadIdx.x; it < nitems; it += nthr) {
        const int t = it / PER_TILE, pr = (it % PER_TILE) / PACK_ROWS;
        const KTileSrc ks = ksrc[jb.kt0 + t];
        if (pr >= 4 * pack_chunks(t, ks.kvalid)) continue;
        if (nitems > nthr) pack_load(v, ks, b, jb.row0 + r, live, pr);
        pack_digits<SL, 2>(v, mxb, r, pr, out + jb.out_off + int64_t(t) * SL * tile_bytes,
                           tile_bytes);
    }
}

// k-split pack for operands with long k: the k tiles of every job are divided among
// gridDim.y CTAs (kper tiles each).  Pass 1 (split_rowmax_kernel) folds each row's max |x|
// (IEEE bit pattern, an exact and order-independent maximum) into gmax with atomicMax;
// pass 2 (split_pack_part_kernel) writes the digits of its k tiles with the exponents taken
// from gmax.  Same digits as split_pack_kernel, many more CTAs.
__global__ void __launch_bounds__(PACK_THREADS)
split_rowmax_kernel(const PackJob* __restrict__ jobs, const KTileSrc* __restrict__ ksrc,
                    const __grid_constant__ Bases b, unsigned long long* __restrict__ gmax,
                    int kper) {
    __shared__ unsigned long long rowmax[BM];
    const PackJob jb = jobs[blockIdx.x];
    const int t0 = blockIdx.y * kper;
    if (t0 >= jb.nkt) return;
    const int t1 = (t0 + kper) < jb.nkt ? (t0 + kper) : jb.nkt;
    const int per_tile = jb.rows * 8;
    const int nitems = per_tile * (t1 - t0);
    for (int r = threadIdx.x; r < jb.rows; r += blockDim.x) rowmax[r] = 0ull;
    __syncthreads();
    for (int it = threadIdx.x; it < nitems; it += blockDim.x) {
        const int t = t0 + it / per_tile, rem = it % per_tile;
        const int r = rem % jb.rows, ch = rem / jb.rows;
        const KTileSrc ks = ksrc[jb.kt0 + t];
        long long v[8];
        const unsigned long long mx = pack_load(v, ks, b, jb.row0 + r, true, ch);
        if (mx) atomicMax(&rowmax[r], mx);
    }
    __syncthreads();
    for (int r = threadIdx.x; r < jb.rows; r += blockDim.x)
        if (rowmax[r]) atomicMax(&gmax[jb.eoff + r], rowmax[r]);
}

template <int SL>
__global__ void __launch_bounds__(PACK_THREADS)
split_pack_part_kernel(const PackJob* __restrict__ jobs, const KTileSrc* __restrict__ ksrc,
                       const __grid_constant__ Bases b, uint8_t* __restrict__ out,
                       int* __restrict__ expo, const unsigned long long* __restrict__ gmax,
                       int tile_rows, int kper) {
    const PackJob jb = jobs[blockIdx.x];
    const int t0 = blockIdx.y * kper;
    if (t0 >= jb.nkt) return;
    const int t1 = (t0 + kper) < jb.nkt ? (t0 + kper) : jb.nkt;
    const int tile_bytes = tile_rows * BKT * 2;
    const int rows8 = (jb.rows + 7) & ~7;
    const int per_tile = rows8 * 8;
    const int nitems = per_tile * (t1 - t0);
    if (blockIdx.y == 0 && blockIdx.z == 0)
        for (int r = threadIdx.x; r < jb.rows; r += blockDim.x) {
            const unsigned long long m = gmax[jb.eoff + r];
            expo[jb.eoff + r] = m ? int((m >> 52) & 0x7ff) - 1022 : 0;
        }
    for (int it = blockIdx.z * blockDim.x + threadIdx.x; it < nitems; it += gridDim.z * blockDim.x) {
        const int t = t0 + it / per_tile, rem = it % per_tile;
        const int r = rem % rows8, ch = rem / rows8;
        const KTileSrc ks = ksrc[jb.kt0 + t];
        if (ch >= pack_chunks(t, ks.kvalid)) continue;
        const bool live = r < jb.rows;
        const unsigned long long mxb = live ? gmax[jb.eoff + r] : 0ull;
        long long v[8];
        pack_load(v, ks, b, jb.row0 + r, live, ch);
        pack_digits<SL, 8>(v, mxb, r, ch, out + jb.out_off + int64_t(t) * SL * tile_bytes,
                           tile_bytes);
    }
}

// ------------------------------------------------------------------------------------
// MMA kernel
// ------------------------------------------------------------------------------------
struct __align__(8) SplitShared {
    uint64_t full[NST];
    uint64_t empty[NST];
    uint64_t tfull[2];
    uint64_t tempty[2];
    uint64_t done;
    uint32_t tmem_base;
    int err;
};

// SL slices per operand.  The issuing code is unrolled over the slice pairs: computing
// the pair, its level, its ring stages and descriptors in loops took it 380 clocks a pair, 5700 a
// k tile, three times what the tensor core needs for 60 products of 128 x 64 x 16.
template <int SL>
__global__ void __launch_bounds__(THREADS, 1)
split_gemm_kernel(const SplitItem* __restrict__ items, int nitems,
                  const SplitTask* __restrict__ tasks, const uint8_t* __restrict__ apack,
                  const uint8_t* __restrict__ bpack, const int* __restrict__ ea,
                  const int* __restrict__ eb, const __grid_constant__ Bases b,
                  int* __restrict__ err) {
    constexpr int slices = SL;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // 1024-byte aligned stage ring (the swizzle atom needs it)
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~uintptr_t(1023));
    SplitShared* sh = reinterpret_cast<SplitShared*>(ring + NST * STAGE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* serr = &sh->err;
    // the first item, on its way during the set-up
    const SplitItem item0 = items[blockIdx.x];
    const SplitTask task0 = tasks[item0.task];

    if (threadIdx.x == 0) {
        for (int i = 0; i < NST; ++i) {
            mbar_init(&sh->full[i], 1);
            mbar_init(&sh->empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh->tfull[i], 1);
            mbar_init(&sh->tempty[i], 8);  // one arrive per epilogue warp
        }
        mbar_init(&sh->done, 1);
        sh->err = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&sh->tmem_base)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = sh->tmem_base;

    if (warp == 0) {
        // ---------------- producer ----------------
        const uint32_t lead = elect_lane();
        // test hook (tn_ctx_inject_wait_timeout, code 1): CTA 0 withholds the copies of its
        // first stage, so that the MMA warp's wait on it runs out and every role drains
        bool withhold = false;
        if (blockIdx.x == 0) withhold = __any_sync(0xffffffffu, lead && atomicCAS(err + 1, 1, 0) == 1);
        uint32_t g = 0;  // global stage counter
        for (int it = blockIdx.x; it < nitems && !warp_err(serr); it += gridDim.x) {
            const SplitItem item = it == int(blockIdx.x) ? item0 : items[it];
            const SplitTask tk = it == int(blockIdx.x) ? task0 : tasks[item.task];
            // the 8-row atoms that hold rows of the block (the rest of the stage keeps
            // what was there: it only reaches outputs that are not stored)
            const uint32_t abytes = uniform(uint32_t(min(BM, tk.m - item.mt * BM) + 7) / 8 * 1024);
            const uint32_t bbytes = uniform(uint32_t(min(BN, tk.n - item.nt * BN) + 7) / 8 * 1024);
            const int nkt = int(uniform(uint32_t(tk.nkt)));
            const uint8_t* asrc = apack + tk.a_off + int64_t(item.mt) * tk.nkt * slices * A_TILE;
            const uint8_t* bsrc = bpack + tk.b_off + int64_t(item.nt) * tk.nkt * slices * B_TILE;
            bool ok = true;
            for (int kt = 0; kt < nkt && ok; ++kt)
                for (int t = 0; t < slices; ++t, ++g, asrc += A_TILE, bsrc += B_TILE) {
                    const int st = g % NST;
                    const uint32_t ph = (g / NST) & 1;
                    ok = __all_sync(0xffffffffu, mbar_wait(&sh->empty[st], ph ^ 1, err, serr));
                    if (!ok) break;
                    if (withhold && g == 0) continue;
                    uint8_t* dst = ring + st * STAGE;
                    mbar_expect_tx(&sh->full[st], abytes + bbytes, lead);
                    bulk_g2s(dst, asrc, abytes, &sh->full[st], lead);
                    bulk_g2s(dst + A_TILE, bsrc, bbytes, &sh->full[st], lead);
                }
        }
        // before the CTA may exit, every copy this warp issued must have landed (in the normal
        // path the MMA warp has consumed them all; after an error this drains)
        for (uint32_t gg = (g > NST ? g - NST : 0); gg < g; ++gg)
            mbar_drain(&sh->full[gg % NST], (gg / NST) & 1);
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        {
            const uint32_t lead = elect_lane();
            const uint32_t ring_lo = uniform(sdesc_lo(smem_u32(ring)));
            const uint32_t tmem_u = uniform(tmem);
            uint32_t g = 0;       // stage counter (matches the producer)
            uint32_t chunk = 0;   // accumulation chunk counter (TMEM double buffer)
            for (int it = blockIdx.x; it < nitems && !warp_err(serr); it += gridDim.x) {
                const SplitItem item = it == int(blockIdx.x) ? item0 : items[it];
                const SplitTask tk = it == int(blockIdx.x) ? task0 : tasks[item.task];
                // N covers the block's columns (a multiple of 16)
                const uint32_t idesc =
                    uniform(idesc_bf16(BM, (min(BN, tk.n - item.nt * BN) + 15) / 16 * 16));
                const int nkt = int(uniform(uint32_t(tk.nkt)));
                const uint64_t kmask = uint64_t(uniform(uint32_t(tk.kmask >> 32))) << 32 |
                                       uniform(uint32_t(tk.kmask));
                for (int k0 = 0; k0 < nkt && !warp_err(serr); k0 += KC, ++chunk) {
                    const int buf = chunk & 1;
                    if (!__all_sync(0xffffffffu, mbar_wait(&sh->tempty[buf], ((chunk >> 1) & 1) ^ 1, err, serr)))
                        break;
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const int k1 = min(k0 + KC, nkt);
                    bool ok = true;
                    for (int kt = k0; kt < k1 && ok; ++kt) {
                        const uint32_t g0 = g;
                        // 16-deep steps with valid k (the others would add zeros)
                        const int nkk = split_ksteps(kmask, kt);
                        const bool fresh = kt == k0;  // the accumulators start anew
                        uint32_t ad[SL], bd[SL];      // descriptors of the slices' tiles
#pragma unroll
                        for (int t = 0; t < SL; ++t) {
                            const uint32_t st = (g0 + t) % NST;
                            if (!__all_sync(0xffffffffu,
                                            mbar_wait(&sh->full[st], ((g0 + t) / NST) & 1, err, serr))) {
                                ok = false;
                                break;
                            }
                            asm volatile("tcgen05.fence::after_thread_sync;");
                            ad[t] = ring_lo + st * (STAGE >> 4);
                            bd[t] = ad[t] + (A_TILE >> 4);
                            // pairs (i, t) and (t, i) with i + t <= slices - 1 (0-based
                            // slices: level = i + t + 2, the fourth accumulator from 5 on); the
                            // first of their accumulators are (0, 0), (0, 1), (1, 1) and (1, 2)
#pragma unroll
                            for (int i = 0; i <= t; ++i) {
                                if (i + t > SL - 1) continue;
                                const int lvl = i + t < NACC - 1 ? i + t : NACC - 1;
                                const uint32_t td = tmem_u + uint32_t(buf * NACC * BN + lvl * BN);
                                const bool first = t < 2 || (i == 1 && t == 2);
#pragma unroll 1
                                for (int kk = 0; kk < nkk; ++kk)
                                    mma_bf16(td, ad[i] + 2 * kk, bd[t] + 2 * kk, idesc,
                                             !(first && kk == 0 && fresh), lead);
                                if (i == t) continue;
#pragma unroll 1
                                for (int kk = 0; kk < nkk; ++kk)
                                    mma_bf16(td, ad[t] + 2 * kk, bd[i] + 2 * kk, idesc, true, lead);
                            }
                        }
                        if (!ok) break;
                        for (int t = 0; t < slices; ++t) mma_commit(&sh->empty[(g0 + t) % NST], lead);
                        g = g0 + slices;
                    }
                    if (!ok) break;
                    // with slices >= 4 every k tile writes all four levels, so every
                    // accumulator of this chunk has been (re)initialised
                    mma_commit(&sh->tfull[buf], lead);
                }
            }
            // every MMA this warp issued completes before TMEM is released
            mma_commit(&sh->done, lead);
            mbar_drain(&sh->done, 0);
        }
    } else {
        // ---------------- epilogue (warps 2..9) ----------------
        // Two warps per lane quadrant, which take the 16-column groups in turn, so that both
        // have work on narrow blocks.  c = 0..31 of a warp: group c / 16, column c % 16.
        constexpr int HC = BN / 2;       // columns per epilogue warp
        const int q = warp & 3;          // TMEM lane quadrant of this warp
        const int h = (warp - 2) >> 2;   // first column group
        const int row = q * 32 + lane;   // row of the output tile
        uint32_t chunk = 0;
        for (int it = blockIdx.x; it < nitems && !*serr; it += gridDim.x) {
            const SplitItem item = it == int(blockIdx.x) ? item0 : items[it];
            const SplitTask tk = it == int(blockIdx.x) ? task0 : tasks[item.task];
            // the block's columns in this tile (none for a quadrant beyond its rows)
            const int ncol = q * 32 < tk.m - item.mt * BM ? min(BN, tk.n - item.nt * BN) : 0;
            const int gr = item.mt * BM + row;
            const int er = gr < tk.m ? ea[tk.ea_off + gr] : 0;
            const int ec = lane + 16 * h + 16 * (lane >> 4) < ncol
                               ? eb[tk.eb_off + item.nt * BN + lane + 16 * h + 16 * (lane >> 4)]
                               : 0;  // exponent of column c = lane
            float hi[HC], lo[HC];
#pragma unroll
            for (int c = 0; c < HC; ++c) { hi[c] = 0.f; lo[c] = 0.f; }
            bool ok = true;
            for (int k0 = 0; k0 < tk.nkt; k0 += KC, ++chunk) {
                const int buf = chunk & 1;
                if (!mbar_wait(&sh->tfull[buf], (chunk >> 1) & 1, err, serr)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t tbase = tmem + (uint32_t(q * 32) << 16) + uint32_t(buf * NACC * BN + h * 16);
                // (the two column groups in a loop, its registers swapped after each pass: straight
                // code of this length waits for its instructions)
#pragma unroll 1
                for (int g = 0; g < 2; ++g) {
                    if (16 * h + 32 * g < ncol) {
                        float v[NACC][16];
#pragma unroll
                        for (int l = 0; l < NACC; ++l) tmem_ld16(tbase + l * BN + 32 * g, v[l]);
                        tmem_wait(v);
#pragma unroll
                        for (int l = 0; l < NACC; ++l)
#pragma unroll
                            for (int c = 0; c < 16; ++c) df_add(hi[c], lo[c], v[l][c]);
                    }
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        const float th = hi[c], tl = lo[c];
                        hi[c] = hi[c + 16];
                        lo[c] = lo[c + 16];
                        hi[c + 16] = th;
                        lo[c + 16] = tl;
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;");
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->tempty[buf]);
            }
            if (!ok) break;
            if (ncol == 0) continue;
            double* C = b.p[tk.cbuf] + tk.coff + gr + int64_t(item.nt * BN) * tk.ldc;
            // Four columns at a time, their chains (exponent, widening, sum, scaling) side by side,
            // in a loop that takes columns 0 to 3 of the registers and moves the rest down.  One
            // FP64 operation a column, two with accumulation; what the integer forms do not cover
            // (subnormals, infinities, NaN, exponents beyond any product of normal operands) takes
            // a branch of its own.  One column after the other, each with a branch at every special
            // value, took 470 clocks a column; this takes 350 (230 eight at a time, which lose more
            // on the blocks of a few columns than they gain on the wide ones: 281 against 279 ms
            // on a chi = 50 chain).
            // The lanes beyond the block hold whatever the accumulators did: zero here.
            constexpr int GC = 4;
            if (gr >= tk.m) {
#pragma unroll
                for (int c = 0; c < HC; ++c) { hi[c] = 0.f; lo[c] = 0.f; }
            }
#pragma unroll 1
            for (int c0 = 0; c0 < HC; c0 += GC) {
                const int tc = c0 + 16 * h + (c0 & 16);  // first column of the four
                if (tc >= ncol) break;
                const int nc = gr < tk.m ? ncol - tc : 0;  // columns that this lane stores
                double* out = C + int64_t(tc) * tk.ldc;
                double old[GC], v[GC];
                if (tk.accum)
#pragma unroll
                    for (int j = 0; j < GC; ++j) old[j] = j < nc ? out[int64_t(j) * tk.ldc] : 0.0;
                int e[GC];
                bool fast = true;
#pragma unroll
                for (int j = 0; j < GC; ++j) {
                    e[j] = er + __shfl_sync(0xffffffffu, ec, c0 + j) - 16;
                    fast = fast && (j >= ncol - tc || (plain(hi[j]) && plain(lo[j]) &&
                                                       unsigned(e[j] + 800) <= 1600u));
                }
                if (__all_sync(0xffffffffu, fast)) {
#pragma unroll
                    for (int j = 0; j < GC; ++j) v[j] = scale2(widen(hi[j]) + widen(lo[j]), e[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < GC; ++j)
                        v[j] = (double(branch_only(hi[j])) + double(branch_only(lo[j]))) * pow2(e[j]);
                }
                if (tk.accum)
#pragma unroll
                    for (int j = 0; j < GC; ++j) v[j] = branch_only(old[j]) + v[j];
#pragma unroll
                for (int j = 0; j < GC; ++j)
                    if (j < nc) out[int64_t(j) * tk.ldc] = v[j];
#pragma unroll
                for (int c = 0; c + GC < HC; ++c) { hi[c] = hi[c + GC]; lo[c] = lo[c + GC]; }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(TMEM_COLS));
}

}  // namespace

int split_tile_bytes_a() { return A_TILE; }
int split_tile_bytes_b() { return B_TILE; }
int split_tile_rows_a() { return BM; }
int split_tile_rows_b() { return BN; }
int split_ktile() { return BKT; }
constexpr int KPER = 2;  // k tiles per CTA of the k-split pack
bool split_pack_needs_max(int max_nkt) { return max_nkt > 2 * KPER; }

void launch_split_pack(const PackJob* jobs, int njobs, const KTileSrc* ksrc, const Bases& b,
                       uint8_t* out, int* expo, int slices, int tile_rows, int max_rows,
                       cudaStream_t s, int max_nkt, unsigned long long* gmax, int64_t nrows) {
    if (njobs <= 0) return;
    TN_REQUIRE(slices >= 4 && slices <= 7, "split precision needs 4..7 slices");
    TN_REQUIRE(tile_rows <= BM, "pack tile taller than the A tile");
    if (!split_pack_needs_max(max_nkt) || !gmax) {
        const dim3 g(njobs, (max_rows + PACK_ROWS - 1) / PACK_ROWS);
        const int nthr = std::min(PACK_MAXTHREADS, PACK_ROWS * BKT / 2 * std::max(max_nkt, 1));
        auto* kernel = slices == 4   ? split_pack_kernel<4>
                       : slices == 5 ? split_pack_kernel<5>
                       : slices == 6 ? split_pack_kernel<6>
                                     : split_pack_kernel<7>;
        kernel<<<g, nthr, 0, s>>>(jobs, ksrc, b, out, expo, tile_rows);
        TN_CUDA(cudaGetLastError());
        count_launch();
        return;
    }
    const dim3 g(njobs, (max_nkt + KPER - 1) / KPER);
    TN_CUDA(cudaMemsetAsync(gmax, 0, size_t(nrows) * sizeof(unsigned long long), s));
    split_rowmax_kernel<<<g, PACK_THREADS, 0, s>>>(jobs, ksrc, b, gmax, KPER);
    TN_CUDA(cudaGetLastError());
    // two items a thread
    const int nz = std::max(1, (max_rows + 7) / 8 * 8 * (BKT / 8) * KPER / (2 * PACK_THREADS));
    auto* kernel = slices == 4   ? split_pack_part_kernel<4>
                   : slices == 5 ? split_pack_part_kernel<5>
                   : slices == 6 ? split_pack_part_kernel<6>
                                 : split_pack_part_kernel<7>;
    kernel<<<dim3(g.x, g.y, nz), PACK_THREADS, 0, s>>>(jobs, ksrc, b, out, expo, gmax, tile_rows,
                                                       KPER);
    TN_CUDA(cudaGetLastError());
    count_launch(2);
}

void launch_split_gemm(const SplitItem* items, int nitems, const SplitTask* tasks,
                       const uint8_t* apack, const uint8_t* bpack, const int* ea, const int* eb,
                       const Bases& b, int slices, int* err, int nsm, cudaStream_t s) {
    if (nitems <= 0) return;
    TN_REQUIRE(slices >= 4 && slices <= 7, "split precision needs 4..7 slices");
    const size_t shm = size_t(NST) * STAGE + sizeof(SplitShared) + 1024;
    auto* kernel = slices == 4   ? split_gemm_kernel<4>
                   : slices == 5 ? split_gemm_kernel<5>
                   : slices == 6 ? split_gemm_kernel<6>
                                 : split_gemm_kernel<7>;
    if (slices == 4) allow_smem<split_gemm_kernel<4>>(shm);
    else if (slices == 5) allow_smem<split_gemm_kernel<5>>(shm);
    else if (slices == 6) allow_smem<split_gemm_kernel<6>>(shm);
    else allow_smem<split_gemm_kernel<7>>(shm);
    const int grid = nitems < nsm ? nitems : nsm;
    kernel<<<grid, THREADS, shm, s>>>(items, nitems, tasks, apack, bpack, ea, eb, b, err);
    TN_CUDA(cudaGetLastError());
    count_launch();
}

}  // namespace tn
