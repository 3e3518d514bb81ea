// Split-precision grouped GEMM on the 5th-generation tensor cores of
// sm_100a (tcgen05.mma kind::i8 with INT32 accumulators in tensor memory,
// operands staged in shared memory by bulk asynchronous copies); see
// gemm_split.cuh for the arithmetic.
//
// Operand packing.  Two passes over the operands: one finds the row exponents,
// one writes the digits as ready-made shared-memory images: op(A) in tiles of
// 128 rows x 32 K-bytes, op(B)^T in tiles of 64 rows x 32 K-bytes, each in the
// canonical K-major layout without swizzle (core matrices of 8 rows x 16
// bytes; consecutive core matrices along K 128 bytes apart, along the rows 256
// bytes apart).  The digits of one (row tile, K chunk) follow each other, so
// one stage of the GEMM is two contiguous bulk copies: D x 4 KB of A and D x
// 2 KB of B.  Both passes are meant to run at the rate of memory: their blocks
// take 128 K entries of a row tile (many blocks also for few problems), an
// element is converted to an integer once, and its digits are the bytes of
// that integer plus a bias.  (One block per row tile for the exponents, and a
// multiply, truncate, subtract and convert per digit, took 0.43 ms for eight
// products of edges 900 to 1500; the two passes take 0.11 ms.)
//
// GEMM kernel.  Persistent CTAs, each over 128 x 64 output tiles: one warp issues
// the bulk copies into a ring of 32-byte-deep chunks (mbarrier transaction
// counts), another the tcgen05.mma instructions: for every chunk the digit pairs
// (p, q) with p + q <= D + 1 into the accumulator of p + q (D accumulators of
// 64 INT32 columns: up to all 512 tensor-memory columns), and commits to the
// stage's "empty" barrier.  Pairs of one p follow each other, so the A
// image is read from shared memory once and kept in the tensor core's collector
// buffer.  After a segment's last chunk a commit to the "done" barrier releases
// eight warps: each reads half the columns of its 32 rows (tensor-memory lanes) with tcgen05.ld,
// recombines the accumulators exactly in 64-bit integers and adds alpha times
// the result into C, while the ring already fills for the next tile.
//
// What bounds it: the shape of the instruction.  D accumulators of N columns
// must fit in 512 columns, so N = 64, and a 128 x 64 x 32 product reads 6 KB of
// operands from shared memory for 32 cycles of arithmetic: measured alone, 48
// cycles an instruction and 45 with the collector (N = 128: 64).  The eight
// products above with 8 slices, 36 products a chunk: 0.74 ms issued by one thread
// of a divergent branch, with a compensated FP64 recombination; 0.34 ms now.
// Every wait on a barrier is bounded; a wait that gives up sets an error flag,
// ends the CTA's work (waiting, bounded, for its copies and products in
// flight), frees the tensor memory and returns.
#include "gemm_split.cuh"

#include <float.h>
#include <limits.h>
#include <math.h>
#include <string.h>

#include <algorithm>

namespace nrgb {

namespace {

constexpr int SBM = 128;              // output rows per CTA (tensor-memory lanes)
constexpr int SBN = 64;               // output columns per CTA
constexpr int SBK = 32;               // K bytes per stage
constexpr int A_TILE = SBM * SBK;     // 4 KB
constexpr int B_TILE = SBN * SBK;     // 2 KB
constexpr int EPI_WARPS = 8;          // two per quarter of the tensor-memory lanes
constexpr int SPLIT_NT = 32 * EPI_WARPS + 64;  // and a warp for the copies, one for the products
constexpr int SLICE_NT = 256;
constexpr int PIECE = 4;              // K chunks per block of the slicing passes
constexpr int MAX_STAGES = 16;
constexpr size_t RING_BYTES = 216 * 1024;
constexpr long long WAIT_LIMIT = 1ll << 24;
constexpr int NO_EXP = (int)0x80808080;  // what memset leaves: a row of zeros

__device__ int g_split_err = 0;

struct SliceJob {
  const double* X;   // X(r, l) = X[r * rs + l * ls], r < rows, l < K
  long long rs, ls;
  int rows, K;
  int tile_rows;     // 128 (A) or 64 (B)
  int kch;           // K chunks of 32
  int pieces;        // blocks of PIECE chunks
  int block0;        // first (row tile, piece) of this job in the launch
  signed char* out;  // packed digits: [row tile][K chunk][digit] images
  int* exps;         // tile rows of exponents (rows of zeros and past `rows`: NO_EXP)
};

struct SplitSeg {
  const signed char* A;  // packed op(A)
  const signed char* B;  // packed op(B)^T
  const int* eA;         // row exponents of op(A)
  const int* eB;         // column exponents of op(B)
  int kch;
  double alpha;
};

struct SplitProb {
  double* C;
  int ldc, m, n;
  double beta;
  int seg0, nseg;
  int tile0, tiles_n, tiles_m;
};

// ------------------------------------------------------------------ slicing
__device__ __forceinline__ int find_job(const SliceJob* jobs, int njobs, int t) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].block0 <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Largest integer whose D balanced digits fit: D bytes 0x7F.
__device__ __forceinline__ long long digit_limit(int D) { return 0x7F7F7F7F7F7F7F7Fll >> (8 * (8 - D)); }

// Exponent of a row whose largest magnitude is mx > 0: the least e for which mx
// scaled by 2^(8 D - 1 - e) rounds to an integer of D balanced digits.
__device__ __forceinline__ int digit_exp(double mx, int D) {
  int e;
  const double f = frexp(fmin(mx, DBL_MAX), &e);  // [0.5, 1)
  return __double2ll_rn(ldexp(f, 8 * D - 1)) > digit_limit(D) ? e + 1 : e;
}

__device__ __forceinline__ int row_exp(const int* exps, int r) {
  const int e = exps[r];
  return e == NO_EXP ? 0 : e;
}

// Row exponents: the largest of the pieces' exponents.
__global__ void __launch_bounds__(SLICE_NT) split_exp_kernel(const SliceJob* __restrict__ jobs, int njobs, int D) {
  const SliceJob J = jobs[find_job(jobs, njobs, blockIdx.x)];
  const int local = blockIdx.x - J.block0;
  const int t = local / J.pieces, l0 = (local % J.pieces) * PIECE * SBK;
  const int l1 = min(J.K, l0 + PIECE * SBK), R = J.tile_rows;
  if (J.rs == 1) {
    // consecutive rows are adjacent: a thread takes one row and every
    // (SLICE_NT / R)-th of its entries
    const int rr = threadIdx.x % R, r = t * R + rr, step = SLICE_NT / R;
    double mx = 0.0;
    if (r < J.rows) {
      const double* x = J.X + r;
#pragma unroll 8
      for (int l = l0 + threadIdx.x / R; l < l1; l += step) mx = fmax(mx, fabs(x[l * J.ls]));
    }
    if (mx > 0.0) atomicMax(&J.exps[t * R + rr], digit_exp(mx, D));
  } else {
    // the K entries of a row are adjacent: one warp per row
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 2
    for (int rr = warp; rr < R; rr += SLICE_NT / 32) {
      const int r = t * R + rr;
      double mx = 0.0;
      if (r < J.rows) {
        const double* x = J.X + r * J.rs;
#pragma unroll
        for (int u = 0; u < PIECE * SBK / 32; ++u) {
          const int l = l0 + lane + 32 * u;
          if (l < l1) mx = fmax(mx, fabs(x[l * J.ls]));
        }
      }
      for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (lane == 0 && mx > 0.0) atomicMax(&J.exps[t * R + rr], digit_exp(mx, D));
    }
  }
}

// Bytes of four words, byte j of word u to byte u of word j.
__device__ __forceinline__ void transpose4(unsigned (&w)[4]) {
  const unsigned a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140);
  const unsigned c = __byte_perm(w[0], w[1], 0x7362), d = __byte_perm(w[2], w[3], 0x7362);
  w[0] = __byte_perm(a, b, 0x5410);
  w[1] = __byte_perm(a, b, 0x7632);
  w[2] = __byte_perm(c, d, 0x5410);
  w[3] = __byte_perm(c, d, 0x7632);
}

// The digits of 16 consecutive K entries x of a row (scaled by f1 * f2 they
// are rounded to integers), 16 bytes into each of the D images.
// With 0x80 in every byte as a bias the balanced digits carry by themselves:
// digit = byte of (y + bias), less 0x80.
__device__ __forceinline__ void write_digits(const double (&x)[16], double f1, double f2, int D, signed char* dst,
                                             size_t image) {
  unsigned out[8][4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    unsigned a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long y = __double2ll_rn(x[4 * q + u] * f1 * f2);
      const unsigned long long z = ((unsigned long long)y + 0x8080808080808080ull) ^ 0x8080808080808080ull;
      a[u] = (unsigned)z;
      b[u] = (unsigned)(z >> 32);
    }
    transpose4(a);
    transpose4(b);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      out[j][q] = a[j];
      out[4 + j][q] = b[j];
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)  // byte j is digit D - j
    if (j < D)
      *reinterpret_cast<uint4*>(dst + (size_t)(D - 1 - j) * image) =
          make_uint4(out[j][0], out[j][1], out[j][2], out[j][3]);
}

// Power of two 2^s, -1022 <= s <= 1023.
__device__ __forceinline__ double pow2(int s) { return __longlong_as_double((long long)(s + 1023) << 52); }

__global__ void __launch_bounds__(SLICE_NT) split_digits_kernel(const SliceJob* __restrict__ jobs, int njobs, int D) {
  __shared__ double tile[SBM][SBK + 1];
  // backwards: what the exponents' pass read last is still in L2
  const int block = gridDim.x - 1 - blockIdx.x;
  const SliceJob J = jobs[find_job(jobs, njobs, block)];
  const int local = block - J.block0;
  const int t = local / J.pieces, c0 = (local % J.pieces) * PIECE, c1 = min(J.kch, c0 + PIECE);
  const int R = J.tile_rows;
  const size_t image = (size_t)R * SBK;
  signed char* base = J.out + (size_t)t * J.kch * D * image;
  // 16 entries of row rr, K group g of chunk c
  auto write = [&](const double(&x)[16], int rr, int c, int g) {
    const int s = 8 * D - 1 - row_exp(J.exps, t * R + rr), h = s / 2;
    write_digits(x, pow2(h), pow2(s - h), D,
                 base + (size_t)c * D * image + (rr >> 3) * 256 + g * 128 + (rr & 7) * 16, image);
  };
  if (J.rs == 1) {  // rows fastest: coalesced reads across the warp
    for (int it = threadIdx.x; it < R * 2 * (c1 - c0); it += SLICE_NT) {
      const int rr = it % R, cg = it / R, c = c0 + (cg >> 1), g = cg & 1;
      const int r = t * R + rr, l0 = c * SBK + g * 16;
      double x[16];
#pragma unroll
      for (int u = 0; u < 16; ++u)
        x[u] = (r < J.rows && l0 + u < J.K) ? J.X[(long long)r + (l0 + u) * J.ls] : 0.0;
      write(x, rr, c, g);
    }
  } else {  // the K entries of a row are adjacent: through shared memory
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = c0; c < c1; ++c) {
      const int l = c * SBK + lane;
#pragma unroll 8
      for (int rr = warp; rr < R; rr += SLICE_NT / 32) {
        const int r = t * R + rr;
        tile[rr][lane] = (r < J.rows && l < J.K) ? J.X[(long long)r * J.rs + l * J.ls] : 0.0;
      }
      __syncthreads();
      for (int it = threadIdx.x; it < R * 2; it += SLICE_NT) {
        const int rr = it % R, g = it / R;
        double x[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) x[u] = tile[rr][16 * g + u];
        write(x, rr, c, g);
      }
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "selp.b32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "selp.b32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait for the phase with parity `parity` to complete.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, volatile int* abort_flag) {
  for (long long it = 0; it < WAIT_LIMIT; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  return false;
}

__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void bulk_g2s(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// Shared-memory matrix descriptor: canonical K-major layout, no swizzle.
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr, unsigned lbo, unsigned sbo) {
  unsigned long long d = 0;
  d |= (unsigned long long)((addr & 0x3FFFFu) >> 4);
  d |= (unsigned long long)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (unsigned long long)((sbo >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;  // descriptor version of tcgen05
  return d;         // base offset 0, relative LBO mode, no swizzle
}

// Instruction descriptor: kind::i8, D = S32, A and B signed 8-bit, both
// K-major, M = 128, N = 64.
constexpr unsigned IDESC_I8 = (2u << 4)            // D format S32
                              | (1u << 7)          // A signed
                              | (1u << 10)         // B signed
                              | ((SBN >> 3) << 17)  // N / 8
                              | ((SBM >> 4) << 24); // M / 16

// Use of the collector buffer of A: filled by the first product of an A image,
// read by the later ones.
enum Collector { A_ONCE, A_FILL, A_USE, A_LASTUSE };

template <Collector COL>
__device__ __forceinline__ void mma_i8(unsigned dtmem, unsigned long long adesc, unsigned long long bdesc,
                                       unsigned accumulate) {
  if constexpr (COL == A_FILL)
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::i8.collector::a::fill [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(IDESC_I8), "r"(accumulate)
      : "memory");
  else if constexpr (COL == A_USE)
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::i8.collector::a::use [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(IDESC_I8), "r"(accumulate)
      : "memory");
  else if constexpr (COL == A_LASTUSE)
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::i8.collector::a::lastuse [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(IDESC_I8), "r"(accumulate)
      : "memory");
  else
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(IDESC_I8), "r"(accumulate)
      : "memory");
}

// True in one lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
  unsigned p;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "elect.sync _|P, 0xffffffff;\n"
      "selp.b32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void mma_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// 16 columns of N accumulators, SBN columns apart (loads and their wait in one
// statement: nothing may read the registers before the wait).
template <int N>
__device__ __forceinline__ void tmem_ld16(unsigned taddr, int (&v)[N][16]) {
  static_assert(N >= 1 && N <= 4);
  if constexpr (N == 1)
    asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(v[0][0]), "=r"(v[0][1]), "=r"(v[0][2]), "=r"(v[0][3]), "=r"(v[0][4]), "=r"(v[0][5]), "=r"(v[0][6]),
        "=r"(v[0][7]), "=r"(v[0][8]), "=r"(v[0][9]), "=r"(v[0][10]), "=r"(v[0][11]), "=r"(v[0][12]), "=r"(v[0][13]),
        "=r"(v[0][14]), "=r"(v[0][15])
      : "r"(taddr + 0 * SBN)
      : "memory");
  else if constexpr (N == 2)
    asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(v[0][0]), "=r"(v[0][1]), "=r"(v[0][2]), "=r"(v[0][3]), "=r"(v[0][4]), "=r"(v[0][5]), "=r"(v[0][6]),
        "=r"(v[0][7]), "=r"(v[0][8]), "=r"(v[0][9]), "=r"(v[0][10]), "=r"(v[0][11]), "=r"(v[0][12]), "=r"(v[0][13]),
        "=r"(v[0][14]), "=r"(v[0][15]), "=r"(v[1][0]), "=r"(v[1][1]), "=r"(v[1][2]), "=r"(v[1][3]), "=r"(v[1][4]),
        "=r"(v[1][5]), "=r"(v[1][6]), "=r"(v[1][7]), "=r"(v[1][8]), "=r"(v[1][9]), "=r"(v[1][10]), "=r"(v[1][11]),
        "=r"(v[1][12]), "=r"(v[1][13]), "=r"(v[1][14]), "=r"(v[1][15])
      : "r"(taddr + 0 * SBN), "r"(taddr + 1 * SBN)
      : "memory");
  else if constexpr (N == 3)
    asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%48];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%49];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%50];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(v[0][0]), "=r"(v[0][1]), "=r"(v[0][2]), "=r"(v[0][3]), "=r"(v[0][4]), "=r"(v[0][5]), "=r"(v[0][6]),
        "=r"(v[0][7]), "=r"(v[0][8]), "=r"(v[0][9]), "=r"(v[0][10]), "=r"(v[0][11]), "=r"(v[0][12]), "=r"(v[0][13]),
        "=r"(v[0][14]), "=r"(v[0][15]), "=r"(v[1][0]), "=r"(v[1][1]), "=r"(v[1][2]), "=r"(v[1][3]), "=r"(v[1][4]),
        "=r"(v[1][5]), "=r"(v[1][6]), "=r"(v[1][7]), "=r"(v[1][8]), "=r"(v[1][9]), "=r"(v[1][10]), "=r"(v[1][11]),
        "=r"(v[1][12]), "=r"(v[1][13]), "=r"(v[1][14]), "=r"(v[1][15]), "=r"(v[2][0]), "=r"(v[2][1]), "=r"(v[2][2]),
        "=r"(v[2][3]), "=r"(v[2][4]), "=r"(v[2][5]), "=r"(v[2][6]), "=r"(v[2][7]), "=r"(v[2][8]), "=r"(v[2][9]),
        "=r"(v[2][10]), "=r"(v[2][11]), "=r"(v[2][12]), "=r"(v[2][13]), "=r"(v[2][14]), "=r"(v[2][15])
      : "r"(taddr + 0 * SBN), "r"(taddr + 1 * SBN), "r"(taddr + 2 * SBN)
      : "memory");
  else if constexpr (N == 4)
    asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%64];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%65];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%66];\n"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%67];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(v[0][0]), "=r"(v[0][1]), "=r"(v[0][2]), "=r"(v[0][3]), "=r"(v[0][4]), "=r"(v[0][5]), "=r"(v[0][6]),
        "=r"(v[0][7]), "=r"(v[0][8]), "=r"(v[0][9]), "=r"(v[0][10]), "=r"(v[0][11]), "=r"(v[0][12]), "=r"(v[0][13]),
        "=r"(v[0][14]), "=r"(v[0][15]), "=r"(v[1][0]), "=r"(v[1][1]), "=r"(v[1][2]), "=r"(v[1][3]), "=r"(v[1][4]),
        "=r"(v[1][5]), "=r"(v[1][6]), "=r"(v[1][7]), "=r"(v[1][8]), "=r"(v[1][9]), "=r"(v[1][10]), "=r"(v[1][11]),
        "=r"(v[1][12]), "=r"(v[1][13]), "=r"(v[1][14]), "=r"(v[1][15]), "=r"(v[2][0]), "=r"(v[2][1]), "=r"(v[2][2]),
        "=r"(v[2][3]), "=r"(v[2][4]), "=r"(v[2][5]), "=r"(v[2][6]), "=r"(v[2][7]), "=r"(v[2][8]), "=r"(v[2][9]),
        "=r"(v[2][10]), "=r"(v[2][11]), "=r"(v[2][12]), "=r"(v[2][13]), "=r"(v[2][14]), "=r"(v[2][15]),
        "=r"(v[3][0]), "=r"(v[3][1]), "=r"(v[3][2]), "=r"(v[3][3]), "=r"(v[3][4]), "=r"(v[3][5]), "=r"(v[3][6]),
        "=r"(v[3][7]), "=r"(v[3][8]), "=r"(v[3][9]), "=r"(v[3][10]), "=r"(v[3][11]), "=r"(v[3][12]), "=r"(v[3][13]),
        "=r"(v[3][14]), "=r"(v[3][15])
      : "r"(taddr + 0 * SBN), "r"(taddr + 1 * SBN), "r"(taddr + 2 * SBN), "r"(taddr + 3 * SBN)
      : "memory");
}

__device__ __forceinline__ int find_prob(const SplitProb* probs, int nprob, int b) {
  int lo = 0, hi = nprob - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (probs[mid].tile0 <= b) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------------------ GEMM
// sum_d v_d 256^(D - 1 - d) of 16 columns as hi 2^L + low, 0 <= low < 2^L: the
// first four terms and the rest are exact in 64 bits each (|v| < 2^31).
template <int D>
struct Recombine {
  static constexpr int NH = D < 4 ? D : 4, NL = D - NH, L = 8 * NL;
  long long hi[16];
  unsigned low[16];

  __device__ __forceinline__ void load(unsigned taddr) {
    {
      int v[NH][16];
      tmem_ld16<NH>(taddr, v);
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        hi[u] = 0;
#pragma unroll
        for (int d = 0; d < NH; ++d) hi[u] += (long long)v[d][u] * (1ll << (8 * (NH - 1 - d)));
      }
    }
    if constexpr (NL > 0) {
      int v[NL][16];
      tmem_ld16<NL>(taddr + NH * SBN, v);
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        long long x = 0;
#pragma unroll
        for (int d = 0; d < NL; ++d) x += (long long)v[d][u] * (1ll << (8 * (NL - 1 - d)));
        hi[u] += x >> L;
        low[u] = (unsigned)x & (unsigned)((1ull << L) - 1);
      }
    }
  }
  // the sum, rounded once to FP64
  __device__ __forceinline__ double value(int u) const {
    long long bottom = (hi[u] & 0xFFFFF) << L;  // below 2^52: exact
    if constexpr (NL > 0) bottom |= low[u];
    return fma((double)(hi[u] >> 20), (double)(1ll << (20 + L)), (double)bottom);
  }
};

// Barriers and the ring of one CTA, as shared-memory addresses.
struct Ring {
  unsigned data, full0, empty0, done, drained, last;
};

constexpr int FIRST = 1, LAST = 2, END = 4;  // of a stage's chunk: see flag_s

// The warp that issues the products.  (A function of its own: inlined beside
// the recombination its loop issues 28 products, those of 7 slices, in 1426 cycles
// instead of 1304.)
template <int D>
__device__ __noinline__ void split_products(Ring ring, unsigned tmem, int stages, const volatile int* flag_s,
                                            volatile int* abort_flag) {
  constexpr unsigned STAGE = (unsigned)D * (A_TILE + B_TILE);
  auto give_up = [&] {
    atomicExch(&g_split_err, 1);
    *abort_flag = 1;
  };
  // products.  The whole warp takes the loop and one lane issues: with the
  // operands' descriptors in uniform registers an issue is short.  The tensor
  // core queues few products, and what the next chunk needs is looked up while
  // the last ones of this chunk wait.
  const bool leader = elect_one();
  int st = 0, round = 0, item = 0;
  bool ready = false;
  for (;;) {
    if (!ready && !mbar_wait(ring.full0 + 8 * st, round & 1, abort_flag)) {
      give_up();
      break;
    }
    const int flag = __shfl_sync(0xffffffffu, flag_s[st], 0);
    if (flag & END) break;
    if ((flag & FIRST) && !mbar_wait(ring.drained, (item & 1) ^ 1, abort_flag)) {
      give_up();
      break;
    }
    tc_fence_after();
    const unsigned sa = ring.data + (unsigned)st * STAGE;
    const unsigned long long ad = smem_desc(sa, 128, 256), bd = smem_desc(sa + D * A_TILE, 128, 256);
    const unsigned more = !(flag & FIRST);
    const unsigned empty = ring.empty0 + 8 * st;
    if (++st == stages) {
      st = 0;
      ++round;
    }
#pragma unroll
    for (int p = 0; p < D; ++p) {
      if (p == (D > 2 ? 2 : 1)) ready = __all_sync(0xffffffffu, mbar_test(ring.full0 + 8 * st, round & 1));
      if (leader) {
#pragma unroll
        for (int q = 0; q < D - p; ++q) {
          const unsigned dt = tmem + (unsigned)((p + q) * SBN);
          const unsigned long long a = ad + (unsigned)(p * A_TILE >> 4), b = bd + (unsigned)(q * B_TILE >> 4);
          const unsigned acc = p > 0 ? 1u : more;
          if (D - p == 1) mma_i8<A_ONCE>(dt, a, b, acc);
          else if (q == 0) mma_i8<A_FILL>(dt, a, b, acc);
          else if (q == D - p - 1) mma_i8<A_LASTUSE>(dt, a, b, acc);
          else mma_i8<A_USE>(dt, a, b, acc);
        }
      }
    }
    if (leader) {
      mma_commit(empty);  // the stage is free once these products have read it
      if (flag & LAST) mma_commit(ring.done);  // every product of the segment has completed
    }
    __syncwarp();
    if (flag & LAST) ++item;
  }
  // nothing is in flight when the tensor memory is released
  if (leader) mma_commit(ring.last);
  for (long long it = 0; it < WAIT_LIMIT && !mbar_try_wait(ring.last, 0); ++it) {
  }
}

template <int D>
__global__ void __launch_bounds__(SPLIT_NT, 1) split_gemm_kernel(const SplitProb* __restrict__ probs, int nprob,
                                                                  const SplitSeg* __restrict__ segs, int tiles,
                                                                  int stages, unsigned tmem_cols) {
  extern __shared__ __align__(1024) unsigned char dsm[];
  // ring of stages, 1024-aligned: [A: D x 4 KB | B: D x 2 KB]
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<size_t>(dsm) + 1023) & ~size_t(1023));
  constexpr unsigned STAGE = (unsigned)D * (A_TILE + B_TILE);
  __shared__ __align__(8) unsigned long long bars[2 * MAX_STAGES + 3];  // full, empty, done, drained, last
  // per stage: first, last chunk of a segment (set by the copies' thread, so that
  // the products' thread looks nothing up), end of the work
  __shared__ volatile int flag_s[MAX_STAGES];
  __shared__ unsigned tmem_base_s;
  __shared__ int abort_s;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const unsigned full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[MAX_STAGES]);
  const unsigned done = smem_u32(&bars[2 * MAX_STAGES]), drained = done + 8, last = done + 16;

  if (tid == 0) {
    for (int i = 0; i < 2 * MAX_STAGES + 3; ++i) mbar_init(smem_u32(&bars[i]), i == 2 * MAX_STAGES + 1 ? EPI_WARPS : 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_base_s;
  volatile int* abort_flag = &abort_s;
  const Ring ring{smem_u32(sm), full0, empty0, done, drained, last};
  auto give_up = [&] {
    atomicExch(&g_split_err, 1);
    *abort_flag = 1;
  };

  if (warp == EPI_WARPS && lane == 0) {
    // copies: each chunk's D images of A and of B
    int st = 0, round = 0;
    for (int t = blockIdx.x; t < tiles && !*abort_flag; t += gridDim.x) {
      const SplitProb P = probs[find_prob(probs, nprob, t)];
      const int local = t - P.tile0, mt = local / P.tiles_n, nt = local % P.tiles_n;
      for (int si = 0; si < P.nseg; ++si) {
        const SplitSeg S = segs[P.seg0 + si];
        const signed char* a = S.A + (size_t)mt * S.kch * D * A_TILE;
        const signed char* b = S.B + (size_t)nt * S.kch * D * B_TILE;
        for (int c = 0; c < S.kch && !*abort_flag; ++c) {
          if (!mbar_wait(empty0 + 8 * st, (round & 1) ^ 1, abort_flag)) {
            give_up();
            break;
          }
          const unsigned dst = smem_u32(sm) + (unsigned)st * STAGE, bar = full0 + 8 * st;
          flag_s[st] = (c == 0 ? FIRST : 0) | (c == S.kch - 1 ? LAST : 0);
          mbar_expect_tx(bar, STAGE);
          bulk_g2s(dst, a + (size_t)c * D * A_TILE, D * A_TILE, bar);
          bulk_g2s(dst + D * A_TILE, b + (size_t)c * D * B_TILE, D * B_TILE, bar);
          if (++st == stages) {
            st = 0;
            ++round;
          }
        }
      }
    }
    if (!*abort_flag) {
      if (mbar_wait(empty0 + 8 * st, (round & 1) ^ 1, abort_flag)) {
        flag_s[st] = END;
        mbar_arrive(full0 + 8 * st);
      } else {
        give_up();
      }
    }
    if (*abort_flag) {  // the copies in flight land before the memory is released
      for (int i = 0; i < stages; ++i) {
        const int n = round + (i < st ? 1 : 0);  // copies into stage i so far
        if (n == 0) continue;
        for (long long it = 0; it < WAIT_LIMIT && !mbar_try_wait(full0 + 8 * i, (n - 1) & 1); ++it) {
        }
      }
    }
  } else if (warp == EPI_WARPS + 1) {
    split_products<D>(ring, tmem, stages, flag_s, &abort_s);
  } else if (warp < EPI_WARPS) {
    // recombination and C: a warp takes 32 rows and half of the columns
    const int quarter = warp & 3, half = warp >> 2;
    int item = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      const SplitProb P = probs[find_prob(probs, nprob, t)];
      const int local = t - P.tile0, mt = local / P.tiles_n, nt = local % P.tiles_n;
      const int row = mt * SBM + quarter * 32 + lane;
      bool ok = true;
      for (int si = 0; si < P.nseg && ok; ++si, ++item) {
        const SplitSeg S = segs[P.seg0 + si];
        // lane u holds the exponent of column u of the half
        const int ea = row_exp(S.eA, row) - 8 * D - 6, eb = row_exp(S.eB, nt * SBN + half * 32 + lane);
        if (lane == 0) ok = mbar_wait(done, item & 1, abort_flag);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) {
          give_up();
          break;
        }
        tc_fence_after();
        Recombine<D> x[2];  // 16 columns each
#pragma unroll
        for (int h = 0; h < 2; ++h)
          x[h].load(tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)(half * 32 + h * 16));
        // the accumulators may be overwritten
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(drained);
        const int col0 = nt * SBN + half * 32;
        double* cp = P.C + (size_t)col0 * P.ldc + row;
#pragma unroll
        for (int u = 0; u < 32; ++u) {
          const int e = ea + __shfl_sync(0xffffffffu, eb, u);
          if (row >= P.m || col0 + u >= P.n) continue;
          const double f = x[u / 16].value(u % 16);
          double val = S.alpha * (abs(e) < 900 ? f * pow2(e) : ldexp(f, e));
          double* c = cp + (size_t)u * P.ldc;
          if (si > 0) val += *c;
          else if (P.beta != 0.0) val += P.beta * *c;
          *c = val;
        }
      }
      if (!ok) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(tmem_cols) : "memory");
  }
}

template <int D>
cudaError_t split_gemm_launch(const SplitProb* probs, int nprob, const SplitSeg* segs, int tiles, cudaStream_t st) {
  constexpr size_t stage = (size_t)D * (A_TILE + B_TILE);
  constexpr int stages = RING_BYTES / stage < MAX_STAGES ? (int)(RING_BYTES / stage) : MAX_STAGES;
  constexpr size_t smem = stages * stage + 1024;
  static std::once_flag once;
  static cudaError_t err = cudaSuccess;
  std::call_once(once, [] {
    err = cudaFuncSetAttribute(split_gemm_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  if (err != cudaSuccess) return err;
  unsigned cols = 32;
  while (cols < (unsigned)(D * SBN)) cols <<= 1;
  split_gemm_kernel<D><<<std::min(tiles, 148), SPLIT_NT, smem, st>>>(probs, nprob, segs, tiles, stages, cols);
  return cudaGetLastError();
}

size_t ceil_div(size_t a, size_t b) { return (a + b - 1) / b; }

}  // namespace

size_t split_gemm_workspace(const GemmProb* probs, int nprob, const GemmSeg* segs, int slices) {
  size_t b = 1 << 16;
  const size_t D = slices;
  for (int p = 0; p < nprob; ++p)
    for (int s = 0; s < probs[p].nseg; ++s) {
      const GemmSeg& g = segs[probs[p].seg0 + s];
      for (int k0 = 0; k0 < g.k; k0 += SPLIT_MAX_K) {
        const size_t kk = std::min(SPLIT_MAX_K, g.k - k0);
        const size_t kch = ceil_div(kk, SBK);
        const size_t tm = ceil_div(probs[p].m, SBM), tn = ceil_div(probs[p].n, SBN);
        b += D * kch * (tm * A_TILE + tn * B_TILE) + 512;
        b += (tm * SBM + tn * SBN) * sizeof(int) + 512;
      }
      b += 2 * sizeof(SliceJob) + sizeof(SplitSeg);
    }
  b += (size_t)nprob * sizeof(SplitProb);
  return b;
}

void split_gemm_grouped(const GemmProb* probs, int nprob, const GemmSeg* segs, int slices, DeviceArena& ws,
                        cudaStream_t st, const char* tag) {
  if (slices < SPLIT_MIN_SLICES || slices > SPLIT_MAX_SLICES)
    throw CudaError("split gemm: slices must be in [2, 8]");
  std::vector<SliceJob> jobs;
  std::vector<SplitSeg> ss;
  std::vector<SplitProb> ps;
  int blocks = 0, tiles = 0;
  double flops = 0;
  const int D = slices;
  std::vector<size_t> eoff;  // per job: its exponents within those of the launch
  size_t nexp = 0;
  for (int p = 0; p < nprob; ++p) {
    const GemmProb& G = probs[p];
    if (G.m <= 0 || G.n <= 0) continue;
    SplitProb sp{};
    sp.C = G.C;
    sp.ldc = G.ldc;
    sp.m = G.m;
    sp.n = G.n;
    sp.beta = G.beta;
    sp.seg0 = (int)ss.size();
    sp.tiles_m = (int)ceil_div(G.m, SBM);
    sp.tiles_n = (int)ceil_div(G.n, SBN);
    for (int s = 0; s < G.nseg; ++s) {
      const GemmSeg& g = segs[G.seg0 + s];
      flops += 2.0 * G.m * G.n * g.k;
      for (int k0 = 0; k0 < g.k; k0 += SPLIT_MAX_K) {
        const int kk = std::min(SPLIT_MAX_K, g.k - k0);
        const int kch = (int)ceil_div(kk, SBK);
        // op(A)(i, l) = A[i + l lda] (as stored) or A[l + i lda] (transposed)
        SliceJob ja{};
        ja.rows = G.m;
        ja.K = kk;
        ja.rs = g.transA ? g.lda : 1;
        ja.ls = g.transA ? 1 : g.lda;
        ja.X = g.A + (size_t)k0 * ja.ls;
        ja.tile_rows = SBM;
        ja.kch = kch;
        ja.out = ws.alloc_n<signed char>((size_t)D * kch * sp.tiles_m * A_TILE);
        // op(B)^T(j, l) = op(B)(l, j) = B[l + j ldb] (as stored) or B[j + l ldb]
        SliceJob jb{};
        jb.rows = G.n;
        jb.K = kk;
        jb.rs = g.transB ? 1 : g.ldb;
        jb.ls = g.transB ? g.ldb : 1;
        jb.X = g.B + (size_t)k0 * jb.ls;
        jb.tile_rows = SBN;
        jb.kch = kch;
        jb.out = ws.alloc_n<signed char>((size_t)D * kch * sp.tiles_n * B_TILE);
        SplitSeg q{};
        q.A = ja.out;
        q.B = jb.out;
        q.kch = kch;
        q.alpha = g.alpha;
        ss.push_back(q);
        for (SliceJob* j : {&ja, &jb}) {
          const int t = (int)ceil_div(j->rows, j->tile_rows);
          j->pieces = (int)ceil_div(kch, PIECE);
          j->block0 = blocks;
          blocks += t * j->pieces;
          jobs.push_back(*j);
          eoff.push_back(nexp);
          nexp += (size_t)t * j->tile_rows;
        }
      }
    }
    sp.nseg = (int)ss.size() - sp.seg0;
    if (sp.nseg == 0) {
      // no inner dimension: C = beta C
      if (G.beta == 0.0) {
        for (int c = 0; c < G.n; ++c)
          NRGB_CUDA(cudaMemsetAsync(G.C + (size_t)c * G.ldc, 0, (size_t)G.m * sizeof(double), st));
        continue;
      }
      throw CudaError("split gemm: a problem without segments and beta != 0");
    }
    sp.tile0 = tiles;
    tiles += sp.tiles_m * sp.tiles_n;
    ps.push_back(sp);
  }
  if (ps.empty()) return;
  // the longest tiles first: the last wave of the persistent CTAs ends with short ones
  auto chunks = [&](const SplitProb& p) {
    int c = 0;
    for (int i = p.seg0; i < p.seg0 + p.nseg; ++i) c += ss[i].kch;
    return c;
  };
  std::stable_sort(ps.begin(), ps.end(), [&](const SplitProb& x, const SplitProb& y) { return chunks(x) > chunks(y); });
  tiles = 0;
  for (SplitProb& p : ps) {
    p.tile0 = tiles;
    tiles += p.tiles_m * p.tiles_n;
  }
  int* exps = ws.alloc_n<int>(nexp);
  for (size_t i = 0; i < jobs.size(); ++i) jobs[i].exps = exps + eoff[i];
  for (size_t i = 0; i < ss.size(); ++i) {  // two jobs per segment, A's and B's
    ss[i].eA = exps + eoff[2 * i];
    ss[i].eB = exps + eoff[2 * i + 1];
  }
  // the descriptors in one copy
  const size_t bj = jobs.size() * sizeof(SliceJob), bs = ss.size() * sizeof(SplitSeg), bp = ps.size() * sizeof(SplitProb);
  std::vector<unsigned char> desc(bj + bs + bp);
  memcpy(desc.data(), jobs.data(), bj);
  memcpy(desc.data() + bj, ss.data(), bs);
  memcpy(desc.data() + bj + bs, ps.data(), bp);
  unsigned char* d = ws.alloc_n<unsigned char>(desc.size());
  NRGB_CUDA(cudaMemcpyAsync(d, desc.data(), desc.size(), cudaMemcpyHostToDevice, st));
  const SliceJob* d_j = reinterpret_cast<const SliceJob*>(d);
  const SplitSeg* d_ss = reinterpret_cast<const SplitSeg*>(d + bj);
  const SplitProb* d_ps = reinterpret_cast<const SplitProb*>(d + bj + bs);
  const int nj = (int)jobs.size(), np = (int)ps.size();
  NRGB_CUDA(cudaMemsetAsync(exps, 0x80, nexp * sizeof(int), st));
  NRGB_LAUNCH("split_slice", st, split_exp_kernel<<<blocks, SLICE_NT, 0, st>>>(d_j, nj, D));
  NRGB_CUDA(cudaGetLastError());
  NRGB_LAUNCH("split_slice", st, split_digits_kernel<<<blocks, SLICE_NT, 0, st>>>(d_j, nj, D));
  NRGB_CUDA(cudaGetLastError());
  cudaError_t (*launch)(const SplitProb*, int, const SplitSeg*, int, cudaStream_t) =
      D == 2 ? split_gemm_launch<2> : D == 3 ? split_gemm_launch<3> : D == 4 ? split_gemm_launch<4>
      : D == 5 ? split_gemm_launch<5> : D == 6 ? split_gemm_launch<6>
      : D == 7 ? split_gemm_launch<7> : split_gemm_launch<8>;
  KernelStats::get().add_work(tag, flops);
  cudaError_t err = cudaSuccess;
  NRGB_LAUNCH(tag, st, err = launch(d_ps, np, d_ss, tiles, st));
  NRGB_CUDA(err);
}

int split_gemm_take_error(cudaStream_t st) {
  int h = 0, z = 0;
  NRGB_CUDA(cudaMemcpyFromSymbolAsync(&h, g_split_err, sizeof(int), 0, cudaMemcpyDeviceToHost, st));
  NRGB_CUDA(cudaStreamSynchronize(st));
  if (h) NRGB_CUDA(cudaMemcpyToSymbolAsync(g_split_err, &z, sizeof(int), 0, cudaMemcpyHostToDevice, st));
  return h;
}

}  // namespace nrgb
