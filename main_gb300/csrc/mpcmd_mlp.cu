// Learned surrogate of the batched ensemble: a multilayer perceptron
// (n_in inputs -> n_layers hidden layers of width H with SiLU -> n_out
// outputs) trained and evaluated by this file's own kernels on the
// fifth-generation tensor cores of sm_103a.
//
// k_chain takes 128 rows of a batch through every layer in one CTA, the
// activations staying in tensor memory.  Inference is one launch of it; a
// training step is four launches:
//   k_chain<FORWARD>   the same pass, which also keeps the pre-activations and
//                      the transposed activations, and ends in the loss and the
//                      output gradient instead of the outputs;
//   k_dx               the gradient of the last hidden layer, the one
//                      contraction over the wide output layer (K = n_out), its
//                      columns spread over CTAs;
//   k_chain<BACKWARD>  the gradients of the other hidden layers, layer after
//                      layer on chip;
//   k_dw               every layer's weight and bias gradients, which no longer
//                      depend on one another, with Adam in the epilogue.
// (A step of 256 rows through four hidden layers of 256 to 2,050 outputs: 87 us
// a call, about 60 of them kernels, where 31 launches through memory took 305.
// All of it is latency: a contraction's MMAs wait for one another.  Each kernel
// starts while the one before it runs; 97 us without that.)
// Every contraction is C[M, N] = A[M, K] . B[N, K]^T with both operands BF16
// and K-major.
//
// Warp roles of all three: one thread streams tiles into a ring of
// shared-memory stages with TMA (cp.async.bulk.tensor, 128-byte swizzle,
// mbarriers); one thread issues tcgen05.mma (kind::f16, BF16 operands, FP32
// accumulator in tensor memory) and releases each stage with tcgen05.commit;
// the epilogue warps read the accumulator back with tcgen05.ld (a warp reaches
// the 32 TMEM lanes of its quarter, a lane holds a row) and apply the fused
// epilogue.  What the next GEMM needs transposed is written from that
// thread-per-row layout, consecutive lanes to consecutive rows, so that every
// operand stays K-major; the pre-activations are kept transposed for the same
// reason.  Every mbarrier wait is bounded (two seconds of globaltimer): on
// expiry the kernel raises an error flag, skips its remaining work, waits for
// its copies and MMAs in flight and still frees its tensor memory.
//
// Weights are kept in FP32 (master copy for Adam) and in BF16 twice: [N, K]
// for the forward GEMM and [K, N] for the input-gradient GEMM.
#include <cuda.h>   // CUtensorMap and the encoder's signature (resolved at run time)
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "mpcmd.h"
#include "mpcmd_device.cuh"   // TripleSum, launch chaining

namespace {

using mpcmd::TripleSum;

constexpr int BM = 128;        // output rows per tile (the MMA's M)
constexpr int BK = 64;         // K per stage: one 128-byte swizzle row of BF16

// ------------------------------------------------------------ PTX ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint64_t globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: false (and the error flag raised) after two seconds.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* err) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer();
  for (;;) {
    if (mbar_try_wait(bar, parity)) return true;
    if (globaltimer() - t0 > 2000000000ull) {
      *reinterpret_cast<volatile int*>(err) = 1;   // (host memory: the host reads it after the stream)
      __threadfence_system();
      return false;
    }
  }
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// Shared-memory matrix descriptor of a K-major BF16 tile written by TMA with
// the 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart
// (stride byte offset), the leading byte offset unused for this layout,
// descriptor version 1 (bits 46-48), swizzle mode 2 (128 B) in bits 61-63.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), BF16
// A and B (bits 7-9, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 in
// bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t f16_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// A from tensor memory: row i in lane i, two consecutive K values per column.
__device__ __forceinline__ void mma_bf16_ta(uint32_t tmem, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem),
      "r"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// 16 columns of a warp's 32 lanes (lane = row, registers = columns).
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ float tmem_ld1(uint32_t taddr) {
  uint32_t r;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\ttcgen05.wait::ld.sync.aligned;" : "=r"(r) : "r"(taddr));
  return __uint_as_float(r);
}
// A 32 x 32 block of the accumulator (lane = row, values = columns).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t u[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
        "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(u[i]);
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = __uint_as_float(r[k]);
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// SiLU and its derivative through the logistic function written with the
// hardware's approximate hyperbolic tangent, sigma(z) = (1 + tanh(z / 2)) / 2:
// one special-function instruction per element (the epilogue of a hidden
// layer is bound by them; an exponential and a division take two).  Its
// relative error (about 2^-11) is below the BF16 rounding that follows.
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float silu_f(float z) {
  const float h = 0.5f * z;
  return fmaf(h, tanh_approx(h), h);
}
__device__ __forceinline__ float dsilu_f(float z) {
  const float s = fmaf(0.5f, tanh_approx(0.5f * z), 0.5f);
  return s * (1.f + z * (1.f - s));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&p);
}

// ------------------------------------------------- chain of layers ----
// The layers of 128 rows in one CTA; the modes share everything but what enters
// the chain, what an epilogue computes and where it goes.  Bound by the FP32 output it
// writes (n_out values a row, 537 MB for the surrogate's 65,536 points, 81 us
// at the measured HBM rate) and the weights it streams from L2 for large calls,
// and by the chain of layers for small ones, so:
//   * the activations never leave the SM: an epilogue writes a hidden layer's
//     BF16 activations into tensor memory, where the next layer's MMAs read
//     their A operand (in place: those MMAs start after the layer's own have
//     completed); the input rows are converted into it by the epilogue warps;
//   * shared memory is left to the weights and the stores: one producer thread
//     walks the weight boxes of all layers in order (64 columns of K by the
//     layer's width, or two boxes by 128 output columns) through a ring of
//     32 KB stages, running ahead across layers and row tiles (one load of each
//     box for two CTAs, by multicast, gained nothing: a call of 65,536 points took
//     192.8 us with it and 192.5 without, of 64 points 40.2 and 38.7);
//   * tensor memory holds A (128 columns) and three 128-column accumulators;
//     a hidden layer uses the first two.  Three groups of four epilogue warps
//     (one warp per lane quarter) take the output tiles in turn, so that the
//     stores of three tiles and the MMAs of the next overlap, and the next row
//     tile enters while the last ones are stored;
//   * row tiles that do not fill a wave are split over several CTAs by output
//     columns, each repeating the (much cheaper) hidden layers: with fewer row
//     tiles than SMs all of them, else the last partial wave.
// Inference: one launch instead of six (one conversion and five GEMMs with the
// activations through L2): with the call's own cost, 64 points take 39 us against
// 81, 65,536 points 192 against 284.  A hidden layer takes 3 us (1 us of MMAs, then
// its epilogue, then the next: a chain), two output tiles of 128 columns 4.4 us.
constexpr int INF_GROUPS = 3;                      // epilogue groups of four warps
constexpr int INF_EPI = 4 * INF_GROUPS;
constexpr int INF_THREADS = 64 + 32 * INF_EPI;
constexpr int INF_BN = 128;                        // output columns per job
constexpr int INF_STAGE = 2 * INF_BN * BK * 2;     // 32 KB: a 64 x 256 hidden box or two 64 x 128 output boxes
constexpr int INF_STAGES = 3;
constexpr int INF_WIDE = 64;                       // columns of y a warp stores together
constexpr int INF_PITCH = INF_WIDE + 4;            // staging words per row (16-byte rows, conflict-free quarter warps)
constexpr int INF_CHUNKS = 4;                      // 32-column chunks of a warp, at most
constexpr int MAX_HIDDEN = 16;                     // hidden layers of a configuration
constexpr uint32_t TM_ACC = 128;                   // first accumulator column (A before it)

enum ChainMode : int { INFER = 0, FORWARD = 1, BACKWARD = 2 };

struct InferMaps {
  CUtensorMap w[MAX_HIDDEN];   // hidden layer l: 64 x H
  CUtensorMap out, tail;       // output layer: 64 x 128 and 64 x tail_n
};
struct InferArgs {
  int layers, H, n_in, rows;   // layers of the chain (BACKWARD: all hidden ones but the last)
  int tiles;            // output jobs per row tile (BACKWARD: none)
  int tail_n;           // width of the last output job (a multiple of 16)
  int whole, part, split;   // rounds of whole row tiles; row tiles left over, each split this many ways
  int n_out;
  const float* x;       // [rows, n_in]
  const float* bias[MAX_HIDDEN];
  const float* bias_out;
  float* y;             // [rows, n_out]
  // Training.  FORWARD keeps x^T [64, rows], the pre-activations [H, rows] and
  // the activations [H, rows] of every layer and writes the output gradient as
  // [rows, npad] and [npad, rows]; BACKWARD takes the last hidden layer's
  // gradient [rows, H] and writes those of the layers below, [H, rows], last
  // first (zt and at in the same order).
  const float *t, *w;   // targets [rows, n_out], output weights [n_out]
  float inv_rows;       // 1 / rows where that is exact, else 0
  int npad;
  float* zt[MAX_HIDDEN];
  __nv_bfloat16* at[MAX_HIDDEN];
  __nv_bfloat16 *xt, *dy, *dyt;
  const __nv_bfloat16* dz;
  double* loss;         // [CTAs * INF_EPI] partial sums of w (y - t)^2
  int* err;
};

constexpr size_t INF_SMEM = 1024 + (size_t)INF_STAGES * INF_STAGE + (size_t)INF_EPI * 32 * (INF_PITCH + INF_CHUNKS) * 4 +
                            (2 * INF_STAGES + 2 * INF_GROUPS + 3) * 8 + 16;
static_assert(INF_SMEM <= 232448, "shared memory of one CTA");

// Work item v of this CTA: its row tile and its output jobs [t0, t1).
__device__ __forceinline__ bool infer_item(const InferArgs& a, int v, int& mt, int& t0, int& t1) {
  const int g = (int)gridDim.x, b = (int)blockIdx.x;
  if (v < a.whole) { mt = v * g + b; t0 = 0; t1 = a.tiles; return true; }
  if (v > a.whole || a.part == 0 || b >= a.part * a.split) return false;
  const int q = b / a.part;
  mt = a.whole * g + b % a.part;
  t0 = a.tiles * q / a.split;
  t1 = a.tiles * (q + 1) / a.split;
  return true;
}

// Whether this CTA keeps piece i of what a training pass keeps (32 columns of
// a layer, counted through the layers): the CTAs that share a row tile all
// compute its layers, and take turns in writing them.
__device__ __forceinline__ bool keeps(const InferArgs& a, int v, int i) {
  return v < a.whole || i % a.split == (int)blockIdx.x / a.part;
}

// 4 or 16 bytes to shared memory (this thread sees them after cp.async.wait_all).
template <int N>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
  if constexpr (N == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Consecutive columns of a lane's row, packed in pairs, as a column each of a
// transposed matrix (consecutive lanes: consecutive rows).
template <int N>
__device__ __forceinline__ void put_columns(__nv_bfloat16* dst, size_t ld, const uint32_t (&w)[N]) {
  unsigned short* d = reinterpret_cast<unsigned short*>(dst);
#pragma unroll
  for (int q = 0; q < N; ++q) {
    d[(size_t)(2 * q) * ld] = (unsigned short)(w[q] & 0xFFFFu);
    d[(size_t)(2 * q + 1) * ld] = (unsigned short)(w[q] >> 16);
  }
}

// A 32-row block of y of INF_WIDE columns through the warp's staging tile: the
// values of 32 columns are staged a lane per row, and when the block is
// complete every instruction writes VB bytes a lane (VB: what the rows'
// alignment allows) of as few rows as that covers.  L2 takes one request per
// 128-byte line a piece of a row touches, whole or not, and rows of 2,050
// values start anywhere in a line: 64-column pieces touch 3 lines for 2 and 256
// columns of 128 rows take 4.4 us, 32-column pieces 2 for 1 and 5.7 us
// (aligned rows: 3.1 us).  Measured and not kept: lines assembled whole in the
// staging tile across chunks (7.6 us, the rotated staging costs more than the
// requests saved), 128-column pieces of 16 or 8 rows at a time (4.7 and 6.1 us).
__device__ __forceinline__ void stage_chunk(uint32_t* buf, int lane, int c, const float (&v)[32], const float* bias) {
  const float4* bp = reinterpret_cast<const float4*>(bias);
#pragma unroll
  for (int q = 0; q < 32; q += 4) {
    const float4 b = bp[q / 4];
    *reinterpret_cast<float4*>(buf + lane * INF_PITCH + c + q) =
        make_float4(v[q] + b.x, v[q + 1] + b.y, v[q + 2] + b.z, v[q + 3] + b.w);
  }
}
template <int VB>
__device__ __forceinline__ void store_block(const uint32_t* buf, int lane, char* base, size_t pitch) {
  constexpr int LPR = INF_WIDE * 4 / VB;            // lanes per row (more than a warp's: a row in parts)
  constexpr int RPI = LPR < 32 ? 32 / LPR : 1;      // rows per instruction
  constexpr int PPR = LPR > 32 ? LPR / 32 : 1;      // instructions per row
  const int sub = LPR < 32 ? lane / LPR : 0, q = LPR < 32 ? lane % LPR : lane;
  const uint32_t* src = buf + sub * INF_PITCH + q * (VB / 4);
  char* dst = base + (size_t)sub * pitch + q * VB;
  const size_t step = RPI * pitch;
#pragma unroll 8
  for (int it = 0; it < 32 / RPI; ++it, dst += step) {
#pragma unroll
    for (int h = 0; h < PPR; ++h) {
      const uint32_t* s = src + it * RPI * INF_PITCH + h * 32 * (VB / 4);
      char* d = dst + h * 32 * VB;
      if constexpr (VB == 16) *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(s);
      else if constexpr (VB == 8) *reinterpret_cast<uint2*>(d) = *reinterpret_cast<const uint2*>(s);
      else *reinterpret_cast<uint32_t*>(d) = *s;
    }
  }
}

// A ragged piece of it: 32 columns staged a lane per row, of which `rows` rows
// and `cols` columns are written.
__device__ __forceinline__ void store_ragged(uint32_t* buf, const uint32_t (&w)[32], int lane, char* base, size_t pitch,
                                             int rows, int cols) {
#pragma unroll
  for (int q = 0; q < 32; q += 4)
    *reinterpret_cast<uint4*>(buf + lane * INF_PITCH + q) = make_uint4(w[q], w[q + 1], w[q + 2], w[q + 3]);
  __syncwarp();
#pragma unroll 4
  for (int r = 0; r < 32; ++r)
    if (r < rows && lane < cols) *reinterpret_cast<uint32_t*>(base + r * pitch + 4 * lane) = buf[r * INF_PITCH + lane];
  __syncwarp();
}

// VB (INFER): the largest of 16, 8 and 4 bytes that divides the address of
// every row of y
template <int MODE, int VB>
__global__ void __launch_bounds__(INF_THREADS, 1)
    k_chain(const __grid_constant__ InferMaps maps, const __grid_constant__ InferArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sRing = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint32_t* stage_all = reinterpret_cast<uint32_t*>(sRing + INF_STAGES * INF_STAGE);
  float* bias_all = reinterpret_cast<float*>(stage_all + INF_EPI * 32 * INF_PITCH);   // a job's biases, per warp
  uint64_t* bars = reinterpret_cast<uint64_t*>(bias_all + INF_EPI * 32 * INF_CHUNKS);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * INF_STAGES + 2 * INF_GROUPS + 3);
  __shared__ volatile int bail;   // a wait of this CTA expired
  __shared__ int issued;          // stages the producer filled
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nkh = a.H / BK, nk0 = MODE == BACKWARD ? nkh : 1;   // K boxes of a layer, of the first
  // barriers: full, empty (ring), accf, acce (output accumulators), hacc (a
  // hidden layer's MMAs have completed), hready (the A operand of the next
  // layer is written and the accumulator read), done
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * INF_STAGES, accf0 = empty0 + 8 * INF_STAGES,
                 acce0 = accf0 + 8 * INF_GROUPS, hacc = acce0 + 8 * INF_GROUPS, hready = hacc + 8, done = hacc + 16;
  if (threadIdx.x == 0) {
    bail = 0;
    issued = 0;
    for (int s = 0; s < INF_STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
    for (int b = 0; b < INF_GROUPS; ++b) { mbar_init(accf0 + 8 * b, 1); mbar_init(acce0 + 8 * b, MODE == FORWARD ? INF_EPI : 4); }
    mbar_init(hacc, 1);
    mbar_init(hready, INF_EPI);
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const uint32_t tmem = *tmem_slot;
  if constexpr (MODE == FORWARD) mpcmd::let_next_start();   // (an ordinary launch: nothing before it still runs)
  if constexpr (MODE == BACKWARD) mpcmd::after_previous();

  if (warp == 0) {
    if (lane == 0) {
      // weight producer
      int g = 0, mt, t0, t1;
      // one stage: boxes k..k+nb-1 of a layer, `n` rows of weights from `row` each
      auto fill = [&](const CUtensorMap* m, int k, int nb, int row, int n) -> bool {
        const int s = g % INF_STAGES;
        if (g >= INF_STAGES && !mbar_wait(empty0 + 8 * s, ((uint32_t)(g / INF_STAGES) & 1u) ^ 1u, a.err)) {
          bail = 1;
          return false;
        }
        mbar_expect_tx(full0 + 8 * s, (uint32_t)(nb * n * BK * 2));
        for (int q = 0; q < nb; ++q)
          tma_load_2d(smem_u32(sRing + s * INF_STAGE + q * (INF_STAGE / 2)), m, full0 + 8 * s, (k + q) * BK, row);
        ++g;
        return true;
      };
      bool ok = true;
      for (int v = 0; ok && !bail && infer_item(a, v, mt, t0, t1); ++v) {
        for (int l = 0; l < a.layers && ok; ++l)
          for (int k = 0; k < (l == 0 ? nk0 : nkh) && ok; ++k) ok = fill(&maps.w[l], k, 1, 0, a.H);
        for (int t = t0; t < t1 && ok; ++t) {
          const bool tail = t == a.tiles - 1;
          for (int k = 0; k < nkh && ok; k += 2)
            ok = fill(tail ? &maps.tail : &maps.out, k, min(2, nkh - k), t * INF_BN, tail ? a.tail_n : INF_BN);
        }
      }
      issued = g;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // MMA issuer: output job o accumulates into buffer o % 3
      int g = 0, o = 0, hp = 0, mt, t0, t1;
      auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
        if (mbar_wait(bar, parity, a.err)) return true;
        bail = 1;
        return false;
      };
      // boxes k..k+nb-1 of the stage against A's columns
      auto stage = [&](uint32_t acc, uint32_t idesc, int k, int nb) -> bool {
        const int s = g % INF_STAGES;
        if (!wait(full0 + 8 * s, (uint32_t)(g / INF_STAGES) & 1u)) return false;
        tmem_fence_after();
        for (int q = 0; q < nb; ++q) {
          const uint32_t b0 = smem_u32(sRing + s * INF_STAGE + q * (INF_STAGE / 2));
          const uint32_t a0 = tmem + (uint32_t)((k + q) * (BK / 2));
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            mma_bf16_ta(acc, a0 + 8 * kk, sw128_desc(b0 + 32 * kk), idesc, (k + q > 0 || kk > 0) ? 1u : 0u);
        }
        mma_commit(empty0 + 8 * s);
        ++g;
        return true;
      };
      const uint32_t hid = f16_idesc(BM, a.H);
      bool ok = true;
      for (int v = 0; ok && !bail && infer_item(a, v, mt, t0, t1); ++v) {
        // the accumulators a hidden layer covers: their last output tiles have been read
        for (int b = 0; b < 2 && ok; ++b) {
          const int uses = (o + 2 - b) / 3;   // output jobs so far in buffer b
          if (uses > 0) ok = wait(acce0 + 8 * b, (uint32_t)(uses - 1) & 1u);
        }
        for (int l = 0; l < a.layers && ok; ++l) {
          if (!(ok = wait(hready, (uint32_t)hp++ & 1u))) break;
          tmem_fence_after();
          for (int k = 0; k < (l == 0 ? nk0 : nkh) && ok; ++k) ok = stage(tmem + TM_ACC, hid, k, 1);
          if (ok) mma_commit(hacc);
        }
        if (ok) ok = wait(hready, (uint32_t)hp++ & 1u);
        // (BACKWARD has no output job: the next input may enter.  The epilogue waits
        // for this and not for hready itself, whose next phase its own input
        // completes: this thread must have seen the one before by then.)
        if (MODE == BACKWARD && ok) mbar_arrive(accf0);
        for (int t = t0; t < t1 && ok; ++t, ++o) {
          const int b = o % 3;
          if (o >= 3 && !(ok = wait(acce0 + 8 * b, ((uint32_t)(o / 3) & 1u) ^ 1u))) break;
          tmem_fence_after();
          const uint32_t idesc = f16_idesc(BM, t == a.tiles - 1 ? a.tail_n : INF_BN);
          for (int k = 0; k < nkh && ok; k += 2)
            ok = stage(tmem + TM_ACC + (uint32_t)(b * INF_BN), idesc, k, min(2, nkh - k));
          if (ok) mma_commit(accf0 + 8 * b);   // arrives when the job's MMAs have completed
        }
      }
      mma_commit(done);   // arrives when every MMA issued above has completed
    }
  } else {
    const int ew = warp - 2;
    const int quarter = warp & 3;          // the TMEM lanes this warp reaches
    const int group = ew >> 2;
    uint32_t* buf = stage_all + ew * 32 * INF_PITCH;
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
    // A's columns and the reads of the accumulator before it are done
    auto publish = [&]() {
      tmem_wait_st();
      tmem_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(hready);
    };
    // what enters the chain: the input rows as 64 columns of K (zero-padded),
    // 32 by each of two groups, or the rows of a gradient
    auto load_input = [&](int mt, bool keep) {
      const int64_t row = (int64_t)mt * BM + quarter * 32 + lane;
      if constexpr (MODE == BACKWARD) {
        // Through the staging tile, four lanes to a row's 64 bytes (a lane per row
        // costs 32 lines an instruction: 3 us).
        constexpr int P = 16 * (INF_CHUNKS - 1) + 4;
        const int64_t r0 = (int64_t)mt * BM + quarter * 32 + (lane >> 2);
#pragma unroll
        for (int i = 0; i < INF_CHUNKS - 1; ++i) {
          const int c0 = 32 * (group + INF_GROUPS * i) + 8 * (lane & 3);
#pragma unroll
          for (int q = 0; q < 32; q += 8)
            if (c0 < a.H && r0 + q < a.rows)
              copy_async<16>(buf + ((lane >> 2) + q) * P + 16 * i + 4 * (lane & 3), a.dz + (r0 + q) * a.H + c0);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
#pragma unroll
        for (int i = 0; i < INF_CHUNKS - 1; ++i) {
          uint32_t w[16];
#pragma unroll
          for (int q = 0; q < 16; q += 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(buf + lane * P + 16 * i + q);
            w[q] = v.x; w[q + 1] = v.y; w[q + 2] = v.z; w[q + 3] = v.w;
          }
          if (32 * (group + INF_GROUPS * i) < a.H) tmem_st16(lanes + (uint32_t)(16 * (group + INF_GROUPS * i)), w);
        }
        __syncwarp();
      } else if (group < 2) {
        const float* xr = a.x + row * a.n_in;
        const int have = row < a.rows ? a.n_in : 0;
        uint32_t w[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const int c = 32 * group + 2 * q;
          w[q] = pack_bf16(c < have ? xr[c] : 0.f, c + 1 < have ? xr[c + 1] : 0.f);
        }
        tmem_st16(lanes + (uint32_t)(16 * group), w);
        if (MODE == FORWARD && keep && row < a.rows) put_columns(a.xt + (size_t)(32 * group) * a.rows + row, a.rows, w);
      }
      publish();
    };
    // The biases of a job travel through registers, fetched one job ahead (their
    // latency was a quarter of an output tile's time).  A hidden layer's chunks
    // go round the groups; an output tile is one group's.
    float* bias = bias_all + ew * 32 * INF_CHUNKS;
    float ahead[INF_CHUNKS];
    auto fetch_hidden = [&](int l) {
#pragma unroll
      for (int i = 0; i < INF_CHUNKS; ++i) {
        const int c = 32 * (group + INF_GROUPS * i) + lane;
        ahead[i] = MODE != BACKWARD && c < a.H ? a.bias[l][c] : 0.f;
      }
    };
    auto fetch_out = [&](int t) {
#pragma unroll
      for (int i = 0; i < INF_CHUNKS; ++i) {
        const int c = t * INF_BN + 32 * i + lane;
        ahead[i] = c < a.n_out ? a.bias_out[c] : 0.f;
      }
    };
    auto put_bias = [&]() {
      __syncwarp();
#pragma unroll
      for (int i = 0; i < INF_CHUNKS; ++i) bias[32 * i + lane] = ahead[i];
      __syncwarp();
    };
    auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
      if (mbar_wait(bar, parity, a.err)) { tmem_fence_after(); return true; }
      bail = 1;
      return false;
    };
    const size_t pitch = (size_t)a.n_out * 4;
    int o = 0, h = 0, mt, t0, t1;
    bool ok = infer_item(a, 0, mt, t0, t1);
    if (ok) { load_input(mt, keeps(a, 0, a.layers * a.H / 32)); fetch_hidden(0); }
    double loss = 0.;
    // FORWARD: this warp's 32 target rows of a job's columns into its staging
    // tile, its chunks side by side
    auto load_targets = [&](int row0, int rows, int t) {
#pragma unroll 1
      for (int r0 = 0; r0 < 32; r0 += 16) {
        float v[32];   // 32 loads in flight
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int r = r0 + (i >> 1), c = 32 * (group + INF_GROUPS * (i & 1)) + lane, col = t * INF_BN + c;
          v[i] = r < rows && c < INF_BN && col < a.n_out ? a.t[(int64_t)(row0 + r) * a.n_out + col] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 32; ++i)
          reinterpret_cast<float*>(buf)[(r0 + (i >> 1)) * INF_PITCH + 32 * (i & 1) + lane] = v[i];
      }
      __syncwarp();
    };
    for (int v = 0; ok; ++v) {
      const int64_t row = (int64_t)mt * BM + quarter * 32 + lane;
      const int row0 = mt * BM + quarter * 32;
      const int rows = a.rows - row0 < 32 ? a.rows - row0 : 32;
      // this group's first output job of the item (FORWARD: the groups share every
      // job, a training batch leaves a CTA one or two)
      const int first = MODE == FORWARD ? t0 : t0 + (group - o % 3 + 3) % 3;
      constexpr int stride = MODE == FORWARD ? 1 : 3;
      if (MODE == FORWARD) load_targets(row0, rows, first);
      for (int l = 0; l < a.layers && ok; ++l, ++h) {
        put_bias();
        if (l + 1 < a.layers) fetch_hidden(l + 1);
        else if (first < t1) fetch_out(first);
        // BACKWARD: this warp's pre-activations arrive while the MMAs run, the
        // first chunk's in registers
        float z0[MODE == BACKWARD ? 32 : 1];
        if constexpr (MODE == BACKWARD) {
          const bool real = row < a.rows;
          const float* zp = a.zt[l] + (real ? row : 0);
#pragma unroll
          for (int i = 1; i < INF_CHUNKS - 1; ++i) {
            const int c0 = 32 * (group + INF_GROUPS * i);
            if (c0 < a.H)
#pragma unroll
              for (int q = 0; q < 32; ++q)
                copy_async<4>(buf + (32 * (i - 1) + q) * 32 + lane, zp + (size_t)(c0 + q) * a.rows);
          }
          if (32 * group < a.H)
#pragma unroll
            for (int q = 0; q < 32; ++q) z0[q] = zp[(size_t)(32 * group + q) * a.rows];
          asm volatile("cp.async.wait_all;" ::: "memory");
        }
        if (!(ok = wait(hacc, (uint32_t)h & 1u))) break;
        int i = 0;
#pragma unroll 1
        for (int c0 = 32 * group; c0 < a.H; c0 += 32 * INF_GROUPS, ++i) {
          float z[32];
          const bool keep = MODE != INFER && row < a.rows && keeps(a, v, (l * a.H + c0) / 32);
          tmem_ld32(lanes + TM_ACC + (uint32_t)c0, z);
          uint32_t w[16];
          if constexpr (MODE == BACKWARD) {
            // through SiLU' of the pre-activations below
            if (i > 0) {
#pragma unroll
              for (int q = 0; q < 32; ++q) z0[q] = __uint_as_float(buf[(32 * (i - 1) + q) * 32 + lane]);
            }
#pragma unroll
            for (int q = 0; q < 16; ++q)
              w[q] = pack_bf16(z[2 * q] * dsilu_f(z0[2 * q]), z[2 * q + 1] * dsilu_f(z0[2 * q + 1]));
          } else {
            const float4* bp = reinterpret_cast<const float4*>(bias + 32 * i);
#pragma unroll
            for (int q = 0; q < 32; q += 4) {
              const float4 b4 = bp[q / 4];
              z[q] += b4.x; z[q + 1] += b4.y; z[q + 2] += b4.z; z[q + 3] += b4.w;
              w[q / 2] = pack_bf16(silu_f(z[q]), silu_f(z[q + 1]));
              w[q / 2 + 1] = pack_bf16(silu_f(z[q + 2]), silu_f(z[q + 3]));
            }
            if (MODE == FORWARD && keep) {
              float* zp = a.zt[l] + (size_t)c0 * a.rows + row;
#pragma unroll
              for (int q = 0; q < 32; ++q) zp[(size_t)q * a.rows] = z[q];
            }
          }
          if (MODE != INFER && keep) put_columns(a.at[l] + (size_t)c0 * a.rows + row, a.rows, w);
          tmem_st16(lanes + (uint32_t)(c0 / 2), w);
        }
        publish();
      }
      if (!ok) break;
      int nmt = 0, nt0 = 0, nt1 = 0;
      const bool more = infer_item(a, v + 1, nmt, nt0, nt1);
      const int last = o + t1 - t0 - 1;   // the item's last output job
      bool entered = false;
      for (int t = first; t < t1; t += stride) {
        const int jo = o + t - t0, b = MODE == FORWARD ? jo % 3 : group;
        put_bias();
        if (t + stride < t1) fetch_out(t + stride);
        else fetch_hidden(0);
        if (MODE == FORWARD && t > first) load_targets(row0, rows, t);
        if (!(ok = wait(accf0 + 8 * b, (uint32_t)(jo / 3) & 1u))) break;
        // the row tile's last MMAs have read A: the next row tile enters
        if (jo == last && more) { load_input(nmt, keeps(a, v + 1, a.layers * a.H / 32)); entered = true; }
        const int cols = min(a.n_out - t * INF_BN, INF_BN);
        const bool full = rows == 32 && cols == INF_BN;
        char* yb = reinterpret_cast<char*>(a.y + t * INF_BN) + (size_t)row0 * pitch;
#pragma unroll 1
        for (int c0 = MODE == FORWARD ? 32 * group : 0; c0 < cols; c0 += MODE == FORWARD ? 32 * INF_GROUPS : 32) {
          float y[32];
          tmem_ld32(lanes + TM_ACC + (uint32_t)(b * INF_BN + c0), y);
          if constexpr (MODE == FORWARD) {
            // Weighted squared error and its gradient 2 w (y - t) / rows.  The 32
            // terms of a chunk add up in three floats, without loss against FP64, and
            // its chunks in FP64 (an FP64 add a term would take 8 us: the pipe has two
            // lanes an SM).
            const int col = t * INF_BN + c0;
            const float4* tp = reinterpret_cast<const float4*>(buf + lane * INF_PITCH + (c0 < 32 * INF_GROUPS ? 0 : 32));
            const float wl = col + lane < a.n_out ? a.w[col + lane] : 0.f;
            TripleSum part{};
            uint32_t g[16];
#pragma unroll
            for (int q = 0; q < 32; q += 4) {
              const float4 t4 = tp[q / 4];
              const float tq[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float wt = __shfl_sync(0xffffffffu, wl, q + e);
                float d = (y[q + e] + bias[c0 + q + e]) - tq[e];
                d = row < a.rows && col + q + e < a.n_out ? d : 0.f;
                mpcmd::triple_add(part, __fmul_rn(__fmul_rn(wt, d), d));
                y[q + e] = 2.f * wt * d;
              }
            }
            const bool beyond = __any_sync(0xffffffffu, !isfinite(part.hi));
            if (!beyond) loss += mpcmd::triple_value(part);
            // (a power of two divides exactly as its reciprocal multiplies)
            if (a.inv_rows != 0.f) {
#pragma unroll
              for (int q = 0; q < 32; ++q) y[q] *= a.inv_rows;
            } else {
#pragma unroll
              for (int q = 0; q < 32; ++q) y[q] /= (float)a.rows;
            }
#pragma unroll
            for (int q = 0; q < 16; ++q) g[q] = pack_bf16(y[2 * q], y[2 * q + 1]);
            if (row < a.rows) {
              uint4* dst = reinterpret_cast<uint4*>(a.dy + row * a.npad + col);
#pragma unroll
              for (int q = 0; q < 4; ++q) dst[q] = make_uint4(g[4 * q], g[4 * q + 1], g[4 * q + 2], g[4 * q + 3]);
              put_columns(a.dyt + (size_t)col * a.rows + row, a.rows, g);
            }
            if (beyond) {
              // a sum beyond FP32's largest number: the terms once more, in FP64
#pragma unroll 1
              for (int q = 0; q < 32; ++q) {
                const float wt = __shfl_sync(0xffffffffu, wl, q);
                float d = tmem_ld1(lanes + TM_ACC + (uint32_t)(b * INF_BN + c0 + q)) + bias[c0 + q];
                d = row < a.rows && col + q < a.n_out ? d - reinterpret_cast<const float*>(tp)[q] : 0.f;
                loss += (double)__fmul_rn(__fmul_rn(wt, d), d);
              }
            }
          } else if (full) {
            stage_chunk(buf, lane, c0 % INF_WIDE, y, bias + c0);
            if ((c0 + 32) % INF_WIDE == 0) {
              __syncwarp();
              store_block<VB>(buf, lane, yb + 4 * (c0 + 32 - INF_WIDE), pitch);
              __syncwarp();
            }
          } else {
            uint32_t w[32];
#pragma unroll
            for (int q = 0; q < 32; ++q) w[q] = __float_as_uint(y[q] + bias[c0 + q]);
            store_ragged(buf, w, lane, yb + 4 * c0, pitch, rows, cols - c0);
          }
        }
        tmem_fence_before();
        __syncwarp();   // (FORWARD: the staging tile has been read, too)
        if (lane == 0) mbar_arrive(acce0 + 8 * b);
      }
      if (ok && more && !entered) {
        // another group has the last output job
        if (first >= t1) fetch_hidden(0);
        if constexpr (MODE == BACKWARD) {
          // no output job: the next input may enter when the issuer has seen that
          // every warp has read the last accumulator
          if ((ok = wait(accf0, (uint32_t)v & 1u))) load_input(nmt, true);
        } else if ((ok = wait(accf0 + 8 * (last % 3), (uint32_t)(last / 3) & 1u))) {
          load_input(nmt, keeps(a, v + 1, a.layers * a.H / 32));
        }
      }
      o += t1 - t0;
      mt = nmt; t0 = nt0; t1 = nt1;
      ok = ok && more;
    }
    if constexpr (MODE == FORWARD) {
      for (int q = 16; q > 0; q >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, q);
      if (lane == 0) a.loss[(size_t)blockIdx.x * INF_EPI + ew] = loss;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // every MMA and every load that was issued has completed before the
    // tensor memory is freed and the CTA exits
    mbar_wait(done, 0, a.err);
    const int g1 = issued;
    for (int g = g1 - INF_STAGES < 0 ? 0 : g1 - INF_STAGES; g < g1; ++g)
      mbar_wait(full0 + 8 * (g % INF_STAGES), (uint32_t)(g / INF_STAGES) & 1u, a.err);
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ------------------------------------------------- training GEMMs ----
// Pipeline of the two kernels below: tiles of 128 x BN, A and B boxes of a K
// step in one stage, two accumulators.  Barriers full[S], empty[S], accf[2],
// acce[2], done.
template <int BN, int S, int EPI>
struct Pipe {
  static constexpr int A_STAGE = BM * BK * 2, BOX = A_STAGE + BN * BK * 2;
  static constexpr int THREADS = 64 + 32 * EPI;
  static constexpr uint32_t COLS = 2 * BN < 32 ? 32 : 2 * BN;
  uint8_t* ring;
  uint32_t full, empty, accf, acce, done, tmem;
  int* err;
  volatile int* bail;

  static constexpr size_t bytes(size_t extra) {
    return 1024 + (size_t)S * BOX + (2 * S + 5) * 8 + 16 + (extra ? extra + 16 : 0);
  }

  // Shared memory, barriers and tensor memory; returns what follows the ring.
  __device__ __forceinline__ uint8_t* open(uint8_t* raw, volatile int* bail_, int* issued, int* err_) {
    ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring + S * BOX);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 5);
    full = smem_u32(bars); empty = full + 8 * S; accf = empty + 8 * S; acce = accf + 16; done = acce + 16;
    err = err_; bail = bail_;
    if (threadIdx.x == 0) {
      *bail = 0;
      *issued = 0;
      for (int s = 0; s < S; ++s) { mbar_init(full + 8 * s, 1); mbar_init(empty + 8 * s, 1); }
      for (int b = 0; b < 2; ++b) { mbar_init(accf + 8 * b, 1); mbar_init(acce + 8 * b, EPI); }
      mbar_init(done, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if ((threadIdx.x >> 5) == 1) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    tmem = *slot;
    return reinterpret_cast<uint8_t*>(bars) + (2 * S + 5) * 8 + 16;
  }
  // one tile's loads (producer thread); g counts stages
  __device__ __forceinline__ bool load(int& g, int nk, const CUtensorMap* ta, int row_a, const CUtensorMap* tb,
                                       int row_b) {
    for (int k = 0; k < nk; ++k) {
      const int s = g % S;
      if (g >= S && !mbar_wait(empty + 8 * s, ((uint32_t)(g / S) & 1u) ^ 1u, err)) { *bail = 1; return false; }
      mbar_expect_tx(full + 8 * s, BOX);
      tma_load_2d(smem_u32(ring + s * BOX), ta, full + 8 * s, k * BK, row_a);
      tma_load_2d(smem_u32(ring + s * BOX + A_STAGE), tb, full + 8 * s, k * BK, row_b);
      ++g;
    }
    return true;
  }
  // tile j's MMAs (issuer thread)
  __device__ __forceinline__ bool multiply(int& g, int j, int nk) {
    constexpr uint32_t idesc = f16_idesc(BM, BN);
    const int b = j & 1;
    if (j >= 2 && !mbar_wait(acce + 8 * b, ((uint32_t)(j >> 1) & 1u) ^ 1u, err)) { *bail = 1; return false; }
    tmem_fence_after();
    const uint32_t acc = tmem + (uint32_t)(b * BN);
    for (int k = 0; k < nk; ++k, ++g) {
      const int s = g % S;
      if (!mbar_wait(full + 8 * s, (uint32_t)(g / S) & 1u, err)) { *bail = 1; return false; }
      tmem_fence_after();
      const uint32_t a0 = smem_u32(ring + s * BOX), b0 = a0 + A_STAGE;
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk)
        mma_bf16(acc, sw128_desc(a0 + 32 * kk), sw128_desc(b0 + 32 * kk), idesc, (k > 0 || kk > 0) ? 1u : 0u);
      mma_commit(empty + 8 * s);
    }
    mma_commit(accf + 8 * b);
    return true;
  }
  // columns c0.. of tile j's accumulator of this warp's quarter (epilogue warps)
  __device__ __forceinline__ bool ready(int j) {
    if (!mbar_wait(accf + 8 * (j & 1), (uint32_t)(j >> 1) & 1u, err)) { *bail = 1; return false; }
    tmem_fence_after();
    return true;
  }
  template <int N>
  __device__ __forceinline__ void read(int j, int quarter, int c0, float (&v)[N]) {
    const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((j & 1) * BN + c0);
    if constexpr (N == 32) tmem_ld32(at, v);
    else tmem_ld16(at, v);
  }
  __device__ __forceinline__ void release(int j) {
    tmem_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(acce + 8 * (j & 1));
  }
  // every MMA and every load that was issued has completed before the tensor
  // memory is freed and the CTA exits
  __device__ __forceinline__ void close(const int* issued) {
    __syncthreads();
    if (threadIdx.x == 0) {
      mbar_wait(done, 0, err);
      const int g1 = *issued;
      for (int g = g1 - S < 0 ? 0 : g1 - S; g < g1; ++g) mbar_wait(full + 8 * (g % S), (uint32_t)(g / S) & 1u, err);
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    if ((threadIdx.x >> 5) == 1)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
  }
};

// Gradient of the last hidden layer: dz = (dY . W_out) * SiLU'(z) as [rows, H]
// and [H, rows].  Bound by its chain of MMAs: each adds 16 of K to the sum of
// the one before, and takes 134 cycles whatever its width (64-row tiles, or 16
// stages in flight: the same 540 cycles for 64 of K; 12 us for 2,050 outputs).
// So the columns are spread over CTAs, 32 to each.  Block 0 also adds up the
// loss.
struct DxArgs {
  int rows, H, nk;      // nk: K boxes that hold outputs (the padding is zero)
  const float* zt;      // [H, rows]
  __nv_bfloat16 *dz, *dzt;
  const double* loss;   // partial sums
  int n_loss;
  double* loss_out;     // host memory: sum / rows
  int* err;
};
using DxPipe = Pipe<32, 10, 4>;

__global__ void __launch_bounds__(DxPipe::THREADS, 1)
    k_dx(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, DxArgs a) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int bail;
  __shared__ int issued;
  DxPipe p;
  p.open(smem_raw, &bail, &issued, a.err);
  mpcmd::after_previous();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_n = a.H / 32, units = (a.rows / BM) * tiles_n;
  if (warp == 0) {
    if (lane == 0) {
      int g = 0;
      for (int u = blockIdx.x; u < units && !bail; u += gridDim.x)
        if (!p.load(g, a.nk, &ta, (u / tiles_n) * BM, &tb, (u % tiles_n) * 32)) break;
      issued = g;
    }
    __syncwarp();
    if (blockIdx.x == 0) {
      double s = 0.;
#pragma unroll 8
      for (int i = lane; i < a.n_loss; i += 32) s += a.loss[i];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) *a.loss_out = s / (double)a.rows;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int g = 0, j = 0;
      for (int u = blockIdx.x; u < units && !bail; u += gridDim.x, ++j)
        if (!p.multiply(g, j, a.nk)) break;
      mma_commit(p.done);
    }
  } else {
    const int quarter = warp & 3;
    int j = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++j) {
      const int row = (u / tiles_n) * BM + quarter * 32 + lane, n = (u % tiles_n) * 32;
      float z[32];   // fetched while the MMAs run
#pragma unroll
      for (int q = 0; q < 32; ++q) z[q] = a.zt[(size_t)(n + q) * a.rows + row];
      if (!p.ready(j)) break;
      float v[32];
      p.read(j, quarter, 0, v);
      uint32_t w[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) w[q] = pack_bf16(v[2 * q] * dsilu_f(z[2 * q]), v[2 * q + 1] * dsilu_f(z[2 * q + 1]));
      uint4* dst = reinterpret_cast<uint4*>(a.dz + (size_t)row * a.H + n);
#pragma unroll
      for (int q = 0; q < 4; ++q) dst[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
      put_columns(a.dzt + (size_t)n * a.rows + row, a.rows, w);
      p.release(j);
    }
  }
  p.close(&issued);
}

// Weight and bias gradients of every layer, dW = dZ^T . X^T^T over the batch and
// db = row sums of dZ^T, and either written out or applied: Adam (Kingma & Ba,
// 2015) on the FP32 master tensors with the step's bias corrections, which
// refreshes the BF16 copies [n, k] and [k, n].  Work units: the 128 x 64 tiles of
// every layer, then blocks of 64 biases; 5 of its 8 us are Adam's divisions and
// root, so 16 warps share a tile (8: 7 us); the parameters and moments (24 bytes a
// weight, in L2) are fetched before the previous kernel has ended (__ldcg: see
// after_previous): only this kernel writes them, in the step before, and every
// kernel of a step lets the next one start after its own wait.
struct AdamArgs {
  float lr, b1, b2, eps, c1, c2;
};
struct DwLayer {
  int n, k;             // padded widths of W [n, k]
  int first, first_bias;   // first work unit of its tiles and of its biases
  float *w, *m, *v, *g;
  float *bw, *bm, *bv, *bg;
  __nv_bfloat16 *wb, *wt;
  const __nv_bfloat16* dzt;   // [n, rows]
};
struct DwMaps {
  CUtensorMap a[MAX_HIDDEN + 1], b[MAX_HIDDEN + 1];   // dZ^T [n, rows], X^T [k, rows]
};
struct DwArgs {
  int layers, rows, tiles, units;   // tiles: units with MMAs
  DwLayer l[MAX_HIDDEN + 1];
  AdamArgs adam;
  int* err;
};
constexpr int DW_EPI = 16;
using DwPipe = Pipe<64, 4, DW_EPI>;
constexpr int DW_PITCH = 20;   // words of a staged row
constexpr size_t DW_SMEM = DwPipe::bytes((size_t)DW_EPI * 32 * DW_PITCH * 4);

// (Zero moments, those of all padding and of inputs that are always zero, leave
// the parameter alone; their divisions and root would take the slow path of
// special operands: 22 us for a tile of them instead of 6.)
__device__ __forceinline__ float adam_step(float p, float gr, float& m1, float& m2, const AdamArgs& a) {
  const float a1 = __fmaf_rn(1.f - a.b1, gr, __fmul_rn(a.b1, m1));
  const float a2 = __fmaf_rn(__fmul_rn(1.f - a.b2, gr), gr, __fmul_rn(a.b2, m2));
  m1 = a1;
  m2 = a2;
  const bool still = a1 == 0.f && a2 == 0.f;
  const float q = a.lr * ((still ? 1.f : a1) / a.c1) / (sqrtf((still ? 1.f : a2) / a.c2) + a.eps);
  return still ? p : p - q;
}

template <bool UPDATE>
__global__ void __launch_bounds__(DwPipe::THREADS, 1)
    k_dw(const __grid_constant__ DwMaps maps, const __grid_constant__ DwArgs a) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int bail;
  __shared__ int issued;
  DwPipe p;
  uint8_t* rest = p.open(smem_raw, &bail, &issued, a.err);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nk = a.rows / BK;
  // layer and tile of unit u
  auto tile_of = [&](int u, int& l, int& mt, int& nt) {
    l = 0;
    while (l + 1 < a.layers && u >= a.l[l + 1].first) ++l;
    const int q = u - a.l[l].first, tn = a.l[l].k / 64;
    mt = q / tn;
    nt = q % tn;
  };
  if (warp == 0) {
    if (lane == 0) {
      mpcmd::wait_for_previous();
      int g = 0, l, mt, nt;
      for (int u = blockIdx.x; u < a.tiles && !bail; u += gridDim.x) {
        tile_of(u, l, mt, nt);
        if (!p.load(g, nk, &maps.a[l], mt * BM, &maps.b[l], nt * 64)) break;
      }
      issued = g;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int g = 0, j = 0;
      for (int u = blockIdx.x; u < a.tiles && !bail; u += gridDim.x, ++j)
        if (!p.multiply(g, j, nk)) break;
      mma_commit(p.done);
    }
  } else {
    const int ew = warp - 2, quarter = warp & 3, c0 = (ew >> 2) * 16;
    float* buf = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(rest) + 15) & ~(uintptr_t)15) + ew * 32 * DW_PITCH;
    int j = 0, l, mt, nt;
    for (int u = blockIdx.x; u < a.units; u += gridDim.x) {
      if (u < a.tiles) {
        tile_of(u, l, mt, nt);
        const DwLayer& ly = a.l[l];
        // this lane's part of the 32 x 16 block: 4 columns of every eighth row
        const int row0 = mt * BM + quarter * 32, col = nt * 64 + c0, sub = lane >> 2, q0 = 4 * (lane & 3);
        const bool real = row0 < ly.n;   // (widths are multiples of 64)
        const size_t at = (size_t)(row0 + sub) * ly.k + col + q0, step = 8 * (size_t)ly.k;
        float4 x[4], m1[4], m2[4];       // fetched while the MMAs run
        if (UPDATE && real) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            x[i] = __ldcg(reinterpret_cast<const float4*>(ly.w + at + i * step));
            m1[i] = __ldcg(reinterpret_cast<const float4*>(ly.m + at + i * step));
            m2[i] = __ldcg(reinterpret_cast<const float4*>(ly.v + at + i * step));
          }
        }
        if (!p.ready(j)) break;
        {
          float v[16];
          p.read(j, quarter, c0, v);
          p.release(j);
#pragma unroll
          for (int q = 0; q < 16; q += 4)
            *reinterpret_cast<float4*>(buf + lane * DW_PITCH + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
        }
        __syncwarp();
        ++j;
        if (real) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float4* cell = reinterpret_cast<float4*>(buf + (8 * i + sub) * DW_PITCH + q0);
            const float4 gr = *cell;
            if constexpr (UPDATE) {
              x[i].x = adam_step(x[i].x, gr.x, m1[i].x, m2[i].x, a.adam);
              x[i].y = adam_step(x[i].y, gr.y, m1[i].y, m2[i].y, a.adam);
              x[i].z = adam_step(x[i].z, gr.z, m1[i].z, m2[i].z, a.adam);
              x[i].w = adam_step(x[i].w, gr.w, m1[i].w, m2[i].w, a.adam);
              *reinterpret_cast<float4*>(ly.w + at + i * step) = x[i];
              *reinterpret_cast<float4*>(ly.m + at + i * step) = m1[i];
              *reinterpret_cast<float4*>(ly.v + at + i * step) = m2[i];
              *reinterpret_cast<uint2*>(ly.wb + at + i * step) =
                  make_uint2(pack_bf16(x[i].x, x[i].y), pack_bf16(x[i].z, x[i].w));
              *cell = x[i];
            } else {
              *reinterpret_cast<float4*>(ly.g + at + i * step) = gr;
            }
          }
          if constexpr (UPDATE) {
            // the transposed copy from the thread-per-row layout
            __syncwarp();
            uint32_t w[8];
#pragma unroll
            for (int q = 0; q < 16; q += 4) {
              const float4 p4 = *reinterpret_cast<const float4*>(buf + lane * DW_PITCH + q);
              w[q / 2] = pack_bf16(p4.x, p4.y);
              w[q / 2 + 1] = pack_bf16(p4.z, p4.w);
            }
            put_columns(ly.wt + (size_t)col * ly.n + row0 + lane, ly.n, w);
          }
        }
        __syncwarp();
      } else {
        l = 0;
        while (l + 1 < a.layers && u >= a.l[l + 1].first_bias) ++l;
        const DwLayer& ly = a.l[l];
        // four rows a warp, their loads in flight together; lane r finishes row r
        const int n0 = (u - ly.first_bias) * 64 + 4 * ew, n = n0 + (lane & 3);
        float b = 0.f, m1 = 0.f, m2 = 0.f;
        if constexpr (UPDATE) { b = __ldcg(ly.bw + n); m1 = __ldcg(ly.bm + n); m2 = __ldcg(ly.bv + n); }
        mpcmd::wait_for_previous();
        float s[4] = {};
        const __nv_bfloat16* zp = ly.dzt + (size_t)n0 * a.rows + lane;
#pragma unroll 4
        for (int c = 0; c < a.rows; c += 32)
#pragma unroll
          for (int r = 0; r < 4; ++r) s[r] += __bfloat162float(zp[(size_t)r * a.rows + c]);
        float sum = 0.f;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          for (int o = 16; o > 0; o >>= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
          if (lane == r) sum = s[r];
        }
        if (lane < 4) {
          if constexpr (UPDATE) {
            ly.bw[n] = adam_step(b, sum, m1, m2, a.adam);
            ly.bm[n] = m1;
            ly.bv[n] = m2;
          } else {
            ly.bg[n] = sum;
          }
        }
      }
    }
  }
  p.close(&issued);
}

__global__ void k_to_bf16(const float* p, int64_t count, int k, int n, __nv_bfloat16* wb, __nv_bfloat16* wt) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < count; e += (int64_t)gridDim.x * blockDim.x) {
    const __nv_bfloat16 b = __float2bfloat16_rn(p[e]);
    wb[e] = b;
    wt[(size_t)(e % k) * n + e / k] = b;
  }
}

// ---------------------------------------------------------------- host ----
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encoder() {
  static EncodeTiled fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(p);
  }
  return fn;
}

// 2-D map of a row-major BF16 matrix [rows, cols] with boxes of 64 columns x box_rows rows, 128-byte swizzle.
bool make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int box_rows) {
  EncodeTiled enc = encoder();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  const cuuint32_t es[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct Layer {
  int n, k;               // padded output and input widths: W [n, k]
  int n_real, k_real;     // logical widths
  float *w, *b, *gw, *gb, *mw, *vw, *mb, *vb;
  __nv_bfloat16 *wb, *wt;  // [n, k], [k, n]
};

}  // namespace

struct mpcmd_mlp {
  mpcmd_mlp_config cfg{};
  int kin = 64, H = 256, L = 4, nout = 0, npad = 0, B = 256;
  int64_t R = 0;           // largest inference call (>= batch, >= max_rows, multiple of 128)
  std::vector<Layer> layers;
  std::vector<void*> allocs;
  // one training batch: x^T [64, B]; per hidden layer activations and gradients
  // [H, B], pre-activations [H, B]; the last hidden layer's gradient [B, H];
  // the output gradient [B, npad] and [npad, B]
  __nv_bfloat16 *x0t = nullptr, *dz = nullptr, *dy = nullptr, *dyt = nullptr;
  std::vector<__nv_bfloat16*> ht, dzt;
  std::vector<float*> zt;
  double* loss_part = nullptr;
  double* loss = nullptr;  // the last batch's loss (page-locked host memory)
  int* err = nullptr;      // raised by a kernel whose wait expired (page-locked host memory)
  InferMaps maps{}, back{};   // weight boxes of the forward and backward chains (the weights stay where they are)
  CUtensorMap dx_a{}, dx_b{};
  DwMaps dw_maps{};
  DwArgs dw{};
  int64_t step = 0;
  int sms = 1;             // SMs of the device
  cudaStream_t st = nullptr;

  ~mpcmd_mlp() {
    if (st) cudaStreamDestroy(st);
    for (void* p : allocs) cudaFree(p);
    if (err) cudaFreeHost(err);
    if (loss) cudaFreeHost(loss);
  }
  template <class U>
  int alloc(U*& p, int64_t n) {
    void* q = nullptr;
    if (cudaMalloc(&q, sizeof(U) * (size_t)std::max<int64_t>(n, 1)) != cudaSuccess) return MPCMD_ERR_ALLOC;
    allocs.push_back(q);
    cudaMemset(q, 0, sizeof(U) * (size_t)std::max<int64_t>(n, 1));
    p = static_cast<U*>(q);
    return MPCMD_OK;
  }
};

namespace {

// (the stream's kernels have ended: their stores to the flag are visible)
int status_of(mpcmd_mlp* m) {
  if (cudaStreamSynchronize(m->st) != cudaSuccess) return MPCMD_ERR_CUDA;
  return *reinterpret_cast<volatile int*>(m->err) ? MPCMD_ERR_CUDA : MPCMD_OK;
}

template <int MODE, int VB>
bool allow_chain() {
  return cudaFuncSetAttribute(k_chain<MODE, VB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)INF_SMEM) ==
         cudaSuccess;
}
template <bool UPDATE>
bool allow_dw() {
  return cudaFuncSetAttribute(k_dw<UPDATE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DW_SMEM) == cudaSuccess;
}

// Output jobs of a row tile and the width of the last one's MMA (a multiple
// of 16, as the instruction takes it).
int infer_tiles(const mpcmd_mlp* m) { return (m->nout + INF_BN - 1) / INF_BN; }
int infer_tail(const mpcmd_mlp* m) { return (m->nout - (infer_tiles(m) - 1) * INF_BN + 15) / 16 * 16; }

bool make_infer_maps(mpcmd_mlp* m) {
  for (int l = 0; l < m->L; ++l)
    if (!make_map(&m->maps.w[l], m->layers[l].wb, m->layers[l].n, m->layers[l].k, m->H)) return false;
  const Layer& lo = m->layers[m->L];
  return make_map(&m->maps.out, lo.wb, lo.n, lo.k, INF_BN) &&
         make_map(&m->maps.tail, lo.wb, lo.n, lo.k, infer_tail(m));
}

// Operands and work units of the training step's other launches.
bool make_train_maps(mpcmd_mlp* m) {
  for (int j = 0; j + 1 < m->L; ++j) {
    const Layer& ly = m->layers[m->L - 1 - j];
    if (!make_map(&m->back.w[j], ly.wt, ly.k, ly.n, m->H)) return false;
  }
  const Layer& lo = m->layers[m->L];
  if (!make_map(&m->dx_a, m->dy, m->B, m->npad, BM) || !make_map(&m->dx_b, lo.wt, lo.k, lo.n, 32)) return false;
  DwArgs& d = m->dw;
  d.layers = m->L + 1; d.rows = m->B; d.err = m->err;
  int u = 0;
  for (int l = 0; l <= m->L; ++l) {
    const Layer& ly = m->layers[l];
    DwLayer& q = d.l[l];
    q.n = ly.n; q.k = ly.k;
    q.w = ly.w; q.m = ly.mw; q.v = ly.vw; q.g = ly.gw;
    q.bw = ly.b; q.bm = ly.mb; q.bv = ly.vb; q.bg = ly.gb;
    q.wb = ly.wb; q.wt = ly.wt;
    q.dzt = l == m->L ? m->dyt : m->dzt[l];
    q.first = u;
    u += (ly.n + BM - 1) / BM * (ly.k / 64);
    const __nv_bfloat16* xt = l == 0 ? m->x0t : m->ht[l - 1];
    if (!make_map(&m->dw_maps.a[l], q.dzt, ly.n, m->B, BM) || !make_map(&m->dw_maps.b[l], xt, ly.k, m->B, 64))
      return false;
  }
  d.tiles = u;
  for (int l = 0; l <= m->L; ++l) { d.l[l].first_bias = u; u += m->layers[l].n / 64; }
  d.units = u;
  return true;
}

// Row tiles of a chain over the CTAs: whole rounds of one row tile per SM, then
// the left-over row tiles shared as far as the SMs go.
int chain_grid(const mpcmd_mlp* m, int64_t rows, InferArgs& a) {
  const int tiles = (int)((rows + BM - 1) / BM);
  a.whole = tiles / m->sms;
  a.part = tiles % m->sms;
  const int shares = a.tiles ? a.tiles : a.layers * a.H / 32;   // (BACKWARD: the pieces kept)
  a.split = a.part ? std::min(shares, m->sms / a.part) : 1;
  return a.whole ? m->sms : a.part * a.split;
}

// y [rows, nout] = network(x [rows, n_in]) (device, FP32).
int infer(mpcmd_mlp* m, const float* x, int64_t rows, float* y) {
  InferArgs a{};
  a.layers = m->L; a.H = m->H; a.n_in = m->cfg.n_in; a.rows = (int)rows;
  a.tiles = infer_tiles(m); a.tail_n = infer_tail(m);
  a.x = x;
  for (int l = 0; l < m->L; ++l) a.bias[l] = m->layers[l].b;
  a.n_out = m->nout; a.y = y; a.bias_out = m->layers[m->L].b;
  a.err = m->err;
  const int grid = chain_grid(m, rows, a);
  const uintptr_t align = reinterpret_cast<uintptr_t>(y) | ((uintptr_t)m->nout * 4);
  if (align % 16 == 0) k_chain<INFER, 16><<<grid, INF_THREADS, INF_SMEM, m->st>>>(m->maps, a);
  else if (align % 8 == 0) k_chain<INFER, 8><<<grid, INF_THREADS, INF_SMEM, m->st>>>(m->maps, a);
  else k_chain<INFER, 4><<<grid, INF_THREADS, INF_SMEM, m->st>>>(m->maps, a);
  return cudaPeekAtLastError() == cudaSuccess ? MPCMD_OK : MPCMD_ERR_CUDA;
}

// Loss and gradients of one batch (inputs x, targets t [B, nout], output
// weights w [nout], device): written out (gw, gb), or applied when `adam` is given.
int train_batch(mpcmd_mlp* m, const float* x, const float* t, const float* w, const AdamArgs* adam) {
  const int B = m->B, L = m->L;
  InferArgs a{};
  a.layers = L; a.H = m->H; a.n_in = m->cfg.n_in; a.rows = B;
  a.tiles = infer_tiles(m); a.tail_n = infer_tail(m);
  a.n_out = m->nout; a.npad = m->npad;
  a.x = x; a.t = t; a.w = w;
  a.inv_rows = (B & (B - 1)) == 0 ? 1.f / (float)B : 0.f;
  a.bias_out = m->layers[L].b;
  for (int l = 0; l < L; ++l) { a.bias[l] = m->layers[l].b; a.zt[l] = m->zt[l]; a.at[l] = m->ht[l]; }
  a.xt = m->x0t; a.dy = m->dy; a.dyt = m->dyt;
  a.loss = m->loss_part; a.err = m->err;
  const int grid = chain_grid(m, B, a);
  k_chain<FORWARD, 4><<<grid, INF_THREADS, INF_SMEM, m->st>>>(m->maps, a);
  DxArgs d{};
  d.rows = B; d.H = m->H; d.nk = (m->nout + BK - 1) / BK;
  d.zt = m->zt[L - 1]; d.dz = m->dz; d.dzt = m->dzt[L - 1];
  d.loss = m->loss_part; d.n_loss = grid * INF_EPI; d.loss_out = m->loss;
  d.err = m->err;
  mpcmd::launch_next_smem(k_dx, std::min((B / BM) * (m->H / 32), m->sms), DxPipe::THREADS, DxPipe::bytes(0), m->st,
                          m->dx_a, m->dx_b, d);
  if (L > 1) {
    InferArgs r{};
    r.layers = L - 1; r.H = m->H; r.rows = B;
    r.dz = m->dz; r.err = m->err;
    for (int j = 0; j + 1 < L; ++j) { r.zt[j] = m->zt[L - 2 - j]; r.at[j] = m->dzt[L - 2 - j]; }
    const int rg = chain_grid(m, B, r);
    mpcmd::launch_next_smem(k_chain<BACKWARD, 4>, rg, INF_THREADS, INF_SMEM, m->st, m->back, r);
  }
  DwArgs g = m->dw;
  if (adam) g.adam = *adam;
  const int dg = std::min(g.units, m->sms);
  mpcmd::launch_next_smem(adam ? k_dw<true> : k_dw<false>, dg, DwPipe::THREADS, DW_SMEM, m->st, m->dw_maps, g);
  return cudaPeekAtLastError() == cudaSuccess ? MPCMD_OK : MPCMD_ERR_CUDA;
}

void refresh_bf16(mpcmd_mlp* m) {
  for (Layer& ly : m->layers)
    k_to_bf16<<<256, 256, 0, m->st>>>(ly.w, (int64_t)ly.n * ly.k, ly.k, ly.n, ly.wb, ly.wt);
}

}  // namespace

// ------------------------------------------------------------- C ABI ----
namespace {

uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

int64_t round_up(int64_t v, int64_t q) { return (v + q - 1) / q * q; }

// Logical (unpadded) parameter layout: per layer W [n_real, k_real] row-major, then b [n_real].
int64_t logical_count(const mpcmd_mlp* m) {
  int64_t c = 0;
  for (const Layer& ly : m->layers) c += (int64_t)ly.n_real * ly.k_real + ly.n_real;
  return c;
}

// Tensors to the logical layout or from it: the padding stays on the device.
int copy_params(mpcmd_mlp* m, float* host, bool to_host, bool grads) {
  int64_t off = 0;
  for (Layer& ly : m->layers) {
    float* dw = grads ? ly.gw : ly.w;
    float* db = grads ? ly.gb : ly.b;
    const size_t hp = 4 * (size_t)ly.k_real, dp = 4 * (size_t)ly.k;
    float* hw = host + off;
    float* hb = hw + (int64_t)ly.n_real * ly.k_real;
    const cudaError_t e1 = to_host ? cudaMemcpy2D(hw, hp, dw, dp, hp, ly.n_real, cudaMemcpyDeviceToHost)
                                   : cudaMemcpy2D(dw, dp, hw, hp, hp, ly.n_real, cudaMemcpyHostToDevice);
    const cudaError_t e2 = to_host ? cudaMemcpy(hb, db, 4 * (size_t)ly.n_real, cudaMemcpyDeviceToHost)
                                   : cudaMemcpy(db, hb, 4 * (size_t)ly.n_real, cudaMemcpyHostToDevice);
    if (e1 != cudaSuccess || e2 != cudaSuccess) return MPCMD_ERR_CUDA;
    off += (int64_t)ly.n_real * ly.k_real + ly.n_real;
  }
  return MPCMD_OK;
}

}  // namespace

extern "C" {

int mpcmd_mlp_create(const mpcmd_mlp_config* cfg, mpcmd_mlp** out) {
  if (!cfg || !out) return MPCMD_ERR_CONFIG;
  *out = nullptr;
  const mpcmd_mlp_config& c = *cfg;
  if (c.n_in < 1 || c.n_in > 64 || c.n_hidden < 64 || c.n_hidden > 256 || c.n_hidden % 64 || c.n_layers < 1 ||
      c.n_layers > 16 || c.n_out < 1 || c.n_out > (1 << 16) || c.batch < 128 || c.batch % 128 || c.max_rows < 0 ||
      !(c.lr > 0) || !(c.beta1 >= 0 && c.beta1 < 1) || !(c.beta2 >= 0 && c.beta2 < 1) || !(c.eps > 0))
    return MPCMD_ERR_CONFIG;
  if (!encoder()) return MPCMD_ERR_CUDA;
  mpcmd_mlp* m = new mpcmd_mlp();
  m->cfg = c;
  m->kin = 64; m->H = c.n_hidden; m->L = c.n_layers; m->nout = c.n_out; m->B = c.batch;
  m->npad = (int)round_up(c.n_out, 128);
  m->R = round_up(std::max<int64_t>(c.batch, c.max_rows), BM);
  int s = 0;
  if (cudaStreamCreate(&m->st) != cudaSuccess) { delete m; return MPCMD_ERR_CUDA; }
  uint64_t rs = c.seed ? c.seed : 1;
  for (int l = 0; l <= m->L; ++l) {
    Layer ly{};
    const bool out_layer = l == m->L;
    ly.n = out_layer ? m->npad : m->H;
    ly.k = l == 0 ? m->kin : m->H;
    ly.n_real = out_layer ? c.n_out : m->H;
    ly.k_real = l == 0 ? c.n_in : m->H;
    const int64_t nk = (int64_t)ly.n * ly.k;
    s |= m->alloc(ly.w, nk); s |= m->alloc(ly.gw, nk); s |= m->alloc(ly.mw, nk); s |= m->alloc(ly.vw, nk);
    s |= m->alloc(ly.b, ly.n); s |= m->alloc(ly.gb, ly.n); s |= m->alloc(ly.mb, ly.n); s |= m->alloc(ly.vb, ly.n);
    s |= m->alloc(ly.wb, nk); s |= m->alloc(ly.wt, nk);
    if (s) break;
    // Glorot-uniform initial weights on the logical block, zero padding and biases
    std::vector<float> w((size_t)nk, 0.f);
    const double a = std::sqrt(6.0 / (ly.n_real + ly.k_real));
    for (int i = 0; i < ly.n_real; ++i)
      for (int j = 0; j < ly.k_real; ++j)
        w[(size_t)i * ly.k + j] = (float)(a * (2.0 * ((splitmix(rs) >> 11) * (1.0 / 9007199254740992.0)) - 1.0));
    if (cudaMemcpy(ly.w, w.data(), 4 * w.size(), cudaMemcpyHostToDevice) != cudaSuccess) s = MPCMD_ERR_CUDA;
    m->layers.push_back(ly);
  }
  const int64_t BH = (int64_t)m->B * m->H;
  s |= m->alloc(m->x0t, (int64_t)m->B * m->kin);
  m->ht.resize(m->L); m->zt.resize(m->L); m->dzt.resize(m->L);
  for (int l = 0; l < m->L && !s; ++l) {
    s |= m->alloc(m->ht[l], BH);
    s |= m->alloc(m->zt[l], BH);
    s |= m->alloc(m->dzt[l], BH);
  }
  s |= m->alloc(m->dz, BH);
  s |= m->alloc(m->dy, (int64_t)m->B * m->npad);
  s |= m->alloc(m->dyt, (int64_t)m->B * m->npad);
  if (s || cudaHostAlloc(reinterpret_cast<void**>(&m->err), sizeof(int), cudaHostAllocDefault) != cudaSuccess ||
      cudaHostAlloc(reinterpret_cast<void**>(&m->loss), sizeof(double), cudaHostAllocDefault) != cudaSuccess) {
    delete m;
    return MPCMD_ERR_ALLOC;
  }
  *m->err = 0;
  *m->loss = 0.0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    delete m;
    return MPCMD_ERR_CUDA;
  }
  if (m->alloc(m->loss_part, (int64_t)m->sms * INF_EPI) != MPCMD_OK) {
    delete m;
    return MPCMD_ERR_ALLOC;
  }
  if (!allow_chain<INFER, 16>() || !allow_chain<INFER, 8>() || !allow_chain<INFER, 4>() ||
      !allow_chain<FORWARD, 4>() || !allow_chain<BACKWARD, 4>() ||
      cudaFuncSetAttribute(k_dx, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DxPipe::bytes(0)) != cudaSuccess ||
      !allow_dw<true>() || !allow_dw<false>() || !make_infer_maps(m) || !make_train_maps(m)) {
    delete m;
    return MPCMD_ERR_CUDA;
  }
  refresh_bf16(m);
  if (status_of(m)) { delete m; return MPCMD_ERR_CUDA; }
  *out = m;
  return MPCMD_OK;
}

int mpcmd_mlp_destroy(mpcmd_mlp* m) {
  delete m;
  return MPCMD_OK;
}

int mpcmd_mlp_param_count(const mpcmd_mlp* m, int64_t* n) {
  if (!m || !n) return MPCMD_ERR_CONFIG;
  *n = logical_count(m);
  return MPCMD_OK;
}

int mpcmd_mlp_get_params(mpcmd_mlp* m, float* host) {
  if (!m || !host) return MPCMD_ERR_CONFIG;
  if (cudaStreamSynchronize(m->st) != cudaSuccess) return MPCMD_ERR_CUDA;
  return copy_params(m, host, true, false);
}

int mpcmd_mlp_set_params(mpcmd_mlp* m, const float* host) {
  if (!m || !host) return MPCMD_ERR_CONFIG;
  if (cudaStreamSynchronize(m->st) != cudaSuccess) return MPCMD_ERR_CUDA;
  // (zero padding, whatever training left there: infinite activations make it NaN)
  for (Layer& ly : m->layers)
    if (cudaMemset(ly.w, 0, 4 * (size_t)ly.n * ly.k) != cudaSuccess || cudaMemset(ly.b, 0, 4 * (size_t)ly.n) != cudaSuccess)
      return MPCMD_ERR_CUDA;
  int r = copy_params(m, const_cast<float*>(host), false, false);
  if (r) return r;
  for (Layer& ly : m->layers) {   // a new starting point: fresh moments
    cudaMemsetAsync(ly.mw, 0, 4 * (size_t)ly.n * ly.k, m->st);
    cudaMemsetAsync(ly.vw, 0, 4 * (size_t)ly.n * ly.k, m->st);
    cudaMemsetAsync(ly.mb, 0, 4 * (size_t)ly.n, m->st);
    cudaMemsetAsync(ly.vb, 0, 4 * (size_t)ly.n, m->st);
  }
  m->step = 0;
  refresh_bf16(m);
  return status_of(m);
}

int mpcmd_mlp_forward(mpcmd_mlp* m, const float* x, int64_t rows, float* y) {
  if (!m || !x || !y || rows < 1 || rows > m->R) return MPCMD_ERR_CONFIG;
  int r = infer(m, x, rows, y);
  if (r) return r;
  return status_of(m);
}

int mpcmd_mlp_gradients(mpcmd_mlp* m, const float* x, const float* t, const float* w, float* grads, double* loss) {
  if (!m || !x || !t || !w) return MPCMD_ERR_CONFIG;
  int r = train_batch(m, x, t, w, nullptr);
  if (r) return r;
  if ((r = status_of(m))) return r;
  if (loss) *loss = *m->loss;
  return grads ? copy_params(m, grads, true, true) : MPCMD_OK;
}

int mpcmd_mlp_train_step(mpcmd_mlp* m, const float* x, const float* t, const float* w, double* loss) {
  if (!m || !x || !t || !w) return MPCMD_ERR_CONFIG;
  AdamArgs a;
  a.lr = (float)m->cfg.lr; a.b1 = (float)m->cfg.beta1; a.b2 = (float)m->cfg.beta2; a.eps = (float)m->cfg.eps;
  a.c1 = (float)(1.0 - std::pow(m->cfg.beta1, (double)(m->step + 1)));
  a.c2 = (float)(1.0 - std::pow(m->cfg.beta2, (double)(m->step + 1)));
  int r = train_batch(m, x, t, w, &a);
  if (r) return r;
  m->step += 1;
  if (loss) {
    if ((r = status_of(m))) return r;
    *loss = *m->loss;
  }
  return MPCMD_OK;
}

int mpcmd_mlp_synchronize(mpcmd_mlp* m) {
  if (!m) return MPCMD_ERR_CONFIG;
  return status_of(m);
}

}  // extern "C"
