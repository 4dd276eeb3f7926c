// The surrogate's network (in <= 64 -> 3 x 256 GELU -> out <= 128) as whole
// passes: one kernel carries a 128-row tile through every layer, forward and
// back, with the activations in shared and tensor memory; a second forms
// every weight gradient; a third sums their parts, applies Adam and lays the
// new weights out for the next pass.
//
// A layer at a time (umma_gemm_persistent.cuh and the kernels of mlp.cu) a
// training step was 52 launches of 2-10 us on 2048-4096 rows (0.33 ms, of
// which the tensor cores worked under 1 %), and a prediction wrote every
// layer's FP32 and BF16 activations to memory.  Here a step is four
// launches, and a prediction reads its inputs and writes its outputs.
// Whole calls: predictions for 100003 rows 0.42 -> 0.17 ms, loss and
// gradients of 4000 rows 0.67 -> 0.34 ms, a fit of 57 steps of 2048 rows
// from new weights 35 -> 10 ms, ranking 300000 candidates with four networks
// 13.8 -> 11.8 ms (10 ms of it the copy of the candidates from pageable
// memory; 1.5 ms the kernel).
//
// Layouts.  Every operand of an MMA is a "chunk": 64 BF16 (128 bytes) of one
// dimension for each of R rows of the other, row r at 128 r, its 16-byte
// piece j at position j ^ (r & 7) -- the 128-byte-swizzled layout that the
// tcgen05 descriptors name, K-major where the 64 run along K, MN-major where
// they run along M or N.  The weights are kept as such chunks in global
// memory (pack_kernel), so a chunk is one untiled bulk copy.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "dense_b200_network.h"

#include <atomic>
#include <cmath>
#include <cstdint>
#include <mutex>

#include "umma_gemm.cuh"

#if defined(__GNUC__)
#define CHAIN_API extern "C" __attribute__((visibility("default")))
#else
#define CHAIN_API extern "C"
#endif

using namespace dense_b200::mlp;

namespace {

constexpr int kHid = 256;        // hidden width
constexpr int kInPad = 64;       // inputs, zero padded
constexpr int kOutPad = 128;     // rows of the output layer's weight matrix
constexpr int kRows = 128;       // rows of a tile
constexpr int kChunkW = 256 * 128;     // bytes of a chunk of 256 rows
constexpr int kChunkA = kRows * 128;   // bytes of a chunk of 128 rows
constexpr int kHalf = 64 * 128;        // bytes of a chunk of 64 rows
constexpr int kRing = 4;         // weight chunks in flight
constexpr int kEpi = 16;         // epilogue warps
constexpr int kChainThreads = 64 + 32 * kEpi;
constexpr int kMaxNets = 64;     // networks of an ensemble in one launch (their pointers are kernel arguments)

// A network's packed weights: forward chunks of layers 0..3, then the
// transposed ones of layers 3, 2, 1 for the input gradients.
constexpr int kFwd0 = 0, kFwd1 = kChunkW, kFwd2 = 5 * kChunkW, kFwd3 = 9 * kChunkW;  // layer 3: 4 x kOutPad x 128
constexpr int kBwd3 = kFwd3 + 4 * kOutPad * 128, kBwd2 = kBwd3 + 2 * kChunkW, kBwd1 = kBwd2 + 4 * kChunkW;
constexpr int kPacked = kBwd1 + 4 * kChunkW;

__host__ __device__ constexpr int out_cols(int n_out) { return (n_out + 15) / 16 * 16; }  // columns computed
__host__ __device__ constexpr int out_chunks(int n_out) { return (n_out + 63) / 64; }     // 64-column chunks of dY

// Byte position of element (row, col) of a chunk (col < 64).
__device__ __forceinline__ int chunk_at(int row, int col) {
  return row * 128 + ((((col >> 3) ^ row) & 7) << 4) + ((col & 7) << 1);
}

// Shared-memory descriptor of a 128-byte-swizzled operand.  K-major: 8-row
// groups 1024 bytes apart (lbo unused).  MN-major: 8 k-rows are 1024 bytes,
// 64-element groups of M or N `lbo` bytes apart.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr, uint32_t lbo) {
  return static_cast<uint64_t>((addr & 0x3FFFF) >> 4) | (static_cast<uint64_t>(lbo >> 4) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void mma_bf16(uint32_t acc, uint64_t da, uint64_t db, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(acc),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate ? 1u : 0u));
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Waits for a phase for at most ~2^31 cycles, or until another role gave up.
__device__ __forceinline__ bool mbar_wait_or(uint64_t* bar, uint32_t parity, const volatile int* abort) {
  const uint32_t b = smem_u32(bar);
  const long long t0 = clock64();
  while (!mbar_try_wait(b, parity)) {
    if (*abort) return false;
    if (clock64() - t0 > (1ll << 31)) return false;
  }
  return true;
}

// One bulk copy of `bytes` (a multiple of 16) from global to shared memory.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// One bulk copy of `bytes` from shared to global memory (a bulk group's).
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void expect_bytes(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// The kernels of a training step are launched to start while the one before
// ends (launch_next): their set-up runs under its tail.  Waits for the
// kernels before to be complete and their writes visible; nothing of theirs
// is read, or written over, before.  Then lets the next one start.  (Every
// kernel of the sequence waits, so that each also follows the ones before
// the one before.)  A kernel that calls this is resident while the one before
// still writes what it reads, so its global loads are plain ones through
// unqualified pointers: __restrict__ and the read-only and cache-hinted load
// functions let the compiler take the memory for constant and move a load
// above the wait.  2048 rows, pass, bias sums and weight gradients: 49 us
// one after the other, 43 so.
__device__ __forceinline__ void follow_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// GELU(z) and GELU'(z), the expressions of gelu and gelu_grad with one erff.
__device__ __forceinline__ float gelu_both(float z, float* grad) {
  const float e = 1.0f + erff(z * 0.70710678118654752f);
  const float cdf = 0.5f * e;
  const float pdf = 0.3989422804014327f * expf(-0.5f * z * z);
  *grad = cdf + z * pdf;
  return 0.5f * z * e;
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// ------------------------------------------------------------------ packing

struct Weights {
  const float* W[4];  // [out][in] FP32: [256][64], [256][256], [256][256], [128][256]
};

// The BF16 chunk positions of weight (layer, o, k): forward (rows o, 64 k's)
// and, for layers 1..3, transposed (rows k, 64 o's).
__device__ __forceinline__ int fwd_at(int layer, int o, int k) {
  const int rows = layer == 3 ? kOutPad : kHid;
  const int base = layer == 0 ? kFwd0 : (layer == 1 ? kFwd1 : (layer == 2 ? kFwd2 : kFwd3));
  return base + (k >> 6) * rows * 128 + chunk_at(o, k & 63);
}
__device__ __forceinline__ int bwd_at(int layer, int o, int k) {
  const int base = layer == 1 ? kBwd1 : (layer == 2 ? kBwd2 : kBwd3);
  return base + (o >> 6) * kChunkW + chunk_at(k, o & 63);
}

__device__ __forceinline__ int layer_of(int i, int* within) {
  constexpr int s0 = kHid * kInPad, s1 = s0 + kHid * kHid, s2 = s1 + kHid * kHid;
  if (i < s0) return *within = i, 0;
  if (i < s1) return *within = i - s0, 1;
  if (i < s2) return *within = i - s1, 2;
  return *within = i - s2, 3;
}
constexpr int kOutWeights = kOutPad * kHid;
constexpr int kHidWeights = kHid * kInPad + 2 * kHid * kHid;
constexpr int kWeights = kHidWeights + kOutWeights;

// Four consecutive weights of a row at a time.
__device__ __forceinline__ void pack_quad(unsigned char* packed, int layer, int at, const float (&w)[4], bool backward) {
  const int width = layer == 0 ? kInPad : kHid;
  const int o = at / width, k = at % width;
  *reinterpret_cast<uint2*>(packed + fwd_at(layer, o, k)) = make_uint2(pack2(w[0], w[1]), pack2(w[2], w[3]));
  if (backward && layer > 0) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<__nv_bfloat16*>(packed + bwd_at(layer, o, k + j)) = __float2bfloat16(w[j]);
  }
}

__global__ void pack_kernel(const Weights w, unsigned char* __restrict__ packed, int backward) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i >= kWeights) return;
  int at;
  const int layer = layer_of(i, &at);
  const float4 x = *reinterpret_cast<const float4*>(w.W[layer] + at);
  const float v[4] = {x.x, x.y, x.z, x.w};
  pack_quad(packed, layer, at, v, backward != 0);
}

// ------------------------------------------------------------------- passes

enum ChainMode : int {
  kPredict,  // FP32 inputs -> outputs
  kRank,     // FP64 candidates -> encoding -> every network of an ensemble -> score
  kTrain,    // gathered rows -> loss, activations, output and layer gradients
};

struct ScoreArgs {
  float mu[8], sd[8];
  float nets;
  double weight, period, tol, log_amp_min, ramp;
};

struct ChainArgs {
  int rows;       // rows of the batch (the tiles' tail rows are zeros)
  int tiles;      // ceil(rows / 128)
  int n_in, n_out;
  int nets;       // kRank: networks; else 1
  const unsigned char* packed[kMaxNets];
  const float* bias[kMaxNets][4];
  int* err;
  // kPredict, kTrain: rows of X; kTrain: idx (null: row r of X is row r of the batch)
  const float* X;
  int ldx, x_rows;
  const int* idx;
  // kPredict
  float* out;     // [rows][n_out]
  // kRank
  const double* P;
  int ldp;
  const int* cols;
  const double* tmpl;
  double log_spread;
  ScoreArgs score;
  double* scores;
  // kTrain
  const float *T, *mask;     // [x_rows][n_out]
  const float* inv_count;    // device, or null: inv_value
  float inv_value;
  float* loss;
  unsigned char* act;        // chunks of 64 rows: [layer input 0][1..3], see act_at
  unsigned char* grad;       // chunks of 64 rows of dZ_0, dZ_1, dZ_2, dY
  float* dz;                 // [3][tiles] tiles of 128 x 256: GELU', then dZ_0, dZ_1, dZ_2 in FP32 (see piece_at)
  float* dy;                 // [tiles] tiles of 128 x 64 out_chunks
};

// FP32 tiles as the epilogue holds them: piece j (4 columns) of chunk c of
// epilogue thread t (0..511) at float4 (4 c + j) 512 + t of the tile, so that
// a warp's accesses are whole lines.  (Row by row, 16 columns a thread, they
// cost a sector each: the pass over 2048 rows took 91 us instead of 55.)
__host__ __device__ constexpr int piece_at(int c, int j, int t) { return ((4 * c + j) * 512 + t) * 4; }
// The epilogue thread of a tile's row and column.
__device__ __forceinline__ int epi_thread(int row, int col) {
  const int q = row >> 5, g = (col & 63) >> 4;
  return (g * 4 + ((q + 2) & 3)) * 32 + (row & 31);
}

// Activations and gradients as weight-gradient operands: blocks of 64 batch
// rows, in each the 64-column chunks side by side.  Inputs of layer 0 have
// one chunk per block, the others four; dY has out_chunks.
__host__ __device__ inline int64_t act_base(int layer, int64_t blocks) {
  return layer == 0 ? 0 : (1 + 4 * static_cast<int64_t>(layer - 1)) * blocks * kHalf;
}
__host__ __device__ inline int64_t grad_base(int layer, int64_t blocks) {
  return 4 * static_cast<int64_t>(layer) * blocks * kHalf;
}

// One CTA per SM, walking tiles.  Warp 0: a thread streams the weight chunks
// of the layers, in order, into a ring.  Warp 1: a thread issues the MMAs of
// a layer (M = 128, N = the layer's outputs) chunk by chunk as the chunks of
// its input appear, into the accumulator (256 TMEM columns) the layer before
// did not use.  Warps 2-17: the epilogue; warp e takes TMEM lanes
// 32 (warp % 4) .. +31 and, of every 64-column chunk, columns 16 (e / 4) ..
// +15, so that a chunk of the next layer's input is complete as early as
// possible and its MMAs run under the rest of the epilogue.  What bounds a
// layer is its GELU arithmetic (24 instructions per element, 32768 elements
// per tile and layer: 6 k issue cycles per SM); the MMAs take 1 k.
template <int MODE>
__global__ void __launch_bounds__(kChainThreads, 1) mlp_chain_kernel(const __grid_constant__ ChainArgs a) {
  extern __shared__ __align__(16) unsigned char chain_raw[];
  __shared__ __align__(8) uint64_t full_bar[kRing], empty_bar[kRing], a_ready[4], acc_full[2], done_bar;
  __shared__ uint32_t tmem_sh;
  __shared__ volatile int abort_flag;
  __shared__ float s_loss[kEpi];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* smem = chain_raw + ((1024u - (smem_u32(chain_raw) & 1023u)) & 1023u);
  unsigned char* sA = smem;                                // the layer input, four chunks
  unsigned char* ring = sA + 4 * kChunkA;
  unsigned char* sX = ring + kRing * kChunkW;              // kRank: the encoded inputs of the tile

  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 4; ++i) mbar_init(&a_ready[i], kEpi);
    for (int i = 0; i < 2; ++i) mbar_init(&acc_full[i], 1);
    mbar_init(&done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (MODE == kTrain) follow_previous();
  const uint32_t tmem = tmem_sh;
  const int n_cols = out_cols(a.n_out);
  const int oc = out_chunks(a.n_out);
  const int passes = MODE == kRank ? a.nets : 1;
  // the layers of a pass: 0..3 forward, 4..6 backward (kTrain)
  constexpr int kLayers = MODE == kTrain ? 7 : 4;
  auto chunks_of = [&](int layer) { return layer == 0 ? 1 : (layer == 4 ? oc : 4); };

  if (warp == 0) {
    if (lane == 0) {
      // -------------------------------------------------------- weight ring
      uint32_t it = 0;
      bool bad = false;
      for (int tile = blockIdx.x; tile < a.tiles && !bad; tile += gridDim.x)
        for (int net = 0; net < passes && !bad; ++net)
          for (int layer = 0; layer < kLayers && !bad; ++layer) {
            const int base = layer == 0   ? kFwd0
                             : layer == 1 ? kFwd1
                             : layer == 2 ? kFwd2
                             : layer == 3 ? kFwd3
                             : layer == 4 ? kBwd3
                             : layer == 5 ? kBwd2
                                          : kBwd1;
            const int stride = layer == 3 ? kOutPad * 128 : kChunkW;
            const uint32_t bytes = layer == 3 ? static_cast<uint32_t>(n_cols) * 128u : static_cast<uint32_t>(kChunkW);
            const int chunks = chunks_of(layer);
            for (int c = 0; c < chunks; ++c, ++it) {
              const int s = static_cast<int>(it % kRing);
              if (it >= kRing && !mbar_wait_or(&empty_bar[s], ((it / kRing) - 1) & 1u, &abort_flag)) {
                bad = true;
                break;
              }
              expect_bytes(&full_bar[s], bytes);
              bulk_load(ring + s * kChunkW, a.packed[net] + base + c * stride, bytes, &full_bar[s]);
            }
          }
      if (bad) {
        atomicOr(a.err, kErrTimeout);
        abort_flag = 1;
      }
      // the copies issued last into each stage land before the CTA ends
      for (int s = 0; s < kRing && static_cast<uint32_t>(s) < it; ++s) {
        const uint32_t last = it - 1u - ((it - 1u - static_cast<uint32_t>(s)) % kRing);
        mbar_wait_bounded(smem_u32(&full_bar[s]), (last / kRing) & 1u);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------------------------------------------------------- MMAs
      uint32_t it = 0, seen[4] = {0, 0, 0, 0};
      const int64_t blocks = static_cast<int64_t>(a.tiles) * 2;
      int turn = 0;
      bool bad = false;
      for (int tile = blockIdx.x; tile < a.tiles && !bad; tile += gridDim.x)
        for (int net = 0; net < passes && !bad; ++net)
          // (kTrain: an eighth, without products, stores dZ_0)
          for (int layer = 0; layer < kLayers + (MODE == kTrain ? 1 : 0) && !bad; ++layer, ++turn) {
            const int n = layer == 3 ? n_cols : kHid;
            const uint32_t idesc = umma_idesc_bf16(kRows, n);
            const uint32_t acc = tmem + (turn & 1) * kHid;
            const int chunks = chunks_of(layer);
            for (int c = 0; c < chunks; ++c) {
              if (!mbar_wait_or(&a_ready[c], seen[c] & 1u, &abort_flag)) {
                bad = true;
                break;
              }
              ++seen[c];
              const uint32_t pa = smem_u32(sA + c * kChunkA);
              if (MODE == kTrain) {
                // the chunk is also an operand of the weight gradients:
                // inputs of layers 0-3, then dY, dZ_2, dZ_1, dZ_0
                unsigned char* to = layer < 4 ? a.act + act_base(layer, blocks) : a.grad + grad_base(7 - layer, blocks);
                for (int h = 0; h < 2; ++h)
                  bulk_store(to + ((static_cast<int64_t>(tile) * 2 + h) * chunks + c) * kHalf,
                             sA + c * kChunkA + h * kHalf, kHalf);
                if (layer == kLayers) continue;
              }
              const int s = static_cast<int>(it % kRing);
              if (!mbar_wait_or(&full_bar[s], (it / kRing) & 1u, &abort_flag)) {
                bad = true;
                break;
              }
              ++it;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              const uint32_t pb = smem_u32(ring + s * kChunkW);
#pragma unroll
              for (int j = 0; j < 4; ++j)
                mma_bf16(acc, sw128_desc(pa + 32 * j, 16), sw128_desc(pb + 32 * j, 16), idesc, c > 0 || j > 0);
              mma_commit(&empty_bar[s]);
            }
            if (MODE == kTrain) {
              // the epilogue overwrites the chunks once this layer is complete
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
            if (!bad) mma_commit(&acc_full[turn & 1]);
          }
      if (MODE == kTrain) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
      if (bad) {
        atomicOr(a.err, kErrTimeout);
        abort_flag = 1;
      }
      // every MMA issued has completed before the tensor memory is freed
      mma_commit(&done_bar);
      mbar_wait_bounded(smem_u32(&done_bar), 0u);
    }
  } else {
    // ------------------------------------------------------------- epilogue
    const int e = warp - 2, q = warp & 3, g = e >> 2;
    const int row = q * 32 + lane;          // of the tile
    const int et = tid - 64;                // 0 .. 511
    const uint32_t lanes = tmem + (static_cast<uint32_t>(q * 32) << 16);
    int turn = 0;
    float loss = 0.f;

    auto ready = [&](int c) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_ready[c]);
    };
    // Once a role has given up, every wait returns at once; the epilogue then
    // runs its course on whatever the accumulators hold (the error bit tells),
    // so that no warp is missing at the named barrier.
    auto accumulator = [&]() {
      if (!mbar_wait_or(&acc_full[turn & 1], (turn >> 1) & 1u, &abort_flag)) {
        atomicOr(a.err, kErrTimeout);
        abort_flag = 1;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    // 16 BF16 columns (first: of the chunk) of this thread's row
    auto put = [&](unsigned char* chunk, int r, int col, const uint32_t (&h)[8]) {
      *reinterpret_cast<uint4*>(chunk + chunk_at(r, col)) = make_uint4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint4*>(chunk + chunk_at(r, col + 8)) = make_uint4(h[4], h[5], h[6], h[7]);
    };
    for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
      const int r0 = tile * kRows;
      // ---- the tile's inputs, 16 columns of a row per thread (four threads
      // per row side by side, so that a row's reads share its sectors)
      {
        const int xr = et >> 2, xc = (et & 3) * 16;
        float x[16];
        const int b = r0 + xr;
        int src = -1;
        if (b < a.rows) src = MODE == kTrain && a.idx ? a.idx[b] : b;
        if (MODE != kRank && src >= a.x_rows) src = -1;
        if (MODE == kRank) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int k = xc + j;
            x[j] = src >= 0 && k < a.n_in
                       ? static_cast<float>(log(a.P[static_cast<int64_t>(src) * a.ldp + a.cols[k]] / a.tmpl[k]) /
                                            a.log_spread)
                       : 0.f;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            x[j] = src >= 0 && xc + j < a.n_in ? a.X[static_cast<int64_t>(src) * a.ldx + xc + j] : 0.f;
        }
        uint32_t h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) h[j] = pack2(x[2 * j], x[2 * j + 1]);
        // (the MMAs that read chunk 0 last are complete: this thread waited
        // for the accumulator they filled)
        put(MODE == kRank ? sX : sA, xr, xc, h);
      }
      if (MODE == kRank) {
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpi) : "memory");
      } else {
        ready(0);
      }
      float ensemble[16];
      for (int net = 0; net < passes; ++net) {
        if (MODE == kRank) {
          // 16 KB, 32 bytes a thread
          const uint4* from = reinterpret_cast<const uint4*>(sX) + et * 2;
          uint4* to = reinterpret_cast<uint4*>(sA) + et * 2;
          to[0] = from[0];
          to[1] = from[1];
          ready(0);
        }
        // ---- hidden layers
        for (int layer = 0; layer < 3; ++layer, ++turn) {
          accumulator();
          const uint32_t acc = lanes + (turn & 1) * kHid;
          const float* bias = a.bias[net][layer];
          for (int c = 0; c < 4; ++c) {
            const int col = c * 64 + g * 16;
            float v[16];
            tmem_ld16(acc + col, v);
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const float4 b = *reinterpret_cast<const float4*>(bias + col + j);
              v[j] += b.x;
              v[j + 1] += b.y;
              v[j + 2] += b.z;
              v[j + 3] += b.w;
            }
            uint32_t h[8];
            if (MODE == kTrain) {
              float d[16];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float u0 = gelu_both(v[2 * j], &d[2 * j]), u1 = gelu_both(v[2 * j + 1], &d[2 * j + 1]);
                h[j] = pack2(u0, u1);
              }
              float* to = a.dz + (static_cast<int64_t>(layer) * a.tiles + tile) * kRows * kHid;
#pragma unroll
              for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(to + piece_at(c, j, et)) =
                    make_float4(d[4 * j], d[4 * j + 1], d[4 * j + 2], d[4 * j + 3]);
            } else {
#pragma unroll
              for (int j = 0; j < 8; ++j) h[j] = pack2(gelu(v[2 * j]), gelu(v[2 * j + 1]));
            }
            put(sA + c * kChunkA, row, g * 16, h);
            ready(c);
          }
        }
        // ---- outputs
        accumulator();
        const uint32_t acc = lanes + (turn & 1) * kHid;
        ++turn;
        const float* bias = a.bias[net][3];
        const int b = r0 + row;
        if (MODE == kPredict) {
          for (int col = g * 16; col < n_cols; col += 64) {
            float v[16];
            tmem_ld16(acc + col, v);
            if (b < a.rows) {
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (col + j < a.n_out) a.out[static_cast<int64_t>(b) * a.n_out + col + j] = v[j] + bias[col + j];
            }
          }
        } else if (MODE == kRank) {
          if (g == 0) {
            float v[16];
            tmem_ld16(acc, v);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float y = v[j] + bias[j];
              ensemble[j] = net == 0 ? y : __fadd_rn(ensemble[j], y);
            }
          }
          // every warp is past the accumulator (and so the MMAs past sA)
          // before the next network's inputs overwrite chunk 0
        } else {
          // loss and dY: 2 mask (y - t) / count, BF16 for the products
          const float inv = a.inv_count ? *a.inv_count : a.inv_value;
          int src = -1;
          if (b < a.rows) src = a.idx ? a.idx[b] : b;
          if (src >= a.x_rows) src = -1;
          for (int c = 0; c < oc; ++c) {
            const int col = c * 64 + g * 16;
            float v[16];
            if (col < n_cols) tmem_ld16(acc + col, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              float dy = 0.f;
              if (src >= 0 && col + j < a.n_out) {
                const int64_t at = static_cast<int64_t>(src) * a.n_out + col + j;
                const float m = a.mask[at], d = (v[j] + bias[col + j]) - a.T[at];
                loss += m * d * d * inv;
                dy = 2.f * m * d * inv;
              }
              v[j] = dy;
            }
            uint32_t h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = pack2(v[2 * j], v[2 * j + 1]);
            put(sA + c * kChunkA, row, g * 16, h);
            ready(c);
            float* to = a.dy + static_cast<int64_t>(tile) * kRows * oc * 64;
#pragma unroll
            for (int j = 0; j < 4; ++j)
              *reinterpret_cast<float4*>(to + piece_at(c, j, et)) =
                  make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
        }
      }
      if (MODE == kRank && g == 0) {
        const int b = r0 + row;
        if (b < a.rows) {
          double y[5];
#pragma unroll
          for (int j = 0; j < 5; ++j) {
            const float m = __fdiv_rn(ensemble[j], a.score.nets);
            y[j] = static_cast<double>(__fadd_rn(__fmul_rn(m, a.score.sd[j]), a.score.mu[j]));
          }
          const double per = exp(fmin(fmax(y[0], -10.0), 10.0));
          const double amp_term = fmin(fmax((y[1] - a.score.log_amp_min) / a.score.ramp + 0.5, 0.0), 1.0);
          const double osc_term = fmin(fmax(y[3], 0.0), 1.0);
          const double region = -fabs(per - a.score.period) / a.score.tol + 0.5 * amp_term + 0.5 * osc_term;
          a.scores[b] = y[4] + a.score.weight * region;
        }
      }
      if (MODE == kTrain) {
        // ---- dZ_2, dZ_1, dZ_0: the input gradients times GELU'
        for (int layer = 2; layer >= 0; --layer, ++turn) {
          accumulator();
          const uint32_t acc = lanes + (turn & 1) * kHid;
          float* dz = a.dz + (static_cast<int64_t>(layer) * a.tiles + tile) * kRows * kHid;
          for (int c = 0; c < 4; ++c) {
            const int col = c * 64 + g * 16;
            float d[16], v[16];
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const float4 x = *reinterpret_cast<const float4*>(dz + piece_at(c, j / 4, et));
              d[j] = x.x;
              d[j + 1] = x.y;
              d[j + 2] = x.z;
              d[j + 3] = x.w;
            }
            tmem_ld16(acc + col, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] *= d[j];
            uint32_t h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = pack2(v[2 * j], v[2 * j + 1]);
            put(sA + c * kChunkA, row, g * 16, h);
            ready(c);
#pragma unroll
            for (int j = 0; j < 16; j += 4)
              *reinterpret_cast<float4*>(dz + piece_at(c, j / 4, et)) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
          }
        }
        // dZ_0 has left the chunks: the next tile may write them
        accumulator();
        ++turn;
      }
    }
    if (MODE == kTrain) {
      for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
      if (lane == 0) s_loss[e] = loss;
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpi) : "memory");
      if (et == 0) {
        float s = 0.f;
        for (int i = 0; i < kEpi; ++i) s += s_loss[i];
        atomicAdd(a.loss, s);
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// The training pass of a batch whose tiles leave most SMs idle: a cluster of
// four CTAs carries a tile, each computing 64 of a layer's 256 columns.
// Column chunk r of a layer's result is CTA r's; it is written to its own
// shared memory and copied from there into the three others', whose next
// products wait for it on a barrier of that chunk.  The output layer and dY
// are computed by all four (a fraction of a hidden layer), stored by CTA 0.
// What bounds the pass is the chain of its layers: per layer an epilogue of
// 8192 elements, a copy of 16 KB over distributed shared memory and the
// products; GELU' stays in registers between the passes.  4000 rows: 49 us
// with one CTA a tile, 33 with four.
//
// Three buffers of layer inputs: H0, H2 and dZ1 in the first, H1, dY and dZ0
// in the second, X and dZ2 in the third.  A chunk is sent only once its
// sender has the chunks of the layer before from every CTA, so the receiver
// has completed the products that read that buffer last: those of L0 (X) for
// H1's sender, L1 (H0) for H2's, L4 (dY) and so L3 (H2) for dZ1's; dZ2 goes
// where only X was.
constexpr int kSplit = 4;
constexpr int kSplitRing = 4;    // weight pieces in flight
constexpr int kPiece = 64 * 128;  // 64 output rows of a weight chunk
constexpr int kExchanges = 5;    // H0, H1, H2, dZ2, dZ1

__device__ __forceinline__ uint32_t in_cta(uint32_t addr, int rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(rank));
  return out;
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__global__ void __cluster_dims__(kSplit, 1, 1) __launch_bounds__(kChainThreads, 1)
    mlp_train_split_kernel(const __grid_constant__ ChainArgs a) {
  extern __shared__ __align__(16) unsigned char split_raw[];
  __shared__ __align__(8) uint64_t full_bar[kSplitRing], empty_bar[kSplitRing], own_ready, acc_full[2], done_bar;
  __shared__ __align__(8) uint64_t in_bar[kExchanges][kSplit];
  __shared__ uint32_t tmem_sh;
  __shared__ volatile int abort_flag;
  __shared__ float s_loss[kEpi];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x % kSplit, tile = blockIdx.x / kSplit;
  unsigned char* smem = split_raw + ((1024u - (smem_u32(split_raw) & 1023u)) & 1023u);
  unsigned char* ring = smem + 12 * kChunkA;
  auto buffer = [&](int i) { return smem + i * 4 * kChunkA; };

  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)), "r"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < kSplitRing; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(&own_ready, kEpi);
    for (int i = 0; i < 2; ++i) mbar_init(&acc_full[i], 1);
    mbar_init(&done_bar, 1);
    for (int x = 0; x < kExchanges; ++x)
      for (int c = 0; c < kSplit; ++c) mbar_init(&in_bar[x][c], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int x = 0; x < kExchanges; ++x)
      for (int c = 0; c < kSplit; ++c)
        if (c != rank) expect_bytes(&in_bar[x][c], kChunkA);
    abort_flag = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  cluster_sync();  // every CTA's barriers stand before a chunk is sent
  follow_previous();
  const uint32_t tmem = tmem_sh;
  const int n_cols = out_cols(a.n_out);
  const int oc = out_chunks(a.n_out);
  // layers 0..3 forward, 4..6 back; the chunks of a layer's input, and the
  // 64-row pieces of each weight chunk
  auto chunks_of = [&](int layer) { return layer == 0 ? 1 : (layer == 4 ? oc : 4); };

  if (warp == 0) {
    if (lane == 0) {
      // -------------------------------------------------------- weight ring
      uint32_t it = 0;
      bool bad = false;
      for (int layer = 0; layer < 7 && !bad; ++layer) {
        const int base = layer == 0   ? kFwd0
                         : layer == 1 ? kFwd1
                         : layer == 2 ? kFwd2
                         : layer == 3 ? kFwd3
                         : layer == 4 ? kBwd3
                         : layer == 5 ? kBwd2
                                      : kBwd1;
        const int stride = layer == 3 ? kOutPad * 128 : kChunkW;
        for (int c = 0; c < chunks_of(layer) && !bad; ++c)
          for (int h = 0; h < (layer == 3 ? oc : 1); ++h, ++it) {
            const int s = static_cast<int>(it % kSplitRing);
            if (it >= kSplitRing && !mbar_wait_or(&empty_bar[s], ((it / kSplitRing) - 1) & 1u, &abort_flag)) {
              bad = true;
              break;
            }
            const int rows = layer == 3 ? (n_cols - 64 * h < 64 ? n_cols - 64 * h : 64) : 64;
            const int piece = layer == 3 ? h : rank;
            expect_bytes(&full_bar[s], rows * 128);
            bulk_load(ring + s * kPiece, a.packed[0] + base + c * stride + piece * kPiece, rows * 128, &full_bar[s]);
          }
      }
      if (bad) {
        atomicOr(a.err, kErrTimeout);
        abort_flag = 1;
      }
      // the copies issued last into each stage land before the CTA ends
      for (int s = 0; s < kSplitRing && static_cast<uint32_t>(s) < it; ++s) {
        const uint32_t last = it - 1u - ((it - 1u - static_cast<uint32_t>(s)) % kSplitRing);
        mbar_wait_bounded(smem_u32(&full_bar[s]), (last / kSplitRing) & 1u);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ------------------------------------------- products, copies, stores
      uint32_t it = 0;
      const int64_t blocks = static_cast<int64_t>(a.tiles) * 2;
      bool bad = false;
      // (an eighth, without products, stores dZ_0)
      for (int layer = 0; layer < 8 && !bad; ++layer) {
        // input of layer: X, H0, H1, H2, dY, dZ2, dZ1; then dZ0
        const int where = layer == 0 || layer == 5 ? 2 : (layer == 1 || layer == 3 || layer == 6 ? 0 : 1);
        const bool shared = layer != 0 && layer != 4;  // chunk c comes from CTA c
        const int exchange = layer < 4 ? layer - 1 : layer - 2;
        const int chunks = layer == 7 ? 4 : chunks_of(layer);
        unsigned char* in = buffer(where);
        if (!mbar_wait_or(&own_ready, layer & 1u, &abort_flag)) {
          bad = true;
          break;
        }
        if (shared && layer < 7) {
          const uint32_t src = smem_u32(in + rank * kChunkA), bar = smem_u32(&in_bar[exchange][rank]);
          for (int k = 1; k < kSplit; ++k) {
            const int to = (rank + k) % kSplit;
            asm volatile(
                "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    in_cta(src, to)),
                "r"(src), "r"(kChunkA), "r"(in_cta(bar, to))
                : "memory");
          }
        }
        // the chunks are also operands of the weight gradients: inputs of
        // layers 0-3, then dY, dZ_2, dZ_1, dZ_0
        unsigned char* to = layer < 4 ? a.act + act_base(layer, blocks) : a.grad + grad_base(7 - layer, blocks);
        for (int c = 0; c < chunks; ++c)
          if (shared ? c == rank : rank == 0)
            for (int h = 0; h < 2; ++h)
              bulk_store(to + ((static_cast<int64_t>(tile) * 2 + h) * chunks + c) * kHalf, in + c * kChunkA + h * kHalf,
                         kHalf);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        if (layer == 7) break;
        const uint32_t acc = tmem + (layer & 1) * 128;
        for (int c = 0; c < chunks && !bad; ++c) {
          if (shared && c != rank && !mbar_wait_or(&in_bar[exchange][c], 0u, &abort_flag)) {
            bad = true;
            break;
          }
          const uint32_t pa = smem_u32(in + c * kChunkA);
          for (int h = 0; h < (layer == 3 ? oc : 1); ++h, ++it) {
            const int s = static_cast<int>(it % kSplitRing);
            if (!mbar_wait_or(&full_bar[s], (it / kSplitRing) & 1u, &abort_flag)) {
              bad = true;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int n = layer == 3 ? (n_cols - 64 * h < 64 ? n_cols - 64 * h : 64) : 64;
            const uint32_t pb = smem_u32(ring + s * kPiece), idesc = umma_idesc_bf16(kRows, n);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              mma_bf16(acc + 64 * h, sw128_desc(pa + 32 * j, 16), sw128_desc(pb + 32 * j, 16), idesc, c > 0 || j > 0);
            mma_commit(&empty_bar[s]);
          }
        }
        // the epilogue may overwrite the chunks stored once this layer is
        // complete
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        if (!bad) mma_commit(&acc_full[layer & 1]);
      }
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
      if (bad) {
        atomicOr(a.err, kErrTimeout);
        abort_flag = 1;
      }
      // every MMA issued has completed before the tensor memory is freed
      mma_commit(&done_bar);
      mbar_wait_bounded(smem_u32(&done_bar), 0u);
    }
  } else {
    // ------------------------------------------------------------- epilogue
    const int e = warp - 2, q = warp & 3, g = e >> 2;
    const int row = q * 32 + lane;          // of the tile
    const int et = tid - 64;                // 0 .. 511
    const uint32_t lanes = tmem + (static_cast<uint32_t>(q * 32) << 16);
    const int r0 = tile * kRows;
    float loss = 0.f;

    auto ready = [&]() {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&own_ready);
    };
    // (once a role has given up, every wait returns at once)
    auto accumulator = [&](int layer) {
      if (!mbar_wait_or(&acc_full[layer & 1], (layer >> 1) & 1u, &abort_flag)) {
        atomicOr(a.err, kErrTimeout);
        abort_flag = 1;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    // 16 BF16 columns (first: of the chunk) of a row
    auto put = [&](unsigned char* chunk, int r, int col, const float (&v)[16]) {
      uint32_t h[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) h[j] = pack2(v[2 * j], v[2 * j + 1]);
      *reinterpret_cast<uint4*>(chunk + chunk_at(r, col)) = make_uint4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint4*>(chunk + chunk_at(r, col + 8)) = make_uint4(h[4], h[5], h[6], h[7]);
    };
    // ---- the tile's inputs, 16 columns of a row per thread
    {
      const int xr = et >> 2, xc = (et & 3) * 16;
      float x[16];
      const int b = r0 + xr;
      int src = -1;
      if (b < a.rows) src = a.idx ? a.idx[b] : b;
      if (src >= a.x_rows) src = -1;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        x[j] = src >= 0 && xc + j < a.n_in ? a.X[static_cast<int64_t>(src) * a.ldx + xc + j] : 0.f;
      put(buffer(2), xr, xc, x);
      ready();
    }
    // ---- hidden layers: this CTA's 64 columns, 16 of a row per thread
    float d[3][16];
#pragma unroll
    for (int layer = 0; layer < 3; ++layer) {
      accumulator(layer);
      const float* bias = a.bias[0][layer] + rank * 64 + g * 16;
      float v[16];
      tmem_ld16(lanes + (layer & 1) * 128 + g * 16, v);
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const float4 b = *reinterpret_cast<const float4*>(bias + j);
        v[j] += b.x;
        v[j + 1] += b.y;
        v[j + 2] += b.z;
        v[j + 3] += b.w;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = gelu_both(v[j], &d[layer][j]);
      put(buffer(layer == 1 ? 1 : 0) + rank * kChunkA, row, g * 16, v);
      ready();
    }
    // ---- outputs, loss and dY: 2 mask (y - t) / count
    {
      const float inv = a.inv_count ? *a.inv_count : a.inv_value;
      const float* bias = a.bias[0][3];
      const int b = r0 + row;
      int src = -1;
      if (b < a.rows) src = a.idx ? a.idx[b] : b;
      if (src >= a.x_rows) src = -1;
      accumulator(3);
      for (int c = 0; c < oc; ++c) {
        const int col = c * 64 + g * 16;
        float v[16];
        if (col < n_cols) tmem_ld16(lanes + 128 + col, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float dy = 0.f;
          if (src >= 0 && col + j < a.n_out) {
            const int64_t at = static_cast<int64_t>(src) * a.n_out + col + j;
            const float m = a.mask[at], diff = (v[j] + bias[col + j]) - a.T[at];
            loss += m * diff * diff * inv;
            dy = 2.f * m * diff * inv;
          }
          v[j] = dy;
        }
        put(buffer(1) + c * kChunkA, row, g * 16, v);
        if (rank == 0) {
          float* to = a.dy + static_cast<int64_t>(tile) * kRows * oc * 64;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(to + piece_at(c, j, et)) =
                make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
      }
      ready();
    }
    // ---- dZ_2, dZ_1, dZ_0: the input gradients times GELU'
#pragma unroll
    for (int layer = 2; layer >= 0; --layer) {
      const int product = 6 - layer;
      accumulator(product);
      float v[16];
      tmem_ld16(lanes + (product & 1) * 128 + g * 16, v);
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] *= d[layer][j];
      put(buffer(layer == 2 ? 2 : 1 - layer) + rank * kChunkA, row, g * 16, v);
      ready();
      float* dz = a.dz + (static_cast<int64_t>(layer) * a.tiles + tile) * kRows * kHid;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4*>(dz + piece_at(rank, j, et)) =
            make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    if (rank == 0) {
      for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
      if (lane == 0) s_loss[e] = loss;
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpi) : "memory");
      if (et == 0) {
        float sum = 0.f;
        for (int i = 0; i < kEpi; ++i) sum += s_loss[i];
        atomicAdd(a.loss, sum);
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256));
  cluster_sync();  // no CTA ends while another may read or write its memory
  if (abort_flag) {
    // after a wait that ran out: time for a copy still on its way to land
    const long long t0 = clock64();
    while (clock64() - t0 < (1ll << 20)) {
    }
  }
}

// --------------------------------------------------------- weight gradients

struct WgradArgs {
  const unsigned char *act, *grad;
  int64_t blocks;   // 64-row blocks of the batch
  int oc;           // 64-column chunks of dY
  int splits, per;          // layers 0-2: ranges of `per` blocks
  int out_splits, out_per;  // the output layer's
  float* parts;             // [splits][kHidWeights]
  float* out_parts;         // [out_splits][kOutWeights]
  int* err;
};

constexpr int kWgradThreads = 192;
constexpr int kWgradStage = 2 * kHalf + 4 * kHalf;  // A: 128 columns of dZ, B: up to 256 of the layer's input

// dW_i = dZ_i^T . input_i over a range of 64-row blocks, both operands
// MN-major straight from the chain kernel's chunks (no transposed copies).
// A unit is 128 output rows of one layer (seven of them: two each of layers
// 0-2, one of the output layer) and one range; its FP32 part goes to the
// workspace, and finish_kernel adds the ranges in order.
__global__ void __launch_bounds__(kWgradThreads, 1) mlp_wgrad_kernel(const WgradArgs a) {
  extern __shared__ __align__(16) unsigned char wgrad_raw[];
  __shared__ __align__(8) uint64_t full_bar[kRing], empty_bar[kRing], acc_full;
  __shared__ uint32_t tmem_sh;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* ring = wgrad_raw + ((1024u - (smem_u32(wgrad_raw) & 1023u)) & 1023u);
  const bool output = static_cast<int>(blockIdx.x) >= 6 * a.splits;
  const int unit = output ? 6 : blockIdx.x % 6, split = output ? blockIdx.x - 6 * a.splits : blockIdx.x / 6;
  const int layer = unit >> 1, half = unit & 1;
  const int per = output ? a.out_per : a.per;
  const int n = layer == 0 ? kInPad : kHid;
  const int nc = n / 64;                            // chunks of the layer input
  const int ac = layer == 3 ? a.oc : 4;             // chunks of dZ
  const int take = layer == 3 ? a.oc : 2;           // of them, this unit's
  const int64_t b0 = static_cast<int64_t>(split) * per;
  const int count = static_cast<int>(a.blocks - b0 < per ? a.blocks - b0 : per);

  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)), "r"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(&acc_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  follow_previous();
  const uint32_t tmem = tmem_sh;

  if (warp == 0) {
    if (lane == 0) {
      bool bad = false;
      int i = 0;
      const unsigned char* ga = a.grad + grad_base(layer, a.blocks) + static_cast<int64_t>(half) * 2 * kHalf;
      const unsigned char* gb = a.act + act_base(layer, a.blocks);
      const uint32_t abytes = take * kHalf, bbytes = nc * kHalf;
      for (; i < count; ++i) {
        const int s = i % kRing;
        if (i >= kRing && !mbar_wait_or(&empty_bar[s], ((i / kRing) - 1) & 1, &abort_flag)) {
          bad = true;
          break;
        }
        expect_bytes(&full_bar[s], abytes + bbytes);
        bulk_load(ring + s * kWgradStage, ga + (b0 + i) * ac * kHalf, abytes, &full_bar[s]);
        bulk_load(ring + s * kWgradStage + 2 * kHalf, gb + (b0 + i) * nc * kHalf, bbytes, &full_bar[s]);
      }
      if (bad) {
        atomicOr(a.err, kErrTimeout);
        abort_flag = 1;
      }
      for (int s = 0; s < kRing && s < i; ++s) {
        const int last = i - 1 - ((i - 1 - s) % kRing);
        mbar_wait_bounded(smem_u32(&full_bar[s]), (last / kRing) & 1);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // both operands MN-major
      const uint32_t idesc = umma_idesc_bf16(128, n) | (1u << 15) | (1u << 16);
      bool bad = false;
      for (int i = 0; i < count; ++i) {
        const int s = i % kRing;
        if (!mbar_wait_or(&full_bar[s], (i / kRing) & 1, &abort_flag)) {
          bad = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t pa = smem_u32(ring + s * kWgradStage), pb = pa + 2 * kHalf;
#pragma unroll
        for (int j = 0; j < 4; ++j)  // 16 batch rows: 2048 bytes
          mma_bf16(tmem, sw128_desc(pa + 2048 * j, kHalf), sw128_desc(pb + 2048 * j, kHalf), idesc, i > 0 || j > 0);
        mma_commit(&empty_bar[s]);
      }
      if (bad) {
        atomicOr(a.err, kErrTimeout);
        abort_flag = 1;
      }
      mma_commit(&acc_full);
      mbar_wait_bounded(smem_u32(&acc_full), 0u);  // before the tensor memory is freed
    }
  } else {
    const int q = warp & 3;
    if (mbar_wait_or(&acc_full, 0u, &abort_flag) && !abort_flag) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int o = half * 128 + q * 32 + lane;  // output row of the layer
      constexpr int first[3] = {0, kHid * kInPad, kHid * kInPad + kHid * kHid};
      float* dst = (output ? a.out_parts + static_cast<int64_t>(split) * kOutWeights
                           : a.parts + static_cast<int64_t>(split) * kHidWeights + first[layer]) +
                   static_cast<int64_t>(o) * n;
      // rows of the output layer past dY's chunks have no gradient
      const bool live = layer < 3 || q * 32 + lane < a.oc * 64;
      for (int c = 0; c < n; c += 16) {
        float v[16];
        tmem_ld16(tmem + (static_cast<uint32_t>(q * 32) << 16) + c, v);
        float4* to = reinterpret_cast<float4*>(dst + c);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          to[j] = live ? make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
      atomicOr(a.err, kErrTimeout);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256));
}

// ------------------------------------------------------------ bias gradients

// Column sums of dZ_0, dZ_1, dZ_2 and dY over one of eight slices of the
// rows, in colsum_kernel's order of additions (eight strided sums per row
// lane, combined pairwise, then the 32 row lanes in order; finish_kernel
// adds the slices in order), so a bias gradient is the same from either.
// Block (column group of 32, slice).
constexpr int kColSlices = 8;

__global__ void __launch_bounds__(256) mlp_bias_sums_kernel(const float* dz, const float* dy, int tiles, int oc,
                                                            float* db_part) {
  __shared__ float part[32][33];
  follow_previous();
  const int y = threadIdx.x & 31, w = threadIdx.x >> 5;  // row lane, four columns
  const int layer = blockIdx.x / 8 < 3 ? blockIdx.x / 8 : 3;
  const int c0 = (layer < 3 ? blockIdx.x % 8 : blockIdx.x - 24) * 32;
  const int col = c0 + 4 * w;
  const int per_tile = kRows * (layer < 3 ? kHid : oc * 64);
  const float* p = layer < 3 ? dz + static_cast<int64_t>(layer) * tiles * per_tile : dy;
  auto at = [&](int r) {
    return *reinterpret_cast<const float4*>(p + static_cast<int64_t>(r >> 7) * per_tile +
                                            piece_at(col >> 6, (col & 15) >> 2, epi_thread(r & 127, col)));
  };
  const int rows = tiles * kRows, per = rows / kColSlices;
  const int r0 = blockIdx.y * per, r1 = r0 + per;
  float acc[8][4] = {};
  int r = r0 + y;
  for (; r + 7 * 32 < r1; r += 8 * 32) {
    float4 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = at(r + j * 32);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      acc[j][0] += v[j].x;
      acc[j][1] += v[j].y;
      acc[j][2] += v[j].z;
      acc[j][3] += v[j].w;
    }
  }
  for (; r < r1; r += 32) {
    const float4 v = at(r);
    acc[0][0] += v.x;
    acc[0][1] += v.y;
    acc[0][2] += v.z;
    acc[0][3] += v.w;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    part[y][4 * w + k] = ((acc[0][k] + acc[1][k]) + (acc[2][k] + acc[3][k])) +
                         ((acc[4][k] + acc[5][k]) + (acc[6][k] + acc[7][k]));
  __syncthreads();
  if (threadIdx.x < 32) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) s += part[i][threadIdx.x];
    db_part[(layer * kColSlices + blockIdx.y) * kHid + c0 + threadIdx.x] = s;
  }
}

// ------------------------------------------------------------------- finish

struct FinishArgs {
  const float* parts;      // [splits][kHidWeights]
  const float* out_parts;  // [out_splits][kOutWeights]
  const float* db_part;    // [4][8][256]
  int splits, out_splits, oc;
  float *dW[4], *db[4];  // written when dW[0] is not null
  // Adam, when hyper is not null: {lr, b1, b2, eps, 1 - b1^t, 1 - b2^t}
  const float* hyper;
  float *W[4], *b[4], *mW[4], *vW[4], *mb[4], *vb[4];
  unsigned char* packed;
};

constexpr int kBiases = 3 * kHid + kOutPad;

__device__ __forceinline__ float adam_update(float w, float g, float* m, float* v, const float* hyper) {
  const float lr = hyper[0], b1 = hyper[1], b2 = hyper[2], eps = hyper[3], c1 = hyper[4], c2 = hyper[5];
  // (the contractions of adam_kernel, spelled out so that both give the same)
  const float mi = __fmaf_rn(1.f - b1, g, __fmul_rn(b1, *m));
  const float vi = __fmaf_rn(__fmul_rn(1.f - b2, g), g, __fmul_rn(b2, *v));
  *m = mi;
  *v = vi;
  return w - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// Four weights, or one bias, per thread: the parts summed in range (slice)
// order, the gradients written out, Adam applied and the new weights packed.
__global__ void __launch_bounds__(256) mlp_finish_kernel(const __grid_constant__ FinishArgs a) {
  follow_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < kWeights / 4) {
    int at;
    const int layer = layer_of(t * 4, &at);
    const float4* p = reinterpret_cast<const float4*>(layer == 3 ? a.out_parts + at : a.parts + t * 4);
    const int splits = layer == 3 ? a.out_splits : a.splits;
    const int64_t stride = (layer == 3 ? kOutWeights : kHidWeights) / 4;
    float4 s = *p;
    for (int k = 1; k < splits; ++k) {
      const float4 x = p[k * stride];
      s.x += x.x;
      s.y += x.y;
      s.z += x.z;
      s.w += x.w;
    }
    if (a.dW[0]) *reinterpret_cast<float4*>(a.dW[layer] + at) = s;
    if (a.hyper) {
      float4 w = *reinterpret_cast<const float4*>(a.W[layer] + at);
      float4 m = *reinterpret_cast<const float4*>(a.mW[layer] + at), v = *reinterpret_cast<const float4*>(a.vW[layer] + at);
      w.x = adam_update(w.x, s.x, &m.x, &v.x, a.hyper);
      w.y = adam_update(w.y, s.y, &m.y, &v.y, a.hyper);
      w.z = adam_update(w.z, s.z, &m.z, &v.z, a.hyper);
      w.w = adam_update(w.w, s.w, &m.w, &v.w, a.hyper);
      *reinterpret_cast<float4*>(a.W[layer] + at) = w;
      *reinterpret_cast<float4*>(a.mW[layer] + at) = m;
      *reinterpret_cast<float4*>(a.vW[layer] + at) = v;
      const float u[4] = {w.x, w.y, w.z, w.w};
      pack_quad(a.packed, layer, at, u, true);
    }
  } else if (t < kWeights / 4 + kBiases) {
    const int i = t - kWeights / 4;
    const int layer = i / kHid, c = i % kHid;
    float s = 0.f;
    if (layer < 3 || c < a.oc * 64)
      for (int k = 0; k < kColSlices; ++k) s += a.db_part[(layer * kColSlices + k) * kHid + c];
    if (a.db[0]) a.db[layer][c] = s;
    if (a.hyper) a.b[layer][c] = adam_update(a.b[layer][c], s, &a.mb[layer][c], &a.vb[layer][c], a.hyper);
  }
}

// -------------------------------------------------------------------- hosts

int device_sms() {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> cached[kMaxDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  cached[dev].store(n, std::memory_order_relaxed);
  return n;
}

constexpr size_t kChainSmem = 4 * kChunkA + kRing * kChunkW + 1024;
constexpr size_t kRankSmem = kChainSmem + kChunkA;
constexpr size_t kSplitSmem = 12 * kChunkA + kSplitRing * kPiece + 1024;
constexpr size_t kWgradSmem = kRing * kWgradStage + 1024;

// Opt-in to the shared memory, once per device (no attribute calls inside a
// graph capture after the first launch).
template <auto kernel>
cudaError_t opt_in(size_t bytes) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static bool done[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (done[dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  done[dev] = e == cudaSuccess;
  return e;
}

// Launches a kernel that calls follow_previous.
template <typename... Params, typename... Args>
cudaError_t launch_next(void (*kernel)(Params...), dim3 grid, int block, size_t smem, cudaStream_t s,
                        const Args&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// Clusters of mlp_train_split_kernel that the GPU holds at once (33 on a
// B200: four SMs of one GPC each), 0 where it cannot run.
int split_clusters() {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> cached[kMaxDevices] = {};  // one more than the count
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  const int known = cached[dev].load(std::memory_order_relaxed);
  if (known > 0) return known - 1;
  if (opt_in<mlp_train_split_kernel>(kSplitSmem) != cudaSuccess) return 0;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kSplit;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kSplit);
  cfg.blockDim = dim3(kChainThreads);
  cfg.dynamicSmemBytes = kSplitSmem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, mlp_train_split_kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cached[dev].store(n + 1, std::memory_order_relaxed);
  return n;
}

template <int MODE>
int launch_chain(const ChainArgs& a, size_t smem, cudaStream_t s) {
  const int sms = device_sms();
  if (sms <= 0) return 2;
  if (opt_in<mlp_chain_kernel<MODE>>(smem) != cudaSuccess) return 2;
  const int grid = a.tiles < sms ? a.tiles : sms;
  if (MODE == kTrain) return launch_next(mlp_chain_kernel<MODE>, dim3(grid), kChainThreads, smem, s, a) ? 2 : 0;
  mlp_chain_kernel<MODE><<<grid, kChainThreads, smem, s>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

bool aligned(const void* p, size_t n) { return p && reinterpret_cast<uintptr_t>(p) % n == 0; }

}  // namespace

CHAIN_API int64_t dense_mlp_packed_bytes(void) { return kPacked; }

CHAIN_API int dense_mlp_pack(const float* const* W, void* packed, int backward, void* stream) {
  if (!W || !aligned(packed, 16)) return 1;
  Weights w;
  for (int i = 0; i < 4; ++i) {
    if (!aligned(W[i], 16)) return 1;
    w.W[i] = W[i];
  }
  pack_kernel<<<(kWeights / 4 + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      w, static_cast<unsigned char*>(packed), backward);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

CHAIN_API int dense_mlp_predict(const float* X, int ldx, int rows, int n_in, const void* packed,
                                const float* const* bias, int n_out, float* out, int* err, void* stream) {
  if (rows < 0 || n_in < 1 || n_in > kInPad || ldx < n_in || n_out < 1 || n_out > kOutPad || !aligned(packed, 16) ||
      !bias || !err)
    return 1;
  if (rows == 0) return 0;
  if (!X || !out) return 1;
  ChainArgs a{};
  a.rows = a.x_rows = rows;
  a.tiles = (rows - 1) / kRows + 1;
  a.n_in = n_in;
  a.n_out = n_out;
  a.nets = 1;
  a.packed[0] = static_cast<const unsigned char*>(packed);
  for (int i = 0; i < 4; ++i) {
    if (!aligned(bias[i], 16)) return 1;
    a.bias[0][i] = bias[i];
  }
  a.err = err;
  a.X = X;
  a.ldx = ldx;
  a.out = out;
  return launch_chain<kPredict>(a, kChainSmem, static_cast<cudaStream_t>(stream));
}

CHAIN_API int dense_mlp_rank(const double* P, int ldp, int rows, const int* cols, const double* tmpl, int n_in,
                             double log_spread, int nets, const void* const* packed, const float* const* bias,
                             int n_out, const float* mu, const float* sd, double weight, double period, double tol,
                             double amp_min, double ramp, double* out, int* err, void* stream) {
  if (rows < 0 || n_in < 1 || n_in > kInPad || n_out < 5 || n_out > 8 || nets < 1 || nets > kMaxNets || !packed ||
      !bias || !mu || !sd || !err || !(log_spread != 0.0) || !(amp_min > 0.0) || !(tol > 0.0) || !(ramp > 0.0))
    return 1;
  if (rows == 0) return 0;
  if (!P || !cols || !tmpl || !out) return 1;
  ChainArgs a{};
  a.rows = a.x_rows = rows;
  a.tiles = (rows - 1) / kRows + 1;
  a.n_in = n_in;
  a.n_out = n_out;
  a.nets = nets;
  for (int k = 0; k < nets; ++k) {
    if (!aligned(packed[k], 16)) return 1;
    a.packed[k] = static_cast<const unsigned char*>(packed[k]);
    for (int i = 0; i < 4; ++i) {
      if (!aligned(bias[4 * k + i], 16)) return 1;
      a.bias[k][i] = bias[4 * k + i];
    }
  }
  a.err = err;
  a.P = P;
  a.ldp = ldp;
  a.cols = cols;
  a.tmpl = tmpl;
  a.log_spread = log_spread;
  for (int j = 0; j < n_out; ++j) {
    a.score.mu[j] = mu[j];
    a.score.sd[j] = sd[j];
  }
  a.score.nets = static_cast<float>(nets);
  a.score.weight = weight;
  a.score.period = period;
  a.score.tol = tol;
  a.score.log_amp_min = std::log(amp_min);
  a.score.ramp = ramp;
  a.scores = out;
  return launch_chain<kRank>(a, kRankSmem, static_cast<cudaStream_t>(stream));
}

// Work buffers of a training pass over `rows` rows, in one allocation:
// activations, gradients, GELU' and the column sums, then the parts.
namespace {
struct TrainBuffers {
  int64_t tiles, blocks, per, splits, out_per, out_splits;
  int64_t grad, dz, dy, db_part, parts, out_parts, bytes;
  TrainBuffers(int rows, int n_out) {
    tiles = (static_cast<int64_t>(rows) + kRows - 1) / kRows;
    blocks = 2 * tiles;
    // Ranges of four blocks or a little more (the bulk copies of a range are
    // then all in flight), longer ones past as many ranges as one layer's
    // units fill the GPU's SMs with: each FP32 sum runs over so many rows,
    // the same as in dense_mlp_gemm_ws, whose results these equal.
    auto ranges = [&](int64_t most, int64_t* n, int64_t* each) {
      *n = blocks < 8 ? 1 : blocks / 4;
      if (*n > most) *n = most;
      *each = (blocks + *n - 1) / *n;
      *n = (blocks + *each - 1) / *each;
    };
    ranges(148 / 2, &splits, &per);
    ranges(148, &out_splits, &out_per);
    grad = 13 * blocks * kHalf;
    dz = grad + (12 + out_chunks(n_out)) * blocks * kHalf;
    dy = dz + 3 * tiles * kRows * kHid * 4;
    db_part = dy + tiles * kRows * out_chunks(n_out) * 64 * 4;
    parts = db_part + 4 * kColSlices * kHid * 4;
    out_parts = parts + splits * kHidWeights * 4;
    bytes = out_parts + out_splits * kOutWeights * 4;
  }
};
}  // namespace

CHAIN_API int64_t dense_mlp_train_bytes(int rows, int n_out) {
  if (rows < 1 || n_out < 1 || n_out > kOutPad) return 0;
  return TrainBuffers(rows, n_out).bytes;
}

CHAIN_API int dense_mlp_train_pass(const float* X, int ldx, int x_rows, int n_in, const float* T, const float* mask,
                                   int n_out, const int* idx, int rows, const void* packed, const float* const* bias,
                                   const float* inv_count, float inv_value, float* loss, void* work,
                                   int64_t work_bytes, int* err, void* stream) {
  if (rows < 1 || x_rows < 1 || n_in < 1 || n_in > kInPad || ldx < n_in || n_out < 1 || n_out > kOutPad || !X || !T ||
      !mask || !aligned(packed, 16) || !bias || !loss || !aligned(work, 256) || !err)
    return 1;
  const TrainBuffers t(rows, n_out);
  if (work_bytes < t.bytes || t.tiles > (1 << 20)) return 1;
  unsigned char* w = static_cast<unsigned char*>(work);
  ChainArgs a{};
  a.rows = rows;
  a.x_rows = x_rows;
  a.tiles = static_cast<int>(t.tiles);
  a.n_in = n_in;
  a.n_out = n_out;
  a.nets = 1;
  a.packed[0] = static_cast<const unsigned char*>(packed);
  for (int i = 0; i < 4; ++i) {
    if (!aligned(bias[i], 16)) return 1;
    a.bias[0][i] = bias[i];
  }
  a.err = err;
  a.X = X;
  a.ldx = ldx;
  a.idx = idx;
  a.T = T;
  a.mask = mask;
  a.inv_count = inv_count;
  a.inv_value = inv_value;
  a.loss = loss;
  a.act = w;
  a.grad = w + t.grad;
  a.dz = reinterpret_cast<float*>(w + t.dz);
  a.dy = reinterpret_cast<float*>(w + t.dy);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // four CTAs a tile while the GPU holds all of the clusters at once, else
  // one (pass, bias sums and weight gradients, each launch after the one
  // before: 4096 rows 67 us with one CTA a tile and 52 with four; 4480 rows,
  // two clusters more than fit, 68 and 80)
  if (a.tiles <= split_clusters()) {
    if (launch_next(mlp_train_split_kernel, dim3(kSplit * a.tiles), kChainThreads, kSplitSmem, s, a)) return 2;
  } else {
    const int rc = launch_chain<kTrain>(a, kChainSmem, s);
    if (rc) return rc;
  }
  if (launch_next(mlp_bias_sums_kernel, dim3(24 + 2 * out_chunks(n_out), kColSlices), 256, 0, s, a.dz, a.dy, t.tiles,
                  out_chunks(n_out), reinterpret_cast<float*>(w + t.db_part)))
    return 2;
  if (opt_in<mlp_wgrad_kernel>(kWgradSmem) != cudaSuccess) return 2;
  WgradArgs g{};
  g.act = w;
  g.grad = w + t.grad;
  g.blocks = t.blocks;
  g.oc = out_chunks(n_out);
  g.splits = static_cast<int>(t.splits);
  g.per = static_cast<int>(t.per);
  g.out_splits = static_cast<int>(t.out_splits);
  g.out_per = static_cast<int>(t.out_per);
  g.parts = reinterpret_cast<float*>(w + t.parts);
  g.out_parts = reinterpret_cast<float*>(w + t.out_parts);
  g.err = err;
  return launch_next(mlp_wgrad_kernel, dim3(6 * g.splits + g.out_splits), kWgradThreads, kWgradSmem, s, g) ? 2 : 0;
}

CHAIN_API int dense_mlp_train_finish(const void* work, int64_t work_bytes, int rows, int n_out, float* const* dW,
                                     float* const* db, const float* hyper, float* const* W, float* const* b,
                                     float* const* mW, float* const* vW, float* const* mb, float* const* vb,
                                     void* packed, void* stream) {
  if (rows < 1 || n_out < 1 || n_out > kOutPad || !aligned(work, 256) || (!dW != !db) || (!dW && !hyper) ||
      (hyper && (!W || !b || !mW || !vW || !mb || !vb || !aligned(packed, 16))))
    return 1;
  const TrainBuffers t(rows, n_out);
  if (work_bytes < t.bytes) return 1;
  const unsigned char* w = static_cast<const unsigned char*>(work);
  FinishArgs a{};
  a.parts = reinterpret_cast<const float*>(w + t.parts);
  a.out_parts = reinterpret_cast<const float*>(w + t.out_parts);
  a.db_part = reinterpret_cast<const float*>(w + t.db_part);
  a.splits = static_cast<int>(t.splits);
  a.out_splits = static_cast<int>(t.out_splits);
  a.oc = out_chunks(n_out);
  a.hyper = hyper;
  for (int i = 0; i < 4; ++i) {
    if (dW) {
      if (!aligned(dW[i], 16) || !db[i]) return 1;
      a.dW[i] = dW[i];
      a.db[i] = db[i];
    }
    if (hyper) {
      if (!aligned(W[i], 16) || !aligned(mW[i], 16) || !aligned(vW[i], 16) || !b[i] || !mb[i] || !vb[i]) return 1;
      a.W[i] = W[i];
      a.b[i] = b[i];
      a.mW[i] = mW[i];
      a.vW[i] = vW[i];
      a.mb[i] = mb[i];
      a.vb[i] = vb[i];
    }
  }
  a.packed = static_cast<unsigned char*>(packed);
  return launch_next(mlp_finish_kernel, dim3((kWeights / 4 + kBiases + 255) / 256), 256, 0,
                     static_cast<cudaStream_t>(stream), a)
             ? 2
             : 0;
}

CHAIN_API int dense_mlp_train_epoch(const float* X, int ldx, int x_rows, int n_in, const float* T, const float* mask,
                                    int n_out, const int* idx, int rows, int steps, const float* hyper, float* loss,
                                    void* work, int64_t work_bytes, float* const* W, float* const* b,
                                    float* const* mW, float* const* vW, float* const* mb, float* const* vb,
                                    void* packed, int* err, void* stream) {
  if (steps < 0 || !idx || !hyper) return 1;
  for (int j = 0; j < steps; ++j) {
    const int64_t at = static_cast<int64_t>(j) * rows;
    int rc = dense_mlp_train_pass(X, ldx, x_rows, n_in, T, mask, n_out, idx + at, rows, packed, b, hyper + 8 * j + 6,
                                  0.f, loss, work, work_bytes, err, stream);
    if (rc == 0)
      rc = dense_mlp_train_finish(work, work_bytes, rows, n_out, nullptr, nullptr, hyper + 8 * j, W, b, mW, vW, mb, vb,
                                  packed, stream);
    if (rc) return rc;
  }
  return 0;
}
