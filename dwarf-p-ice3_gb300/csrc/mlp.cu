// mlp.cu — BF16 tensor-core (tcgen05) GEMM with fused epilogues, and the
// per-point MLP of the slow-process surrogate built on it (forward,
// hand-written backward, Adam).
//
// tc_gemm_kernel: one CTA (8 warps) computes a 128 x 128 tile (N <= 256) of
//   C[m][n] = sum_k A(m, k) B(n, k),  A(m, k) = A[m*sam + k*sak],  B(n, k) = B[n*sbn + k*sbk]
// in FP32 in TMEM.  K is walked in chunks of 64 through a ring of G_NST
// shared-memory stages in the K-major core-matrix layout, filled with 16-byte
// asynchronous copies where K is the contiguous index (element loads
// otherwise, which also transpose); one thread issues the K/16 tcgen05.mma of
// a chunk and commits them to the stage's mbarrier, and a stage is refilled
// once its MMAs are done (bounded waits).  Rows >= M and k >= K are staged as
// zeros.  The epilogue reads the tile back with tcgen05.ld (warp w: rows
// 32 (w % 4) .. + 31, every second group of 16 columns) and applies:
//   EPI_STORE     C -> f32 (split-K partials at C + split * M * ldc)
//   EPI_BIAS_GELU Z = C + bias -> f32 Zout (optional), H = GELU(Z) -> bf16
//   EPI_BIAS      Y = C + bias -> f32
//   EPI_DGELU     dZ = C * GELU'(Zin) -> bf16 H and f32 C
// H also goes to HT, transposed ([n][m], zeros up to the tile's last row),
// where the caller wants it: the weight gradients contract over m, and with
// HT their operands have m contiguous too.
// Bound: at the training batch (16,384 rows) the latency of filling the ring
// and the epilogue's stores; four warps, one stage and element-wise transposing
// took 122 us per hidden layer forward, 299 us backward and 776 us per weight
// gradient.  Tiles of 128 columns with three stages put two CTAs on an SM: a
// gradient of 16,384 rows 407 -> 387 us against tiles of 256 with four.
// The epilogue's rows go through the ring's shared memory, four lanes to a
// row: 387 -> 359 us against a lane to a row, whose accesses touch 32 lines.
// On a barrier timeout the kernel sets *err, stops issuing and frees its
// TMEM after a second bounded wait.
#include <cuda_bf16.h>
#include <math.h>

#include "ice3gb_kernels.h"
#include "tc_sm103.cuh"

namespace {

constexpr int KC = 64;                 // K chunk per stage
constexpr long WAIT_ITERS = 1L << 22;  // bounded mbarrier wait (about a second at most)

// GELU in its tanh form, 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3)))
// (Hendrycks & Gimpel 2016), with the hardware tanh.approx.f32: one MUFU
// operation and five FP32 operations per activation, the same function in
// training and inference.
__device__ __forceinline__ float tanh_hw(float x)
{
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float gelu(float z)
{
  const float u = z * fmaf(0.035677408136300125f, z * z, 0.7978845608028654f);
  const float h = 0.5f * z;
  return fmaf(h, tanh_hw(u), h);
}
__device__ __forceinline__ float dgelu(float z)
{
  const float z2 = z * z;
  const float th = tanh_hw(z * fmaf(0.035677408136300125f, z2, 0.7978845608028654f));
  const float du = fmaf(0.10703222440890037f, z2, 0.7978845608028654f);
  return 0.5f * (1.0f + th) + 0.5f * z * (1.0f - th * th) * du;
}

constexpr int G_THREADS = 256, G_NST = 3, G_NT = 128;             // G_NT: columns of a CTA's tile
constexpr int G_A = 128 * KC, G_STAGE = (128 + G_NT) * KC;        // elements of a stage (A, then B)

// 16 bytes global -> shared, or zeros
__device__ __forceinline__ void copy16(__nv_bfloat16 *dst, const __nv_bfloat16 *src, bool in)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}

// Rows r0 .. r0 + nrows - 1 (those below `rows`) and k0 .. k0 + KC - 1 (below
// K) of an operand with strides sr, sk into a stage's tile.
__device__ __forceinline__ void stage_tile(__nv_bfloat16 *tile, const __nv_bfloat16 *x, long sr, long sk, long r0, int nrows,
                                           long rows, int k0, int K, bool vec, int tid)
{
  if (vec) {
    for (int i = tid; i < nrows * (KC / 8); i += G_THREADS) {
      const int r = i / (KC / 8), q = i % (KC / 8), k = k0 + 8 * q;
      const bool in = r0 + r < rows && k < K;
      copy16(tile + tc::core_off(r, 8 * q, KC), in ? x + (r0 + r) * sr + k : x, in);
    }
  } else {
    for (int i = tid; i < nrows * KC; i += G_THREADS) {
      int r, kk;
      if (sr == 1) { r = i % nrows; kk = i / nrows; } else { r = i / KC; kk = i % KC; }
      __nv_bfloat16 v = __float2bfloat16(0.0f);
      if (r0 + r < rows && k0 + kk < K) v = x[(r0 + r) * sr + (long)(k0 + kk) * sk];
      tile[tc::core_off(r, kk, KC)] = v;
    }
  }
}

__device__ __forceinline__ uint32_t bf16x2_bits(float a, float b)
{
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ bool aligned_rows(const void *p, long ld, int elem)
{
  return (((uintptr_t)p | (uintptr_t)(ld * elem)) & 15) == 0;
}

// A warp's 32 rows x 16 values (row = lane, in v) to rows of x, and back,
// through its part of shared memory: four lanes take a row's 64 bytes (two a
// row's 32 for BF16), so that an access touches 8 (16) lines instead of 32.
// rows: how many of the 32 there are.  All lanes call.
constexpr int G_LINE = 20;                                        // words per row in the buffer (16 bytes apart)
__device__ __forceinline__ void store_rows(float *x, long ld, int rows, const float v[16], float *buf, int lane)
{
#pragma unroll
  for (int q = 0; q < 4; ++q)
    *reinterpret_cast<float4 *>(buf + lane * G_LINE + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 8 * i + (lane >> 2), q = lane & 3;
    if (r < rows) *reinterpret_cast<float4 *>(x + r * ld + 4 * q) = *reinterpret_cast<const float4 *>(buf + r * G_LINE + 4 * q);
  }
  __syncwarp();
}
__device__ __forceinline__ void load_rows(const float *x, long ld, int rows, float v[16], float *buf, int lane)
{
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 8 * i + (lane >> 2), q = lane & 3;
    *reinterpret_cast<float4 *>(buf + r * G_LINE + 4 * q) =
        r < rows ? __ldg(reinterpret_cast<const float4 *>(x + r * ld + 4 * q)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 t = *reinterpret_cast<const float4 *>(buf + lane * G_LINE + 4 * q);
    v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
  }
  __syncwarp();
}
__device__ __forceinline__ void store_rows(__nv_bfloat16 *x, long ld, int rows, const float h[16], float *buf, int lane)
{
#pragma unroll
  for (int q = 0; q < 2; ++q)
    *reinterpret_cast<uint4 *>(buf + lane * G_LINE + 4 * q) =
        make_uint4(bf16x2_bits(h[8 * q], h[8 * q + 1]), bf16x2_bits(h[8 * q + 2], h[8 * q + 3]),
                   bf16x2_bits(h[8 * q + 4], h[8 * q + 5]), bf16x2_bits(h[8 * q + 6], h[8 * q + 7]));
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = 16 * i + (lane >> 1), q = lane & 1;
    if (r < rows) *reinterpret_cast<uint4 *>(x + r * ld + 8 * q) = *reinterpret_cast<const uint4 *>(buf + r * G_LINE + 4 * q);
  }
  __syncwarp();
}

__global__ void __launch_bounds__(G_THREADS) tc_gemm_kernel(const TcGemmArgs a)
{
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __nv_bfloat16 *const ring = reinterpret_cast<__nv_bfloat16 *>(smem_raw);
  __shared__ __align__(8) uint64_t mbar[G_NST];
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.z * G_NT, nt = min(a.N - n0, G_NT), np = (nt + 15) & ~15;
  const uint32_t ncols = np <= 32 ? 32u : np <= 64 ? 64u : 128u;
  const long m0 = (long)blockIdx.x * 128;
  // K range of this split
  const int kpad = (a.K + 15) & ~15;
  const int ksplit = ((kpad / 16 + a.k_split - 1) / a.k_split) * 16;
  const int kbeg = blockIdx.y * ksplit;
  const int kend = min(kpad, kbeg + ksplit);
  const int nch = kend > kbeg ? (kend - kbeg + KC - 1) / KC : 0;
  if (tid == 0) {
    for (int i = 0; i < G_NST; ++i) tc::mbar_init(&mbar[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc(&tmem_base, ncols);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_base;
  const uint32_t idesc = tc::idesc_bf16_f32(128, np);
  // (a padded operand holds zeros from K to the next multiple of 8)
  const bool k8 = a.padded || (a.K % 8) == 0;
  const bool a_vec = k8 && a.sak == 1 && aligned_rows(a.A, a.sam, 2);
  const bool b_vec = k8 && a.sbk == 1 && aligned_rows(a.B, a.sbn, 2);
  auto fill = [&](int ch) {
    __nv_bfloat16 *sA = ring + (ch % G_NST) * G_STAGE;
    // (nothing past this split's range is read: its chunk count ends there)
    const int k0 = kbeg + ch * KC, K = min(a.K, kend);
    stage_tile(sA, a.A, a.sam, a.sak, m0, 128, a.M, k0, K, a_vec, tid);
    stage_tile(sA + G_A, a.B, a.sbn, a.sbk, n0, np, a.N, k0, K, b_vec, tid);
  };
  for (int ch = 0; ch < G_NST - 1; ++ch) {
    if (ch < nch) fill(ch);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  bool ok = true;
  int issued = 0;
  for (int ch = 0; ch < nch; ++ch) {
    asm volatile("cp.async.wait_group %0;" ::"n"(G_NST - 2) : "memory");   // this thread's copies of chunk ch
    tc::fence_async_smem();
    ok = __syncthreads_and(ok) != 0;                   // block-uniform
    if (!ok) break;
    if (tid == 0) {
      tc::fence_after();
      const uint32_t sA = tc::smem_u32(ring + (ch % G_NST) * G_STAGE), sB = sA + G_A * 2;
      const int steps = min(KC, kend - kbeg - ch * KC) / 16;
      for (int ks = 0; ks < steps; ++ks)
        tc::mma_bf16(tmem, tc::desc(sA + ks * 256, 128u, (KC / 8) * 128u), tc::desc(sB + ks * 256, 128u, (KC / 8) * 128u),
                     idesc, ch > 0 || ks > 0);
      tc::commit(&mbar[ch % G_NST]);
    }
    issued = ch + 1;
    // refill the stage of chunk ch - 1 once its MMAs are done
    if (ch + G_NST - 1 < nch) {
      if (ch > 0) ok = tc::mbar_wait(&mbar[(ch - 1) % G_NST], (uint32_t)(((ch - 1) / G_NST) & 1), WAIT_ITERS);
      if (ok) fill(ch + G_NST - 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // every MMA of the tile is done when the last commit is
  if (ok && issued > 0)
    ok = tc::mbar_wait(&mbar[(issued - 1) % G_NST], (uint32_t)(((issued - 1) / G_NST) & 1), WAIT_ITERS);
  ok = __syncthreads_and(ok) != 0;
  tc::fence_after();
  if (!ok) {
    if (tid == 0) atomicExch(a.err, 1);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // let MMAs in flight finish before freeing TMEM
    if (issued > 0) tc::mbar_wait(&mbar[(issued - 1) % G_NST], (uint32_t)(((issued - 1) / G_NST) & 1), WAIT_ITERS);
  }
  // ---- epilogue
  if (ok) {
    const int row = (warp & 3) * 32 + lane;
    const long m = m0 + row, mw = m - lane;            // the lane's row, the warp's first
    const bool in = m < a.M;
    const int rows = (int)min(32L, (long)a.M - mw);
    float *const buf = reinterpret_cast<float *>(smem_raw) + warp * 32 * G_LINE;   // (the ring: its MMAs are done)
    const bool c4 = aligned_rows(a.C, a.ldc, 4), z4 = aligned_rows(a.Zout ? a.Zout : a.Zin, a.ldz, 4);
    const bool h8 = aligned_rows(a.H, a.ldh, 2);
    for (int c0 = 16 * (warp >> 2); c0 < np; c0 += 32) {
      const int gc = n0 + c0;                          // the column of C
      float v[16];
      if (issued) tc::tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
      else
        for (int j = 0; j < 16; ++j) v[j] = 0.0f;
      const bool full = c0 + 16 <= nt;
      float h[16];                                     // what H takes
      if (a.epi == EPI_DGELU) {
        float z[16];
        if (full && z4) {
          load_rows(a.Zin + mw * a.ldz + gc, a.ldz, rows, z, buf, lane);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) z[j] = (in && c0 + j < nt) ? a.Zin[m * a.ldz + gc + j] : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) h[j] = v[j] *= dgelu(z[j]);
      } else if (a.epi != EPI_STORE) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (c0 + j < nt) v[j] += a.bias[gc + j];
          h[j] = a.epi == EPI_BIAS_GELU ? gelu(v[j]) : 0.0f;
        }
      }
      // FP32 result: Z of the forward, C of the others
      float *const o = a.epi == EPI_BIAS_GELU ? a.Zout : a.C;
      if (o) {
        const long ld = a.epi == EPI_BIAS_GELU ? a.ldz : a.ldc;
        float *const d = o + (a.epi == EPI_STORE ? (long)blockIdx.y * a.M * a.ldc : 0L) + mw * ld + gc;
        if (full && (a.epi == EPI_BIAS_GELU ? z4 : (c4 && (a.epi != EPI_STORE || ((a.M * a.ldc) & 3) == 0)))) {
          store_rows(d, ld, rows, v, buf, lane);
        } else if (in) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c0 + j < nt) d[lane * ld + j] = v[j];
        }
      }
      if (a.epi != EPI_BIAS_GELU && a.epi != EPI_DGELU) continue;
      __nv_bfloat16 *const d = a.H + mw * a.ldh + gc;
      if (full && h8) {
        store_rows(d, a.ldh, rows, h, buf, lane);
      } else if (in) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (c0 + j < nt) d[lane * a.ldh + j] = __float2bfloat16(h[j]);
      }
      if (a.HT) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (c0 + j < nt) a.HT[(long)(gc + j) * a.ldht + m] = __float2bfloat16(in ? h[j] : 0.0f);
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, ncols);
}

// ---------------------------------------------------------------------------
// Fused inference of the surrogate's MLP shape (16 -> 256 -> 256 -> 256 ->
// n_out <= 16, GELU): one persistent CTA per SM walks 128-row tiles, two of
// them in flight (slots 0 and 1).  Each slot has a 128 x 256 FP32 accumulator
// in TMEM (all 512 columns together) and a BF16 activation tile in shared
// memory (64 KB, K-major core matrices); W1 and the output layer stay
// resident in shared memory, and W2 / W3 stream from L2 in 16 KB K-chunks
// (pre-packed in the core-matrix layout) through a four-stage ring of bulk
// asynchronous copies.  The warps have roles:
//   0-15   bias + GELU of a hidden layer's accumulator into the activation
//          tile (warp w: rows 32 (w % 4) .. + 31, columns 64 (w / 4) .. + 63)
//   16-19  the input rows -> BF16, and the output rows
//   20     one thread issues the tcgen05.mma: layer by layer, slot 0 then 1
//   21     one thread issues the weight copies
// so that the MMAs of one slot run while the other slot's GELU does.
// Bound: the GELU warps (32,768 hardware tanh per layer and tile at 16 per
// clock and the FP32 operations around them, which take two values per
// instruction) and their reads of TMEM.  2 M rows take 0.745 ms (775
// TFLOP/s); 0.844 ms with one value per instruction; 1.21 ms with one tile in
// flight and all warps in step, MMAs and GELU largely in turn.
constexpr int FZ_NST = 4;                               // weight ring stages
constexpr int FZ_KC = 32;                               // K of a weight chunk
constexpr int FZ_GELU_WARPS = 16, FZ_IO_WARP = 16, FZ_MMA_WARP = 20, FZ_COPY_WARP = 21, FZ_THREADS = 32 * 22;
constexpr uint32_t FZ_CHUNK_BYTES = 256 * FZ_KC * 2;
constexpr int FZ_CHUNKS = 256 / FZ_KC;                  // per hidden layer
constexpr int FZ_OFF_H = 0, FZ_OFF_STAGE = 2 * 65536, FZ_OFF_W1 = FZ_OFF_STAGE + FZ_NST * FZ_CHUNK_BYTES;
constexpr int FZ_OFF_W4 = FZ_OFF_W1 + 8192, FZ_OFF_X = FZ_OFF_W4 + 8192, FZ_OFF_B = FZ_OFF_X + 2 * 4096;
constexpr int FZ_SMEM = FZ_OFF_B + (3 * 256 + 16) * 4;

// Two FP32 operations per instruction (sm_100 and later), each rounded as the
// scalar one.
__device__ __forceinline__ uint64_t f32x2(float a, float b)
{
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b)
{
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b)
{
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c)
{
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// gelu() of the two values r + b, packed to BF16: the same operations in the
// same order, two at a time.
__device__ __forceinline__ uint32_t fz_gelu2(uint32_t r0, uint32_t r1, uint64_t b)
{
  const uint64_t z = add_f32x2(f32x2(__uint_as_float(r0), __uint_as_float(r1)), b);
  const uint64_t k1 = f32x2(0.035677408136300125f, 0.035677408136300125f), k0 = f32x2(0.7978845608028654f, 0.7978845608028654f);
  const uint64_t u = mul_f32x2(z, fma_f32x2(k1, mul_f32x2(z, z), k0)), h = mul_f32x2(f32x2(0.5f, 0.5f), z);
  float ux, uy, gx, gy;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(ux), "=f"(uy) : "l"(u));
  const uint64_t g = fma_f32x2(h, f32x2(tanh_hw(ux), tanh_hw(uy)), h);
  asm("mov.b64 {%0, %1}, %2;" : "=f"(gx), "=f"(gy) : "l"(g));
  return bf16x2_bits(gx, gy);
}

// Bias + GELU of 32 accumulator columns (from cb0) of one row into the
// activation tile; the biases are read four at a time (the same address for
// the whole warp).
__device__ __forceinline__ void fz_gelu32(const uint32_t r[32], const float *bias, int cb0, int row, __nv_bfloat16 *sH)
{
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int cb = cb0 + 8 * g;
    const ulonglong2 b0 = *reinterpret_cast<const ulonglong2 *>(bias + cb);
    const ulonglong2 b1 = *reinterpret_cast<const ulonglong2 *>(bias + cb + 4);
    const uint32_t *q = r + 8 * g;
    *reinterpret_cast<uint4 *>(sH + tc::core_off(row, cb, 256)) =
        make_uint4(fz_gelu2(q[0], q[1], b0.x), fz_gelu2(q[2], q[3], b0.y), fz_gelu2(q[4], q[5], b1.x),
                   fz_gelu2(q[6], q[7], b1.y));
  }
}

__global__ void __launch_bounds__(FZ_THREADS, 1) mlp_fused_kernel(const MlpFusedArgs a)
{
  extern __shared__ __align__(1024) unsigned char smem[];
  float *sB = reinterpret_cast<float *>(smem + FZ_OFF_B);
  // acc: a hidden layer's accumulator is ready; out: the output layer's; in:
  // the input tile is written (and the slot's last output read); act: the
  // activation tile is written (and the accumulator read)
  __shared__ __align__(8) uint64_t bar_acc[2], bar_out[2], bar_in[2], bar_act[2], bar_full[FZ_NST], bar_free[FZ_NST],
      bar_end;
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long ntiles = (a.n + 127) / 128;
  const long my_tiles = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  // resident operands: W1 (256 x 16), output layer (16 x 256), biases
  for (int i = tid; i < 4096 / 8; i += FZ_THREADS) {
    reinterpret_cast<uint4 *>(smem + FZ_OFF_W1)[i] = __ldg(reinterpret_cast<const uint4 *>(a.w1) + i);
    reinterpret_cast<uint4 *>(smem + FZ_OFF_W4)[i] = __ldg(reinterpret_cast<const uint4 *>(a.w4) + i);
  }
  for (int i = tid; i < 256; i += FZ_THREADS) {
    sB[i] = a.b1[i];
    sB[256 + i] = a.b2[i];
    sB[512 + i] = a.b3[i];
  }
  if (tid < 16) sB[768 + tid] = tid < a.n_out ? a.b4[tid] : 0.0f;
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(&bar_acc[s], 1);
      tc::mbar_init(&bar_out[s], 1);
      tc::mbar_init(&bar_in[s], 4);
      tc::mbar_init(&bar_act[s], FZ_GELU_WARPS);
    }
    for (int s = 0; s < FZ_NST; ++s) {
      tc::mbar_init(&bar_full[s], 1);
      tc::mbar_init(&bar_free[s], 1);
    }
    tc::mbar_init(&bar_end, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc(&tmem_base, 512);
  tc::fence_async_smem();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_base;
  bool ok = true;
  // this warp's writes to shared memory and reads of TMEM are done
  auto warp_arrive = [&](uint64_t *bar) {
    tc::fence_async_smem();
    tc::fence_before();
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(bar);
  };
  if (warp < FZ_GELU_WARPS) {
    const int row = 32 * (warp & 3) + lane, c0 = 64 * (warp >> 2);
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    uint32_t phase[2] = {0u, 0u};
    for (long t0 = 0; t0 < my_tiles && ok; t0 += 2)
      for (int layer = 0; layer < 3 && ok; ++layer)
        for (int s = 0; s < 2 && t0 + s < my_tiles; ++s) {
          ok = tc::mbar_wait(&bar_acc[s], phase[s], WAIT_ITERS);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          phase[s] ^= 1u;
          tc::fence_after();
          const uint32_t acc = tmem + 256u * s + lanes + (uint32_t)c0;
          __nv_bfloat16 *sH = reinterpret_cast<__nv_bfloat16 *>(smem + FZ_OFF_H + 65536 * s);
          uint32_t r0[32], r1[32];
          tc::tmem_ld32_nowait(acc, r0);
          tc::tmem_wait_ld();
          tc::tmem_ld32_nowait(acc + 32u, r1);       // in flight during the first half
          fz_gelu32(r0, sB + 256 * layer, c0, row, sH);
          tc::tmem_wait_ld();
          fz_gelu32(r1, sB + 256 * layer, c0 + 32, row, sH);
          warp_arrive(&bar_act[s]);
        }
  } else if (warp < FZ_MMA_WARP) {
    // ---- input and output rows (thread = row of the tile)
    const int row = 32 * (warp & 3) + lane;
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    float4 x[4];
    auto load = [&](long t) {
      const long rw = ((long)blockIdx.x + t * gridDim.x) * 128 + row;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        x[q] = rw < a.n ? __ldg(reinterpret_cast<const float4 *>(a.x + rw * 16) + q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    auto put = [&](int s) {
      __nv_bfloat16 *sX = reinterpret_cast<__nv_bfloat16 *>(smem + FZ_OFF_X + 4096 * s);
#pragma unroll
      for (int q = 0; q < 2; ++q)
        *reinterpret_cast<uint4 *>(sX + tc::core_off(row, 8 * q, 16)) =
            make_uint4(bf16x2_bits(x[2 * q].x, x[2 * q].y), bf16x2_bits(x[2 * q].z, x[2 * q].w),
                       bf16x2_bits(x[2 * q + 1].x, x[2 * q + 1].y), bf16x2_bits(x[2 * q + 1].z, x[2 * q + 1].w));
      warp_arrive(&bar_in[s]);
    };
    for (long t = 0; t < 2 && t < my_tiles; ++t) {
      load(t);
      put((int)t);
    }
    for (long t = 0; t < my_tiles && ok; ++t) {
      const int s = (int)(t & 1);
      if (t + 2 < my_tiles) load(t + 2);               // in flight while the tile is computed
      ok = tc::mbar_wait(&bar_out[s], (uint32_t)((t >> 1) & 1), WAIT_ITERS);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      tc::fence_after();
      float v[16];
      tc::tmem_ld16(tmem + 256u * s + lanes, v);
      const long rw = ((long)blockIdx.x + t * gridDim.x) * 128 + row;
      if (rw < a.n) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (j < a.n_out) a.y[rw * a.n_out + j] = v[j] + sB[768 + j];
      }
      if (t + 2 < my_tiles) put(s);
    }
  } else if (warp == FZ_MMA_WARP) {
    if (lane == 0) {
      const uint32_t id256 = tc::idesc_bf16_f32(128, 256), id16 = tc::idesc_bf16_f32(128, 16);
      const uint32_t aW1 = tc::smem_u32(smem + FZ_OFF_W1), aW4 = tc::smem_u32(smem + FZ_OFF_W4);
      uint32_t ph_act[2] = {0u, 0u};
      long g = 0;                                      // weight chunks consumed
      for (long t0 = 0; t0 < my_tiles && ok; t0 += 2)
        for (int layer = 0; layer < 4 && ok; ++layer)
          for (int s = 0; s < 2 && t0 + s < my_tiles && ok; ++s) {
            const uint32_t acc = tmem + 256u * s, aH = tc::smem_u32(smem + FZ_OFF_H + 65536 * s);
            if (layer == 0) {
              ok = tc::mbar_wait(&bar_in[s], (uint32_t)((t0 >> 1) & 1), WAIT_ITERS);
            } else {
              ok = tc::mbar_wait(&bar_act[s], ph_act[s], WAIT_ITERS);
              ph_act[s] ^= 1u;
            }
            if (!ok) break;
            tc::fence_after();
            if (layer == 0) {
              tc::mma_bf16(acc, tc::desc(tc::smem_u32(smem + FZ_OFF_X + 4096 * s), 128u, 256u), tc::desc(aW1, 128u, 256u),
                           id256, false);
            } else if (layer < 3) {
              for (int c = 0; c < FZ_CHUNKS; ++c, ++g) {
                const int st = (int)(g % FZ_NST);
                if (!(ok = tc::mbar_wait(&bar_full[st], (uint32_t)((g / FZ_NST) & 1), WAIT_ITERS))) break;
                tc::fence_after();
                const uint32_t aS = tc::smem_u32(smem + FZ_OFF_STAGE + st * FZ_CHUNK_BYTES);
#pragma unroll
                for (int j = 0; j < FZ_KC / 16; ++j)
                  tc::mma_bf16(acc, tc::desc(aH + (uint32_t)(c * (FZ_KC / 8) + 2 * j) * 128u, 128u, 4096u),
                               tc::desc(aS + (uint32_t)(2 * j) * 128u, 128u, (FZ_KC / 8) * 128u), id256, c > 0 || j > 0);
                tc::commit(&bar_free[st]);
              }
              if (!ok) break;
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j)
                tc::mma_bf16(acc, tc::desc(aH + (uint32_t)(2 * j) * 128u, 128u, 4096u),
                             tc::desc(aW4 + (uint32_t)(2 * j) * 128u, 128u, 4096u), id16, j > 0);
            }
            tc::commit(layer < 3 ? &bar_acc[s] : &bar_out[s]);
          }
      // every MMA issued is done before the shared memory and TMEM are released
      tc::commit(&bar_end);
      if (!tc::mbar_wait(&bar_end, 0u, WAIT_ITERS)) ok = false;
    }
  } else if (lane == 0) {
    // ---- weight chunks in the order of the MMAs: per pair of tiles W2 for
    // slot 0, for slot 1, then W3 likewise
    long g = 0;
    auto copy = [&](const __nv_bfloat16 *w, int c) -> bool {
      const int st = (int)(g % FZ_NST);
      if (g >= FZ_NST && !tc::mbar_wait(&bar_free[st], (uint32_t)((g / FZ_NST - 1) & 1), WAIT_ITERS)) return false;
      tc::mbar_expect_tx(&bar_full[st], FZ_CHUNK_BYTES);
      tc::bulk_g2s(smem + FZ_OFF_STAGE + st * FZ_CHUNK_BYTES, w + (long)c * (256 * FZ_KC), FZ_CHUNK_BYTES, &bar_full[st]);
      ++g;
      return true;
    };
    for (long t0 = 0; t0 < my_tiles && ok; t0 += 2)
      for (int layer = 0; layer < 2 && ok; ++layer)
        for (int s = 0; s < 2 && t0 + s < my_tiles && ok; ++s)
          for (int c = 0; c < FZ_CHUNKS && ok; ++c) ok = copy(layer == 0 ? a.w2 : a.w3, c);
    // the copies in flight land before the shared memory is released
    for (long i = g > FZ_NST ? g - FZ_NST : 0; i < g; ++i)
      if (!tc::mbar_wait(&bar_full[i % FZ_NST], (uint32_t)((i / FZ_NST) & 1), WAIT_ITERS)) ok = false;
  }
  if (!ok) failed = 1;
  tc::fence_before();
  __syncthreads();
  if (tid == 0 && failed) atomicExch(a.err, 1);
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// FP32 master weights -> the fused kernel's BF16 layouts: W1 [256][16] and
// the output layer [16][256] (rows >= n_out zero) as K-major core-matrix
// tiles, W2 / W3 [256][256] as K-chunks of 256 x FZ_KC each.
__global__ void mlp_pack_kernel(const float *__restrict__ p, long w1, long w2, long w3, long w4, int n_out,
                                __nv_bfloat16 *__restrict__ out)
{
  const long total = 4096 + 65536 + 65536 + 4096;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    float v;
    long dst;
    if (i < 4096) {                                   // W1: n = i / 16, k = i % 16
      const int n = (int)(i / 16), k = (int)(i % 16);
      v = p[w1 + i];
      dst = tc::core_off(n, k, 16);
    } else if (i < 4096 + 131072) {                   // W2 / W3: n, k in 256 x 256
      const long j = i - 4096;
      const int l = (int)(j / 65536);
      const int n = (int)((j % 65536) / 256), k = (int)(j % 256);
      v = p[(l == 0 ? w2 : w3) + (long)n * 256 + k];
      dst = 4096 + (long)l * 65536 + (long)(k / FZ_KC) * (256 * FZ_KC) + tc::core_off(n, k % FZ_KC, FZ_KC);
    } else {                                          // output layer: n < 16, k < 256
      const long j = i - 4096 - 131072;
      const int n = (int)(j / 256), k = (int)(j % 256);
      v = n < n_out ? p[w4 + (long)n * 256 + k] : 0.0f;
      dst = 4096 + 131072 + tc::core_off(n, k, 256);
    }
    out[dst] = __float2bfloat16(v);
  }
}

// Sum of the split-K partials in a fixed order: out[i] = sum_s part[s * n + i].
__global__ void sum_splits_kernel(const float *__restrict__ part, float *__restrict__ out, long n, int splits)
{
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    float s = 0.0f;
#pragma unroll 8
    for (int j = 0; j < splits; ++j) s += part[(long)j * n + i];
    out[i] = s;
  }
}

// Column sums (bias gradients) of a range of rows per block, in a fixed order:
// part[b][n] = sum of x[m * ld + n] over the block's rows, eight rows side by
// side for 32 columns; sum_splits_kernel adds the blocks.  (A thread per
// column over all rows took 0.93 ms for 16,384 x 256.)
__global__ void __launch_bounds__(256) col_sum_kernel(const float *__restrict__ x, float *__restrict__ part, int rows,
                                                      int cols, long ld, int rows_per)
{
  __shared__ float red[8][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, n = blockIdx.x * 32 + tx;
  const int r1 = min(rows, (int)(blockIdx.y + 1) * rows_per);
  float s = 0.0f;
  if (n < cols) {
#pragma unroll 4
    for (int m = blockIdx.y * rows_per + ty; m < r1; m += 8) s += x[(long)m * ld + n];
  }
  red[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && n < cols) {
#pragma unroll
    for (int j = 1; j < 8; ++j) s += red[j][tx];
    part[(long)blockIdx.y * cols + n] = s;
  }
}

// Loss of the surrogate head: per rate r, y[2r] is the logit of "the rate is
// nonzero" (binary cross-entropy against act), y[2r+1] the transformed rate
// (squared error against val where the rate is nonzero).  Writes dY
// ([rows][16], mean over the batch) in bf16 for the GEMMs (also transposed,
// [16][ldt]) and in f32 for the output-bias gradient, and accumulates the loss.
__global__ void surrogate_loss_kernel(const float *__restrict__ y, const float *__restrict__ tgt, int rows, int nrates,
                                      __nv_bfloat16 *__restrict__ dy, __nv_bfloat16 *__restrict__ dyt, long ldt,
                                      float *__restrict__ dyf, float *__restrict__ loss)
{
  __shared__ float red[128];
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  float l = 0.0f;
  if (m < rows) {
    const float inv = 1.0f / (float)rows;
    for (int r = 0; r < nrates; ++r) {
      const float logit = y[(long)m * 16 + 2 * r], pred = y[(long)m * 16 + 2 * r + 1];
      const float act = tgt[(long)m * 16 + 2 * r], val = tgt[(long)m * 16 + 2 * r + 1];
      const float p = 1.0f / (1.0f + expf(-logit));
      l += -(act * logf(fmaxf(p, 1e-12f)) + (1.0f - act) * logf(fmaxf(1.0f - p, 1e-12f)));
      const float e = act > 0.5f ? pred - val : 0.0f;
      l += e * e;
      const float g0 = (p - act) * inv, g1 = 2.0f * e * inv;
      dy[(long)m * 16 + 2 * r] = __float2bfloat16(g0);
      dy[(long)m * 16 + 2 * r + 1] = __float2bfloat16(g1);
      dyf[(long)m * 16 + 2 * r] = g0;
      dyf[(long)m * 16 + 2 * r + 1] = g1;
    }
    for (int j = 2 * nrates; j < 16; ++j) {
      dy[(long)m * 16 + j] = __float2bfloat16(0.0f);
      dyf[(long)m * 16 + j] = 0.0f;
    }
    for (int j = 0; j < 16; ++j) dyt[j * ldt + m] = dy[(long)m * 16 + j];
  } else {
    for (int j = 0; j < 16; ++j) dyt[j * ldt + m] = __float2bfloat16(0.0f);   // zeros to the block's last row
  }
  red[threadIdx.x] = l;
  __syncthreads();
  for (int s = 64; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, red[0] / (float)rows);
}

// Adam on FP32 master weights; refreshes the BF16 copies used by the GEMMs
// (w16 [out][din], w16t [din][ldt]).
__global__ void adam_kernel(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m1,
                            float *__restrict__ m2, __nv_bfloat16 *__restrict__ w16, __nv_bfloat16 *__restrict__ w16t,
                            int din, long ldt, long n, float lr, float b1, float b2, float eps, float c1, float c2)
{
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float a = b1 * m1[i] + (1.0f - b1) * gi, b = b2 * m2[i] + (1.0f - b2) * gi * gi;
    m1[i] = a;
    m2[i] = b;
    const float wi = w[i] - lr * (a * c1) / (sqrtf(b * c2) + eps);
    w[i] = wi;
    if (w16) w16[i] = __float2bfloat16(wi);
    if (w16t) w16t[(i % din) * ldt + i / din] = __float2bfloat16(wi);
  }
}

__global__ void to_bf16_kernel(const float *__restrict__ x, __nv_bfloat16 *__restrict__ y, long n)
{
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16(x[i]);
}

// x [rows][cols] (f32) -> y (BF16, [rows][cols], or NULL) and yt (BF16,
// [cols][ldt]), the transpose with zeros for rows .. pad_rows - 1.
__global__ void to_bf16_t_kernel(const float *__restrict__ x, __nv_bfloat16 *__restrict__ y, __nv_bfloat16 *__restrict__ yt,
                                 long rows, int cols, long pad_rows, long ldt)
{
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < pad_rows * cols; i += (long)gridDim.x * blockDim.x) {
    const long r = i / cols;
    const int k = (int)(i - r * cols);
    const __nv_bfloat16 v = __float2bfloat16(r < rows ? x[i] : 0.0f);
    if (y && r < rows) y[i] = v;
    yt[k * ldt + r] = v;
  }
}

}  // namespace

// The stage ring takes 96 KB of an SM's 227 KB, so at most two CTAs are resident
// per SM, with at most G_NT of the 512 TMEM columns each: no tcgen05.alloc has to
// wait for another CTA of this kernel.
constexpr int SM_SMEM = 227 * 1024, TMEM_COLS = 512;
static_assert(SM_SMEM / (G_NST * G_STAGE * 2) * G_NT <= TMEM_COLS, "TMEM columns of the CTAs of an SM");
static_assert(G_NST * G_STAGE * 2 >= G_THREADS * G_LINE * 4, "the epilogue's buffers fit in the ring");
size_t tc_gemm_smem_bytes() { return (size_t)G_NST * G_STAGE * sizeof(__nv_bfloat16); }

cudaError_t launch_tc_gemm(const TcGemmArgs &a, cudaStream_t s)
{
  if (a.N < 1 || a.N > 256 || a.M < 1 || a.K < 1 || a.k_split < 1) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(tc_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)tc_gemm_smem_bytes());
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)((a.M + 127) / 128), (unsigned)a.k_split, (unsigned)((a.N + G_NT - 1) / G_NT));
  tc_gemm_kernel<<<grid, G_THREADS, tc_gemm_smem_bytes(), s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_mlp_pack(const float *p, long w1, long w2, long w3, long w4, int n_out, __nv_bfloat16 *out,
                            cudaStream_t s)
{
  mlp_pack_kernel<<<136, 1024, 0, s>>>(p, w1, w2, w3, w4, n_out, out);
  return cudaGetLastError();
}

cudaError_t launch_mlp_fused(const MlpFusedArgs &a, int num_sms, cudaStream_t s)
{
  cudaError_t e = cudaFuncSetAttribute(mlp_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FZ_SMEM);
  if (e != cudaSuccess) return e;
  const long tiles = (a.n + 127) / 128;
  long blocks = num_sms;
  if (blocks > tiles) blocks = tiles;
  if (blocks < 1) return cudaSuccess;
  mlp_fused_kernel<<<(unsigned)blocks, FZ_THREADS, FZ_SMEM, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_sum_splits(const float *part, float *out, long n, int splits, cudaStream_t s)
{
  long blocks = (n + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  sum_splits_kernel<<<(unsigned)blocks, 256, 0, s>>>(part, out, n, splits);
  return cudaGetLastError();
}

cudaError_t launch_col_sum(const float *x, float *part, float *out, int rows, int cols, long ld, cudaStream_t s)
{
  const int rows_per = (rows + COL_SUM_BLOCKS - 1) / COL_SUM_BLOCKS, blocks = (rows + rows_per - 1) / rows_per;
  col_sum_kernel<<<dim3((unsigned)((cols + 31) / 32), (unsigned)blocks), 256, 0, s>>>(x, part, rows, cols, ld, rows_per);
  cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? e : launch_sum_splits(part, out, cols, blocks, s);
}

cudaError_t launch_surrogate_loss(const float *y, const float *tgt, int rows, int nrates, __nv_bfloat16 *dy,
                                  __nv_bfloat16 *dyt, long ldt, float *dyf, float *loss, cudaStream_t s)
{
  surrogate_loss_kernel<<<(unsigned)((rows + 127) / 128), 128, 0, s>>>(y, tgt, rows, nrates, dy, dyt, ldt, dyf, loss);
  return cudaGetLastError();
}

cudaError_t launch_adam(float *w, const float *g, float *m1, float *m2, __nv_bfloat16 *w16, __nv_bfloat16 *w16t, int din,
                        long ldt, long n, float lr, float b1, float b2, float eps, int step, cudaStream_t s)
{
  const float c1 = 1.0f / (1.0f - powf(b1, (float)step)), c2 = 1.0f / (1.0f - powf(b2, (float)step));
  long blocks = (n + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  adam_kernel<<<(unsigned)blocks, 256, 0, s>>>(w, g, m1, m2, w16, w16t, din, ldt, n, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError();
}

cudaError_t launch_to_bf16_t(const float *x, __nv_bfloat16 *y, __nv_bfloat16 *yt, long rows, int cols, long pad_rows,
                             long ldt, cudaStream_t s)
{
  long blocks = (pad_rows * cols + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  to_bf16_t_kernel<<<(unsigned)blocks, 256, 0, s>>>(x, y, yt, rows, cols, pad_rows, ldt);
  return cudaGetLastError();
}

cudaError_t launch_to_bf16(const float *x, __nv_bfloat16 *y, long n, cudaStream_t s)
{
  long blocks = (n + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  to_bf16_kernel<<<(unsigned)blocks, 256, 0, s>>>(x, y, n);
  return cudaGetLastError();
}
