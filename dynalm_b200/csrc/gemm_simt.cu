// y = x W^T (+ bias): the plain matrix product, fp32 accumulation on the CUDA cores.
//
// The 32-bit path's product for matrices with fewer than 512 features or numbers of k (larger ones: gemm_split.cu) and
// the fallback for shapes the tensor-core kernels refuse; no reduced-precision mode. x: [M, K] (row stride ldx), W: [N, K] row-major,
// y: [M, N] (row stride ldy), bias: fp32 [N] or null.
//
// Every output element is a sum in an order that K alone fixes, so its value does not depend on the number of rows in the
// call nor on where the row sits (the reference's matmul accumulates in fp32 too,
// dynacore/cpu/generic/kernels_generic.cpp:23-34): k is cut into SPANS spans of equal length (a multiple of 32); a span's
// sum is a running fused multiply-add in the order of k; four spans in a row are added up in their order to a quarter,
// the quarters in their order to the result. Both kernels below follow it, and either may deal spans (the few-row kernel)
// or quarters (the tiled kernel, over a thread-block cluster) to different threads without changing a bit.
//
// * gemm_rows_kernel, few rows of aligned float32 (decode steps): bound by the bytes of W. A block owns 16 features,
//   up to 16 rows and all of K, a half-warp one span of them; every warp streams its own two spans through a two-stage
//   cp.async ring (no block barrier before the end), the first stage requested before the wait on the kernel in front.
// * gemm_tile_kernel, everything else: bound by the multiply-add lanes, which outrun shared memory unless a number read is
//   used often: 128 x 128 outputs a block of 128 threads, 8 x 16 a thread (six 16-byte reads for 128 multiply-adds; with
//   8 x 8 a thread, four for 64, 2048 x 16384 x 2048 ran at 38.6 TFLOP/s), as packed pairs (fma.rn.f32x2, each half an fma of
//   its own); tiles of 16 k double-buffered in shared memory, the next tile's loads in registers meanwhile. Four blocks of a
//   cluster share a tile, a quarter of k each; the running quarter waits in shared memory, which leaves the registers to the
//   span, and the blocks add the four up there. (A block that walked all of k kept the quarters so far in y: 2,790 us for
//   2048 x 16384 x 2048 against 2,736, 1,223 against 1,039 for 700 rows, 160 against 46 for 17 rows x 2048 x 2048.)
//
// Measured on B200 (float32, us; before: one kernel of 64 x 64 tiles, 4 x 4 outputs a thread, k in one chain):
//   rows x features x k     2048 x 2048    16384 x 2048    2048 x 8192
//   1                       335 -> 11      363 -> 36       1,330 -> 24
//   16                      333 -> 15      363 -> 67       1,337 -> 37
//   64                      337 -> 41      363 -> 121      1,356 -> 142
//   700                     307 -> 162     1,788 -> 1,049  1,205 -> 577
//   2,048                   675 -> 394      4,919 -> 2,736  2,686 -> 1,449
#include "qkv_rope.cuh"

#include <cooperative_groups.h>

#include <type_traits>

namespace dl {

namespace cg = cooperative_groups;

constexpr int SPANS = 16, QUARTERS = 4;

__host__ __device__ inline int span_length(int K) { return ((K + SPANS - 1) / SPANS + 31) / 32 * 32; }

__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(bytes)
               : "memory");
}

// ---- few rows -----------------------------------------------------------------------------------------------

constexpr int RF = 16;                    // features of a block
constexpr int RK = 32;                    // k of a stage, per span
constexpr int RW = RK + 4;                // a feature's padded row: eight features' 16-byte reads fall into different banks
constexpr int RWARPS = SPANS / 2;         // two spans a warp

template <int R>
__host__ __device__ constexpr int rows_stage_floats() { return 2 * RF * RW + 2 * R * RK; }

// What becomes of the sums of up to 16 rows on their way out: the gated activation silu(gate) up of W = [gate; up] (a block holds eight
// gate and the eight matching up features), or the rotary encoding and the cache write of the q | k | v projection (qkv_rope.cuh;
// a block of a q or k head holds eight rotary pairs). Both as activation.cu and rope_cache.cu work them out, which were launches of
// their own (a step of a tiny model, 5 rows and 3 layers: 32 launches, now 26).
enum { ROWS_STORE = 0, ROWS_SWIGLU = 1, ROWS_ROPE = 2 };

template <int R, int OUT>
__global__ void __launch_bounds__(RWARPS * 32)
gemm_rows_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w, const float* __restrict__ bias,
                 float* __restrict__ y, int ldy, int M, int N, int K, float out_scale, const QkvRopeOf<float> rope) {
  extern __shared__ __align__(16) float rows_smem[];
  const int m_first = blockIdx.y * R;
  x += static_cast<size_t>(m_first) * ldx;
  y += static_cast<size_t>(m_first) * ldy;
  M -= m_first;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, f = lane & 15, half = lane >> 4;
  const int span = span_length(K);
  // the block's features: eight from n0 on, eight from n1 on
  int n0 = blockIdx.x * RF, n1 = n0 + RF / 2, head = 0;
  bool turned = false;
  if constexpr (OUT == ROWS_SWIGLU) n0 = blockIdx.x * (RF / 2), n1 = N / 2 + n0;
  if constexpr (OUT == ROWS_ROPE) {
    const int per_head = rope.head_dim / RF;
    head = blockIdx.x / per_head;                   // q heads, then k heads, then v heads
    turned = head < rope.n_heads + rope.n_kv_heads;
    if (turned) {
      n0 = head * rope.head_dim + blockIdx.x % per_head * (RF / 2);
      n1 = n0 + rope.head_dim / 2;
    }
  }
  float* ring = rows_smem + warp * 2 * rows_stage_floats<R>();
  const int steps = span / RK;

  // a stage: RK numbers of both spans' 16 features, then of the R rows; past K zeros
  auto load_w = [&](int s) {
    float* st = ring + (s & 1) * rows_stage_floats<R>();
#pragma unroll
    for (int i = 0; i < 2 * RF * RK / 4 / 32; ++i) {
      const int e = i * 32 + lane, c = e & 7, row = e >> 3;         // row: half * 16 + feature
      const int k = (2 * warp + (row >> 4)) * span + s * RK + c * 4;
      const int n = min((row & 8 ? n1 : n0) + (row & 7), N - 1);
      cp_async16_zfill(st + row * RW + c * 4, w + static_cast<size_t>(n) * K + (k < K ? k : 0), k < K ? 16 : 0);
    }
  };
  auto load_x = [&](int s) {
    float* st = ring + (s & 1) * rows_stage_floats<R>() + 2 * RF * RW;
    for (int e = lane; e < 2 * R * RK / 4; e += 32) {
      const int c = e & 7, row = e >> 3;                            // row: half * R + row of x
      const int h = row / R, m = row - h * R;
      const int k = (2 * warp + h) * span + s * RK + c * 4;
      const bool there = k < K && m < M;
      cp_async16_zfill(st + row * RK + c * 4, there ? x + static_cast<size_t>(m) * ldx + k : x, there ? 16 : 0);
    }
  };

  load_w(0);
  pdl_wait();
  load_x(0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  pdl_trigger();
  float acc[R];
#pragma unroll
  for (int m = 0; m < R; ++m) acc[m] = 0.0f;
  for (int s = 0; s < steps; ++s) {
    if (s + 1 < steps) {
      load_w(s + 1);
      load_x(s + 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const float* st = ring + (s & 1) * rows_stage_floats<R>();
    const float4* wr = reinterpret_cast<const float4*>(st + (half * RF + f) * RW);
    const float4* xr = reinterpret_cast<const float4*>(st + 2 * RF * RW + half * R * RK);
#pragma unroll
    for (int c = 0; c < RK / 4; ++c) {
      const float4 b = wr[c];
#pragma unroll
      for (int m = 0; m < R; ++m) {
        const float4 a = xr[m * (RK / 4) + c];
        acc[m] = fmaf(a.x, b.x, acc[m]);
        acc[m] = fmaf(a.y, b.y, acc[m]);
        acc[m] = fmaf(a.z, b.z, acc[m]);
        acc[m] = fmaf(a.w, b.w, acc[m]);
      }
    }
    __syncwarp();          // the stage may be overwritten
  }
  __syncthreads();         // the rings are not read any more: the spans' sums go there
#pragma unroll
  for (int m = 0; m < R; ++m) rows_smem[((2 * warp + half) * R + m) * RF + f] = acc[m];
  __syncthreads();
  const int t = threadIdx.x;
  auto sum_of = [&](int m, int i) {
    const float* s = rows_smem + m * RF + i;
    float total = 0.0f;
#pragma unroll
    for (int q = 0; q < QUARTERS; ++q) {
      float part = s[4 * q * R * RF];
#pragma unroll
      for (int j = 1; j < SPANS / QUARTERS; ++j) part += s[(4 * q + j) * R * RF];
      total = q == 0 ? part : total + part;
    }
    return total;
  };
  if constexpr (OUT == ROWS_STORE) {
    const int m = t >> 4, n = n0 + f;
    if (t >= RF * R || m >= M || n >= N) return;
    float total = sum_of(m, f);
    if (bias) total += bias[n];
    y[static_cast<size_t>(m) * ldy + n] = total * out_scale;
  } else {
    const int m = t >> 3, i = t & 7;
    if (t >= RF / 2 * R || m >= M) return;
    float a = sum_of(m, i), b = sum_of(m, i + RF / 2);
    if constexpr (OUT == ROWS_SWIGLU) {
      if (n0 + i < N / 2) y[static_cast<size_t>(m) * ldy + n0 + i] = a / (1.0f + expf(-a)) * b;
    } else {
      const int pos = rope.positions[m], hd = rope.head_dim, in_head = n0 + i - head * hd;
      if (turned) {
        const float theta = static_cast<float>(pos) * rope.pos_scale * rope.inv_freq[in_head];
        float s, c;
        sincosf(theta, &s, &c);
        const float ra = a * c - b * s, rb = a * s + b * c;
        a = ra, b = rb;
      }
      float* to;
      if (head < rope.n_heads) {
        to = y + static_cast<size_t>(m) * ldy + n0 + i;
      } else {
        const size_t slot = qkv_rope_slot(rope, m, pos);
        if (slot == QKV_NO_SLOT) return;
        const int kvh = head - rope.n_heads - (turned ? 0 : rope.n_kv_heads);
        to = (turned ? rope.k_cache : rope.v_cache) + (slot * rope.n_kv_heads + kvh) * hd + in_head;
      }
      to[0] = a;
      to[n1 - n0] = b;
    }
  }
}

// ---- any number of rows ------------------------------------------------------------------------------------------

constexpr int TK = 16;

// acc.{lo, hi} = fma(a, b.{lo, hi}, acc.{lo, hi}): two multiply-adds in one instruction, each rounded by itself
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}

constexpr int BN = 128;

// BM x 128 outputs, 8 x TN a thread (BM 128: TN 16; BM 64: TN 8), 128 threads; `wide`: four numbers of a row of x and of W may
// be loaded at once. A quarter of k for each of the CL blocks of a cluster: QUARTERS, or one where k has no more than a quarter (up
// to 128: 1,000 x 499 x 80 float32 took 20.3 us with three blocks of four that had nothing to do, 11.0 without).
template <typename TX, typename TO, int BM, int TN, int CL>
__global__ void __launch_bounds__(128, 2)
gemm_tile_kernel(const TX* __restrict__ x, int ldx, const TX* __restrict__ w, const float* __restrict__ bias,
                 TO* __restrict__ y, int ldy, int M, int N, int K, float out_scale, int wide) {
  constexpr int THREADS = 128, COLS = BN / TN, XS = BM + 4, WS = BN + 4;
  static_assert(BM / 8 * COLS == THREADS, "");
  constexpr int XV = BM * TK / 4 / THREADS, WV = BN * TK / 4 / THREADS;       // runs of four numbers a thread loads
  extern __shared__ __align__(16) float tile_smem[];
  float* xs = tile_smem;                              // [2][TK][XS]
  float* ws = xs + 2 * TK * XS;                       // [2][TK][WS]
  float* quarter = ws + 2 * TK * WS;                  // [8 TN][THREADS]: the running quarter
  const int tid = threadIdx.x;
  const int part = blockIdx.x % CL;
  const int m0 = blockIdx.y * BM, n0 = (blockIdx.x / CL) * BN;
  const int tm = tid / COLS * 4, tn = tid % COLS * 4;    // rows tm.. and BM/2 + tm.., columns tn + 4 COLS j ..
  const int span = span_length(K), quarter_k = span * (SPANS / QUARTERS);
  const int k_begin = part * quarter_k, k_end = min(K, k_begin + quarter_k);

  // the next tile's numbers on their way: float32, or bfloat16 as they lie, which are converted only when they are kept (with the
  // conversion beside the load every run waited for its own: 40 x 499 x 80 15.0 us, now 11.3)
  float xv[XV][4], wv[WV][4];
  ushort4 xh[XV], wh[WV];
  auto fetch = [&](int k0) {
    if constexpr (sizeof(TX) == 2) {
      auto run = [&](ushort4& v, const TX* base, int ld, int row, int rows, int e, bool at_once) {
        const int k = k0 + e % (TK / 4) * 4, there = row < rows ? K - k : 0;
        const TX* p = base + static_cast<size_t>(row) * ld + k;
        v = make_ushort4(0, 0, 0, 0);
        if (at_once) {                                  // (K is a multiple of four)
          if (there > 0) v = *reinterpret_cast<const ushort4*>(p);
        } else {
          const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
          if (there > 0) v.x = q[0];
          if (there > 1) v.y = q[1];
          if (there > 2) v.z = q[2];
          if (there > 3) v.w = q[3];
        }
      };
      auto all = [&](auto at_once) {
        constexpr bool O = decltype(at_once)::value;
#pragma unroll
        for (int i = 0; i < XV; ++i) run(xh[i], x, ldx, m0 + (i * THREADS + tid) / (TK / 4), M, i * THREADS + tid, O);
#pragma unroll
        for (int i = 0; i < WV; ++i) run(wh[i], w, K, n0 + (i * THREADS + tid) / (TK / 4), N, i * THREADS + tid, O);
      };
      if (wide) all(std::true_type());
      else all(std::false_type());
    } else {
#pragma unroll
      for (int i = 0; i < XV; ++i) {
        const int e = i * THREADS + tid, k = k0 + (e % (TK / 4)) * 4, m = m0 + e / (TK / 4);
        const TX* p = x + static_cast<size_t>(m) * ldx + k;
        if (wide && m < M && k + 3 < K) {
          const float4 v = *reinterpret_cast<const float4*>(p);
          xv[i][0] = v.x, xv[i][1] = v.y, xv[i][2] = v.z, xv[i][3] = v.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) xv[i][j] = (m < M && k + j < K) ? to_float(p[j]) : 0.0f;
        }
      }
#pragma unroll
      for (int i = 0; i < WV; ++i) {
        const int e = i * THREADS + tid, k = k0 + (e % (TK / 4)) * 4, n = n0 + e / (TK / 4);
        const TX* p = w + static_cast<size_t>(n) * K + k;
        if (wide && n < N && k + 3 < K) {
          const float4 v = *reinterpret_cast<const float4*>(p);
          wv[i][0] = v.x, wv[i][1] = v.y, wv[i][2] = v.z, wv[i][3] = v.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) wv[i][j] = (n < N && k + j < K) ? to_float(p[j]) : 0.0f;
        }
      }
    }
  };
  auto keep = [&](int buf) {
    if constexpr (sizeof(TX) == 2) {
      auto numbers = [](float (&v)[4], const ushort4& h) {
        v[0] = __bfloat162float(__ushort_as_bfloat16(h.x)), v[1] = __bfloat162float(__ushort_as_bfloat16(h.y));
        v[2] = __bfloat162float(__ushort_as_bfloat16(h.z)), v[3] = __bfloat162float(__ushort_as_bfloat16(h.w));
      };
#pragma unroll
      for (int i = 0; i < XV; ++i) numbers(xv[i], xh[i]);
#pragma unroll
      for (int i = 0; i < WV; ++i) numbers(wv[i], wh[i]);
    }
#pragma unroll
    for (int i = 0; i < XV; ++i) {
      const int e = i * THREADS + tid, k = (e % (TK / 4)) * 4, r = e / (TK / 4);
#pragma unroll
      for (int j = 0; j < 4; ++j) xs[(buf * TK + k + j) * XS + r] = xv[i][j];
    }
#pragma unroll
    for (int i = 0; i < WV; ++i) {
      const int e = i * THREADS + tid, k = (e % (TK / 4)) * 4, r = e / (TK / 4);
#pragma unroll
      for (int j = 0; j < 4; ++j) ws[(buf * TK + k + j) * WS + r] = wv[i][j];
    }
  };

  unsigned long long acc[8][TN / 2];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
  int buf = 0;
  if (k_begin < k_end) {
    fetch(k_begin);
    keep(0);
  }
  __syncthreads();
  for (int k0 = k_begin; k0 < k_end; k0 += TK) {
    const bool more = k0 + TK < k_end;
    if (more) fetch(k0 + TK);
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      const float* xr = xs + (buf * TK + k) * XS + tm;
      const float* wr = ws + (buf * TK + k) * WS + tn;
      const float4 a0 = *reinterpret_cast<const float4*>(xr), a1 = *reinterpret_cast<const float4*>(xr + BM / 2);
      unsigned long long b[TN / 2];
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(wr + 4 * COLS * j);
        b[2 * j] = v.x, b[2 * j + 1] = v.y;
      }
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned long long aa = twice(a[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, b[j]);
      }
    }
    if (more) keep(buf ^ 1);
    if ((k0 + TK) % span == 0 || !more) {              // a span ends (spans are multiples of TK): into the running quarter
      const bool opens = k0 - k_begin < span;
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int at = (i * TN + 2 * j + h) * THREADS + tid;
            const float v = __uint_as_float(static_cast<unsigned>(h ? acc[i][j] >> 32 : acc[i][j]));
            quarter[at] = opens ? v : quarter[at] + v;
          }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
    }
    __syncthreads();
    buf ^= 1;
  }

  // every block of the cluster adds up the quarters of a share of the outputs
  cg::cluster_group cluster = cg::this_cluster();
  if constexpr (CL > 1) cluster.sync();
  const int have = min(CL, (K + quarter_k - 1) / quarter_k);      // quarters that hold any k
  const float* theirs[CL];
#pragma unroll
  for (int q = 0; q < CL; ++q) theirs[q] = CL > 1 ? cluster.map_shared_rank(quarter, q) : quarter;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i % CL != part) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int at = (i * TN + j) * THREADS + tid;
      float v = theirs[0][at];
#pragma unroll
      for (int q = 1; q < CL; ++q)
        if (q < have) v += theirs[q][at];
      const int m = m0 + (i < 4 ? tm + i : BM / 2 + tm + i - 4), n = n0 + tn + j / 4 * 4 * COLS + j % 4;
      if (m < M && n < N) {
        if (bias) v += bias[n];
        y[static_cast<size_t>(m) * ldy + n] = from_float<TO>(v * out_scale);
      }
    }
  }
  if constexpr (CL > 1) cluster.sync();                 // nobody leaves while its quarter is being read
}

template <typename TX, typename TO, int BM, int TN, int CL>
int launch_tiles(const void* x, int ldx, const void* w, const float* bias, void* y, int ldy, int M, int N, int K,
                 float out_scale, int wide, cudaStream_t stream) {
  constexpr int THREADS = 128;
  constexpr int SMEM = (2 * TK * (BM + 4 + BN + 4) + 8 * TN * THREADS) * 4;
  auto kernel = gemm_tile_kernel<TX, TO, BM, TN, CL>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + BN - 1) / BN * CL, (M + BM - 1) / BM, 1);
  cfg.blockDim = THREADS;
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CL > 1 ? 1 : 0;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, static_cast<const TX*>(x), ldx, static_cast<const TX*>(w), bias,
                                             static_cast<TO*>(y), ldy, M, N, K, out_scale, wide));
}

template <int R, int OUT = ROWS_STORE>
int launch_rows(const float* x, int ldx, const float* w, const float* bias, float* y, int ldy, int M, int N, int K,
                float out_scale, cudaStream_t stream, const QkvRopeOf<float>& rope = {}) {
  constexpr int SMEM = RWARPS * 2 * rows_stage_floats<R>() * 4;
  auto kernel = gemm_rows_kernel<R, OUT>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int blocks = OUT == ROWS_SWIGLU ? (N / 2 + RF / 2 - 1) / (RF / 2) : (N + RF - 1) / RF;
  return launch_streaming(kernel, dim3(blocks, (M + R - 1) / R), dim3(RWARPS * 32), SMEM, stream, x, ldx, w, bias, y, ldy, M, N, K,
                          out_scale, rope);
}

}  // namespace dl

// in_dtype (x and W) / out_dtype: 0 = float32, 1 = bfloat16.
DL_EXPORT int dl_gemm_simt(int in_dtype, int out_dtype, const void* x, int ldx, const void* w, const float* bias,
                           void* y, int ldy, int M, int N, int K, float out_scale, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return DL_ERR_UNSUPPORTED;
  if ((M + 63) / 64 > 65535) return DL_ERR_UNSUPPORTED;
  // four numbers of a row at once: 16 bytes of float32, 8 of bfloat16
  const bool aligned = K % 4 == 0 && ldx % 4 == 0 &&
                       ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & (in_dtype == 0 ? 15 : 7)) == 0;
  // The few-row kernel up to 16 rows, and for narrow products of up to 64 rows in groups of 16 that share W in L2, up to about
  // four blocks an SM. Measured, groups / tiles, us: 64 x 2048 x 2048 41 / 45, 48 x 3072 x 2048 41 / 46, 64 x 3072 x 2048 57 /
  // 45, 32 x 2048 x 8192 66 / 143, 32 x 16384 x 2048 125 / 119; 16 x 128256 x 2048 461 / 735.
  const long long row_blocks = static_cast<long long>((N + dl::RF - 1) / dl::RF) * ((M + 15) / 16);
  if (aligned && in_dtype == 0 && out_dtype == 0 && (M <= 16 || (M <= 64 && row_blocks <= 4 * dl::sm_count()))) {
    const float* xf = static_cast<const float*>(x);
    const float* wf = static_cast<const float*>(w);
    float* yf = static_cast<float*>(y);
#define DL_ROWS(R) return dl::launch_rows<R>(xf, ldx, wf, bias, yf, ldy, M, N, K, out_scale, stream)
    if (M == 1) DL_ROWS(1);
    if (M == 2) DL_ROWS(2);
    if (M <= 4) DL_ROWS(4);
    if (M <= 8) DL_ROWS(8);
    DL_ROWS(16);
#undef DL_ROWS
  }
  // Tiles of 128 rows or of 64, by the rounds of blocks over the SMs (of 148, clusters of four fill 140): an SM
  // takes about 33 us for every block of 64 rows and 50 for one of 128 that it gets, at k 2048. Measured, 64 / 128, us: 128 x
  // 2048 x 2048 46 / 69, 128 x 16384 x 2048 237 / 218, 300 x 3072 x 2048 131 / 159, 700 x 2048 x 2048 181 / 162, 1000 x 16384
  // x 2048 1,656 / 1,382.
  const bool alone = K <= dl::span_length(K) * (dl::SPANS / dl::QUARTERS);
  const long long blocks = alone ? 1 : dl::QUARTERS, filled = alone ? dl::sm_count() : (dl::sm_count() * 35ll + 36) / 37;
  auto rounds = [&](int rows) { return (blocks * ((N + dl::BN - 1) / dl::BN) * ((M + rows - 1) / rows) + filled - 1) / filled; };
  const bool tall = 50 * rounds(128) < 33 * rounds(64);
#define DL_TILES(TI, TO, CL)                                                                                           \
  return tall ? dl::launch_tiles<TI, TO, 128, 16, CL>(x, ldx, w, bias, y, ldy, M, N, K, out_scale, aligned, stream)    \
              : dl::launch_tiles<TI, TO, 64, 8, CL>(x, ldx, w, bias, y, ldy, M, N, K, out_scale, aligned, stream)
#define DL_LAUNCH(TI, TO)                       \
  do {                                          \
    if (alone) DL_TILES(TI, TO, 1);             \
    DL_TILES(TI, TO, dl::QUARTERS);             \
  } while (0)
  if (in_dtype == 0 && out_dtype == 0) DL_LAUNCH(float, float);
  if (in_dtype == 1 && out_dtype == 1) DL_LAUNCH(dl::bf16, dl::bf16);
  if (in_dtype == 1 && out_dtype == 0) DL_LAUNCH(dl::bf16, float);
#undef DL_LAUNCH
#undef DL_TILES
  return DL_ERR_UNSUPPORTED;
}

// The gated feed-forward's first half for up to 16 rows, float32: w = [Wg; Wu] with 2 F rows, y [M, F] = silu(x Wg^T) (x Wu^T), the
// same bits as the product followed by dl_silu_mul. x and w 16-byte aligned, K and ldx multiples of 4.
DL_EXPORT int dl_gemm_simt_swiglu(const float* x, int ldx, const float* w, float* y, int ldy, int M, int F, int K, cudaStream_t stream) {
  if (M <= 0 || F <= 0) return 0;
  if (K <= 0 || (K & 3) || (ldx & 3) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) || M > 16 || F > (1 << 29))
    return DL_ERR_UNSUPPORTED;
#define DL_ROWS(R) return dl::launch_rows<R, dl::ROWS_SWIGLU>(x, ldx, w, nullptr, y, ldy, M, 2 * F, K, 1.0f, stream)
  if (M == 1) DL_ROWS(1);
  if (M == 2) DL_ROWS(2);
  if (M <= 4) DL_ROWS(4);
  if (M <= 8) DL_ROWS(8);
  DL_ROWS(16);
#undef DL_ROWS
}

// The q | k | v projection of up to 16 rows, float32, with the rotary encoding and the cache write: as dl_gemm_split_qkv_rope, the
// same bits as dl_gemm_simt followed by dl_rope_cache_write.
DL_EXPORT int dl_gemm_simt_qkv_rope(const float* x, int ldx, const float* w, float* q_out, int ldq, int M, int K, const int* positions,
                                    const int* row_request, const int* block_table, int max_blocks, float* k_cache, float* v_cache,
                                    const float* inv_freq, float pos_scale, int n_heads, int n_kv_heads, int head_dim, int page_size,
                                    cudaStream_t stream) {
  if (M <= 0) return 0;
  if (K <= 0 || (K & 3) || (ldx & 3) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) || M > 16 ||
      head_dim <= 0 || head_dim % dl::RF || n_heads <= 0 || n_kv_heads <= 0 || page_size <= 0 || inv_freq == nullptr)
    return DL_ERR_UNSUPPORTED;
  const dl::QkvRopeOf<float> rope = {positions, row_request, block_table, max_blocks, k_cache, v_cache, inv_freq, nullptr, pos_scale,
                                     n_heads, n_kv_heads, head_dim, page_size};
  const int N = (n_heads + 2 * n_kv_heads) * head_dim;
#define DL_ROWS(R) return dl::launch_rows<R, dl::ROWS_ROPE>(x, ldx, w, nullptr, q_out, ldq, M, N, K, 1.0f, stream, rope)
  if (M == 1) DL_ROWS(1);
  if (M == 2) DL_ROWS(2);
  if (M <= 4) DL_ROWS(4);
  if (M <= 8) DL_ROWS(8);
  DL_ROWS(16);
#undef DL_ROWS
}
