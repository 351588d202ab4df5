// The two passes over the segments of long portions (see ssm.cu) in matrix form, for bfloat16 inputs.
//
// Within a segment of n tokens with step sizes d_t, write e(t, s) = exp(-rate (d_{s+1} + .. + d_t)). Then
//   added   = sum_s  e(n - 1, s) d_s B_s x_s^T                                       (what the segment adds to the state)
//   y_t     = sum_{s <= t} (C_t . B_s) e(t, s) d_s x_s  +  e(t, -1) S_start^T C_t  +  D x_t
// which are products of matrices: the recurrence walks none of its tokens. B, C and x are bfloat16 numbers as stored, so
// their products are exact in the tensor cores; every float32 factor (weights e d, the start state, C . B) is cut into three
// bfloat16 terms of 8 bits each, which hold its 24 bits, and multiplied three times. All sums are float32. The exponents are
// sums of step sizes, kept as a float and the float that it misses, so that a difference of two of them is as exact as the
// product of the single decays would be.
//
// ssm_added_kernel: block = (segment, head), a warp 16 rows of the state. ssm_outputs_kernel: block = (segment, head), a warp
// 16 tokens: C S_start first, then over the tokens up to its own in steps of 16 the scores C B^T (from registers to
// registers, as in a flash attention: a score tile's accumulator is the next product's left operand). No chain over the tokens is
// left; a block asks for all that it reads at its start, but its conversions and products follow one another, and two blocks an SM
// hide little of that.
//
// A token's numbers reach itself and the tokens behind it alone, infinities and NaNs among them: runs of sixteen tokens with such
// an x are added token by token (ssm_outputs_kernel).
//
// Both passes of the walk in ssm.cu issue five multiply-adds per number of the state and token; here it is about two and a half,
// three times over, on the tensor pipe. Figures at the launch rule in ssm.cu.
#pragma once

namespace dl {

constexpr int SEG_T = 128;             // most tokens of a segment

__device__ __forceinline__ void seg_ldm4(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
}
__device__ __forceinline__ void seg_ldm4t(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
}
__device__ __forceinline__ void seg_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// a and b as three pairs of bfloat16 whose sums they are (to the 24 bits of a float). What has no finite bfloat16 next to it
// stays in the first term alone.
__device__ __forceinline__ void seg_split(float a, float b, uint32_t (&out)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    out[i] = *reinterpret_cast<const uint32_t*>(&v);
    a = fabsf(__low2float(v)) <= 3.3895e38f ? a - __low2float(v) : 0.0f;
    b = fabsf(__high2float(v)) <= 3.3895e38f ? b - __high2float(v) : 0.0f;
  }
}

// Whether one of eight bfloat16 numbers is an infinity or no number.
__device__ __forceinline__ bool seg_not_finite(const uint4& v) {
  constexpr unsigned EXPONENTS = 0x7f807f80u;
  return (__vcmpeq2(v.x & EXPONENTS, EXPONENTS) | __vcmpeq2(v.y & EXPONENTS, EXPONENTS) | __vcmpeq2(v.z & EXPONENTS, EXPONENTS) |
          __vcmpeq2(v.w & EXPONENTS, EXPONENTS)) != 0u;
}

// 16 bytes to shared memory, or zeros.
__device__ __forceinline__ void seg_copy16(void* dst, const void* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src),
               "r"(there ? 16 : 0)
               : "memory");
}

// The segment's step sizes and running exponents: at[t] = (exponent, what it misses, step size, 0); zeros past the end.
// Called by the whole block (at least SEG_T threads); ends with a barrier.
__device__ __forceinline__ void seg_exponents(float4* at, double* warp_sums, const bf16* proj, int proj_stride, int col, int r0,
                                              int n, float bias, float rate) {
  const int t = threadIdx.x;
  float dt = 0.0f;
  double run = 0.0;
  if (t < SEG_T) {
    if (t < n) dt = softplus_f(to_float(proj[static_cast<size_t>(r0 + t) * proj_stride + col]) + bias);
    const float one = rate * dt;                      // e^-200 is 0 in float32: so far, and sums of them stay finite
    run = one > 200.0f ? 200.0 : static_cast<double>(rate) * static_cast<double>(dt);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, run, o);
      if ((t & 31) >= o) run += v;
    }
    if ((t & 31) == 31) warp_sums[t >> 5] = run;
  }
  __syncthreads();
  if (t < SEG_T) {
    for (int w = 0; w < (t >> 5); ++w) run += warp_sums[w];
    const float hi = static_cast<float>(run);
    at[t] = make_float4(hi, static_cast<float>(run - static_cast<double>(hi)), dt, 0.0f);
  }
  __syncthreads();
}

template <int N, int P>
__global__ void __launch_bounds__(256)
ssm_added_kernel(const bf16* __restrict__ u, int u_stride, const bf16* __restrict__ proj, int proj_stride, int dt_col,
                 const float* __restrict__ dt_bias, const float* __restrict__ a_log, const int* __restrict__ segments,
                 float* __restrict__ scratch, float* __restrict__ seg_decay, int H, int G) {
  constexpr int BS = N + 8, XS = P + 8, UNITS = N / 16 * (P / 64);
  extern __shared__ __align__(16) unsigned char seg_smem[];
  bf16* sb = reinterpret_cast<bf16*>(seg_smem);       // [SEG_T][BS]
  bf16* sx = sb + SEG_T * BS;                         // [3][SEG_T][XS]
  __shared__ float4 at[SEG_T];
  __shared__ double warp_sums[SEG_T / 32];
  const int4 seg = reinterpret_cast<const int4*>(segments)[blockIdx.x];
  const int h = blockIdx.y, g = h / (H / G), r0 = seg.y, n = seg.z, inner = H * P, tid = threadIdx.x;
  // everything the block reads is asked for at once: a trip to memory takes as long as the products
  const bf16* rows = u + static_cast<size_t>(r0) * u_stride;
#pragma unroll
  for (int i = 0; i < SEG_T * (N / 8) / 256; ++i) {
    const int e = i * 256 + tid, t = e / (N / 8), c = e % (N / 8) * 8;
    seg_copy16(sb + t * BS + c, rows + (t < n ? static_cast<size_t>(t) * u_stride + inner + g * N + c : 0), t < n);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  constexpr int XI = SEG_T * (P / 8) / 256;
  Vec16 xv[XI];
#pragma unroll
  for (int i = 0; i < XI; ++i) {
    const int e = i * 256 + tid, t = e / (P / 8), c = e % (P / 8) * 8;
    xv[i].raw = make_uint4(0, 0, 0, 0);
    if (t < n) xv[i] = *reinterpret_cast<const Vec16*>(rows + static_cast<size_t>(t) * u_stride + h * P + c);
  }
  seg_exponents(at, warp_sums, proj, proj_stride, dt_col + h, r0, n, dt_bias[h], expf(a_log[h]));
  const float4 end = at[n - 1];
#pragma unroll
  for (int xi = 0; xi < XI; ++xi) {
    const int e = xi * 256 + tid, t = e / (P / 8), c = e % (P / 8) * 8;
    float v[8];
    const float4 a = at[t];
    const float w = t < n ? expf(-((end.x - a.x) + (end.y - a.y))) * a.z : 0.0f;
    unpack<bf16>(xv[xi], v);
    uint32_t parts[4][3];
#pragma unroll
    for (int j = 0; j < 4; ++j) seg_split(t < n ? v[2 * j] * w : 0.0f, t < n ? v[2 * j + 1] * w : 0.0f, parts[j]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint4*>(sx + (i * SEG_T + t) * XS + c) = make_uint4(parts[0][i], parts[1][i], parts[2][i], parts[3][i]);
  }
  if (tid == 0) seg_decay[static_cast<size_t>(blockIdx.x) * H + h] = expf(-(end.x + end.y));
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31, j = lane >> 3, l8 = lane & 7;
  float* S = scratch + (static_cast<size_t>(blockIdx.x) * H + h) * N * P;
  for (int unit = warp; unit < UNITS; unit += 8) {
    const int n0 = unit % (N / 16) * 16, p0 = unit / (N / 16) * 64;
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[i][k] = 0.0f;
    for (int k0 = 0; k0 < (n + 15) / 16 * 16; k0 += 16) {
      uint32_t a[4];
      seg_ldm4t(a, sb + (k0 + (j >> 1) * 8 + l8) * BS + n0 + (j & 1) * 8);
#pragma unroll
      for (int i = 2; i >= 0; --i)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t b[4];
          seg_ldm4t(b, sx + (i * SEG_T + k0 + (j & 1) * 8 + l8) * XS + p0 + q * 16 + (j >> 1) * 8);
          seg_mma(acc[2 * q], a, b[0], b[1]);
          seg_mma(acc[2 * q + 1], a, b[2], b[3]);
        }
    }
    float* row = S + static_cast<size_t>(n0 + (lane >> 2)) * P + p0 + (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      *reinterpret_cast<float2*>(row + i * 8) = make_float2(acc[i][0], acc[i][1]);
      *reinterpret_cast<float2*>(row + 8 * P + i * 8) = make_float2(acc[i][2], acc[i][3]);
    }
  }
}

template <int N, int P>
__global__ void __launch_bounds__(256, P == 64 ? 2 : 1)
ssm_outputs_kernel(const bf16* __restrict__ u, int u_stride, const bf16* __restrict__ proj, int proj_stride, int dt_col,
                   const float* __restrict__ dt_bias, const float* __restrict__ a_log, const float* __restrict__ d_skip,
                   const int* __restrict__ segments, const float* __restrict__ scratch, float* __restrict__ y, int H, int G) {
  constexpr int BS = N + 8, XS = P + 8;
  extern __shared__ __align__(16) unsigned char seg_smem[];
  bf16* sb = reinterpret_cast<bf16*>(seg_smem);       // [SEG_T][BS]
  bf16* sx = sb + SEG_T * BS;                         // [SEG_T][XS]
  bf16* ss = sx + SEG_T * XS;                         // C [SEG_T][BS] first, then the start state's terms [3][N][XS]
  __shared__ float4 at[SEG_T];
  __shared__ double warp_sums[SEG_T / 32];
  __shared__ unsigned not_finite;                     // bit i: of the tokens 16 i .. 16 i + 15 one has an x that is not finite
  const int4 seg = reinterpret_cast<const int4*>(segments)[blockIdx.x];
  const int h = blockIdx.y, g = h / (H / G), r0 = seg.y, n = seg.z, inner = H * P, tid = threadIdx.x;
  // everything the block reads is asked for at once (73 -> 63 us for the sizes of the profile; what a segment adds to the state
  // 41 -> 34)
  const bf16* rows = u + static_cast<size_t>(r0) * u_stride;
#pragma unroll
  for (int i = 0; i < SEG_T * (N / 8) / 256; ++i) {
    const int e = i * 256 + tid, t = e / (N / 8), c = e % (N / 8) * 8;
    const bf16* row = rows + (t < n ? static_cast<size_t>(t) * u_stride + inner + g * N + c : 0);
    seg_copy16(ss + t * BS + c, row + (t < n ? G * N : 0), t < n);
    seg_copy16(sb + t * BS + c, row, t < n);
  }
#pragma unroll
  for (int i = 0; i < SEG_T * (P / 8) / 256; ++i) {
    const int e = i * 256 + tid, t = e / (P / 8), c = e % (P / 8) * 8;
    seg_copy16(sx + t * XS + c, rows + (t < n ? static_cast<size_t>(t) * u_stride + h * P + c : 0), t < n);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  const float* S = scratch + (static_cast<size_t>(blockIdx.x) * H + h) * N * P;
  constexpr int SI = N * (P / 8) / 256;
  float4 start[SI][2];
#pragma unroll
  for (int i = 0; i < SI; ++i) {
    const float* from = S + static_cast<size_t>(i * 256 + tid) * 8;
    start[i][0] = *reinterpret_cast<const float4*>(from);
    start[i][1] = *reinterpret_cast<const float4*>(from + 4);
  }
  if (tid == 0) not_finite = 0u;
  seg_exponents(at, warp_sums, proj, proj_stride, dt_col + h, r0, n, dt_bias[h], expf(a_log[h]));
  asm volatile("cp.async.wait_all;" ::: "memory");
  unsigned mine = 0u;
#pragma unroll
  for (int i = 0; i < SEG_T * (P / 8) / 256; ++i) {    // (what the thread copied itself)
    const int e = i * 256 + tid, t = e / (P / 8), c = e % (P / 8) * 8;
    if (seg_not_finite(reinterpret_cast<const Vec16*>(sx + t * XS + c)->raw)) mine |= 1u << (t >> 4);
  }
  __syncthreads();
  if (mine != 0u) atomicOr(&not_finite, mine);        // (set to zero in front of the barriers of seg_exponents, read behind the next two)
  const int warp = tid >> 5, lane = tid & 31, j = lane >> 3, l8 = lane & 7;
  const int tile = warp < 4 ? warp : 11 - warp;        // 16 tokens; a scheduler's two warps have nine steps together
  const int t0 = tile * 16, ta = t0 + (lane >> 2), tb = ta + 8;
  uint32_t c_frag[N / 16][4];
#pragma unroll
  for (int k = 0; k < N / 16; ++k) seg_ldm4(c_frag[k], ss + (t0 + (j & 1) * 8 + l8) * BS + k * 16 + (j >> 1) * 8);
  __syncthreads();                                     // C is in registers: its place takes the start state
#pragma unroll
  for (int si = 0; si < SI; ++si) {
    const int e = si * 256 + tid, r = e / (P / 8), c = e % (P / 8) * 8;
    const float4 a = start[si][0], b = start[si][1];
    uint32_t parts[4][3];
    seg_split(a.x, a.y, parts[0]);
    seg_split(a.z, a.w, parts[1]);
    seg_split(b.x, b.y, parts[2]);
    seg_split(b.z, b.w, parts[3]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint4*>(ss + (i * N + r) * XS + c) = make_uint4(parts[0][i], parts[1][i], parts[2][i], parts[3][i]);
  }
  __syncthreads();
  if (t0 >= n) return;
  float acc[P / 8][4];
#pragma unroll
  for (int i = 0; i < P / 8; ++i)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[i][k] = 0.0f;
#pragma unroll
  for (int k = 0; k < N / 16; ++k)
#pragma unroll
    for (int i = 2; i >= 0; --i)
#pragma unroll
      for (int q = 0; q < P / 16; ++q) {
        uint32_t b[4];
        seg_ldm4t(b, ss + (i * N + k * 16 + (j & 1) * 8 + l8) * XS + q * 16 + (j >> 1) * 8);
        seg_mma(acc[2 * q], c_frag[k], b[0], b[1]);
        seg_mma(acc[2 * q + 1], c_frag[k], b[2], b[3]);
      }
  const float4 ea = at[ta], eb = at[tb];
  {
    const float wa = expf(-(ea.x + ea.y)), wb = expf(-(eb.x + eb.y));
#pragma unroll
    for (int i = 0; i < P / 8; ++i) acc[i][0] *= wa, acc[i][1] *= wa, acc[i][2] *= wb, acc[i][3] *= wb;
  }
  for (int s0 = 0; s0 <= t0; s0 += 16) {
    float gc[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) gc[i][k] = 0.0f;
#pragma unroll
    for (int k = 0; k < N / 16; ++k) {
      uint32_t b[4];
      seg_ldm4(b, sb + (s0 + (j >> 1) * 8 + l8) * BS + k * 16 + (j & 1) * 8);
      seg_mma(gc[0], c_frag[k], b[0], b[1]);
      seg_mma(gc[1], c_frag[k], b[2], b[3]);
    }
    float v[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int s = s0 + i * 8 + (lane & 3) * 2 + k;
        const float4 es = at[s];
        v[i][k] = s <= ta ? gc[i][k] * (expf(-((ea.x - es.x) + (ea.y - es.y))) * es.z) : 0.0f;
        v[i][2 + k] = s <= tb ? gc[i][2 + k] * (expf(-((eb.x - es.x) + (eb.y - es.y))) * es.z) : 0.0f;
      }
    if (not_finite >> (s0 >> 4) & 1u) {
      // In the product the weight 0 of a token that a row does not see, or of a term of a weight that needs no third one, would
      // meet the infinity: these sixteen tokens are added one by one, each to the rows that see it.
#pragma unroll 1
      for (int k = 0; k < 16; ++k) {
        const int from = (lane & ~3) | (k >> 1 & 3);
        const float wa = __shfl_sync(0xffffffffu, k & 8 ? (k & 1 ? v[1][1] : v[1][0]) : (k & 1 ? v[0][1] : v[0][0]), from);
        const float wb = __shfl_sync(0xffffffffu, k & 8 ? (k & 1 ? v[1][3] : v[1][2]) : (k & 1 ? v[0][3] : v[0][2]), from);
        const bool seen_a = s0 + k <= ta, seen_b = s0 + k <= tb;
        const bf16* xr = sx + (s0 + k) * XS + (lane & 3) * 2;
#pragma unroll
        for (int i = 0; i < P / 8; ++i) {
          const __nv_bfloat162 xv = *reinterpret_cast<const __nv_bfloat162*>(xr + i * 8);
          if (seen_a) acc[i][0] = fmaf(wa, __low2float(xv), acc[i][0]), acc[i][1] = fmaf(wa, __high2float(xv), acc[i][1]);
          if (seen_b) acc[i][2] = fmaf(wb, __low2float(xv), acc[i][2]), acc[i][3] = fmaf(wb, __high2float(xv), acc[i][3]);
        }
      }
      continue;
    }
    uint32_t a[3][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t p0[3], p1[3];
      seg_split(v[i][0], v[i][1], p0);
      seg_split(v[i][2], v[i][3], p1);
#pragma unroll
      for (int m = 0; m < 3; ++m) a[m][2 * i] = p0[m], a[m][2 * i + 1] = p1[m];
    }
#pragma unroll
    for (int q = 0; q < P / 16; ++q) {
      uint32_t b[4];
      seg_ldm4t(b, sx + (s0 + (j & 1) * 8 + l8) * XS + q * 16 + (j >> 1) * 8);
#pragma unroll
      for (int m = 2; m >= 0; --m) {
        seg_mma(acc[2 * q], a[m], b[0], b[1]);
        seg_mma(acc[2 * q + 1], a[m], b[2], b[3]);
      }
    }
  }
  const float skip = d_skip[h];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int t = half ? tb : ta;
    if (t >= n) continue;
    float* row = y + static_cast<size_t>(r0 + t) * inner + h * P + (lane & 3) * 2;
    const bf16* xr = sx + t * XS + (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < P / 8; ++i) {
      const __nv_bfloat162 xv = *reinterpret_cast<const __nv_bfloat162*>(xr + i * 8);
      *reinterpret_cast<float2*>(row + i * 8) = make_float2(fmaf(skip, __low2float(xv), acc[i][2 * half]),
                                                            fmaf(skip, __high2float(xv), acc[i][2 * half + 1]));
    }
  }
}

template <int N, int P>
int launch_added(const bf16* u, int u_stride, const bf16* proj, int proj_stride, int dt_col, const float* dt_bias,
                 const float* a_log, const int* segments, int n_segments, float* scratch, float* seg_decay, int H, int G,
                 cudaStream_t stream) {
  constexpr int SMEM = (SEG_T * (N + 8) + 3 * SEG_T * (P + 8)) * 2;
  const cudaError_t e = cudaFuncSetAttribute(ssm_added_kernel<N, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  ssm_added_kernel<N, P><<<dim3(n_segments, H), 256, SMEM, stream>>>(u, u_stride, proj, proj_stride, dt_col, dt_bias, a_log,
                                                                      segments, scratch, seg_decay, H, G);
  return launch_status();
}

template <int N, int P>
int launch_outputs(const bf16* u, int u_stride, const bf16* proj, int proj_stride, int dt_col, const float* dt_bias,
                   const float* a_log, const float* d_skip, const int* segments, int n_segments, const float* scratch, float* y,
                   int H, int G, cudaStream_t stream) {
  constexpr int SHARED_PLACE = 3 * N * (P + 8) > SEG_T * (N + 8) ? 3 * N * (P + 8) : SEG_T * (N + 8);      // C, then the start state
  constexpr int SMEM = (SEG_T * (N + 8) + SEG_T * (P + 8) + SHARED_PLACE) * 2;
  static_assert(SMEM + 4096 <= 232448, "with the static arrays within the 227 KiB of a block");
  const cudaError_t e = cudaFuncSetAttribute(ssm_outputs_kernel<N, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  ssm_outputs_kernel<N, P><<<dim3(n_segments, H), 256, SMEM, stream>>>(u, u_stride, proj, proj_stride, dt_col, dt_bias, a_log,
                                                                        d_skip, segments, scratch, y, H, G);
  return launch_status();
}

}  // namespace dl
