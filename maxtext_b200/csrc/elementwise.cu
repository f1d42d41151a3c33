// Memory-bound kernels of the decoder layer: RMSNorm (forward, backward), rotary embedding on a packed
// q|k|v tensor, gated activation (SwiGLU / GeGLU), embedding gather and its scatter-add backward.
// All are HBM-bandwidth bound: 16-byte vector accesses, one pass over the data where the row fits in
// registers, fp32 math.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mt {

// Eight bf16 numbers as one 16-byte word. (As a struct of four __nv_bfloat162, whose copies go through their assignment operators, every load and store
// became four of 4 bytes: the L1 ran at 90 % while HBM idled at half of its rate.)
struct bf16x8 { uint4 q; };

__device__ __forceinline__ void unpack8(const bf16x8& p, float (&f)[8]) {
  const uint32_t w[4] = {p.q.x, p.q.y, p.q.z, p.q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&t);
}
__device__ __forceinline__ bf16x8 pack8(const float (&f)[8]) {
  return {make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]))};
}
__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {        // two bf16 products, each rounded once
  const __nv_bfloat162 t = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&t);
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum over the TPR threads that share a row. TPR == 32: one warp per row; TPR == 256: one block per row, whose warps meet in `smem` (8 floats). A block that
// sums one row after the other gives two buffers in turn, so that one barrier per row is enough.
template <int TPR>
__device__ __forceinline__ float row_sum(float v, float* smem) {
  v = warp_sum(v);
  if (TPR == 32) return v;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) smem[w] = v;
  __syncthreads();
  float t = (l < TPR / 32) ? smem[l] : 0.f;
  return warp_sum(t);
}

// ------------------------------------------------------------------------------------------------ RMSNorm forward
// y = bf16(x * rstd) * bf16(scale + offset), both roundings as in the reference layer. With `add` the row is bf16(x + add), which also goes to
// `sum`: the residual add in front of a norm, in the norm's own pass. Bandwidth-bound; at 16384 rows of 4096 lanes the add and the norm took 65 + 85 us
// as two kernels (402 + 268 MB) and take 90 us as one (537 MB).
// Blocks stride over the rows and fetch the next row before they sum the present one: with one row per block, every load waited for a block to start and
// every store for a barrier (75 us for the plain norm and 117 us for add and norm at 16384 x 4096, 3.6 - 4.6 TB/s; 46 and 90 us now).
// blocks that share an SM: the kernel is compiled for that many, and the grid counts on them
constexpr int rms_fwd_resident(int tpr, int vpt, bool add) { return vpt <= 1 ? (tpr == 32 ? 5 : 6) : vpt <= 2 ? 4 : vpt <= 4 || !add ? 2 : 1; }
template <int TPR, int VPT, bool ADD>
__global__ void __launch_bounds__(256, rms_fwd_resident(TPR, VPT, ADD)) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ add,
                                                          __nv_bfloat16* __restrict__ sum, const __nv_bfloat16* __restrict__ scale, float eps, float offset,
                                                          __nv_bfloat16* __restrict__ y, float* __restrict__ rstd_out, int rows, int D) {
  __shared__ float red[2][8];
  constexpr int RPB = 256 / TPR;
  const int tid = threadIdx.x % TPR;
  const long step = (long)gridDim.x * RPB;
  long row = (long)blockIdx.x * RPB + threadIdx.x / TPR;
  bf16x8 nx[VPT], na[ADD ? VPT : 1], sc[VPT];               // sc: bf16(scale + offset), the same for every row
  if (scale) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int col = (i * TPR + tid) * 8;
      if (col < D) {
        float f[8];
        unpack8(*reinterpret_cast<const bf16x8*>(scale + col), f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += offset;
        sc[i] = pack8(f);
      }
    }
  }
  auto fetch = [&](long r) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int col = (i * TPR + tid) * 8;
      if (r < rows && col < D) {
        nx[i] = *reinterpret_cast<const bf16x8*>(x + r * D + col);
        if (ADD) na[i] = *reinterpret_cast<const bf16x8*>(add + r * D + col);
      }
    }
  };
  fetch(row);
  int buf = 0;
  for (long top = (long)blockIdx.x * RPB; top < rows; top += step, row += step, buf ^= 1) {   // top: the block's first row, the same for all its threads
    const bool active = row < rows;
    bf16x8 v[VPT];                                           // the row as it is stored
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int col = (i * TPR + tid) * 8;
      if (active && col < D) {
        float f[8];
        v[i] = nx[i];
        if (ADD) {
          float a[8];
          unpack8(nx[i], f);
          unpack8(na[i], a);
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] += a[e];
          v[i] = pack8(f);
          *reinterpret_cast<bf16x8*>(sum + row * D + col) = v[i];
        }
        unpack8(v[i], f);                                    // the norm reads the stream as it is stored
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
      }
    }
    fetch(row + step);
    ss = row_sum<TPR>(ss, red[buf]);
    const float rstd = rsqrtf(ss / (float)D + eps);
    if (active && tid == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int col = (i * TPR + tid) * 8;
      if (active && col < D) {
        float o[8];
        unpack8(v[i], o);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = o[e] * rstd;
        bf16x8 r = pack8(o);
        if (scale) r.q = make_uint4(mul2(r.q.x, sc[i].q.x), mul2(r.q.y, sc[i].q.y), mul2(r.q.z, sc[i].q.z), mul2(r.q.w, sc[i].q.w));
        *reinterpret_cast<bf16x8*>(y + row * D + col) = r;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ RMSNorm backward
// dx = rstd * (g - xhat * mean(g * xhat)) [+ dres], g = dy * (scale + offset);  dscale += sum_rows dy * xhat. `dres` is what reaches the same row past
// the norm (the residual stream's own gradient): added here, it costs no pass of its own. It joins the norm's gradient as that is stored (bf16), so the sum
// is the same bits as of a norm and an add on their own.
// Blocks stride over rows and keep per-column dscale partials in registers; each (block, row slot) writes its partial row into `partial`, and
// rms_dscale_reduce_kernel adds the rows up in a fixed order: no atomics, so the result is bitwise reproducible.
// As in the forward pass the next row is fetched before the present one is summed: 110 us for 16384 x 4096 with a stream gradient and a scale's (537 MB), of
// which the reduction below is 6, 192 us without.
template <int TPR, int VPT>
__global__ void __launch_bounds__(256, TPR == 32 ? (VPT == 1 ? 4 : 1) : VPT == 1 ? 3 : VPT == 2 ? 2 : 1) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                   const __nv_bfloat16* __restrict__ scale, const float* __restrict__ rstd_in, float offset,
                                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx, float* __restrict__ partial, int rows,
                                   int D) {
  __shared__ float red[2][8];
  const int rows_per_block = blockDim.x / TPR;
  const int r_in_block = threadIdx.x / TPR;
  const int tid = threadIdx.x % TPR;
  float ds[VPT][8];
  auto factor = [&](int col, float (&f)[8]) {                // from L1 each time: the registers are worth more to the next row
    if (scale) {
      unpack8(*reinterpret_cast<const bf16x8*>(scale + col), f);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] += offset;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = 1.f;
    }
  };
#pragma unroll
  for (int i = 0; i < VPT; ++i)
#pragma unroll
    for (int e = 0; e < 8; ++e) ds[i][e] = 0.f;
  const long n_groups = ((long)rows + rows_per_block - 1) / rows_per_block;
  constexpr bool AHEAD = TPR == 256 && VPT <= 2;             // a warp per row has enough rows under way; wider rows have no registers left for it
  bf16x8 nd[VPT], nx[VPT];                                   // the next row
  float nrstd = 0.f;
  auto fetch = [&](long grp) {
    const long row = grp * rows_per_block + r_in_block;
    if (row >= rows) return;
    nrstd = rstd_in[row];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int col = (i * TPR + tid) * 8;
      if (col < D) {
        nd[i] = *reinterpret_cast<const bf16x8*>(dy + row * D + col);
        nx[i] = *reinterpret_cast<const bf16x8*>(x + row * D + col);
      }
    }
  };
  if (AHEAD) fetch(blockIdx.x);
  int buf = 0;
  for (long grp = blockIdx.x; grp < n_groups; grp += gridDim.x, buf ^= 1) {
    const long row = grp * rows_per_block + r_in_block;
    const bool active = row < rows;
    if (!AHEAD) fetch(grp);
    const float rstd = active ? nrstd : 0.f;
    bf16x8 cd[VPT], cx[VPT], cr[VPT];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int col = (i * TPR + tid) * 8;
      cd[i] = nd[i]; cx[i] = nx[i];
      if (active && col < D) {
        if (dres) cr[i] = *reinterpret_cast<const bf16x8*>(dres + row * D + col);
        float a[8], b[8], sc[8];
        unpack8(cd[i], a);
        unpack8(cx[i], b);
        factor(col, sc);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = b[e] * rstd;
          dot += a[e] * sc[e] * xh;
          ds[i][e] += a[e] * xh;
        }
      }
    }
    if (AHEAD) fetch(grp + gridDim.x);
    dot = row_sum<TPR>(dot, red[buf]) / (float)D;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int col = (i * TPR + tid) * 8;
      if (active && col < D) {
        float a[8], b[8], sc[8], o[8];
        unpack8(cd[i], a);
        unpack8(cx[i], b);
        factor(col, sc);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = rstd * __fmaf_rn(-__fmul_rn(b[e], rstd), dot, __fmul_rn(a[e], sc[e]));   // g and xhat rounded as in the sums
        if (dres) {
          unpack8(cr[i], a);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] = bf16_round(o[e]) + a[e];
        }
        *reinterpret_cast<bf16x8*>(dx + row * D + col) = pack8(o);
      }
    }
  }
  if (partial) {
    float* prow = partial + ((long)blockIdx.x * rows_per_block + r_in_block) * D;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int col = (i * TPR + tid) * 8;
      if (col < D) {
        *reinterpret_cast<float4*>(prow + col) = make_float4(ds[i][0], ds[i][1], ds[i][2], ds[i][3]);
        *reinterpret_cast<float4*>(prow + col + 4) = make_float4(ds[i][4], ds[i][5], ds[i][6], ds[i][7]);
      }
    }
  }
}

// dscale[c] += sum over partial rows, in a fixed order: row r joins sum r % 4 (the last, incomplete four rows all join sum 0), and the four sums meet in
// pairs. The four serial chains per column are what bounds it, so nothing else may wait in them: a block of 256 threads fetches 16 KB of its COLS columns ahead,
// and a thread per column and sum adds up the rows that wait in shared memory. Narrow widths have more blocks with eight columns (32-byte pieces); from 1024
// columns on there are enough with 32. A thread per column that loads what it adds (16 - 32 blocks at the usual widths) took 47 us for 592 rows of 4096
// columns and 95 us for the 4736 rows of a 128-wide head norm; 6.4 and 11 us now.
template <int COLS>
__global__ void __launch_bounds__(256) rms_dscale_reduce_kernel(const float* __restrict__ partial, int nrows, int D, float* __restrict__ dscale) {
  constexpr int ROWS = 4096 / COLS, V = COLS / 4, STEP = 256 / V, PER = ROWS / STEP;      // V 16-byte pieces per row, PER of a thread per tile
  __shared__ __align__(16) float tile[2][ROWS][COLS];
  __shared__ float sums[4][COLS];
  const int c0 = blockIdx.x * COLS, piece = (threadIdx.x % V) * 4, r0 = threadIdx.x / V;
  const int c = threadIdx.x % COLS, j = threadIdx.x / COLS;                                 // column and sum of a thread below 4 COLS
  const int whole = nrows / 4 * 4;
  float4 next[PER];
  auto fetch = [&](int top) {
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int r = top + r0 + k * STEP;
      if (r < nrows) next[k] = *reinterpret_cast<const float4*>(partial + (long)r * D + c0 + piece);
    }
  };
  fetch(0);
  float a = 0.f;
  int buf = 0;
  for (int top = 0; top < nrows; top += ROWS, buf ^= 1) {
#pragma unroll
    for (int k = 0; k < PER; ++k) *reinterpret_cast<float4*>(&tile[buf][r0 + k * STEP][piece]) = next[k];
    fetch(top + ROWS);
    __syncthreads();                                         // two buffers in turn: one barrier per tile is enough
    if (j < 4) {
      const int n = (whole - top < ROWS ? whole - top : ROWS) / 4;
#pragma unroll 32
      for (int i = 0; i < n; ++i) a += tile[buf][4 * i + j][c];
      if (j == 0 && nrows - top <= ROWS)
        for (int r = whole - top; r < nrows - top; ++r) a += tile[buf][r][c];
    }
  }
  if (j < 4) sums[j][c] = a;
  __syncthreads();
  if (j == 0) dscale[c0 + c] += (sums[0][c] + sums[1][c]) + (sums[2][c] + sums[3][c]);
}

// ------------------------------------------------------------------------------------------------ rotary embedding
// In-place rotation of the first n_rot heads of x [tokens, heads, dh]; one block per token, thread per
// rotated pair (sin/cos evaluated once per pair and reused across heads).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const int* __restrict__ pos, const float* __restrict__ inv_ts,
                            int heads, int dh, int n_rot, int rot_dim, int interleaved, int inverse) {
  const long tok = blockIdx.x;
  const int half = rot_dim / 2;
  const float p = (float)pos[tok];
  for (int j = threadIdx.x; j < half; j += blockDim.x) {
    float s, c;
    sincosf(p * inv_ts[j], &s, &c);
    if (inverse) s = -s;
    const int i0 = interleaved ? 2 * j : j;
    const int i1 = interleaved ? 2 * j + 1 : j + half;
    __nv_bfloat16* base = x + tok * (long)heads * dh;
    for (int h = 0; h < n_rot; ++h) {
      const float a = __bfloat162float(base[h * dh + i0]);
      const float b = __bfloat162float(base[h * dh + i1]);
      // written out like the rotation of the inference kernels, so that both round alike
      base[h * dh + i0] = __float2bfloat16_rn(__fmaf_rn(a, c, -__fmul_rn(b, s)));
      base[h * dh + i1] = __float2bfloat16_rn(__fmaf_rn(a, s, __fmul_rn(b, c)));
    }
  }
}

// The same with 16-byte accesses: heads, rotated halves (or, paired, the rotated lanes) and rows in multiples of 8 elements. A block per token; the
// angles are worked out once and wait in shared memory, then a thread turns 8 pairs of one head at a time, two heads in flight. The kernel above moves
// 2 bytes per access: 116 us for 40 heads of 128 lanes at 16384 tokens (335 MB), against 80 us here.
template <bool PAIRED>
__global__ void __launch_bounds__(512) rope_vec_kernel(__nv_bfloat16* __restrict__ x, const int* __restrict__ pos, const float* __restrict__ inv_ts,
                                                       int heads, int dh, int n_rot, int rot_dim, int inverse) {
  extern __shared__ __align__(16) float2 cs[];              // rot_dim / 2 angles
  const long tok = blockIdx.x;
  const int half = rot_dim / 2, nt = blockDim.x;
  const int per_head = (PAIRED ? rot_dim : half) / 8, items = n_rot * per_head;
  __nv_bfloat16* base = x + tok * (long)heads * dh;
  bf16x8 u[2], w[2];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = i0 + k * nt;
      if (i < items) {
        const __nv_bfloat16* at = base + (i / per_head) * dh + (i % per_head) * 8;
        u[k] = *reinterpret_cast<const bf16x8*>(at);
        if (!PAIRED) w[k] = *reinterpret_cast<const bf16x8*>(at + half);
      }
    }
  };
  fetch(threadIdx.x);                                       // on their way while the angles are worked out
  const float p = (float)pos[tok];
  for (int j = threadIdx.x; j < half; j += nt) {
    float s, c;
    sincosf(p * inv_ts[j], &s, &c);
    cs[j] = make_float2(c, inverse ? -s : s);
  }
  __syncthreads();
  auto low = [](float a, float b, float2 c) { return __fmaf_rn(a, c.x, -__fmul_rn(b, c.y)); };
  auto high = [](float a, float b, float2 c) { return __fmaf_rn(a, c.y, __fmul_rn(b, c.x)); };
  for (int i0 = threadIdx.x; i0 < items; i0 += 2 * nt) {
    if (i0 >= 2 * nt) fetch(i0);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = i0 + k * nt;
      if (i < items) {
        const int j = (i % per_head) * 8;
        __nv_bfloat16* at = base + (i / per_head) * dh + j;
        float a[8], b[8], o[8];
        unpack8(u[k], a);
        if (PAIRED) {
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const float2 c = cs[(j + e) / 2];
            o[e] = low(a[e], a[e + 1], c);
            o[e + 1] = high(a[e], a[e + 1], c);
          }
          *reinterpret_cast<bf16x8*>(at) = pack8(o);
        } else {
          unpack8(w[k], b);
          float t[8];
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const float4 c = *reinterpret_cast<const float4*>(cs + j + e);
            o[e] = low(a[e], b[e], make_float2(c.x, c.y));
            t[e] = high(a[e], b[e], make_float2(c.x, c.y));
            o[e + 1] = low(a[e + 1], b[e + 1], make_float2(c.z, c.w));
            t[e + 1] = high(a[e + 1], b[e + 1], make_float2(c.z, c.w));
          }
          *reinterpret_cast<bf16x8*>(at) = pack8(o);
          *reinterpret_cast<bf16x8*>(at + half) = pack8(t);
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ gated activation
__device__ __forceinline__ float act_apply(float g, int code) {
  switch (code) {
    case 0: return g / (1.f + __expf(-g));                                                         // silu
    case 1: { const float k = 0.7978845608028654f; return 0.5f * g * (1.f + tanhf(k * (g + 0.044715f * g * g * g))); }  // gelu (tanh)
    case 2: return g > 0.f ? g : 0.f;                                                              // relu
    default: return g;                                                                             // linear
  }
}
__device__ __forceinline__ float act_grad(float g, int code) {
  switch (code) {
    case 0: { const float s = 1.f / (1.f + __expf(-g)); return s * (1.f + g * (1.f - s)); }
    case 1: {
      const float k = 0.7978845608028654f;
      const float u = k * (g + 0.044715f * g * g * g);
      const float t = tanhf(u);
      return 0.5f * (1.f + t) + 0.5f * g * (1.f - t * t) * k * (1.f + 3.f * 0.044715f * g * g);
    }
    case 2: return g > 0.f ? 1.f : 0.f;
    default: return 1.f;
  }
}

// gu [rows, 2F] = [gate | up] -> out [rows, F]. Bandwidth-bound: a thread takes a 16-byte column of two rows at a time, so that it has four (backward: six)
// loads in flight and no index to divide; a block is as wide as the row needs (gated_block) and takes several pairs of rows where that is less than 256
// threads. One vector per thread out of a flat index with 64-bit divisions took 281 us forward and 479 us backward for 16384 x 14336 and 51 and 80 us for
// 24576 x 1408; 217, 360, 43 and 68 us here (6.5 TB/s). A division of the block's index for its row and column cost 30 and 10 us at the first size.
template <int CODE>
__global__ void __launch_bounds__(256) gated_act_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, long rows, int F) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  const long r = ((blockIdx.z * (long)gridDim.y + blockIdx.y) * blockDim.y + threadIdx.y) * 2;
  if (c >= F) return;
  bf16x8 g[2], u[2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (r + k < rows) {
      g[k] = *reinterpret_cast<const bf16x8*>(gu + (r + k) * 2 * F + c);
      u[k] = *reinterpret_cast<const bf16x8*>(gu + (r + k) * 2 * F + F + c);
    }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (r + k < rows) {
      float a[8], b[8], o[8];
      unpack8(g[k], a);
      unpack8(u[k], b);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = act_apply(a[e], CODE) * b[e];
      *reinterpret_cast<bf16x8*>(out + (r + k) * F + c) = pack8(o);
    }
}

template <int CODE>
__global__ void __launch_bounds__(256, 5) gated_act_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ gu,
                                                            __nv_bfloat16* __restrict__ dgu, long rows, int F) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  const long r = ((blockIdx.z * (long)gridDim.y + blockIdx.y) * blockDim.y + threadIdx.y) * 2;
  if (c >= F) return;
  bf16x8 g[2], u[2], d[2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (r + k < rows) {
      g[k] = *reinterpret_cast<const bf16x8*>(gu + (r + k) * 2 * F + c);
      u[k] = *reinterpret_cast<const bf16x8*>(gu + (r + k) * 2 * F + F + c);
      d[k] = *reinterpret_cast<const bf16x8*>(dy + (r + k) * F + c);
    }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (r + k < rows) {
      float a[8], b[8], t[8], dg[8], du[8];
      unpack8(g[k], a);
      unpack8(u[k], b);
      unpack8(d[k], t);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        dg[e] = t[e] * b[e] * act_grad(a[e], CODE);
        du[e] = t[e] * act_apply(a[e], CODE);
      }
      *reinterpret_cast<bf16x8*>(dgu + (r + k) * 2 * F + c) = pack8(dg);
      *reinterpret_cast<bf16x8*>(dgu + (r + k) * 2 * F + F + c) = pack8(du);
    }
}

// ------------------------------------------------------------------------------------------------ embedding
__global__ void embedding_fwd_kernel(const int* __restrict__ tok, const __nv_bfloat16* __restrict__ table,
                                     __nv_bfloat16* __restrict__ out, int D, int V) {
  const long t = blockIdx.x;
  int id = tok[t];
  id = id < 0 ? 0 : (id >= V ? V - 1 : id);
  const uint4* src = reinterpret_cast<const uint4*>(table + (long)id * D);
  uint4* dst = reinterpret_cast<uint4*>(out + t * D);
  for (int i = threadIdx.x; i < D / 8; i += blockDim.x) dst[i] = src[i];
}

__global__ void embedding_bwd_kernel(const int* __restrict__ tok, const __nv_bfloat16* __restrict__ dy, float* __restrict__ dtable,
                                     int D, int V) {
  const long t = blockIdx.x;
  int id = tok[t];
  if (id < 0 || id >= V) return;
  for (int i = threadIdx.x; i < D; i += blockDim.x) atomicAdd(dtable + (long)id * D + i, __bfloat162float(dy[t * D + i]));
}

// ------------------------------------------------------------------------------------------------ heads of latent attention
// What latent attention does between its projections and the attention kernel, in one pass over a token:
//   q [H, nope + rope] -> [q_nope | rot(q_rope)] * scale;   k = [kv_nope | rot(kr) for every head];   v = the rest of kv [H, nope + vd]
// with the roundings of the separate steps (after the rotation and after the scale), and the way back: dkr sums over the heads. Bandwidth-bound: a thread
// moves 16-byte columns (rotated ones in pairs). As rotations, concatenations, products, copies and their zero-filled gradients it was about 70 launches and
// 1.0 ms of a training step of two layers at 4096 tokens (16 heads of 128 + 64 and 128); six launches of 41 us now.
struct LatentHeads {
  int H, nope, rope, vd;
  long ldkr;                            // row stride of kr
  float scale;
  const int* pos;
  const float* inv_ts;
};
__device__ __forceinline__ bf16x8 scaled8(const bf16x8& p, float scale) {
  float f[8];
  unpack8(p, f);
#pragma unroll
  for (int e = 0; e < 8; ++e) f[e] *= scale;
  return pack8(f);
}
// lanes j .. j + 7 of a rotated row (PAIRED: neighbours turn together; otherwise lane j with lane j + rope / 2, and `b` holds the second ones)
template <bool PAIRED>
__device__ __forceinline__ void turn8(const float2* cs, int j, bf16x8& a, bf16x8& b) {
  float x[8], y[8], o[8], t[8];
  unpack8(a, x);
  if (PAIRED) {
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const float2 c = cs[(j + e) / 2];
      o[e] = __fmaf_rn(x[e], c.x, -__fmul_rn(x[e + 1], c.y));
      o[e + 1] = __fmaf_rn(x[e], c.y, __fmul_rn(x[e + 1], c.x));
    }
    a = pack8(o);
  } else {
    unpack8(b, y);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float2 c = cs[j + e];
      o[e] = __fmaf_rn(x[e], c.x, -__fmul_rn(y[e], c.y));
      t[e] = __fmaf_rn(x[e], c.y, __fmul_rn(y[e], c.x));
    }
    a = pack8(o);
    b = pack8(t);
  }
}
__device__ __forceinline__ bf16x8 ld8(const __nv_bfloat16* p) { return *reinterpret_cast<const bf16x8*>(p); }
__device__ __forceinline__ void st8(__nv_bfloat16* p, const bf16x8& v) { *reinterpret_cast<bf16x8*>(p) = v; }

template <bool PAIRED>
__global__ void __launch_bounds__(256) latent_heads_fwd_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ kr,
                                                               const __nv_bfloat16* __restrict__ kv, __nv_bfloat16* __restrict__ qo,
                                                               __nv_bfloat16* __restrict__ k, __nv_bfloat16* __restrict__ v, const LatentHeads a) {
  extern __shared__ __align__(16) float2 cs[];
  const long n = blockIdx.x;
  const int half = a.rope / 2, qk = a.nope + a.rope, kvw = a.nope + a.vd;
  const float p = (float)a.pos[n];
  for (int j = threadIdx.x; j < half; j += blockDim.x) {
    float s, c;
    sincosf(p * a.inv_ts[j], &s, &c);
    cs[j] = make_float2(c, s);
  }
  __syncthreads();
  const int un = a.nope / 8, ur = (PAIRED ? a.rope : half) / 8, uv = a.vd / 8, per = un + ur + uv;
  for (int i = threadIdx.x; i < a.H * per; i += blockDim.x) {
    const int h = i / per, u = i % per;
    const __nv_bfloat16 *qh = q + (n * a.H + h) * qk, *kvh = kv + (n * a.H + h) * kvw;
    __nv_bfloat16 *qoh = qo + (n * a.H + h) * qk, *kh = k + (n * a.H + h) * qk;
    if (u < un) {
      st8(qoh + u * 8, scaled8(ld8(qh + u * 8), a.scale));
      st8(kh + u * 8, ld8(kvh + u * 8));
    } else if (u < un + ur) {
      const int j = (u - un) * 8;
      bf16x8 x = ld8(qh + a.nope + j), y, r = ld8(kr + n * a.ldkr + j), t;
      if (!PAIRED) { y = ld8(qh + a.nope + j + half); t = ld8(kr + n * a.ldkr + j + half); }
      turn8<PAIRED>(cs, j, x, y);
      turn8<PAIRED>(cs, j, r, t);
      st8(qoh + a.nope + j, scaled8(x, a.scale));
      st8(kh + a.nope + j, r);
      if (!PAIRED) {
        st8(qoh + a.nope + j + half, scaled8(y, a.scale));
        st8(kh + a.nope + j + half, t);
      }
    } else {
      const int j = (u - un - ur) * 8;
      st8(v + (n * a.H + h) * a.vd + j, ld8(kvh + a.nope + j));
    }
  }
}

template <bool PAIRED>
__global__ void __launch_bounds__(256) latent_heads_bwd_kernel(const __nv_bfloat16* __restrict__ dqo, const __nv_bfloat16* __restrict__ dk,
                                                               const __nv_bfloat16* __restrict__ dv, __nv_bfloat16* __restrict__ dq,
                                                               __nv_bfloat16* __restrict__ dkr, __nv_bfloat16* __restrict__ dkv, const LatentHeads a) {
  extern __shared__ __align__(16) float2 cs[];
  const long n = blockIdx.x;
  const int half = a.rope / 2, qk = a.nope + a.rope, kvw = a.nope + a.vd;
  __nv_bfloat16* sum = reinterpret_cast<__nv_bfloat16*>(cs + half);          // [rope]
  const float p = (float)a.pos[n];
  for (int j = threadIdx.x; j < half; j += blockDim.x) {
    float s, c;
    sincosf(p * a.inv_ts[j], &s, &c);
    cs[j] = make_float2(c, -s);
  }
  for (int j = threadIdx.x; j < a.rope; j += blockDim.x) {
    float t = 0.f;
    for (int h = 0; h < a.H; ++h) t += __bfloat162float(dk[(n * a.H + h) * qk + a.nope + j]);
    sum[j] = __float2bfloat16_rn(t);
  }
  __syncthreads();
  const int un = a.nope / 8, ur = (PAIRED ? a.rope : half) / 8, uv = a.vd / 8, per = un + ur + uv;
  for (int i = threadIdx.x; i < a.H * per + ur; i += blockDim.x) {
    const int h = i / per, u = i % per;
    if (h == a.H) {                                          // the shared rotated key
      const int j = u * 8;
      bf16x8 x = ld8(sum + j), y;
      if (!PAIRED) y = ld8(sum + j + half);
      turn8<PAIRED>(cs, j, x, y);
      st8(dkr + n * a.rope + j, x);
      if (!PAIRED) st8(dkr + n * a.rope + j + half, y);
      continue;
    }
    const __nv_bfloat16 *gq = dqo + (n * a.H + h) * qk, *gk = dk + (n * a.H + h) * qk;
    __nv_bfloat16 *oq = dq + (n * a.H + h) * qk, *okv = dkv + (n * a.H + h) * kvw;
    if (u < un) {
      st8(oq + u * 8, scaled8(ld8(gq + u * 8), a.scale));
      st8(okv + u * 8, ld8(gk + u * 8));
    } else if (u < un + ur) {
      const int j = (u - un) * 8;
      bf16x8 x = scaled8(ld8(gq + a.nope + j), a.scale), y;
      if (!PAIRED) y = scaled8(ld8(gq + a.nope + j + half), a.scale);
      turn8<PAIRED>(cs, j, x, y);
      st8(oq + a.nope + j, x);
      if (!PAIRED) st8(oq + a.nope + j + half, y);
    } else {
      const int j = (u - un - ur) * 8;
      st8(okv + a.nope + j, ld8(dv + (n * a.H + h) * a.vd + j));
    }
  }
}

}  // namespace mt

// ================================================================================================ launchers
using namespace mt;

template <int TPR>
static void launch_rms_fwd(const void* x, const void* add, void* sum, const void* scale, float eps, float offset, void* y, float* rstd, int rows, int D,
                           int sms, cudaStream_t st) {
  const int vpt = (D / 8 + TPR - 1) / TPR;
  const int threads = 256;
  const int rpb = threads / TPR, blocks = (rows + rpb - 1) / rpb;
  const int most = sms * rms_fwd_resident(TPR, vpt, add != nullptr), grid = blocks < most ? blocks : most;   // what is resident at once, so that all blocks have the same rows
#define K(V, A) rmsnorm_fwd_kernel<TPR, V, A><<<grid, threads, 0, st>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)add, (__nv_bfloat16*)sum, \
                                                                        (const __nv_bfloat16*)scale, eps, offset, (__nv_bfloat16*)y, rstd, rows, D)
#define L(V) do { if (add) K(V, true); else K(V, false); } while (0)
  if (vpt <= 1) L(1); else if (vpt <= 2) L(2); else if (vpt <= 4) L(4); else L(8);
#undef L
#undef K
}

// add, sum: both null, or the residual add in front of the norm
extern "C" int mt_rmsnorm_fwd(const void* x, const void* add, void* sum, const void* scale, float eps, float offset, void* y, float* rstd, int rows,
                              int D, int sms, cudaStream_t st) {
  if (D % 8 || D > 8 * 256 * 8 || !add != !sum) return -1;
  if (D <= 512) launch_rms_fwd<32>(x, add, sum, scale, eps, offset, y, rstd, rows, D, sms, st);
  else launch_rms_fwd<256>(x, add, sum, scale, eps, offset, y, rstd, rows, D, sms, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

static int rms_bwd_grid(int rows, int tpr, int sms) {
  const int rpb = 256 / tpr;
  long groups = ((long)rows + rpb - 1) / rpb;
  int grid = (int)(groups < (long)sms * 4 ? groups : (long)sms * 4);
  return grid < 1 ? 1 : grid;
}

template <int TPR>
static void launch_rms_bwd(const void* dy, const void* x, const void* scale, const float* rstd, float offset, const void* dres, void* dx,
                           float* dscale, float* partial, int rows, int D, int sms, cudaStream_t st) {
  const int vpt = (D / 8 + TPR - 1) / TPR;
  const int threads = 256;
  const int grid = rms_bwd_grid(rows, TPR, sms);
  float* part = dscale ? partial : nullptr;
#define L(V) rmsnorm_bwd_kernel<TPR, V><<<grid, threads, 0, st>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,                 \
                                                                  (const __nv_bfloat16*)scale, rstd, offset,                        \
                                                                  (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, part, rows, D)
  if (vpt <= 1) L(1); else if (vpt <= 2) L(2); else if (vpt <= 4) L(4); else L(8);
#undef L
  if (!part) return;
  const int prows = grid * (threads / TPR);
  if (D >= 1024 && D % 32 == 0) rms_dscale_reduce_kernel<32><<<D / 32, 256, 0, st>>>(part, prows, D, dscale);
  else rms_dscale_reduce_kernel<8><<<D / 8, 256, 0, st>>>(part, prows, D, dscale);
}

// number of fp32 rows of length D that `partial` must hold for mt_rmsnorm_bwd with a scale gradient
extern "C" int mt_rmsnorm_bwd_partial_rows(int rows, int D, int sms) {
  const int tpr = D <= 512 ? 32 : 256;
  return rms_bwd_grid(rows, tpr, sms) * (256 / tpr);
}

// `partial`: scratch of mt_rmsnorm_bwd_partial_rows(rows, D, sms) x D floats (needed only when dscale is given); rows of a
// block that saw no input row are written as zeros by the kernel, so the scratch needs no clearing.
extern "C" int mt_rmsnorm_bwd(const void* dy, const void* x, const void* scale, const float* rstd, float offset, const void* dres,
                              void* dx, float* dscale, float* partial, int rows, int D, int sms, cudaStream_t st) {
  if (D % 8 || D > 8 * 256 * 8 || (dscale && !partial)) return -1;
  if (D <= 512) launch_rms_bwd<32>(dy, x, scale, rstd, offset, dres, dx, dscale, partial, rows, D, sms, st);
  else launch_rms_bwd<256>(dy, x, scale, rstd, offset, dres, dx, dscale, partial, rows, D, sms, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int mt_rope(void* x, const int* pos, const float* inv_ts, long tokens, int heads, int dh, int n_rot, int rot_dim,
                       int interleaved, int inverse, cudaStream_t st) {
  if (tokens <= 0) return 0;
  const int step = interleaved ? 8 : 16;
  // One or two heads (a shared rotated key) give the 16-byte kernel no bytes to save, only a barrier and shared memory to wait for: 13.1 us against 15.1 for
  // 16384 tokens with 1 or 2 heads of 64 or 128; with 4 heads 14.1 against 13.6, with 8 17.7 against 13.1.
  if (n_rot > 2 && rot_dim % step == 0 && dh % 8 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 && rot_dim <= 4096) {
    auto k = interleaved ? rope_vec_kernel<true> : rope_vec_kernel<false>;
    const int items = n_rot * (interleaved ? rot_dim : rot_dim / 2) / 8, want = ((items + 1) / 2 + 31) / 32 * 32;     // two items per thread if they fit
    k<<<(unsigned)tokens, want < 32 ? 32 : want > 512 ? 512 : want, rot_dim / 2 * sizeof(float2), st>>>((__nv_bfloat16*)x, pos, inv_ts, heads, dh, n_rot, rot_dim, inverse);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
  }
  int threads = rot_dim / 2;
  threads = threads < 32 ? 32 : (threads > 256 ? 256 : threads);
  rope_kernel<<<(unsigned)tokens, threads, 0, st>>>((__nv_bfloat16*)x, pos, inv_ts, heads, dh, n_rot, rot_dim, interleaved, inverse);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Threads along a row: its 16-byte columns over as few blocks as 256 threads allow, evenly; what is left of the 256 takes further pairs of rows. (Blocks
// of 256 columns whatever the width left 62 to 95 % of the threads without work below 768 lanes.)
static dim3 gated_block(int F) {
  const int n = F / 8, blocks = (n + 255) / 256, x = (n + blocks - 1) / blocks;
  return dim3((unsigned)x, (unsigned)(256 / x));
}
static dim3 gated_grid(long rows, int F) {       // y and z count the groups of rows: y alone ends at 65535
  const dim3 b = gated_block(F);
  const long groups = (rows + 2 * b.y - 1) / (2 * b.y), z = (groups + 65534) / 65535;
  return dim3((F / 8 + b.x - 1) / b.x, (unsigned)((groups + z - 1) / z), (unsigned)z);
}

extern "C" int mt_gated_act_fwd(const void* gu, void* out, long rows, int F, int code, cudaStream_t st) {
  if (F % 8) return -1;
  if (rows <= 0 || F <= 0) return 0;
  auto k = code == 0 ? gated_act_fwd_kernel<0> : code == 1 ? gated_act_fwd_kernel<1> : code == 2 ? gated_act_fwd_kernel<2> : gated_act_fwd_kernel<3>;
  k<<<gated_grid(rows, F), gated_block(F), 0, st>>>((const __nv_bfloat16*)gu, (__nv_bfloat16*)out, rows, F);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int mt_gated_act_bwd(const void* dy, const void* gu, void* dgu, long rows, int F, int code, cudaStream_t st) {
  if (F % 8) return -1;
  if (rows <= 0 || F <= 0) return 0;
  auto k = code == 0 ? gated_act_bwd_kernel<0> : code == 1 ? gated_act_bwd_kernel<1> : code == 2 ? gated_act_bwd_kernel<2> : gated_act_bwd_kernel<3>;
  k<<<gated_grid(rows, F), gated_block(F), 0, st>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)gu, (__nv_bfloat16*)dgu, rows, F);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int mt_embedding_fwd(const int* tok, const void* table, void* out, long tokens, int D, int V, cudaStream_t st) {
  if (D % 8) return -1;
  if (tokens <= 0) return 0;
  embedding_fwd_kernel<<<(unsigned)tokens, 128, 0, st>>>(tok, (const __nv_bfloat16*)table, (__nv_bfloat16*)out, D, V);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int mt_embedding_bwd(const int* tok, const void* dy, float* dtable, long tokens, int D, int V, cudaStream_t st) {
  if (tokens <= 0) return 0;
  embedding_bwd_kernel<<<(unsigned)tokens, 256, 0, st>>>(tok, (const __nv_bfloat16*)dy, dtable, D, V);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Widths in multiples of 8 (rotated halves too), pointers and the row stride of kr aligned to 16 bytes.
extern "C" int mt_latent_heads_ok(int nope, int rope, int vd, int paired) {
  return nope > 0 && rope > 0 && vd > 0 && nope % 8 == 0 && vd % 8 == 0 && rope % (paired ? 8 : 16) == 0 && rope <= 2048;
}

// backward 0: q, kr, kv -> qo, k, v.  backward 1: dqo, dk, dv -> dq, dkr [tokens, rope], dkv.
extern "C" int mt_latent_heads(int backward, const void* in0, const void* in1, const void* in2, void* out0, void* out1, void* out2, const int* pos,
                               const float* inv_ts, long tokens, int H, int nope, int rope, int vd, long ldkr, float scale, int paired, cudaStream_t st) {
  if (!mt_latent_heads_ok(nope, rope, vd, paired) || H < 1 || ldkr % 8) return -1;
  if (tokens <= 0) return 0;
  const LatentHeads a{H, nope, rope, vd, ldkr, scale, pos, inv_ts};
  const int smem = rope / 2 * (int)sizeof(float2) + rope * 2;
  using B = __nv_bfloat16;
  auto k = backward ? (paired ? latent_heads_bwd_kernel<true> : latent_heads_bwd_kernel<false>)
                    : (paired ? latent_heads_fwd_kernel<true> : latent_heads_fwd_kernel<false>);
  k<<<(unsigned)tokens, 256, smem, st>>>((const B*)in0, (const B*)in1, (const B*)in2, (B*)out0, (B*)out1, (B*)out2, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
