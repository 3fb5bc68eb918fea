// Learned right preconditioner: device kernels of the edge message-passing
// network (included into solver.cu inside its anonymous namespace).
//
// The preconditioner has no reference counterpart; it sits where
// CRS<T>::PrecondBackSolve sits (ucs/crs.tcc:591).  Network (sizes and the
// parameter layout are fixed by the PCFD_LP_* constants of pcfd.h):
//   h0   = ReLU(Win x + bin)                                   11 -> 64
//   m_i  = (1/deg_i) sum_j (We e_ij + ce) * h_j   (per channel)
//   h'   = ReLU(Ws h + Wm m + b)                               128 -> 64, x3
//   out  = Wout h3 + bout                                      64 -> 5
// Matrices are BF16 (rounded from the FP32 master copy), biases and all
// accumulation FP32, activations h and m stored BF16.  The 128-row layer
// products [h | m] (128 x 128) x [Ws | Wm]^T (128 x 64) and, in the backward
// pass, dz (128 x 64) x [Ws | Wm] (64 x 128) run on the tensor cores
// (tcgen05.mma, accumulator in TMEM); the weight image reaches shared memory
// through the bulk copy engine.  Gathers, the encoder, the decoder and the
// weight gradients run on the FP32 pipes.
#pragma once

#include "umma.cuh"

constexpr int LP_NIN = PCFD_LP_NIN;
constexpr int LP_H = PCFD_LP_HIDDEN;
constexpr int LP_NE = PCFD_LP_NEDGE;
constexpr int LP_NOUT = PCFD_LP_NOUT;
constexpr int LP_NL = PCFD_LP_LAYERS;
constexpr int LP_OFF_WIN = 0;
constexpr int LP_OFF_BIN = LP_H * LP_NIN;
constexpr int LP_OFF_L0 = LP_OFF_BIN + LP_H;
constexpr int LP_L_WE = 0;
constexpr int LP_L_CE = LP_H * LP_NE;
constexpr int LP_L_WS = LP_L_CE + LP_H;
constexpr int LP_L_WM = LP_L_WS + LP_H * LP_H;
constexpr int LP_L_B = LP_L_WM + LP_H * LP_H;
constexpr int LP_L_SIZE = LP_L_B + LP_H;
constexpr int LP_OFF_WOUT = LP_OFF_L0 + LP_NL * LP_L_SIZE;
constexpr int LP_OFF_BOUT = LP_OFF_WOUT + LP_NOUT * LP_H;
constexpr int LP_NPARAM = LP_OFF_BOUT + LP_NOUT;
static_assert(LP_NPARAM == PCFD_LP_NPARAM, "parameter layout");

constexpr int LP_TILE = 128;                        // nodes per CTA (MMA M)
constexpr int LP_THREADS = 256;                     // 8 warps
constexpr int LP_IMG = LP_H * 2 * LP_H;             // BF16 values in one weight image (64 x 128)
constexpr uint32_t LP_IMG_BYTES = LP_IMG * 2;       // 16 KiB
constexpr int LP_ERR_TIMEOUT = 1;
constexpr int LP_FLIGHT = 8;                        // neighbour rows in flight in a half-warp's gather

// shared memory of the layer kernels: A tile, weight image, barriers
constexpr size_t LP_SMEM_A = (size_t)LP_TILE * 2 * LP_H * 2;  // 32 KiB
constexpr size_t LP_SMEM = 1024 + LP_SMEM_A + LP_IMG_BYTES + 64;

__device__ __forceinline__ float bfr(float v) { return __bfloat162float(__float2bfloat16(v)); }

struct LpSmem {
  unsigned char* a;   // A operand tile (K-major canonical)
  unsigned char* b;   // weight image
  uint64_t* bar_w;    // bulk-copy completion
  uint64_t* bar_mma;  // MMA completion
  uint32_t* tmem_holder;
};
__device__ __forceinline__ LpSmem lp_smem(unsigned char* raw) {
  uintptr_t base = (reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023);
  LpSmem s;
  s.a = reinterpret_cast<unsigned char*>(base);
  s.b = s.a + LP_SMEM_A;
  s.bar_w = reinterpret_cast<uint64_t*>(s.b + LP_IMG_BYTES);
  s.bar_mma = s.bar_w + 1;
  s.tmem_holder = reinterpret_cast<uint32_t*>(s.bar_mma + 1);
  return s;
}

// Start of a layer kernel: barriers, the weight image copy, TMEM columns.
__device__ __forceinline__ void lp_begin(const LpSmem& sm, const __nv_bfloat16* img, uint32_t ncols) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    umma::mbar_init(sm.bar_w, 1);
    umma::mbar_init(sm.bar_mma, 1);
    umma::fence_mbar_init();
  }
  __syncthreads();
  if (tid == 0) {
    umma::mbar_expect_tx(sm.bar_w, LP_IMG_BYTES);
    umma::bulk_g2s(sm.b, img, LP_IMG_BYTES, sm.bar_w);
  }
  if ((tid >> 5) == 0) umma::tmem_alloc(sm.tmem_holder, ncols);
}

// After the A tile is written: one thread issues the K/16 MMAs and commits.
// Returns the TMEM address; *ok is false when a bounded wait expired.
template <int K, int N>
__device__ __forceinline__ uint32_t lp_mma(const LpSmem& sm, bool* ok) {
  umma::fence_async_smem();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *sm.tmem_holder;
  bool good = true;
  if (threadIdx.x == 0) {
    good = umma::mbar_wait(sm.bar_w, 0);
    if (good) {
      constexpr uint32_t idesc = umma::idesc_bf16(LP_TILE, N);
      const uint32_t a0 = umma::smem_addr(sm.a), b0 = umma::smem_addr(sm.b);
#pragma unroll
      for (int ks = 0; ks < K / 16; ks++) {
        const uint64_t ad = umma::smem_desc(a0 + ks * 256, 128, (K / 8) * 128);
        const uint64_t bd = umma::smem_desc(b0 + ks * 256, 128, (K / 8) * 128);
        umma::mma_bf16(tmem, ad, bd, idesc, ks > 0 ? 1u : 0u);
      }
      umma::mma_commit(sm.bar_mma);
    }
  }
  // every thread waits (bounded) for the accumulator
  good = __syncthreads_and(good ? 1 : 0) != 0;
  if (good) good = umma::mbar_wait(sm.bar_mma, 0);
  umma::fence_after_sync();
  *ok = good;
  return tmem;
}

__device__ __forceinline__ void lp_end(uint32_t tmem, uint32_t ncols) {
  umma::fence_before_sync();
  __syncthreads();
  if ((threadIdx.x >> 5) == 0) umma::tmem_dealloc(tmem, ncols);
}

// gates of channels c .. c + 3, as two channel pairs
struct Gate4 {
  float2 w[4][2], c[2];
};
__device__ __forceinline__ Gate4 load_gate(const float* __restrict__ wl, int c) {
  Gate4 g;
#pragma unroll
  for (int p = 0; p < 2; p++) {
    const int c0 = c + 2 * p;
#pragma unroll
    for (int k = 0; k < 4; k++)
      g.w[k][p] = make_float2(bfr(wl[LP_L_WE + c0 * LP_NE + k]), bfr(wl[LP_L_WE + (c0 + 1) * LP_NE + k]));
    g.c[p] = make_float2(wl[LP_L_CE + c0], wl[LP_L_CE + c0 + 1]);
  }
  return g;
}

// Packed FP32 fused multiply-add of two lanes (PTX fma.rn.f32x2): each half
// is rounded as fmaf rounds it.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(d)
      : "l"(*reinterpret_cast<const uint64_t*>(&a)), "l"(*reinterpret_cast<const uint64_t*>(&b)),
        "l"(*reinterpret_cast<const uint64_t*>(&c)));
  return *reinterpret_cast<const float2*>(&d);
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// gate of channel pair p for edge features e
__device__ __forceinline__ float2 gate_eval(const Gate4& g, int p, float4 e) {
  return fma2(g.w[3][p], both(e.w),
              fma2(g.w[2][p], both(e.z), fma2(g.w[1][p], both(e.y), fma2(g.w[0][p], both(e.x), g.c[p]))));
}
__device__ __forceinline__ float4 shfl4(float4 v, int src) {
  return make_float4(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                     __shfl_sync(0xffffffffu, v.z, src), __shfl_sync(0xffffffffu, v.w, src));
}

// four BF16 values in one 8-byte word
__device__ __forceinline__ void unpack4(uint2 u, float2 f[2]) {
  f[0] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  f[1] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
}
__device__ __forceinline__ uint2 pack4(float2 a, float2 b) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(a.x, a.y), q = __floats2bfloat162_rn(b.x, b.y);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&p), *reinterpret_cast<const uint32_t*>(&q));
}

// A half-warp's row of the edge graph: its entries p0 .. p1 - 1 and the first
// 16 of its neighbours (lane k of the half holds the k-th: index and edge
// features).
struct HalfRow {
  int p0, p1, jl;
  float4 el;
};
__device__ __forceinline__ void half_fetch(int p, int p1, int lane, const int* __restrict__ nnbr,
                                           const float4* __restrict__ ef, int& jl, float4& el) {
  jl = 0;
  el = make_float4(0.f, 0.f, 0.f, 0.f);
  if ((lane & 15) < p1 - p) {
    jl = nnbr[p + (lane & 15)];
    el = ef[p + (lane & 15)];
  }
}

// four channels of the A tile's row r from column k on (k a multiple of 4)
__device__ __forceinline__ void st_a4(unsigned char* a, int r, int k, int K, uint2 v) {
  *reinterpret_cast<uint2*>(a + umma::tile_offset(r, k, K)) = v;
}

// ---------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------

// node features (pcfd_lp_features): y/sigma, state, log volume
__global__ void k_lp_features(int n, const double* __restrict__ y, const double* __restrict__ sigma_dev,
                              const double* __restrict__ q, const double* __restrict__ vol, double rho_inf,
                              double p_inf, double c_inf, double vmean, float* __restrict__ x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double sigma = *sigma_dev;
  const double isig = sigma > 0.0 ? 1.0 / sigma : 0.0;
  const double* Q = &q[(size_t)i * NVARS];
  float* xi = &x[(size_t)i * LP_NIN];
#pragma unroll
  for (int k = 0; k < 5; k++) xi[k] = (float)(y[(size_t)i * 5 + k] * isig);
  xi[5] = (float)(Q[0] / rho_inf - 1.0);
  xi[6] = (float)(Q[7] / c_inf);
  xi[7] = (float)(Q[8] / c_inf);
  xi[8] = (float)(Q[9] / c_inf);
  xi[9] = (float)(Q[6] / p_inf - 1.0);
  xi[10] = (float)log(vol[i] / vmean);
}

// sigma = sqrt(sum / count) from the k_sumsq partials
__global__ void k_lp_sigma(int nparts, const double* __restrict__ part, double count, double* __restrict__ sigma) {
  __shared__ double red[256];
  double a = 0.0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) a += part[i];
  red[threadIdx.x] = a;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *sigma = sqrt(red[0] / count);
}

// Encoder: a warp per node, lane l channels 2 l and 2 l + 1 with their weights
// in registers; the node's features arrive in one load and are shuffled
// (40,960 nodes: 23 us with the weights read at every node, 11 now).
__global__ void __launch_bounds__(256) k_lp_encode(int n, const float* __restrict__ x, const float* __restrict__ w,
                                                   __nv_bfloat16* __restrict__ h0) {
  const int lane = threadIdx.x & 31, c = 2 * lane;
  float2 wr[LP_NIN];
#pragma unroll
  for (int k = 0; k < LP_NIN; k++)
    wr[k] = make_float2(bfr(w[LP_OFF_WIN + c * LP_NIN + k]), bfr(w[LP_OFF_WIN + (c + 1) * LP_NIN + k]));
  const float2 bias = make_float2(w[LP_OFF_BIN + c], w[LP_OFF_BIN + c + 1]);
  const int nwarps = gridDim.x * (blockDim.x >> 5);
#pragma unroll 4
  for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += nwarps) {
    const float xl = lane < LP_NIN ? x[(size_t)i * LP_NIN + lane] : 0.f;
    float2 a = bias;
#pragma unroll
    for (int k = 0; k < LP_NIN; k++) a = fma2(wr[k], both(__shfl_sync(0xffffffffu, xl, k)), a);
    *reinterpret_cast<__nv_bfloat162*>(&h0[(size_t)i * LP_H + c]) =
        __floats2bfloat162_rn(fmaxf(a.x, 0.f), fmaxf(a.y, 0.f));
  }
}

// m for up to 16 neighbours of a row a half-warp: lane k of the half holds the
// k-th neighbour's index jl and edge features el; cnt of them are valid, most
// those of the warp's longer row.  The loads of LP_FLIGHT neighbour rows are
// issued together, then summed in neighbour order (the order of the sequential
// sum).  A slot past a row's end reads row 0 and adds a product with zero: a
// branch per neighbour, in which the halves differ, measured 72 us a layer
// of 40,960 nodes instead of 38.
__device__ __forceinline__ void lp_gather_block(const Gate4& g, const __nv_bfloat16* __restrict__ h_in, int c, int hb,
                                                int jl, float4 el, int cnt, int most, float2 (&acc)[2]) {
  for (int t = 0; t < most; t += LP_FLIGHT) {
    uint2 raw[LP_FLIGHT];
#pragma unroll
    for (int u = 0; u < LP_FLIGHT; u++) {
      const int j = __shfl_sync(0xffffffffu, jl, hb + t + u);
      raw[u] = *reinterpret_cast<const uint2*>(&h_in[(size_t)j * LP_H + c]);
    }
#pragma unroll
    for (int u = 0; u < LP_FLIGHT; u++) {
      const float4 e = shfl4(el, hb + t + u);
      float2 hh[2];
      unpack4(t + u < cnt ? raw[u] : make_uint2(0u, 0u), hh);
#pragma unroll
      for (int p = 0; p < 2; p++) acc[p] = fma2(gate_eval(g, p, e), hh[p], acc[p]);
    }
  }
}

// One message-passing layer for ROWS nodes (128, or 64 in the upper half of the
// MMA's rows).  Gather phase: warp w builds rows ROWS / 8 w .. of A = [h | m],
// two at a time: a half-warp has a row and each of its lanes four channels, so
// an index, an edge feature or a row address is handled once for two rows.
// The warp's row pointers arrive in one load; a row's neighbour indices and
// edge features arrive in one load, issued while the previous rows are
// gathered.  Then one 128x64x128 MMA, and the epilogue (a row per thread, TMEM
// read 16 columns at a time) adds the bias, applies ReLU and stores h' in
// BF16; the last layer also applies the decoder and writes either out (FP32)
// or z = y + sigma * out (FP64).
// Bound by issue (47 %) and by the shared-memory port (55 %: shuffles).  A row
// a warp took 23.6 M warp instructions and 49 us for 40,960 nodes, this takes
// 14.8 M and 38 us.
// 64 rows halve the chain of row pairs a warp goes through, 128 rows halve the
// weight images and MMAs: a forward and backward pass with 64 / 128 takes 174 /
// 202 us for 900 nodes, 222 / 247 for 5,120, 454 / 453 for 40,960, 1162 / 1151
// for 147,456 and 7955 / 7538 for 1,179,648, so 64 up to two tiles of 128 rows
// a multiprocessor.
template <bool LAST, int ROWS>
__global__ void __launch_bounds__(LP_THREADS, ROWS == LP_TILE ? 3 : 2) k_lp_layer(
    int n, const int* __restrict__ nptr, const int* __restrict__ nnbr, const float4* __restrict__ ef,
    const float* __restrict__ invdeg, const __nv_bfloat16* __restrict__ h_in, const float* __restrict__ wl,
    const __nv_bfloat16* __restrict__ img, __nv_bfloat16* __restrict__ h_out, __nv_bfloat16* __restrict__ m_out,
    const float* __restrict__ w, float* __restrict__ out, const double* __restrict__ y,
    const double* __restrict__ sigma_dev, double* __restrict__ z, int* __restrict__ err) {
  extern __shared__ unsigned char lp_raw[];
  const LpSmem sm = lp_smem(lp_raw);
  constexpr int K = 2 * LP_H;
  constexpr int RPW = ROWS / 8;  // rows per warp
  lp_begin(sm, img, LP_H);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hb = lane & 16, half = lane >> 4, c = 4 * (lane & 15);
  const int base = blockIdx.x * ROWS;
  const int r0 = warp * RPW;
  {
    const Gate4 g = load_gate(wl, c);
    // lane k <= RPW holds nptr of row r0 + k (nptr has n + 1 entries)
    int pl = 0;
    if (lane <= RPW && base + r0 + lane <= n) pl = nptr[base + r0 + lane];
    auto fetch = [&](int rr) {
      HalfRow f;
      f.p0 = __shfl_sync(0xffffffffu, pl, rr + half);
      f.p1 = __shfl_sync(0xffffffffu, pl, rr + half + 1);
      if (base + r0 + rr + half >= n) f.p1 = f.p0;
      half_fetch(f.p0, f.p1, lane, nnbr, ef, f.jl, f.el);
      return f;
    };
    HalfRow f = fetch(0);
    for (int rr = 0; rr < RPW; rr += 2) {
      const int r = r0 + rr + half;
      const int i = base + r;
      uint2 hv = make_uint2(0u, 0u), mv = hv;
      float id = 0.f;
      if (i < n) {
        hv = *reinterpret_cast<const uint2*>(&h_in[(size_t)i * LP_H + c]);
        id = invdeg[i];
      }
      HalfRow fn = f;
      if (rr + 2 < RPW) fn = fetch(rr + 2);
      float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      for (int o = 0;; o += 16) {
        const int cnt = f.p1 - f.p0 - o, most = __reduce_max_sync(0xffffffffu, cnt);
        if (most <= 0) break;
        if (o) half_fetch(f.p0 + o, f.p1, lane, nnbr, ef, f.jl, f.el);  // neighbours past the first 16
        lp_gather_block(g, h_in, c, hb, f.jl, f.el, cnt, min(most, 16), acc);
      }
      if (i < n) {
        mv = pack4(make_float2(acc[0].x * id, acc[0].y * id), make_float2(acc[1].x * id, acc[1].y * id));
        if (m_out) *reinterpret_cast<uint2*>(&m_out[(size_t)i * LP_H + c]) = mv;
      }
      st_a4(sm.a, r, c, K, hv);
      st_a4(sm.a, r, LP_H + c, K, mv);
      f = fn;
    }
  }
  bool ok;
  const uint32_t tmem = lp_mma<K, LP_H>(sm, &ok);
  if (!ok) {
    if (threadIdx.x == 0) atomicExch(err, LP_ERR_TIMEOUT);
  } else if (warp < ROWS / 32) {
    const int r = warp * 32 + lane;
    const int i = base + r;
    float o[LP_NOUT];
#pragma unroll
    for (int oo = 0; oo < LP_NOUT; oo++) o[oo] = LAST ? w[LP_OFF_BOUT + oo] : 0.f;
#pragma unroll
    for (int cc = 0; cc < LP_H; cc += 16) {
      float v[16];
      umma::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + cc, v);
      if (i < n) {
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = bfr(fmaxf(v[k] + wl[LP_L_B + cc + k], 0.f));
        if (!LAST || h_out) {
          uint4* dst = reinterpret_cast<uint4*>(&h_out[(size_t)i * LP_H + cc]);
#pragma unroll
          for (int q8 = 0; q8 < 2; q8++) {
            __nv_bfloat162 b0 = __floats2bfloat162_rn(v[8 * q8], v[8 * q8 + 1]);
            __nv_bfloat162 b1 = __floats2bfloat162_rn(v[8 * q8 + 2], v[8 * q8 + 3]);
            __nv_bfloat162 b2 = __floats2bfloat162_rn(v[8 * q8 + 4], v[8 * q8 + 5]);
            __nv_bfloat162 b3 = __floats2bfloat162_rn(v[8 * q8 + 6], v[8 * q8 + 7]);
            uint4 u;
            u.x = *reinterpret_cast<uint32_t*>(&b0);
            u.y = *reinterpret_cast<uint32_t*>(&b1);
            u.z = *reinterpret_cast<uint32_t*>(&b2);
            u.w = *reinterpret_cast<uint32_t*>(&b3);
            dst[q8] = u;
          }
        }
        if (LAST) {
#pragma unroll
          for (int oo = 0; oo < LP_NOUT; oo++)
#pragma unroll
            for (int k = 0; k < 16; k++) o[oo] = fmaf(bfr(w[LP_OFF_WOUT + oo * LP_H + cc + k]), v[k], o[oo]);
        }
      }
    }
    if (LAST && i < n) {
      if (out) {
#pragma unroll
        for (int oo = 0; oo < LP_NOUT; oo++) out[(size_t)i * LP_NOUT + oo] = o[oo];
      }
      if (z) {
        const double sg = *sigma_dev;
#pragma unroll
        for (int oo = 0; oo < LP_NOUT; oo++) z[(size_t)i * 5 + oo] = y[(size_t)i * 5 + oo] + sg * (double)o[oo];
      }
    }
  }
  lp_end(tmem, LP_H);
}

// ---------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------

// Per-block partial sums of every backward kernel -> the gradient, in one
// launch at the end of the pass.  Eight warps split the blocks of 32
// consecutive entries into runs, each summed in order, and the eight sums are
// added in order: a fixed order (deterministic).  Latency bound: eight launches
// with one thread per entry took 181 us of a 40,960-node pass, eight of this
// form 69 us, one 12.
constexpr int LP_RED_RUNS = 8;
constexpr int LP_NSEG = 2 * LP_NL + 2;
struct LpSegments {
  int nblk[LP_NSEG], len[LP_NSEG], first[LP_NSEG + 1];  // partial arrays, entries each, first block of the launch
  const float* part[LP_NSEG];
  float* grad[LP_NSEG];
};
__global__ void __launch_bounds__(32 * LP_RED_RUNS) k_lp_reduce(LpSegments sg) {
  __shared__ float red[LP_RED_RUNS][32];
  const int lane = threadIdx.x & 31, run = threadIdx.x >> 5;
  int q = 0;
  while (q + 1 < LP_NSEG && (int)blockIdx.x >= sg.first[q + 1]) q++;
  const int len = sg.len[q], k = (blockIdx.x - sg.first[q]) * 32 + lane;
  const int per = (sg.nblk[q] + LP_RED_RUNS - 1) / LP_RED_RUNS;
  const int b0 = run * per, b1 = min(sg.nblk[q], b0 + per);
  const float* __restrict__ part = sg.part[q] + k;
  float a = 0.f;
  if (k < len) {
#pragma unroll 8
    for (int b = b0; b < b1; b++) a += part[(size_t)b * len];
  }
  red[run][lane] = a;
  __syncthreads();
  if (run == 0 && k < len) {
    float t = red[0][lane];
#pragma unroll
    for (int w = 1; w < LP_RED_RUNS; w++) t += red[w][lane];
    sg.grad[q][k] = t;
  }
}

// block-wide sum of narr arrays in shared memory: red[narr][len] -> out
__device__ __forceinline__ void lp_block_sum(float* red, int narr, int len, float* out) {
  __syncthreads();
  for (int k = threadIdx.x; k < len; k += blockDim.x) {
    float a = 0.f;
    for (int w = 0; w < narr; w++) a += red[w * len + k];
    out[k] = a;
  }
}

// decoder backward: dout = 2 (out - t) / (5 n); dh3 = Wout^T dout; partials
// of dWout, dbout and the loss.  Warp per node stripe, lane = channel pair.
constexpr int LP_DEC_LEN = LP_NOUT * LP_H + LP_NOUT + 1;
__global__ void __launch_bounds__(256) k_lp_dec_bwd(int n, const float* __restrict__ out, const float* __restrict__ t,
                                                    const __nv_bfloat16* __restrict__ h3, const float* __restrict__ w,
                                                    float* __restrict__ dh, float* __restrict__ part) {
  __shared__ float red[8 * LP_DEC_LEN];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = 2 * lane;
  const float scale = 2.0f / (5.0f * (float)n);
  float gw0[LP_NOUT] = {0}, gw1[LP_NOUT] = {0}, gb[LP_NOUT] = {0}, gl = 0.f;
  float wo0[LP_NOUT], wo1[LP_NOUT];
#pragma unroll
  for (int o = 0; o < LP_NOUT; o++) {
    wo0[o] = bfr(w[LP_OFF_WOUT + o * LP_H + c]);
    wo1[o] = bfr(w[LP_OFF_WOUT + o * LP_H + c + 1]);
  }
  const int nwarps = gridDim.x * (blockDim.x >> 5);
  for (int i = blockIdx.x * (blockDim.x >> 5) + warp; i < n; i += nwarps) {
    float d[LP_NOUT];
#pragma unroll
    for (int o = 0; o < LP_NOUT; o++) {
      const float r = out[(size_t)i * LP_NOUT + o] - t[(size_t)i * LP_NOUT + o];
      d[o] = scale * r;
      gl = fmaf(r, r, gl);
      gb[o] += d[o];
    }
    const float2 hv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&h3[(size_t)i * LP_H + c]));
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int o = 0; o < LP_NOUT; o++) {
      a0 = fmaf(wo0[o], d[o], a0);
      a1 = fmaf(wo1[o], d[o], a1);
      gw0[o] = fmaf(d[o], hv.x, gw0[o]);
      gw1[o] = fmaf(d[o], hv.y, gw1[o]);
    }
    *reinterpret_cast<float2*>(&dh[(size_t)i * LP_H + c]) = make_float2(a0, a1);
  }
  float* my = red + warp * LP_DEC_LEN;
#pragma unroll
  for (int o = 0; o < LP_NOUT; o++) {
    my[o * LP_H + c] = gw0[o];
    my[o * LP_H + c + 1] = gw1[o];
  }
  if (lane == 0) {
#pragma unroll
    for (int o = 0; o < LP_NOUT; o++) my[LP_NOUT * LP_H + o] = gb[o];
  }
  // loss: sum over lanes is 32x the node sum (every lane saw every node)
  if (lane == 0) my[LP_NOUT * LP_H + LP_NOUT] = gl;
  lp_block_sum(red, 8, LP_DEC_LEN, part + (size_t)blockIdx.x * LP_DEC_LEN);
}

// Layer backward on the tensor cores: dz = BF16(dh * (h' > 0)) (stored for
// the weight gradients), then [dh_self | dm] = dz x [Ws | Wm] (128 x 128), dm
// stored divided by the node's degree, as every neighbour reads it.  Bound by
// the rows' latency and by writing them (40,960 nodes: 21 us with one row's
// loads in flight a warp, 15 with eight).
__global__ void __launch_bounds__(LP_THREADS) k_lp_layer_bwd(int n, const float* __restrict__ dh,
                                                             const __nv_bfloat16* __restrict__ h_out,
                                                             const __nv_bfloat16* __restrict__ img,
                                                             const float* __restrict__ invdeg,
                                                             __nv_bfloat16* __restrict__ dz_out,
                                                             float* __restrict__ dh_self, float* __restrict__ dm,
                                                             int* __restrict__ err) {
  extern __shared__ unsigned char lp_raw[];
  const LpSmem sm = lp_smem(lp_raw);
  constexpr int K = LP_H;
  lp_begin(sm, img, 2 * LP_H);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = 4 * (lane & 15);
  const int base = blockIdx.x * LP_TILE;
  // two rows a warp at a time, the loads of eight rows in flight together
#pragma unroll
  for (int q = 0; q < LP_TILE / 64; q++) {
    float4 d[4];
    uint2 h[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = base + warp * (LP_TILE / 8) + 8 * q + 2 * u + (lane >> 4);
      d[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      h[u] = make_uint2(0u, 0u);
      if (i < n) {
        d[u] = *reinterpret_cast<const float4*>(&dh[(size_t)i * LP_H + c]);
        h[u] = *reinterpret_cast<const uint2*>(&h_out[(size_t)i * LP_H + c]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int r = warp * (LP_TILE / 8) + 8 * q + 2 * u + (lane >> 4);
      float2 hv[2];
      unpack4(h[u], hv);
      const uint2 dv = pack4(make_float2(hv[0].x > 0.f ? d[u].x : 0.f, hv[0].y > 0.f ? d[u].y : 0.f),
                             make_float2(hv[1].x > 0.f ? d[u].z : 0.f, hv[1].y > 0.f ? d[u].w : 0.f));
      if (base + r < n) *reinterpret_cast<uint2*>(&dz_out[(size_t)(base + r) * LP_H + c]) = dv;
      st_a4(sm.a, r, c, K, dv);
    }
  }
  bool ok;
  const uint32_t tmem = lp_mma<K, 2 * LP_H>(sm, &ok);
  if (!ok) {
    if (threadIdx.x == 0) atomicExch(err, LP_ERR_TIMEOUT);
  } else {
    // 8 warps: warp w reads TMEM lanes 32 (w % 4).., columns 64 (w / 4)..
    const int r = (warp & 3) * 32 + lane;
    const int i = base + r;
    const int half = warp >> 2;
    float v[LP_H];
#pragma unroll
    for (int cc = 0; cc < LP_H; cc += 16)
      umma::tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + half * LP_H + cc, v + cc);
    if (i < n) {
      if (half) {
        const float id = invdeg[i];
#pragma unroll
        for (int k = 0; k < LP_H; k++) v[k] *= id;
      }
      float4* dst = reinterpret_cast<float4*>((half == 0 ? dh_self : dm) + (size_t)i * LP_H);
#pragma unroll
      for (int q4 = 0; q4 < LP_H / 4; q4++) dst[q4] = make_float4(v[4 * q4], v[4 * q4 + 1], v[4 * q4 + 2], v[4 * q4 + 3]);
    }
  }
  lp_end(tmem, 2 * LP_H);
}

// Transpose of the gather: dh_j = dh_self_j + sum_{i in N(j)} g_ij dm_i (dm
// already divided by deg_i) with g_ij the gate seen from i (normal flipped);
// partials of dWe and dce.  As in the layer kernel a half-warp has a node and
// a lane four channels, and eight neighbour rows are in flight together
// (40,960 nodes: a node a warp 45 us, 34 now).
constexpr int LP_GB_LEN = LP_H * LP_NE + LP_H;
constexpr int LP_GB_SM = 2;  // blocks per multiprocessor
__global__ void __launch_bounds__(256, LP_GB_SM) k_lp_gather_bwd(
    int n, const int* __restrict__ nptr, const int* __restrict__ nnbr, const float4* __restrict__ ef,
    const __nv_bfloat16* __restrict__ h_in, const float* __restrict__ wl, const float* __restrict__ dh_self,
    const float* __restrict__ dm, float* __restrict__ dh_next, float* __restrict__ part) {
  __shared__ float red[16 * LP_GB_LEN];
  const int lane = threadIdx.x & 31, hw = threadIdx.x >> 4, hb = lane & 16, c = 4 * (lane & 15);
  const Gate4 g = load_gate(wl, c);
  const float2 zero = make_float2(0.f, 0.f), one = make_float2(1.f, 1.f);
  float2 gw[4][2], gc[2] = {zero, zero};
#pragma unroll
  for (int k = 0; k < 4; k++) gw[k][0] = gw[k][1] = zero;
  auto fetch = [&](int j) {
    HalfRow f;
    f.p0 = f.p1 = 0;
    if (j < n) {
      f.p0 = nptr[j];
      f.p1 = nptr[j + 1];
    }
    half_fetch(f.p0, f.p1, lane, nnbr, ef, f.jl, f.el);
    return f;
  };
  const int step = gridDim.x * 16;
  int j = blockIdx.x * 16 + hw;
  HalfRow f = fetch(j);
  while (j - (hw & 1) < n) {  // the warp's first node
    float2 acc[2] = {zero, zero}, hj[2] = {zero, zero};
    if (j < n) {
      const float4 s4 = *reinterpret_cast<const float4*>(&dh_self[(size_t)j * LP_H + c]);
      acc[0] = make_float2(s4.x, s4.y);
      acc[1] = make_float2(s4.z, s4.w);
      unpack4(*reinterpret_cast<const uint2*>(&h_in[(size_t)j * LP_H + c]), hj);
    }
    const HalfRow fn = fetch(j + step);
    for (int o = 0;; o += 16) {
      const int cnt = f.p1 - f.p0 - o, most = __reduce_max_sync(0xffffffffu, cnt);
      if (most <= 0) break;
      if (o) half_fetch(f.p0 + o, f.p1, lane, nnbr, ef, f.jl, f.el);  // neighbours past the first 16
      for (int t = 0; t < min(most, 16); t += LP_FLIGHT) {
        float4 d[LP_FLIGHT];
#pragma unroll
        for (int u = 0; u < LP_FLIGHT; u++) {
          const int i = __shfl_sync(0xffffffffu, f.jl, hb + t + u);
          d[u] = *reinterpret_cast<const float4*>(&dm[(size_t)i * LP_H + c]);
          if (t + u >= cnt) d[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < LP_FLIGHT; u++) {
          float4 e = shfl4(f.el, hb + t + u);
          {
            e.x = -e.x;
            e.y = -e.y;
            e.z = -e.z;
#pragma unroll
            for (int p = 0; p < 2; p++) {
              const float2 dp = p ? make_float2(d[u].z, d[u].w) : make_float2(d[u].x, d[u].y);
              acc[p] = fma2(gate_eval(g, p, e), dp, acc[p]);
              const float2 dg = make_float2(dp.x * hj[p].x, dp.y * hj[p].y);
              gc[p] = fma2(dg, one, gc[p]);
              gw[0][p] = fma2(dg, both(e.x), gw[0][p]);
              gw[1][p] = fma2(dg, both(e.y), gw[1][p]);
              gw[2][p] = fma2(dg, both(e.z), gw[2][p]);
              gw[3][p] = fma2(dg, both(e.w), gw[3][p]);
            }
          }
        }
      }
    }
    if (j < n)
      *reinterpret_cast<float4*>(&dh_next[(size_t)j * LP_H + c]) = make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
    j += step;
    f = fn;
  }
  float* my = red + hw * LP_GB_LEN;
#pragma unroll
  for (int p = 0; p < 2; p++) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      my[(c + 2 * p) * LP_NE + k] = gw[k][p].x;
      my[(c + 2 * p + 1) * LP_NE + k] = gw[k][p].y;
    }
    my[LP_H * LP_NE + c + 2 * p] = gc[p].x;
    my[LP_H * LP_NE + c + 2 * p + 1] = gc[p].y;
  }
  lp_block_sum(red, 16, LP_GB_LEN, part + (size_t)blockIdx.x * LP_GB_LEN);
}

// Weight gradients of one layer on the FP32 pipes: dWs = dz^T h, dWm = dz^T m,
// db = sum dz.  A block takes a run of nodes in chunks of 32, the next chunk's
// rows on their way to registers while one is summed.  Thread (cg, kg) owns
// rows 4 cg .. + 3 and columns 4 kg .. + 3 of both halves of [h | m], 32
// entries in packed FP32 FMAs: a node costs it three 16-byte shared-memory
// reads and 16 FMAs where a row of 32 columns a thread took 33 reads and 32
// FMAs.  A warp's reads cover 8 cg x 4 kg, neighbouring 16 bytes: no bank
// conflicts.  Bound by the shared-memory
// port (82 %).  40,960 nodes: 90 us before, 20 now.
// A run of LP_WG_RUN nodes is summed on its own and added to the block's sums:
// a block's whole share in one FP32 accumulator, 3,881 nodes of a mesh of
// 1,179,648, lets its roundings grow with the mesh (the backward pass of that
// mesh 4.76 ms with it, 4.78 with runs).
constexpr int LP_WG_LEN = LP_H * 2 * LP_H + LP_H;
constexpr int LP_WG_CHUNK = 32;
constexpr int LP_WG_RUN = 256;
__global__ void __launch_bounds__(256, 2) k_lp_wgrad(int n, int nodes_per_block, const __nv_bfloat16* __restrict__ dz,
                                                     const __nv_bfloat16* __restrict__ h,
                                                     const __nv_bfloat16* __restrict__ m, float* __restrict__ part) {
  __shared__ __align__(16) float sdz[LP_WG_CHUNK][LP_H];
  __shared__ __align__(16) float sh[LP_WG_CHUNK][LP_H];
  __shared__ __align__(16) float smm[LP_WG_CHUNK][LP_H];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int cg = (warp & 1) * 8 + (lane >> 2), kg = (warp >> 1) * 4 + (lane & 3);
  static_assert(LP_H == 64 && LP_WG_CHUNK * LP_H == 256 * 8, "thread tile");
  const int n0 = blockIdx.x * nodes_per_block;
  const int n1 = min(n, n0 + nodes_per_block);
  // [row][column pair: h 0 1, h 2 3, m 0 1, m 2 3], the run's and the block's
  float2 acc[4][4], sum[4][4];
  float accb[4] = {0.f, 0.f, 0.f, 0.f}, sumb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int k = 0; k < 4; k++) acc[r][k] = sum[r][k] = make_float2(0.f, 0.f);
  // eight consecutive channels of one row of each array a thread
  const int fr = t >> 3, fc = (t & 7) * 8;
  uint4 v[3];
  auto fetch = [&](int cb) {
    const int i = cb + fr;
    const size_t o = (size_t)i * LP_H + fc;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    v[0] = i < n1 ? *reinterpret_cast<const uint4*>(dz + o) : zero;
    v[1] = i < n1 ? *reinterpret_cast<const uint4*>(h + o) : zero;
    v[2] = i < n1 ? *reinterpret_cast<const uint4*>(m + o) : zero;
  };
  auto put = [&](float* dst, const uint4& u) {
    const __nv_bfloat162* q = reinterpret_cast<const __nv_bfloat162*>(&u);
    const float2 f0 = __bfloat1622float2(q[0]), f1 = __bfloat1622float2(q[1]);
    const float2 f2 = __bfloat1622float2(q[2]), f3 = __bfloat1622float2(q[3]);
    reinterpret_cast<float4*>(dst)[0] = make_float4(f0.x, f0.y, f1.x, f1.y);
    reinterpret_cast<float4*>(dst)[1] = make_float4(f2.x, f2.y, f3.x, f3.y);
  };
  fetch(n0);
  for (int cb = n0; cb < n1; cb += LP_WG_CHUNK) {
    __syncthreads();
    put(&sdz[fr][fc], v[0]);
    put(&sh[fr][fc], v[1]);
    put(&smm[fr][fc], v[2]);
    __syncthreads();
    fetch(cb + LP_WG_CHUNK);
    const int nr = min(LP_WG_CHUNK, n1 - cb);
#pragma unroll 4
    for (int r = 0; r < nr; r++) {
      const float4 d4 = *reinterpret_cast<const float4*>(&sdz[r][4 * cg]);
      const float4 h4 = *reinterpret_cast<const float4*>(&sh[r][4 * kg]);
      const float4 m4 = *reinterpret_cast<const float4*>(&smm[r][4 * kg]);
      const float d[4] = {d4.x, d4.y, d4.z, d4.w};
      const float2 b[4] = {make_float2(h4.x, h4.y), make_float2(h4.z, h4.w), make_float2(m4.x, m4.y),
                           make_float2(m4.z, m4.w)};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (kg == 0) accb[q] += d[q];
#pragma unroll
        for (int k = 0; k < 4; k++) acc[q][k] = fma2(make_float2(d[q], d[q]), b[k], acc[q][k]);
      }
    }
    if ((cb - n0) % LP_WG_RUN == LP_WG_RUN - LP_WG_CHUNK || cb + LP_WG_CHUNK >= n1) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        sumb[q] += accb[q];
        accb[q] = 0.f;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          sum[q][k].x += acc[q][k].x;
          sum[q][k].y += acc[q][k].y;
          acc[q][k] = make_float2(0.f, 0.f);
        }
      }
    }
  }
  // [Ws | Wm] rows
  float* out = part + (size_t)blockIdx.x * LP_WG_LEN;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int c = 4 * cg + q;
#pragma unroll
    for (int half = 0; half < 2; half++)
      *reinterpret_cast<float4*>(&out[half * LP_H * LP_H + c * LP_H + 4 * kg]) =
          make_float4(sum[q][2 * half].x, sum[q][2 * half].y, sum[q][2 * half + 1].x, sum[q][2 * half + 1].y);
    if (kg == 0) out[2 * LP_H * LP_H + c] = sumb[q];
  }
}

// Encoder backward: dz0 = dh0 (h0 > 0); dWin = dz0^T x, dbin = sum dz0.  A
// warp takes every eighth node of the block's run, lane l channels 2 l and
// 2 l + 1; the node's features arrive in one load and are shuffled, the loads
// of four nodes are in flight together (40,960 nodes: 104 us with one node at
// a time, 9 now).
constexpr int LP_EB_LEN = LP_H * LP_NIN + LP_H;
__global__ void __launch_bounds__(256) k_lp_enc_bwd(int n, int nodes_per_block, const float* __restrict__ dh,
                                                    const __nv_bfloat16* __restrict__ h0, const float* __restrict__ x,
                                                    float* __restrict__ part) {
  __shared__ float red[8 * LP_EB_LEN];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = 2 * lane;
  float2 acc[LP_NIN + 1];  // the last one is the bias
#pragma unroll
  for (int k = 0; k <= LP_NIN; k++) acc[k] = make_float2(0.f, 0.f);
  const int n0 = blockIdx.x * nodes_per_block;
  const int n1 = min(n, n0 + nodes_per_block);
  for (int ib = n0 + warp; ib < n1; ib += 32) {
    float2 d[4];
    __nv_bfloat162 hv[4];
    float xl[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = ib + 8 * u;
      d[u] = make_float2(0.f, 0.f);
      hv[u] = __floats2bfloat162_rn(0.f, 0.f);
      xl[u] = 0.f;
      if (i < n1) {
        d[u] = *reinterpret_cast<const float2*>(&dh[(size_t)i * LP_H + c]);
        hv[u] = *reinterpret_cast<const __nv_bfloat162*>(&h0[(size_t)i * LP_H + c]);
        xl[u] = lane < LP_NIN ? x[(size_t)i * LP_NIN + lane] : 1.f;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const float2 h = __bfloat1622float2(hv[u]);
      const float2 g = make_float2(h.x > 0.f ? d[u].x : 0.f, h.y > 0.f ? d[u].y : 0.f);
#pragma unroll
      for (int k = 0; k <= LP_NIN; k++) acc[k] = fma2(g, both(__shfl_sync(0xffffffffu, xl[u], k)), acc[k]);
    }
  }
  float* my = red + warp * LP_EB_LEN;
#pragma unroll
  for (int k = 0; k < LP_NIN; k++) {
    my[c * LP_NIN + k] = acc[k].x;
    my[(c + 1) * LP_NIN + k] = acc[k].y;
  }
  my[LP_H * LP_NIN + c] = acc[LP_NIN].x;
  my[LP_H * LP_NIN + c + 1] = acc[LP_NIN].y;
  lp_block_sum(red, 8, LP_EB_LEN, part + (size_t)blockIdx.x * LP_EB_LEN);
}

// ---------------------------------------------------------------------------
// parameters
// ---------------------------------------------------------------------------

// BF16 weight images for the tensor cores, per layer: forward [Ws | Wm] as a
// 64 x 128 K-major tile, backward [Ws | Wm]^T as a 128 x 64 K-major tile.
__global__ void k_lp_pack(const float* __restrict__ w, __nv_bfloat16* __restrict__ fwd,
                          __nv_bfloat16* __restrict__ bwd) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= LP_NL * LP_IMG) return;
  const int l = t / LP_IMG, e = t % LP_IMG;
  const float* wl = w + LP_OFF_L0 + l * LP_L_SIZE;
  {
    const int r = e / (2 * LP_H), k = e % (2 * LP_H);
    const float v = k < LP_H ? wl[LP_L_WS + r * LP_H + k] : wl[LP_L_WM + r * LP_H + (k - LP_H)];
    *reinterpret_cast<__nv_bfloat16*>(reinterpret_cast<unsigned char*>(fwd + (size_t)l * LP_IMG) +
                                      umma::tile_offset(r, k, 2 * LP_H)) = __float2bfloat16(v);
  }
  {
    const int r = e / LP_H, k = e % LP_H;  // row r of [Ws | Wm]^T, column k = output channel
    const float v = r < LP_H ? wl[LP_L_WS + k * LP_H + r] : wl[LP_L_WM + k * LP_H + (r - LP_H)];
    *reinterpret_cast<__nv_bfloat16*>(reinterpret_cast<unsigned char*>(bwd + (size_t)l * LP_IMG) +
                                      umma::tile_offset(r, k, LP_H)) = __float2bfloat16(v);
  }
}

__global__ void k_lp_adam(int np, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m1,
                          float* __restrict__ m2, float lr, float b1, float b2, float eps, float bc1, float bc2) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= np) return;
  const float gk = g[k];
  const float a = b1 * m1[k] + (1.f - b1) * gk;
  const float b = b2 * m2[k] + (1.f - b2) * gk * gk;
  m1[k] = a;
  m2[k] = b;
  w[k] -= lr * (a / bc1) / (sqrtf(b / bc2) + eps);
}

// oriented edge features and 1/deg of every node
__global__ void k_lp_graph(int n, const int* __restrict__ nptr, const int* __restrict__ nedg,
                           const int2* __restrict__ en, const D4* __restrict__ ea, const double* __restrict__ xyz,
                           double lmean, float4* __restrict__ ef, float* __restrict__ invdeg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int p0 = nptr[i], p1 = nptr[i + 1];
  invdeg[i] = p1 > p0 ? 1.0f / (float)(p1 - p0) : 0.f;
  for (int p = p0; p < p1; p++) {
    const int se = nedg[p];
    const int e = se < 0 ? ~se : se;
    const float sg = se < 0 ? 1.f : -1.f;  // ~e marks the edge's first node
    const int2 nd = en[e];
    const double dx = xyz[3 * nd.y] - xyz[3 * nd.x], dy = xyz[3 * nd.y + 1] - xyz[3 * nd.x + 1],
                 dz = xyz[3 * nd.y + 2] - xyz[3 * nd.x + 2];
    const D4 a = ea[e];
    ef[p] = make_float4(sg * (float)a.x, sg * (float)a.y, sg * (float)a.z,
                        (float)(sqrt(dx * dx + dy * dy + dz * dz) / lmean));
  }
}

// t = (dq - y) / sigma in FP32 (training target)
__global__ void k_lp_target(long long n5, const double* __restrict__ dq, const double* __restrict__ y,
                            const double* __restrict__ sigma_dev, float* __restrict__ t) {
  const double sg = *sigma_dev;
  const double is = sg > 0.0 ? 1.0 / sg : 0.0;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n5; k += (long long)gridDim.x * blockDim.x)
    t[k] = (float)((dq[k] - y[k]) * is);
}
