// Matrix products of the 16/32-bit decoder layers, each with its layer's elementwise work in the epilogue:
//
//   fr_dense_proj       every projection of the normalised input h as ONE product with the merged weight; the
//                       column ranges leave through their own epilogues (plain store, store into KV-cache
//                       slots, SwiGLU or clamped GLU of interleaved gate / up rows, sigmoid with bias, GELU
//                       times a looked-up row)
//   fr_dense_gated_add  x += g1 * (A1 W1^T) + g2 * (A2 W2^T) on the fp32 residual stream
//
// Three implementations behind each:
//   dense_tc_kernel    bf16, persistent and warp-specialised like gemm_fp8.cu: warp 0 = TMA producer (128-byte
//                      swizzle, 64 bf16 per row), warp 1 = tcgen05.mma issuer (kind::f16, M = 128, fp32
//                      accumulators in TMEM, two buffers), warps 2..9 = epilogue
//   dense_rows_kernel  M <= 8 (decode of one or two rows, few columns, short K, f32): a warp streams four weight rows against all
//                      M activations, so the weights cross HBM once; the warps of a CTA may split K
//   dense_simt_kernel  f32 with more rows: tiles of 64 or 128 x 64, fp32 FMAs
#include "fr_common.cuh"
#include "sm100_ptx.cuh"

namespace fr {

int* device_status_ptr();  // capi.cu

namespace dense {

constexpr int kMaxSegs = 12;
struct Segs {
  fr_out_segment s[kMaxSegs];
  int n;
};
struct Parts {
  fr_gated_part p[2];
  int n;
};

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// eight consecutive elements as fp32
__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void unpack8(const uint4& a, float (&v)[8]) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&v)[8]) {
  unpack8(*reinterpret_cast<const uint4*>(p), v);
}

// z * sigmoid(z) and sigmoid(z); FAST: the bf16 epilogues, whose result is rounded to 8 bits
template <bool FAST>
__device__ __forceinline__ float sigmoid_f(float z) {
  return FAST ? __fdividef(1.0f, 1.0f + __expf(-z)) : 1.0f / (1.0f + expf(-z));
}
template <bool FAST>
__device__ __forceinline__ float silu_f(float z) { return z * sigmoid_f<FAST>(z); }

// gelu with the tanh approximation: 0.5 z (1 + tanh(u)) = z sigmoid(2 u)
template <bool FAST>
__device__ __forceinline__ float gelu_tanh_f(float z) {
  constexpr float kRoot = 0.7978845608028654f;  // sqrt(2 / pi)
  return z * sigmoid_f<FAST>(2.0f * kRoot * (z + 0.044715f * z * z * z));
}

// Ranges whose weight rows come in [32 gate | 32 up] blocks, and the activation of a pair.
__host__ __device__ __forceinline__ bool paired(const fr_out_segment& s) {
  return s.kind == FR_SEG_SWIGLU || s.kind == FR_SEG_GLU_CLAMP;
}
template <bool FAST>
__device__ __forceinline__ float pair_act(const fr_out_segment& s, float g, float u) {
  if (s.kind == FR_SEG_SWIGLU) return silu_f<FAST>(g) * u;
  g = fminf(g, s.limit);
  u = fminf(fmaxf(u, -s.limit), s.limit);
  return g * sigmoid_f<FAST>(s.alpha * g) * (u + s.up_bias);
}

__device__ __forceinline__ int seg_of(const Segs& sg, int col) {
  int i = 0;
#pragma unroll 1
  while (i + 1 < sg.n && col >= sg.s[i + 1].n0) ++i;
  return i;
}

// One value of one column range (column index within the range, already combined for SWIGLU).
template <typename T, bool FAST>
__device__ __forceinline__ void seg_write(const fr_out_segment& s, int64_t row, int c, float z) {
  if (c >= s.n) return;
  const int64_t r = s.row_map != nullptr ? s.row_map[row] : row;
  if (s.kind == FR_SEG_STORE_F32) {
    static_cast<float*>(s.out)[r * s.ldo + c] = z;
    return;
  }
  if (s.kind == FR_SEG_SIGMOID) z = sigmoid_f<FAST>(z + (s.bias != nullptr ? s.bias[c] : 0.f));
  if (s.kind == FR_SEG_GELU_MUL)
    z = gelu_tanh_f<FAST>(z) * to_f<T>(static_cast<const T*>(s.mul)[(s.mul_map != nullptr ? s.mul_map[row] : row) * s.ld_mul + c]);
  static_cast<T*>(s.out)[r * s.ldo + c] = from_f<T>(z);
}

// ---------------------------------------------------------------------------
// M <= 8: a warp takes four weight rows; KS warps of the CTA share them along K
// ---------------------------------------------------------------------------
constexpr int kRowsThreads = 256;

// Four weight rows (pointers) against MB activation rows, this warp's chunks of 256 columns. The first P chunks of weights are loaded
// by begin(), before griddepcontrol.wait, where the caller says that the launch ahead does not write them (FR_DENSE_LAID_OUT), so that
// the products begin as soon as the activations are there. us per launch in a row of launches on new weights, P = 0 / chunks ahead,
// one row: 32768 x 2048 25.6 / 23.6, 2048 x 2048 2.9 / 2.5, 8320 x 4096 14.2 / 13.1; f32 12288 x 2048 20.5 / 17.3. From three rows on
// the registers for the weights cost more than that gave (eight rows of bf16 x 20480 x 2048 61.0 / 66.6).
template <typename T, int MB, int P>
struct RowsDot {
  static constexpr int kVec = 8 * sizeof(T) / 16;  // 16-byte loads of a lane's eight columns
  uint4 ahead[P > 0 ? P : 1][4][kVec];

  static __device__ __forceinline__ void load(uint4 (&raw)[4][kVec], const T* const (&w)[4], int k) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int v = 0; v < kVec; ++v) raw[r][v] = __ldcs(reinterpret_cast<const uint4*>(w[r] + k) + v);
  }
  static __device__ __forceinline__ void add(const uint4 (&raw)[4][kVec], const T* __restrict__ a, int64_t lda, int k, int M,
                                             float (&acc)[4][MB]) {
    float wv[4][8];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if constexpr (sizeof(T) == 2) {
        unpack8(raw[r][0], wv[r]);
      } else {
#pragma unroll
        for (int v = 0; v < kVec; ++v) {
          wv[r][4 * v] = __uint_as_float(raw[r][v].x);
          wv[r][4 * v + 1] = __uint_as_float(raw[r][v].y);
          wv[r][4 * v + 2] = __uint_as_float(raw[r][v].z);
          wv[r][4 * v + 3] = __uint_as_float(raw[r][v].w);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      float av[8];
      load8(a + (m < M ? m : 0) * lda + k, av);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[r][m] = fmaf(wv[r][i], av[i], acc[r][m]);
    }
  }

  __device__ __forceinline__ void begin(const T* const (&w)[4], int K, int kwarp, int ks) {
#pragma unroll
    for (int c = 0; c < P; ++c) {
      const int k = (kwarp + c * ks) * 256 + (threadIdx.x & 31) * 8;
      if (k < K) load(ahead[c], w, k);
    }
  }
  __device__ __forceinline__ void finish(const T* __restrict__ a, int64_t lda, const T* const (&w)[4], int K, int kwarp, int ks, int M,
                                         float (&acc)[4][MB]) {
    const int k0 = kwarp * 256 + (threadIdx.x & 31) * 8;
#pragma unroll
    for (int c = 0; c < P; ++c)
      if (k0 + c * ks * 256 < K) add(ahead[c], a, lda, k0 + c * ks * 256, M, acc);
#pragma unroll 2
    for (int k = k0 + P * ks * 256; k < K; k += ks * 256) {
      uint4 raw[4][kVec];
      load(raw, w, k);
      add(raw, a, lda, k, M, acc);
    }
  }
};
template <typename T, bool AHEAD>
constexpr int kRowsAhead = !AHEAD ? 0 : sizeof(T) == 2 ? 2 : 1;

// Start four weight rows on their way into L2 (weights never change: this may run before griddepcontrol.wait, while
// the previous kernel is still working).
template <typename T>
__device__ __forceinline__ void prefetch_rows(const T* const (&w)[4], int K, int kwarp, int ks, int first) {  // columns from `first` on
  constexpr int kLine = 128 / sizeof(T);
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < 4; ++r)
    for (int k = first + (kwarp * 32 + lane) * kLine; k < K; k += ks * 32 * kLine)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(w[r] + k));
}

template <typename T, int MB, bool AHEAD>
__global__ void __launch_bounds__(kRowsThreads)
dense_rows_proj_kernel(const T* __restrict__ a, int64_t lda, const T* __restrict__ w, int64_t ldw, int M, int N, int K,
                       const __grid_constant__ Segs sg, int ks) {
  constexpr bool kFast = sizeof(T) == 2;
  __shared__ float red[8][4 * MB];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups_per_cta = (kRowsThreads / 32) / ks;
  const int grp = blockIdx.x * groups_per_cta + warp / ks;  // group of four weight rows
  const int kwarp = warp % ks;
  const bool live = grp * 4 < N;
  int si = 0, c0 = 0;
  float acc[4][MB] = {};
  const T* wr[4] = {};
  RowsDot<T, MB, kRowsAhead<T, AHEAD>> dot;
  if (live) {
    si = seg_of(sg, grp * 4);
    const fr_out_segment& s = sg.s[si];
    const int local = grp * 4 - s.n0;
    if (paired(s)) {  // two channels: rows {gate c, gate c + 1, up c, up c + 1}
      c0 = local / 2;
      const int64_t g = s.n0 + (c0 / 32) * 64 + c0 % 32;
      wr[0] = w + g * ldw;
      wr[1] = w + (g + 1) * ldw;
      wr[2] = w + (g + 32) * ldw;
      wr[3] = w + (g + 33) * ldw;
    } else {
      c0 = local;
#pragma unroll
      for (int r = 0; r < 4; ++r) wr[r] = w + static_cast<int64_t>(grp * 4 + r) * ldw;
    }
    dot.begin(wr, K, kwarp, ks);
    prefetch_rows<T>(wr, K, kwarp, ks, kRowsAhead<T, AHEAD> * ks * 256);
  }
  ptx::griddep_wait();
  ptx::griddep_launch_dependents();
  if (live) dot.finish(a, lda, wr, K, kwarp, ks, M, acc);
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const float v = warp_sum(acc[r][m]);
      if (lane == 0) red[warp][r * MB + m] = v;
    }
  __syncthreads();
  if (!live || kwarp != 0) return;
  const fr_out_segment& s = sg.s[si];
  if (paired(s)) {
    if (lane < 2 * MB) {
      const int r = lane / MB, m = lane % MB;
      float g = 0.f, u = 0.f;
      for (int k = 0; k < ks; ++k) {
        g += red[warp + k][r * MB + m];
        u += red[warp + k][(r + 2) * MB + m];
      }
      if (m < M) seg_write<T, kFast>(s, m, c0 + r, pair_act<kFast>(s, g, u));
    }
  } else if (lane < 4 * MB) {
    const int r = lane / MB, m = lane % MB;
    float z = 0.f;
    for (int k = 0; k < ks; ++k) z += red[warp + k][r * MB + m];
    if (m < M) seg_write<T, kFast>(s, m, c0 + r, z);
  }
}

template <typename T, int MB, bool AHEAD>
__global__ void __launch_bounds__(kRowsThreads)
dense_rows_gated_kernel(const __grid_constant__ Parts pt, float* __restrict__ x, int64_t ldx, int M, int N, T* __restrict__ copy,
                        int64_t ldc, int ks) {
  __shared__ float red[8][2][4 * MB];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups_per_cta = (kRowsThreads / 32) / ks;
  const int grp = blockIdx.x * groups_per_cta + warp / ks;
  const int kwarp = warp % ks;
  const bool live = grp * 4 < N;
  auto weight_rows = [&](const fr_gated_part& part, const T* (&wr)[4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
      wr[r] = static_cast<const T*>(part.w) + static_cast<int64_t>(min(grp * 4 + r, N - 1)) * part.ldw;
  };
  // One chunk of the last part ahead (in the models the longer one). More of them, or of two bf16 rows, cost CTAs per SM: us for one
  // row, none / one / two and one of the first part: 2048 x (2048 + 6144) 8.3 / 7.5 / 9.4, 2048 x 6144 6.2 / 5.5 / 7.5,
  // 4096 x 12288 24.5 / 20.0 / 19.0; two rows 9.4 / 11.0 / 10.4, 6.5 / 8.4 / 8.3, 23.0 / 22.8 / 21.9.
  const int last = pt.n - 1;
  constexpr int kAhead = AHEAD ? 1 : 0;
  RowsDot<T, MB, 0> dot0;
  RowsDot<T, MB, kAhead> dot1;
  constexpr bool kLoop = MB > (sizeof(T) == 2 ? 2 : 4);  // see below
  if (kLoop && live) {
    for (int p = 0; p < pt.n; ++p) {
      const T* wr[4];
      weight_rows(pt.p[p], wr);
      prefetch_rows<T>(wr, pt.p[p].K, kwarp, ks, 0);
    }
  } else if (live) {
    const T* wr[4];
    if (last > 0) {
      weight_rows(pt.p[0], wr);
      prefetch_rows<T>(wr, pt.p[0].K, kwarp, ks, 0);
    }
    weight_rows(pt.p[last], wr);
    dot1.begin(wr, pt.p[last].K, kwarp, ks);
    prefetch_rows<T>(wr, pt.p[last].K, kwarp, ks, kAhead * ks * 256);
  }
  ptx::griddep_wait();
  ptx::griddep_launch_dependents();
  auto leave = [&](int p, const float (&acc)[4][MB]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        const float v = warp_sum(acc[r][m]);
        if (lane == 0) red[warp][p][r * MB + m] = v;
      }
  };
  // Few rows: the parts one after the other, the second's loads on their way before the first's sums are joined. Many: a loop, which
  // leaves the compiler room to keep two steps of loads in flight. us, loop / apart: one row, 2048 x 6144 8.4 / 6.2, two 9.8 / 6.5,
  // three of f32 17.9 / 13.7; four of bf16 9.3 / 11.3, eight 18.0 / 19.8, eight of f32 x 4096 x 12288 66 / 76.
  if constexpr (kLoop) {
    for (int p = 0; p < pt.n; ++p) {
      float acc[4][MB] = {};
      if (live) {
        const T* wr[4];
        weight_rows(pt.p[p], wr);
        RowsDot<T, MB, 0>().finish(static_cast<const T*>(pt.p[p].a), pt.p[p].lda, wr, pt.p[p].K, kwarp, ks, M, acc);
      }
      leave(p, acc);
    }
  } else {
    if (last > 0) {
      float acc[4][MB] = {};
      const fr_gated_part& part = pt.p[0];
      const T* wr[4];
      weight_rows(part, wr);
      if (live) dot0.finish(static_cast<const T*>(part.a), part.lda, wr, part.K, kwarp, ks, M, acc);
      leave(0, acc);
    }
    {
      float acc[4][MB] = {};
      const fr_gated_part& part = pt.p[last];
      const T* wr[4];
      weight_rows(part, wr);
      if (live) dot1.finish(static_cast<const T*>(part.a), part.lda, wr, part.K, kwarp, ks, M, acc);
      leave(last, acc);
    }
  }
  __syncthreads();
  if (!live || kwarp != 0 || lane >= 4 * MB) return;
  const int r = lane / MB, m = lane % MB, n = grp * 4 + r;
  if (copy != nullptr && m < M && n >= N - 8)  // the padding behind the last columns
    for (int c = N + (n - (N - 8)); c < (N + 7) / 8 * 8 && c < ldc; c += 8) copy[m * ldc + c] = from_f<T>(0.f);
  if (m >= M || n >= N) return;
  float v = x[m * ldx + n];
  for (int p = 0; p < pt.n; ++p) {
    float z = 0.f;
    for (int k = 0; k < ks; ++k) z += red[warp + k][p][r * MB + m];
    const T* g = static_cast<const T*>(pt.p[p].gate);
    v += (g != nullptr ? to_f<T>(g[m * pt.p[p].ldg + n]) : 1.0f) * z;
  }
  x[m * ldx + n] = v;
  if (copy != nullptr) copy[m * ldc + n] = from_f<T>(v);
}

// ---------------------------------------------------------------------------
// f32, more rows: TM x 64 tiles, 256 threads of TM / 16 x 4 outputs. With tiles enough they reach 34 of the fp32 units' 75 TFLOP/s
// (loads from shared memory and FMAs share the issue slots). Operands arrive by cp.async two steps of 16 ahead and stay as they lie in memory, rows of k, so that one fma.rn.f32x2
// takes two consecutive k of an output without any rearranging (an output is the sum of its even and its odd chain).
// us for 64 / 351 rows of 2048: 20480 columns 286 / 1153 before (64 x 64 tiles through transposed copies, one step ahead), 220 /
// 863 now (34 TFLOP/s); 2048 columns 133 / 226 and 92 / 155. (128 x 128 tiles of 8 x 8 outputs per thread, half the loads from shared
// memory per FMA but one CTA per SM: 1131 for 351 rows x 20480.)
// ---------------------------------------------------------------------------
constexpr int kSimtK = 16, kSimtStages = 3;
constexpr int kSimtPitch = kSimtK + 4;  // floats: eight consecutive rows of 16 bytes meet in no bank

__device__ __forceinline__ uint64_t f32x2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float f32x2_sum(uint64_t v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return lo + hi;
}

template <int TM>
struct Simt {
  static constexpr int RM = TM / 16, CN = 4;
  float as[kSimtStages][TM][kSimtPitch], ws[kSimtStages][64][kSimtPitch];

  // row r of a thread's RM and column c of its four (of a [32 gate | 32 up] block two gates, then their ups), within the tile
  static __device__ __forceinline__ int row_of(int ty, int r) { return ty * RM + r; }
  static __device__ __forceinline__ int col_of(int tx, int c) { return c * 16 + tx; }

  __device__ __forceinline__ void tile(const float* __restrict__ a, int64_t lda, const float* __restrict__ w, int64_t ldw, int M,
                                       int N, int K, int m0, int n0, float (&out)[RM][CN]) {
    const int tid = threadIdx.x, lr = tid >> 2, lk = (tid & 3) * 4, tx = tid & 15, ty = tid >> 4;
    auto copy = [](float* dst, const float* src, bool in) {  // zeros outside; `src` is a valid address either way
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
    };
    const int steps = (K + kSimtK - 1) / kSimtK;
    auto fetch = [&](int step) {
      if (step < steps) {
        const int st = step % kSimtStages, k = step * kSimtK + lk;
        const bool in = k < K;  // K is a multiple of 8
#pragma unroll
        for (int i = 0; i < TM / 64; ++i) {
          const bool row = m0 + lr + 64 * i < M;
          copy(&as[st][lr + 64 * i][lk], a + static_cast<int64_t>(row ? m0 + lr + 64 * i : 0) * lda + (in ? k : 0), in && row);
        }
        const bool col = n0 + lr < N;
        copy(&ws[st][lr][lk], w + static_cast<int64_t>(col ? n0 + lr : 0) * ldw + (in ? k : 0), in && col);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    uint64_t acc[RM][CN] = {};
    __syncthreads();  // the tile before, if any, has been read
    for (int i = 0; i < kSimtStages - 1; ++i) fetch(i);
    for (int step = 0; step < steps; ++step) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kSimtStages - 2) : "memory");
      __syncthreads();  // this step's operands are there, the last one's are read
      fetch(step + kSimtStages - 1);
      const int st = step % kSimtStages;
#pragma unroll
      for (int k = 0; k < kSimtK; k += 4) {
        ulonglong2 wv[CN];
#pragma unroll
        for (int c = 0; c < CN; ++c) wv[c] = *reinterpret_cast<const ulonglong2*>(&ws[st][col_of(tx, c)][k]);
#pragma unroll
        for (int r = 0; r < RM; ++r) {
          const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(&as[st][row_of(ty, r)][k]);
#pragma unroll
          for (int c = 0; c < CN; ++c) {
            acc[r][c] = f32x2_fma(av.x, wv[c].x, acc[r][c]);
            acc[r][c] = f32x2_fma(av.y, wv[c].y, acc[r][c]);
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
      for (int c = 0; c < CN; ++c) out[r][c] = f32x2_sum(acc[r][c]);
  }
};

template <int TM>
__global__ void __launch_bounds__(256, TM == 64 ? 3 : 2)
dense_simt_proj_kernel(const float* __restrict__ a, int64_t lda, const float* __restrict__ w, int64_t ldw, int M, int N, int K,
                       const __grid_constant__ Segs sg) {
  using S = Simt<TM>;
  __shared__ __align__(16) S sm;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * 64;
  float acc[S::RM][S::CN];
  sm.tile(a, lda, w, ldw, M, N, K, m0, n0, acc);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int col0 = n0 + half * 32;  // a 32-column chunk lies in one range
    if (col0 >= N) break;
    const fr_out_segment& s = sg.s[seg_of(sg, col0)];
    const bool pair = paired(s);
    if (pair && half == 1) continue;
#pragma unroll
    for (int r = 0; r < S::RM; ++r) {
      const int row = m0 + S::row_of(ty, r);
      if (row >= M) continue;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float v = acc[r][2 * half + e];
        if (pair)
          seg_write<float, false>(s, row, (col0 - s.n0) / 2 + e * 16 + tx, pair_act<false>(s, v, acc[r][2 + e]));
        else
          seg_write<float, false>(s, row, col0 - s.n0 + e * 16 + tx, v);
      }
    }
  }
}

__global__ void __launch_bounds__(256, 3)
dense_simt_gated_kernel(const __grid_constant__ Parts pt, float* __restrict__ x, int64_t ldx, int M, int N, float* __restrict__ copy,
                        int64_t ldc) {
  using S = Simt<64>;
  __shared__ __align__(16) S sm;
  const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float sum[S::RM][S::CN] = {};
  for (int p = 0; p < pt.n; ++p) {
    const fr_gated_part& part = pt.p[p];
    float acc[S::RM][S::CN];
    sm.tile(static_cast<const float*>(part.a), part.lda, static_cast<const float*>(part.w), part.ldw, M, N, part.K, m0, n0, acc);
    const float* g = static_cast<const float*>(part.gate);
#pragma unroll
    for (int r = 0; r < S::RM; ++r)
#pragma unroll
      for (int c = 0; c < S::CN; ++c) {
        const int row = m0 + S::row_of(ty, r), col = n0 + S::col_of(tx, c);
        if (row < M && col < N) sum[r][c] += (g != nullptr ? g[row * part.ldg + col] : 1.0f) * acc[r][c];
      }
  }
#pragma unroll
  for (int r = 0; r < S::RM; ++r)
#pragma unroll
    for (int c = 0; c < S::CN; ++c) {
      const int row = m0 + S::row_of(ty, r), col = n0 + S::col_of(tx, c);
      if (row < M && col < N) {
        const float v = x[row * ldx + col] + sum[r][c];
        x[row * ldx + col] = v;
        if (copy != nullptr) copy[row * ldc + col] = v;
      } else if (copy != nullptr && row < M && col < (N + 7) / 8 * 8 && col < ldc) {
        copy[row * ldc + col] = 0.f;
      }
    }
}

// One share of K per blockIdx.z, times the part's gate, into its partial [M, N]: the tiles of an update alone leave SMs with one or
// two CTAs of three, each with a chain of thousands of K steps (us: 351 rows x 2048 x 8192 669 -> 371, 128 rows 441 -> 141, 1000
// rows 1241 -> 899; 128 x 4096 x 12288 638 -> 363). Shorter sums are also closer ones: the error against 64 bits goes from 9e-7 of
// the norm to 3 to 6e-7.
__global__ void __launch_bounds__(256, 3)
dense_simt_partial_kernel(const __grid_constant__ Parts pt, int splits0, int splits1, float* __restrict__ partials, int M, int N) {
  using S = Simt<64>;
  __shared__ __align__(16) S sm;
  const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64, slot = blockIdx.z;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const bool second = slot >= splits0;
  const fr_gated_part& part = pt.p[second ? 1 : 0];
  const int i = second ? slot - splits0 : slot, n = second ? splits1 : splits0, steps = (part.K + kSimtK - 1) / kSimtK;
  const int k0 = static_cast<int>(static_cast<int64_t>(steps) * i / n) * kSimtK;
  const int k1 = min(static_cast<int>(static_cast<int64_t>(steps) * (i + 1) / n) * kSimtK, part.K);
  float acc[S::RM][S::CN];
  sm.tile(static_cast<const float*>(part.a) + k0, part.lda, static_cast<const float*>(part.w) + k0, part.ldw, M, N, k1 - k0, m0, n0, acc);
  const float* g = static_cast<const float*>(part.gate);
#pragma unroll
  for (int r = 0; r < S::RM; ++r)
#pragma unroll
    for (int c = 0; c < S::CN; ++c) {
      const int row = m0 + S::row_of(ty, r), col = n0 + S::col_of(tx, c);
      if (row < M && col < N)
        partials[(static_cast<int64_t>(slot) * M + row) * N + col] = (g != nullptr ? g[row * part.ldg + col] : 1.0f) * acc[r][c];
    }
}

// ---------------------------------------------------------------------------
// sum of the K shares of a split product, then the column ranges' epilogues
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
dense_finish_kernel(const float* __restrict__ partials, int n_splits, int M, int N, const __grid_constant__ Segs sg) {
  ptx::griddep_wait();
  ptx::griddep_launch_dependents();
  const int row = blockIdx.y, col = blockIdx.x * 256 + threadIdx.x;
  if (col >= N) return;
  const fr_out_segment& s = sg.s[seg_of(sg, col)];
  auto sum = [&](int c) {
    float z = 0.f;
    for (int i = 0; i < n_splits; ++i) z += partials[(static_cast<int64_t>(i) * M + row) * N + c];
    return z;
  };
  const int local = col - s.n0;
  constexpr bool kFast = sizeof(T) == 2;
  if (!paired(s)) {
    seg_write<T, kFast>(s, row, local, sum(col));
  } else if (local % 64 < 32) {
    seg_write<T, kFast>(s, row, local / 64 * 32 + local % 64, pair_act<kFast>(s, sum(col), sum(col + 32)));
  }
}

// ---------------------------------------------------------------------------
// bf16 on tcgen05
// ---------------------------------------------------------------------------
constexpr int kBlockM = 128;
constexpr int kBlockK = 64;  // bf16 elements: one 128-byte swizzle span
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + kEpiWarps * 32;
enum Epi { kEpiSegs = 0, kEpiAdd = 1, kEpiPartial = 2 };

// Rows a kernel is made for. kAny: stage sizes are constants (a full tile's products take longer than the hand-over, and the
// issuing thread has no time to spare: run-time sizes cost 8192 rows 4 %). kFew: at most 128 rows, stages as planned at launch.
// kOctet: at most 8 rows, which the row kernel sums in fp32 FMAs otherwise. The tensor cores' accumulation loses bits with
// every product added (2.1e-6 of the norm at K = 2048, 1.4e-5 at 12288, where the row kernel has 8e-8 and 9e-8), so here it
// spans one k-block only: the four blocks of a stage go to four accumulators, which a warp adds up in fp32 registers.
// kPair: tiles of 256 rows by two CTAs of a cluster, each with its 128 rows of A and half of the weight rows, one tcgen05.mma for both.
enum Rows { kAny = 0, kFew = 1, kOctet = 2, kPair = 3 };

template <int BLOCK_N, int ROWS>
struct Cfg {
  static constexpr int kTileM = ROWS == kPair ? 2 * kBlockM : kBlockM, kTileB = ROWS == kPair ? BLOCK_N / 2 : BLOCK_N;  // kTileB: a CTA's
  static constexpr int kStageBytes = (kBlockM + kTileB) * kBlockK * 2;
  static constexpr int kStages = kTileB == 256 ? 4 : (kTileB == 128 ? 6 : 8);
  static constexpr int kAcc = ROWS == kOctet ? 8 : 2;  // accumulators in TMEM
  static constexpr int kTmemCols = kAcc * BLOCK_N <= 128 ? 128 : (kAcc * BLOCK_N <= 256 ? 256 : 512);  // a power of two
};

// Operand stages of a few rows (one row block). They bring in only themselves: an SM pulls operands at about 48 bytes per
// clock, and a whole tile of A would be two thirds of that traffic beside 64 weight rows. The product still reads 128 rows
// of A; what lies behind the loaded ones goes into accumulator rows that nobody stores.
// A hand-over between the loading and the issuing warp costs a few hundred clocks whatever the tile's width, more than the 0.07 us of
// a k-block's products of 64 columns: narrow tiles hand over up to four k-blocks at a time, as long as three stages remain.
constexpr int kTileA = kBlockM * kBlockK * 2;
constexpr int kMaxStages = 12;
constexpr int kOperandBytes = 200 * 1024;
constexpr int kBarBytes = (2 * kMaxStages + 4) * 8 + 16;
constexpr int kOctetBlocks = 4;  // k-blocks of a stage of kOctet
constexpr int kOctetBytes = 2 * 8 * 64 * 4 + 16;  // its finished tiles on their way out, two of [8][64], and whether they are whole
struct Stages {
  int a_rows, a_bytes, block_bytes, blocks, n, smem;  // blocks: k-blocks of a stage, each [A rows | weight rows]
  __host__ Stages(int M, int block_n) {  // M <= 128
    a_rows = (M + 7) / 8 * 8;
    a_bytes = a_rows * kBlockK * 2;
    block_bytes = a_bytes + block_n * kBlockK * 2;
    blocks = block_n > 128 ? 1 : 4;
    while (blocks > 1 && 3 * blocks * block_bytes > kOperandBytes) blocks /= 2;
    n = kOperandBytes / (blocks * block_bytes);
    n = n < kMaxStages ? n : kMaxStages;
    smem = 1024 + n * blocks * block_bytes + (kTileA - a_bytes) + kBarBytes;
  }
};

struct TcArgs {
  int M, N;
  int a_bytes, block_bytes, stage_blocks, stages;  // as planned by Stages
  int ahead;         // the first job's weights may be read before griddepcontrol.wait
  int n_parts;
  int kb[2];         // k-blocks per part
  int splits[2];     // kEpiPartial: K splits per part
  Segs segs;         // kEpiSegs
  float* x;          // kEpiAdd
  int64_t ldx;
  const __nv_bfloat16* gate[2];
  int64_t ldg[2];
  float* partials;   // kEpiPartial: [splits, M, N]
  __nv_bfloat16* copy;  // kEpiAdd: the new x as bf16, or null
  int64_t ldc;
};

// Work of a CTA in order: kEpiSegs / kEpiAdd: tile after tile, the parts of a tile back to back (its second
// accumulator is added by the same threads as its first); kEpiPartial: one K share of one part of one tile.
struct Job {
  int mb, nb, part, kb0, kb1, slot;
};
template <int EPI>
__device__ __forceinline__ Job job_at(const TcArgs& g, int unit, int sub, int m_blocks, int n_blocks) {
  Job j;
  int tile = unit;
  j.part = sub;
  j.kb0 = 0;
  j.slot = 0;
  if (EPI == kEpiPartial) {
    const int per_tile = g.splits[0] + g.splits[1];
    tile = unit / per_tile;
    const int s = unit % per_tile;
    j.part = s < g.splits[0] ? 0 : 1;
    const int i = j.part == 0 ? s : s - g.splits[0];
    const int n = g.splits[j.part], kb = g.kb[j.part];
    j.kb0 = static_cast<int>(static_cast<int64_t>(kb) * i / n);
    j.kb1 = static_cast<int>(static_cast<int64_t>(kb) * (i + 1) / n);
    j.slot = s;
  } else {
    j.kb1 = g.kb[sub];
  }
  constexpr int kGroup = 8;  // row blocks per raster group: A streams once, the group's B blocks stay in L2
  const int per_group = kGroup * n_blocks;
  const int first = tile / per_group * kGroup;
  const int rows = min(kGroup, m_blocks - first);
  const int t = tile - tile / per_group * per_group;
  j.mb = first + t % rows;
  j.nb = t / rows;
  return j;
}

__device__ __forceinline__ void store32_bf16(__nv_bfloat16* dst, const float (&v)[32], int nvalid) {
  if (nvalid >= 32 && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
    if ((reinterpret_cast<uintptr_t>(dst) & 31u) == 0) {
      const uint32_t w0[8] = {w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7]};
      const uint32_t w1[8] = {w[8], w[9], w[10], w[11], w[12], w[13], w[14], w[15]};
      ptx::st_global_v8(dst, w0);
      ptx::st_global_v8(dst + 16, w1);
    } else {
      uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
      for (int i = 0; i < 4; ++i) d4[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < nvalid) dst[i] = __float2bfloat16_rn(v[i]);
  }
}

// 32 fp32 values to / from consecutive addresses; vector accesses when the row allows them
__device__ __forceinline__ void store32_f32(float* dst, const float (&v)[32], int nvalid) {
  if (nvalid >= 32 && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
    float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll
    for (int i = 0; i < 8; ++i) d4[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < nvalid) dst[i] = v[i];
  }
}

// Stores the 64 columns of kOctet's tile ([8][64] in shared memory) that begin at n0; thread `t` of `nt`.
template <int EPI>
__device__ __forceinline__ void finish_octet(const TcArgs& g, const Job& j, int n0, const float* v, int t, int nt) {
#pragma unroll 1
  for (int e = t; e < g.M * 64; e += nt) {
    const int row = e / 64, c = e % 64, col = n0 + c;
    if (col >= g.N) continue;
    if constexpr (EPI == kEpiSegs) {
      const fr_out_segment& s = g.segs.s[seg_of(g.segs, col)];
      if (!paired(s))
        seg_write<__nv_bfloat16, true>(s, row, col - s.n0, v[e]);
      else if (c < 32)
        seg_write<__nv_bfloat16, true>(s, row, (n0 - s.n0) / 2 + c, pair_act<true>(s, v[e], v[e + 32]));
    } else {
      const __nv_bfloat16* gp = g.gate[j.part];
      const float gt = gp != nullptr ? __bfloat162float(gp[row * g.ldg[j.part] + col]) : 1.0f;
      g.partials[(static_cast<int64_t>(j.slot) * g.M + row) * g.N + col] = gt * v[e];
    }
  }
}

template <int BLOCK_N, int EPI, int ROWS>
__global__ void __launch_bounds__(kThreads, 1)
dense_tc_kernel(const __grid_constant__ CUtensorMap ta0, const __grid_constant__ CUtensorMap tb0,
                const __grid_constant__ CUtensorMap ta1, const __grid_constant__ CUtensorMap tb1,
                const __grid_constant__ TcArgs g, int* status) {
  using C = Cfg<BLOCK_N, ROWS>;
  constexpr bool FEW = ROWS == kFew || ROWS == kOctet, PAIR = ROWS == kPair;
  static_assert(ROWS != kOctet || (BLOCK_N == 64 && EPI != kEpiAdd), "");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  const uint32_t n_stages = FEW ? g.stages : C::kStages, block_bytes = FEW ? g.block_bytes : C::kStageBytes;
  const uint32_t a_bytes = FEW ? g.a_bytes : kTileA;
  const int stage_blocks = ROWS == kOctet ? kOctetBlocks : (FEW && BLOCK_N <= 128 ? g.stage_blocks : 1);
  const uint32_t stage_bytes = stage_blocks * block_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + n_stages * stage_bytes + (kTileA - a_bytes));
  const uint32_t bar_full = ptx::smem_u32(bars);
  const uint32_t bar_empty = bar_full + 8 * kMaxStages;
  const uint32_t bar_tfull = bar_empty + 8 * kMaxStages;
  const uint32_t bar_tempty = bar_tfull + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* octet = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + kBarBytes);  // kOctet

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? ptx::cluster_ctarank() : 0u;
  const int unit0 = PAIR ? blockIdx.x >> 1 : blockIdx.x, unit_step = PAIR ? gridDim.x >> 1 : gridDim.x;
  const int m_blocks = (g.M + C::kTileM - 1) / C::kTileM;
  const int n_blocks = (g.N + BLOCK_N - 1) / BLOCK_N;
  const int subs = EPI == kEpiPartial ? 1 : g.n_parts;
  const int num_units = m_blocks * n_blocks * (EPI == kEpiPartial ? g.splits[0] + g.splits[1] : 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < static_cast<int>(n_stages); ++s) {
      ptx::mbar_init(bar_full + 8 * s, 1);
      ptx::mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(bar_tfull + 8 * b, 1);
      ptx::mbar_init(bar_tempty + 8 * b, ROWS == kOctet ? 1 : (PAIR ? 2 * kEpiWarps : kEpiWarps));  // PAIR: of both CTAs, in CTA 0
    }
    *abort_flag = 0;
    ptx::mbar_init_fence();
    ptx::prefetch_tmap(&ta0);
    ptx::prefetch_tmap(&tb0);
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      ptx::tmem_alloc_pair(ptx::smem_u32(tmem_slot), C::kTmemCols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(ptx::smem_u32(tmem_slot), C::kTmemCols);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) {  // neither CTA may signal the other's barriers before they are set up
    ptx::cluster_arrive();
    ptx::cluster_wait();
  }
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // the weights of one stage's k-blocks, and the bytes that the stage waits for
  auto load_weights = [&](const Job& j, int kb0, uint32_t stage) {
    const CUtensorMap* tb = j.part == 0 ? &tb0 : &tb1;
    uint32_t sb = base + stage * stage_bytes + a_bytes;
    if constexpr (PAIR) {  // CTA 0 collects both CTAs' bytes
      if (rank == 0) ptx::mbar_expect_tx_one(bar_full + 8 * stage, 2 * C::kStageBytes);
      ptx::tma_load_2d_pair_one(sb, tb, kb0 * kBlockK, j.nb * BLOCK_N + static_cast<int>(rank) * C::kTileB, ptx::mapa(bar_full + 8 * stage, 0));
    } else {
      const int kb1 = stage_blocks == 1 ? kb0 + 1 : min(kb0 + stage_blocks, j.kb1);
      ptx::mbar_expect_tx_one(bar_full + 8 * stage, (kb1 - kb0) * block_bytes);
      for (int kb = kb0; kb < kb1; ++kb, sb += block_bytes)
        ptx::tma_load_2d_one(sb, tb, kb * kBlockK, j.nb * BLOCK_N, bar_full + 8 * stage);
    }
  };
  // Weights that the launch ahead does not write (FR_DENSE_LAID_OUT) fill the first job's stages while that launch still runs: whole
  // passes of 48 and 64 requests 1.011x and 1.003x.
  int loaded = 0;
  if (warp == 0 && g.ahead != 0 && unit0 < num_units) {
    const Job j = job_at<EPI>(g, unit0, 0, m_blocks, n_blocks);
    for (int kb0 = j.kb0; kb0 < j.kb1 && loaded < static_cast<int>(n_stages); kb0 += stage_blocks) load_weights(j, kb0, loaded++);
  }
  ptx::griddep_wait();
  ptx::griddep_launch_dependents();

  if (warp == 0) {
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int unit = unit0; unit < num_units && ok; unit += unit_step) {
      for (int sub = 0; sub < subs && ok; ++sub) {
        const Job j = job_at<EPI>(g, unit, sub, m_blocks, n_blocks);
        const CUtensorMap* ta = j.part == 0 ? &ta0 : &ta1;
        for (int kb0 = j.kb0; kb0 < j.kb1; kb0 += stage_blocks) {
          ok = ptx::mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag, status, 61);
          if (!ok) break;
          if (loaded > 0) --loaded;
          else load_weights(j, kb0, stage);
          uint32_t sa = base + stage * stage_bytes;
          if constexpr (PAIR) {
            ptx::tma_load_2d_pair_one(sa, ta, kb0 * kBlockK, j.mb * C::kTileM + static_cast<int>(rank) * kBlockM,
                                      ptx::mapa(bar_full + 8 * stage, 0));
          } else {
            const int kb1 = stage_blocks == 1 ? kb0 + 1 : min(kb0 + stage_blocks, j.kb1);
            for (int kb = kb0; kb < kb1; ++kb, sa += block_bytes)
              ptx::tma_load_2d_one(sa, ta, kb * kBlockK, j.mb * kBlockM, bar_full + 8 * stage);
          }
          if (++stage == n_stages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = ptx::make_idesc(1u, 1u, C::kTileM, BLOCK_N);
    // both CTAs of a pair, or this one
    auto commit = [&](uint32_t bar) {
      if constexpr (PAIR) {
        ptx::tc_commit_pair_one(ptx::mapa(bar, 0));
        ptx::tc_commit_pair_one(ptx::mapa(bar, 1));
      } else {
        ptx::tc_commit_one(bar);
      }
    };
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    int it = 0;
    for (int unit = unit0; rank == 0 && unit < num_units && ok; unit += unit_step) {  // PAIR: CTA 0 issues for both
      for (int sub = 0; sub < subs && ok; ++sub) {
        const Job j = job_at<EPI>(g, unit, sub, m_blocks, n_blocks);
        // a set of accumulators: of the whole job, or (kOctet) of one stage, one per k-block
        uint32_t set = 0, d_tmem = 0;
        auto next_set = [&]() {
          set = it & 1;
          d_tmem = tmem_base + set * (C::kAcc / 2 * BLOCK_N);
          ok = ptx::mbar_wait_warp(bar_tempty + 8 * set, ((it >> 1) & 1) ^ 1u, abort_flag, status, 62);
          ++it;
          if (ok) ptx::tc_fence_after();
        };
        if (ROWS != kOctet) next_set();
        if (!ok) break;
        for (int kb0 = j.kb0; kb0 < j.kb1; kb0 += stage_blocks) {
          if (ROWS == kOctet) next_set();
          if (!ok) break;
          ok = ptx::mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag, status, 63);
          if (!ok) break;
          ptx::tc_fence_after();
          uint32_t sa = base + stage * stage_bytes;
          const int kb1 = stage_blocks == 1 ? kb0 + 1 : min(kb0 + stage_blocks, j.kb1);
          for (int kb = kb0; kb < kb1; ++kb, sa += block_bytes) {
            const uint64_t a_desc = ptx::smem_desc_sw128(sa), b_desc = ptx::smem_desc_sw128(sa + a_bytes);
            const uint32_t more = ROWS != kOctet && kb > j.kb0 ? 1u : 0u;
            if constexpr (PAIR)
              ptx::mma_k_block_f16_pair(d_tmem, a_desc, b_desc, idesc, more);
            else
              ptx::mma_k_block_f16(d_tmem, a_desc, b_desc, idesc, more);
            if (ROWS == kOctet) d_tmem += BLOCK_N;
          }
          commit(bar_empty + 8 * stage);
          if (ROWS == kOctet) commit(bar_tfull + 8 * set);
          if (++stage == n_stages) { stage = 0; phase ^= 1u; }
        }
        if (ok && ROWS != kOctet) commit(bar_tfull + 8 * set);
      }
    }
  } else if (ROWS == kOctet) {
    // Warp 4 adds up: TMEM lanes 0 .. 31 are open to it, and all rows lie in lanes 0 .. 7. The other seven store the tile that
    // it has left in shared memory while it goes on with the next one; all eight meet once per tile.
    bool ok = true;
    int it = 0, tile = 0;
    for (int unit = unit0; unit < num_units && ok; unit += unit_step) {
      for (int sub = 0; sub < subs && ok; ++sub, ++tile) {
        const Job j = job_at<EPI>(g, unit, sub, m_blocks, n_blocks);
        float* out = octet + (tile & 1) * (8 * 64);
        volatile int* whole = reinterpret_cast<volatile int*>(octet + 2 * 8 * 64) + (tile & 1);
        if (warp == 4) {
          float v[16] = {}, lost[16] = {};
          for (int kb0 = j.kb0; kb0 < j.kb1; kb0 += kOctetBlocks, ++it) {
            const uint32_t set = it & 1;
            int okw = 0;
            if (lane == 0) okw = ptx::mbar_wait(bar_tfull + 8 * set, (it >> 1) & 1, abort_flag, status, 64) ? 1 : 0;
            okw = __shfl_sync(0xffffffffu, okw, 0);
            if (!okw) { ok = false; break; }
            ptx::tc_fence_after();
            float sum[16];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const int n = j.kb1 - kb0 - 2 * half;  // blocks left; what lies behind them is old and not added
              if (n <= 0) break;
              uint32_t r0[32], r1[32];
              const uint32_t taddr = tmem_base + (set * kOctetBlocks + 2 * half) * BLOCK_N;
              ptx::tmem_ld_16x256(taddr, r0);
              ptx::tmem_ld_16x256(taddr + BLOCK_N, r1);
              ptx::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) {  // registers 4 x + 2 and 4 x + 3 hold rows 8 .. 15
                const int x = i / 2 * 4 + i % 2;
                const float two = __uint_as_float(r0[x]) + (n > 1 ? __uint_as_float(r1[x]) : 0.f);
                sum[i] = half == 0 ? two : sum[i] + two;
              }
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar_tempty + 8 * set);
#pragma unroll
            for (int i = 0; i < 16; ++i) {  // Knuth's two-sum: what the addition rounds away is kept beside it
              const float t = v[i] + sum[i], z = t - v[i];
              lost[i] += (v[i] - (t - z)) + (sum[i] - z);
              v[i] = t;
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {  // row lane / 4, columns 8 i + 2 (lane % 4) and the one after
            const float x = fabsf(v[2 * i]) < INFINITY ? v[2 * i] + lost[2 * i] : v[2 * i];
            const float y = fabsf(v[2 * i + 1]) < INFINITY ? v[2 * i + 1] + lost[2 * i + 1] : v[2 * i + 1];
            *reinterpret_cast<float2*>(out + (lane >> 2) * 64 + 8 * i + 2 * (lane & 3)) = make_float2(x, y);
          }
          if (lane == 0) *whole = ok ? 1 : 0;
          __syncwarp();
        }
        // a tile that was given up (a wait that ran out) ends the loop for all eight warps alike
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
        ok = *whole != 0;
        if (ok && warp != 4) {
          const int w = warp - 2 - (warp > 4 ? 1 : 0);
          finish_octet<EPI>(g, j, j.nb * BLOCK_N, out, w * 32 + lane, (kEpiWarps - 1) * 32);
        }
      }
    }
  } else {
    const int quad = warp & 3;
    const int part_of_cols = (warp - 2) >> 2;  // two warps per lane quadrant: even / odd chunks
    bool ok = true;
    int it = 0;
    for (int unit = unit0; unit < num_units && ok; unit += unit_step) {
      for (int sub = 0; sub < subs && ok; ++sub, ++it) {
        const Job j = job_at<EPI>(g, unit, sub, m_blocks, n_blocks);
        const uint32_t buf = it & 1;
        const int row = j.mb * C::kTileM + static_cast<int>(rank) * kBlockM + quad * 32 + lane;
        const int n0 = j.nb * BLOCK_N;
        const bool any_row = row - lane < g.M;
        int okw = 0;
        if (lane == 0) okw = ptx::mbar_wait(bar_tfull + 8 * buf, (it >> 1) & 1, abort_flag, status, 64) ? 1 : 0;
        okw = __shfl_sync(0xffffffffu, okw, 0);
        if (!okw) { ok = false; break; }
        ptx::tc_fence_after();
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * BLOCK_N;
        if constexpr (EPI == kEpiSegs) {
#pragma unroll 1
          for (int c = part_of_cols; any_row && c < BLOCK_N / 64; c += 2) {  // pairs of 32-column chunks
            const int col = n0 + c * 64;
            if (col >= g.N) break;
            uint32_t r0[32], r1[32];
            ptx::tmem_ld_32x32(taddr + c * 64, r0);
            ptx::tmem_ld_32x32(taddr + c * 64 + 32, r1);
            ptx::tmem_ld_wait();
            if (row < g.M) {
            const fr_out_segment& s0 = g.segs.s[seg_of(g.segs, col)];
            if (paired(s0)) {
              const int ch = (col - s0.n0) / 2;
              float v[32];
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = pair_act<true>(s0, __uint_as_float(r0[i]), __uint_as_float(r1[i]));
              const int64_t r = s0.row_map != nullptr ? s0.row_map[row] : row;
              store32_bf16(static_cast<__nv_bfloat16*>(s0.out) + r * s0.ldo + ch, v, s0.n - ch);
            } else {
#pragma unroll
              for (int half = 0; half < 2; ++half) {
                const int hc = col + half * 32;
                if (hc < g.N) {
                  const fr_out_segment& s = g.segs.s[seg_of(g.segs, hc)];
                  const int lc = hc - s.n0, nvalid = s.n - lc;
                  float v[32];
#pragma unroll
                  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(half == 0 ? r0[i] : r1[i]);
                  if (nvalid > 0) {
                    const int64_t r = s.row_map != nullptr ? s.row_map[row] : row;
                    if (s.kind == FR_SEG_STORE_F32) {
                      store32_f32(static_cast<float*>(s.out) + r * s.ldo + lc, v, nvalid);
                    } else {
                      if (s.kind == FR_SEG_SIGMOID) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                          const float b = (s.bias != nullptr && i < nvalid) ? __ldg(s.bias + lc + i) : 0.f;
                          v[i] = sigmoid_f<true>(v[i] + b);
                        }
                      }
                      if (s.kind == FR_SEG_GELU_MUL) {
                        const __nv_bfloat16* mul = static_cast<const __nv_bfloat16*>(s.mul) +
                                                   (s.mul_map != nullptr ? s.mul_map[row] : row) * s.ld_mul + lc;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                          if (i < nvalid) v[i] = gelu_tanh_f<true>(v[i]) * __bfloat162float(__ldg(mul + i));
                      }
                      store32_bf16(static_cast<__nv_bfloat16*>(s.out) + r * s.ldo + lc, v, nvalid);
                    }
                  }
                }
              }
            }
            }
            __syncwarp();  // the next tcgen05.ld is a whole-warp instruction
          }
        } else {
#pragma unroll 1
          for (int c = part_of_cols; any_row && c < BLOCK_N / 32; c += 2) {
            const int col = n0 + c * 32;
            const int nvalid = g.N - col;
            if (nvalid <= 0) break;
            uint32_t r[32];
            ptx::tmem_ld_32x32(taddr + c * 32, r);
            // the operands of the update are in flight while the accumulator is read
            const __nv_bfloat16* gp = g.gate[j.part];
            float gt[32];
            const bool live = row < g.M;
            const __nv_bfloat16* gr = gp + (live ? row : 0) * g.ldg[j.part] + col;
            if (gp != nullptr && nvalid >= 32 && (reinterpret_cast<uintptr_t>(gr) & 15u) == 0) {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                float t[8];
                unpack8(__ldg(reinterpret_cast<const uint4*>(gr) + i), t);
#pragma unroll
                for (int e = 0; e < 8; ++e) gt[i * 8 + e] = t[e];
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) gt[i] = gp == nullptr ? 1.0f : (i < nvalid ? __bfloat162float(gr[i]) : 0.f);
            }
            float v[32];
            if constexpr (EPI == kEpiAdd) {
              float* xr = g.x + (live ? row : 0) * g.ldx + col;
              if (nvalid >= 32 && (reinterpret_cast<uintptr_t>(xr) & 15u) == 0) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const float4 t = reinterpret_cast<const float4*>(xr)[i];
                  v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
                }
              } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = i < nvalid ? xr[i] : 0.f;
              }
              ptx::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = fmaf(gt[i], __uint_as_float(r[i]), v[i]);
              if (live) store32_f32(xr, v, nvalid);
              if (live && g.copy != nullptr && sub + 1 == subs) {
                __nv_bfloat16* cr = g.copy + row * g.ldc + col;
                store32_bf16(cr, v, nvalid);
                if (nvalid < 32)
                  for (int c = nvalid; (col + c) % 8 != 0 && col + c < g.ldc; ++c) cr[c] = __float2bfloat16_rn(0.f);
              }
            } else {
              ptx::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = gt[i] * __uint_as_float(r[i]);
              if (live) store32_f32(g.partials + (static_cast<int64_t>(j.slot) * g.M + row) * g.N + col, v, nvalid);
            }
            __syncwarp();
          }
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (PAIR)
            ptx::mbar_arrive_cluster_relaxed(ptx::mapa(bar_tempty + 8 * buf, 0));
          else
            ptx::mbar_arrive(bar_tempty + 8 * buf);
        }
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if constexpr (PAIR) {  // both converge before either frees tensor memory or leaves
    ptx::cluster_arrive();
    ptx::cluster_wait();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    if constexpr (PAIR)
      ptx::tmem_dealloc_pair(tmem_base, C::kTmemCols);
    else
      ptx::tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess) return nullptr;
    if (q != cudaDriverEntryPointSuccess) return nullptr;
    return reinterpret_cast<EncodeTiledFn>(ptr);
  }();
  return fn;
}

// bf16 [rows, cols] with a row pitch, box of 64 columns x box_rows, 128-byte swizzle, zero fill outside
int make_tmap_bf16_2d(CUtensorMap* map, const void* ptr, uint64_t cols, uint64_t rows, int64_t pitch, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return FR_ERR_CUDA;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch) * 2};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FR_OK : FR_ERR_CUDA;
}

template <int BLOCK_N, int EPI, int ROWS>
static int launch_tc(TcArgs g, const fr_gated_part* parts, cudaStream_t stream) {
  using C = Cfg<BLOCK_N, ROWS>;
  constexpr bool FEW = ROWS == kFew || ROWS == kOctet, PAIR = ROWS == kPair;
  const Stages few(FEW ? g.M : kBlockM, BLOCK_N);
  g.a_bytes = few.a_bytes;
  g.block_bytes = few.block_bytes;
  g.stage_blocks = few.blocks;
  g.stages = few.n;
  const int smem = FEW ? few.smem + (ROWS == kOctet ? kOctetBytes : 0) : 1024 + C::kStages * C::kStageBytes + kBarBytes;
  CUtensorMap ta[2], tb[2];
  for (int p = 0; p < 2; ++p) {
    const fr_gated_part& q = parts[p < g.n_parts ? p : 0];
    int st = make_tmap_bf16_2d(&ta[p], q.a, q.K, g.M, q.lda, FEW ? few.a_rows : kBlockM);
    if (st == FR_OK) st = make_tmap_bf16_2d(&tb[p], q.w, q.K, g.N, q.ldw, C::kTileB);
    if (st != FR_OK) return st;
  }
  auto kern = dense_tc_kernel<BLOCK_N, EPI, ROWS>;
  static PerDeviceFlag attr_done;
  if (ensure_dyn_smem(attr_done, kern, FEW ? 1024 + kOperandBytes + kTileA + kBarBytes + kOctetBytes : smem) != FR_OK) return FR_ERR_CUDA;
  int* status = device_status_ptr();
  if (!status) return FR_ERR_CUDA;
  const int64_t units = static_cast<int64_t>(ceil_div(g.M, C::kTileM)) * ceil_div(g.N, BLOCK_N) *
                        (EPI == kEpiPartial ? g.splits[0] + g.splits[1] : 1);
  const int slots = device_sm_count() / (PAIR ? 2 : 1);
  const int grid = static_cast<int>(units < slots ? units : slots) * (PAIR ? 2 : 1);
  if constexpr (PAIR)
    return launch_cluster(kern, grid, kThreads, smem, stream, 2, g.M <= kPdlRows, ta[0], tb[0], ta[1], tb[1], g, status);
  return launch_kernel(kern, grid, kThreads, smem, stream, g.M <= kPdlRows, ta[0], tb[0], ta[1], tb[1], g, status);
}

// Whether kFew pays: of more than 64 rows little of a row block is left out, and a short product is over before that repays the
// run-time sizes (128 rows x 2048 x 256: 4.46 us with constants, 4.65 with sizes; K = 2048: 12.5 and 11.9; 64 rows x 2048 x 128:
// 3.72 and 3.87; K = 512: 5.5 and 5.2).
static bool few_rows(int M, int64_t K) { return M <= kBlockM && K >= (M <= 64 ? 256 : 1024); }

// Tile width with the least work on the busiest SM: rounds of tiles times the rows of A and B that a tile brings in (`few`: of a
// single row block only its own rows; the update in place brings in whole ones, 16 rows x 20480 x 2048: 32.0 us, 38.4 as if it did not).
// 192 is for a single row block only: there it fills one round of SMs where 256 leaves many idle and 128 begins a second
// (64 rows x 20480 x 2048: 17.9 us; 28 with 80 tiles of 256 and whole tiles of A).
static int pick_block_n(int M, int N, bool few) {
  const int64_t sms = device_sm_count(), mb = ceil_div(M, kBlockM), a_rows = few && M <= kBlockM ? Stages(M, 64).a_rows : kBlockM;
  int best = 0;
  int64_t best_cost = 0;
  for (int bn = 256; bn >= 64; bn -= bn == 128 ? 64 : (few && M <= kBlockM ? 64 : 128)) {
    const int64_t cost = (mb * ceil_div(N, bn) + sms - 1) / sms * (a_rows + bn);
    if (best == 0 || cost < best_cost) {
      best = bn;
      best_cost = cost;
    }
  }
  return best;
}

// Whether tiles of 256 columns are taken by pairs of CTAs: from two rounds of tiles on, unless 256 rows at a time take more rounds. A
// CTA of a pair brings in 32 KB per 128 x 256 x 64 products, alone 48. us, alone / in pairs (same bits): 20480 x 2048 700 rows 55.9 /
// 50.9, 2048 rows 134.7 / 118.4, 8192 rows 516 / 454; 24576 x 4096 2048 rows 304 / 270; update 2048 x 8192 8192 rows 296 / 263; one
// round, 4096 x 2048 700 rows 17.2 / 17.6; three rounds for two, 20480 x 2048 350 rows 33.0 / 36.8.
static bool use_pair(int M, int N) {
  const int64_t sms = device_sm_count(), n_blocks = ceil_div(N, 256);
  const int64_t alone = (ceil_div(M, kBlockM) * n_blocks + sms - 1) / sms, pairs = (ceil_div(M, 2 * kBlockM) * n_blocks + sms / 2 - 1) / (sms / 2);
  return alone >= 2 && pairs <= alone;
}

// Whether a few-row product streams the weights through the row kernel. There a weight costs an FMA per row, rows counted as 1, 2, 4
// or 8: one or two hide them behind the loads, eight do not, four hardly. The tensor cores (kOctet) take 0.18 us per k-block and
// round of tiles and 3 us more, whatever the rows. us, row kernel / tensor cores:
//   8 rows   K = 2048: N = 1536 8.7 / 9.7, 4096 14.2 / 10.3, 20480 60 / 24; K = 4096: 2048 14.2 / 15.9, 2560 17.4 / 15.9; K = 8192:
//            2560 25.7 / 27.7, 4096 35.6 / 28.1; K = 12288: 3072 37.6 / 39.2, 4096 44.7 / 39.6
//   4 rows   K = 2048: 5120 10.2 / 10.2, 8192 14.1 / 10.9, 10240 (two rounds, the second nearly empty) 17.5 / 16.9, 20480 31 / 23;
//            K = 8192: 6144 30.2 / 28.3, 10240 44.6 / 52.1, 14336 57.9 / 52.6
// Below K = 2048 the row kernel's sums are the more accurate ones (6e-8 of the norm at 512, 8e-8 here; 7.5e-8 and 8e-8 at 2048,
// 9.4e-8 and 8e-8 at 12288). With K split over the SMs (a launch that reads the shares follows; K is the sum over the parts):
//   8 rows   K = 2048: 1056 7.9 / 7.2, 4096 16.6 / 11.8; K = 12288: 1056 16.5 / 12.9, 4096 48.6 / 30.6
//   4 rows   K = 2048: 2048 7.7 / 8.4, 4096 9.1 / 11.5; K = 12288: 2048 17.0 / 18.4, 4096 29.1 / 30.4
static bool use_rows(int dtype, int M, int N, int64_t K, bool split_k) {
  if (M > 8) return false;
  if (dtype != 0 || M <= 2 || N <= 1024 || K < 2048) return true;
  if (split_k) return M <= 4;
  if (M > 4) return N <= (K <= 6144 ? 2048 : 3072);
  const int64_t tiles = ceil_div(N, 64), sms = device_sm_count(), rounds = ceil_div(tiles, sms);
  return N <= 4096 || tiles * 5 < rounds * sms * 3;  // less than three fifths of the SMs busy
}

static int rows_ks(int N, int K) {
  // warps per CTA that share a group of four rows along K: several waves of small CTAs, so that the last one is
  // short, as long as a warp keeps two steps of 256 columns
  const int64_t warps = ceil_div(N, 4);
  int ks = 1;
  while (ks < 8 && ((warps * ks < 148 * 16 && K / (ks * 2) >= 256) || (warps * ks < 148 * 96 && K / (ks * 2) >= 512))) ks *= 2;
  return ks;
}

template <typename T>
static int launch_rows_proj(const void* a, int64_t lda, const void* w, int64_t ldw, int M, int N, int K, const Segs& sg,
                            bool ahead, cudaStream_t stream) {
  const int ks = rows_ks(N, K);
  const int grid = ceil_div(ceil_div(N, 4), (kRowsThreads / 32) / ks);
  const T* A = static_cast<const T*>(a);
  const T* W = static_cast<const T*>(w);
  auto go = [&](auto kernel) { return launch_kernel(kernel, grid, kRowsThreads, 0, stream, true, A, lda, W, ldw, M, N, K, sg, ks); };
  if (M == 1) return ahead ? go(dense_rows_proj_kernel<T, 1, true>) : go(dense_rows_proj_kernel<T, 1, false>);
  if (M == 2) return ahead ? go(dense_rows_proj_kernel<T, 2, true>) : go(dense_rows_proj_kernel<T, 2, false>);
  return M <= 4 ? go(dense_rows_proj_kernel<T, 4, false>) : go(dense_rows_proj_kernel<T, 8, false>);
}

template <typename T>
static int launch_rows_gated(const Parts& pt, float* x, int64_t ldx, int M, int N, void* copy_out, int64_t ldc, bool ahead,
                             cudaStream_t stream) {
  T* copy = static_cast<T*>(copy_out);
  int K = 0;
  for (int p = 0; p < pt.n; ++p) K = K > pt.p[p].K ? K : pt.p[p].K;
  const int ks = rows_ks(N, K);
  const int grid = ceil_div(ceil_div(N, 4), (kRowsThreads / 32) / ks);
  auto go = [&](auto kernel) { return launch_kernel(kernel, grid, kRowsThreads, 0, stream, true, pt, x, ldx, M, N, copy, ldc, ks); };
  if (M == 1) return ahead ? go(dense_rows_gated_kernel<T, 1, true>) : go(dense_rows_gated_kernel<T, 1, false>);
  constexpr bool kTwoAhead = sizeof(T) == 4;  // two bf16 rows load nothing ahead
  if (M == 2) return ahead ? go(dense_rows_gated_kernel<T, 2, kTwoAhead>) : go(dense_rows_gated_kernel<T, 2, false>);
  return M <= 4 ? go(dense_rows_gated_kernel<T, 4, false>) : go(dense_rows_gated_kernel<T, 8, false>);
}

static bool operand_ok(const void* p, int64_t ld, int K) {
  return p != nullptr && (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && ld % 8 == 0 && ld >= K && K % 8 == 0 && K > 0;
}

// K shares of the two parts for few-row products: about one work unit per SM in all.
static void plan_splits(int M, int N, int kb0, int kb1, int* s0, int* s1) {
  *s0 = *s1 = 0;
  const int64_t tiles = static_cast<int64_t>(ceil_div(M, kBlockM)) * ceil_div(N, 64);
  if (tiles * 2 > device_sm_count() || M > 1024) return;  // the tiles alone keep the SMs busy
  const int want = static_cast<int>(device_sm_count() / tiles);
  const int total = kb0 + kb1;
  int a = static_cast<int>((static_cast<int64_t>(want) * kb0 + total / 2) / total);
  a = a < 1 ? 1 : (a > (kb0 + 3) / 4 ? (kb0 + 3) / 4 : a);
  int b = 0;
  if (kb1 > 0) {
    b = want - a;
    b = b < 1 ? 1 : (b > (kb1 + 3) / 4 ? (kb1 + 3) / 4 : b);
  }
  *s0 = a;
  *s1 = b;
}

// The same for f32, more than 8 rows: three rounds of CTAs, three of them per SM, with shares of at least 512 columns. Up to 1024
// rows, where the partials that the next launch reads are small beside the product.
static void plan_simt_splits(int M, int N, int K0, int K1, int* s0, int* s1) {
  *s0 = *s1 = 0;
  const int64_t tiles = static_cast<int64_t>(ceil_div(M, 64)) * ceil_div(N, 64), slots = 3 * device_sm_count(), K = static_cast<int64_t>(K0) + K1;
  if (M <= 8 || M > 1024 || tiles >= 2 * slots) return;
  const int64_t want = std::min((3 * slots + tiles - 1) / tiles, K / 512);
  if (want < 2) return;
  const int64_t share = (K / want + kSimtK - 1) / kSimtK * kSimtK;
  *s0 = static_cast<int>((K0 + share - 1) / share);
  *s1 = static_cast<int>((K1 + share - 1) / share);
}

}  // namespace dense

// shared with attn_mix.cu
int make_tmap_bf16_box64(CUtensorMap* map, const void* ptr, uint64_t cols, uint64_t rows, int64_t pitch, uint32_t box_rows) {
  return dense::make_tmap_bf16_2d(map, ptr, cols, rows, pitch, box_rows);
}

}  // namespace fr

using namespace fr;

// Column ranges as the kernels get them; FR_ERR_BAD_ARG when they do not tile the columns as the header says.
static int check_segs(const fr_out_segment* segs, int n_segs, int N, dense::Segs* sg) {
  FR_CHECK_ARG(segs && n_segs > 0 && n_segs <= dense::kMaxSegs);
  sg->n = n_segs;
  for (int i = 0; i < n_segs; ++i) {
    const fr_out_segment& s = segs[i];
    const int end = i + 1 < n_segs ? segs[i + 1].n0 : N;
    FR_CHECK_ARG(s.out && s.n0 % 32 == 0 && s.n > 0 && s.kind >= 0 && s.kind <= FR_SEG_GELU_MUL);
    FR_CHECK_ARG(s.n0 < end && (i > 0 || s.n0 == 0));
    FR_CHECK_ARG(s.kind != FR_SEG_GELU_MUL || s.mul);
    if (dense::paired(s))
      FR_CHECK_ARG(s.n0 % 64 == 0 && (end - s.n0) % 64 == 0 && 2 * s.n <= end - s.n0);
    else
      FR_CHECK_ARG(s.n <= end - s.n0);
    sg->s[i] = s;
  }
  return FR_OK;
}

static bool take_laid_out(int* algo) {
  if (*algo < 0 || (*algo & FR_DENSE_LAID_OUT) == 0) return false;
  *algo &= ~FR_DENSE_LAID_OUT;
  return true;
}

extern "C" int fr_dense_proj(int dtype, const void* a, int64_t lda, const void* w, int64_t ldw, int M, int N, int K,
                             const fr_out_segment* segs, int n_segs, int algo, cudaStream_t stream) {
  FR_CHECK_ARG((dtype == 0 || dtype == 1) && M >= 0 && N > 0);
  if (M == 0) return FR_OK;
  FR_CHECK_ARG(dense::operand_ok(a, lda, K) && dense::operand_ok(w, ldw, K) && N % 4 == 0);
  dense::Segs sg{};
  if (check_segs(segs, n_segs, N, &sg) != FR_OK) return FR_ERR_BAD_ARG;
  const bool ahead = take_laid_out(&algo);
  if (algo == 0) algo = dense::use_rows(dtype, M, N, K, false) ? 1 : 2;
  if (algo == 1) {
    FR_CHECK_SUPPORTED(M <= 8);
    return dtype == 0 ? dense::launch_rows_proj<__nv_bfloat16>(a, lda, w, ldw, M, N, K, sg, ahead, stream)
                      : dense::launch_rows_proj<float>(a, lda, w, ldw, M, N, K, sg, ahead, stream);
  }
  if (dtype == 1) {
    const float* A = static_cast<const float*>(a);
    const float* W = static_cast<const float*>(w);
    // 128 rows per tile take every weight from shared memory half as often; with fewer than a tile per SM 64 spread better, and
    // short products are mostly beginnings and ends of tiles, of which two CTAs per SM hide fewer than three
    // (us, 64 / 128 rows per tile: 128 x 20480 x 64 22.6 / 29.0, 351 x 20480 x 2048 see the kernel)
    const int64_t large = static_cast<int64_t>(ceil_div(N, 64)) * ceil_div(M, 128);
    if (M > 64 && K >= 512 && large >= device_sm_count())
      dense::dense_simt_proj_kernel<128><<<dim3(ceil_div(N, 64), ceil_div(M, 128)), 256, 0, stream>>>(A, lda, W, ldw, M, N, K, sg);
    else
      dense::dense_simt_proj_kernel<64><<<dim3(ceil_div(N, 64), ceil_div(M, 64)), 256, 0, stream>>>(A, lda, W, ldw, M, N, K, sg);
    return launch_status();
  }
  dense::TcArgs g{};
  g.ahead = ahead ? 1 : 0;
  g.M = M;
  g.N = N;
  g.n_parts = 1;
  g.kb[0] = ceil_div(K, dense::kBlockK);
  g.segs = sg;
  fr_gated_part part{a, w, nullptr, lda, ldw, 0, K, 0};
  if (M <= 8) return dense::launch_tc<64, dense::kEpiSegs, dense::kOctet>(g, &part, stream);
  const bool few = dense::few_rows(M, K);
  const int block_n = dense::pick_block_n(M, N, few);
  if (few) {
    switch (block_n) {
      case 256: return dense::launch_tc<256, dense::kEpiSegs, dense::kFew>(g, &part, stream);
      case 192: return dense::launch_tc<192, dense::kEpiSegs, dense::kFew>(g, &part, stream);
      case 128: return dense::launch_tc<128, dense::kEpiSegs, dense::kFew>(g, &part, stream);
      default: return dense::launch_tc<64, dense::kEpiSegs, dense::kFew>(g, &part, stream);
    }
  }
  if (block_n == 256 && dense::use_pair(M, N)) return dense::launch_tc<256, dense::kEpiSegs, dense::kPair>(g, &part, stream);
  switch (block_n) {
    case 256: return dense::launch_tc<256, dense::kEpiSegs, dense::kAny>(g, &part, stream);
    case 128: return dense::launch_tc<128, dense::kEpiSegs, dense::kAny>(g, &part, stream);
    default: return dense::launch_tc<64, dense::kEpiSegs, dense::kAny>(g, &part, stream);
  }
}

extern "C" int fr_dense_proj_split(int dtype, const void* a, int64_t lda, const void* w, int64_t ldw, int M, int N, int K,
                                   const fr_out_segment* segs, int n_segs, float* partials, int n_splits, cudaStream_t stream) {
  FR_CHECK_ARG(M > 0 && M <= 65535 && N > 0 && partials && n_splits > 0);
  dense::Segs sg{};
  if (check_segs(segs, n_segs, N, &sg) != FR_OK) return FR_ERR_BAD_ARG;
  const fr_gated_part part{a, w, nullptr, lda, ldw, 0, K, 0};
  const int r = fr_dense_gated_add(dtype, &part, 1, partials, N, M, N, partials, n_splits, nullptr, 0, 0, stream);  // x is left alone
  if (r != FR_OK) return r;
  auto kern = dtype == 0 ? dense::dense_finish_kernel<__nv_bfloat16> : dense::dense_finish_kernel<float>;
  return launch_kernel(kern, dim3(ceil_div(N, 256), M), 256, 0, stream, M <= kPdlRows, static_cast<const float*>(partials), n_splits, M, N, sg);
}

extern "C" int fr_dense_gated_add_splits(int dtype, int M, int N, int K0, int K1) {
  return M <= 8 || dtype != 0 ? 0 : fr_dense_few_row_splits(dtype, M, N, K0, K1);
}

extern "C" int fr_dense_few_row_splits(int dtype, int M, int N, int K0, int K1) {
  int a, b;
  if (dtype == 1 && M > 0 && N > 0 && K0 > 0) {
    dense::plan_simt_splits(M, N, K0, K1 > 0 ? K1 : 0, &a, &b);
    return a + b;
  }
  if (dtype != 0 || M <= 0 || N <= 0 || K0 <= 0 || dense::use_rows(dtype, M, N, static_cast<int64_t>(K0) + (K1 > 0 ? K1 : 0), true)) return 0;
  dense::plan_splits(M, N, ceil_div(K0, dense::kBlockK), K1 > 0 ? ceil_div(K1, dense::kBlockK) : 0, &a, &b);
  return a + b;
}

extern "C" int fr_dense_gated_add(int dtype, const fr_gated_part* parts, int n_parts, float* x, int64_t ldx, int M, int N,
                                  float* partials, int n_splits, void* copy, int64_t ldc, int algo, cudaStream_t stream) {
  FR_CHECK_ARG((dtype == 0 || dtype == 1) && parts && (n_parts == 1 || n_parts == 2) && M >= 0 && N > 0);
  if (M == 0) return FR_OK;
  FR_CHECK_ARG(x && ldx >= N && (copy == nullptr || (ldc >= N && partials == nullptr)));
  dense::Parts pt{};
  pt.n = n_parts;
  int64_t K = 0;
  for (int p = 0; p < n_parts; ++p) {
    K += parts[p].K;
    FR_CHECK_ARG(dense::operand_ok(parts[p].a, parts[p].lda, parts[p].K) &&
                 dense::operand_ok(parts[p].w, parts[p].ldw, parts[p].K));
    pt.p[p] = parts[p];
  }
  if (partials == nullptr) n_splits = 0;
  const bool ahead = take_laid_out(&algo);
  if (algo == 0) algo = (M <= 8 && n_splits == 0) ? 1 : 2;
  if (algo == 1) {
    FR_CHECK_SUPPORTED(M <= 8 && n_splits == 0);
    return dtype == 0 ? dense::launch_rows_gated<__nv_bfloat16>(pt, x, ldx, M, N, copy, ldc, ahead, stream)
                      : dense::launch_rows_gated<float>(pt, x, ldx, M, N, copy, ldc, ahead, stream);
  }
  if (dtype == 1 && n_splits > 0) {
    int s0, s1;
    dense::plan_simt_splits(M, N, parts[0].K, n_parts > 1 ? parts[1].K : 0, &s0, &s1);
    FR_CHECK_SUPPORTED(s0 > 0 && s0 + s1 == n_splits && (n_parts == 1 || s1 > 0));
    dense::dense_simt_partial_kernel<<<dim3(ceil_div(N, 64), ceil_div(M, 64), n_splits), 256, 0, stream>>>(pt, s0, s1, partials, M, N);
    return launch_status();
  }
  if (dtype == 1) {
    dense::dense_simt_gated_kernel<<<dim3(ceil_div(N, 64), ceil_div(M, 64)), 256, 0, stream>>>(
        pt, x, ldx, M, N, static_cast<float*>(copy), ldc);
    return launch_status();
  }
  dense::TcArgs g{};
  g.ahead = ahead ? 1 : 0;
  g.M = M;
  g.N = N;
  g.n_parts = n_parts;
  g.x = x;
  g.ldx = ldx;
  g.copy = static_cast<__nv_bfloat16*>(copy);
  g.ldc = ldc;
  for (int p = 0; p < n_parts; ++p) {
    g.kb[p] = ceil_div(parts[p].K, dense::kBlockK);
    g.gate[p] = static_cast<const __nv_bfloat16*>(parts[p].gate);
    g.ldg[p] = parts[p].ldg;
  }
  if (n_splits > 0) {
    dense::plan_splits(M, N, g.kb[0], n_parts > 1 ? g.kb[1] : 0, &g.splits[0], &g.splits[1]);
    FR_CHECK_ARG(g.splits[0] > 0 && g.splits[0] + g.splits[1] == n_splits && (n_parts == 1 || g.splits[1] > 0));
    g.partials = partials;
    if (M <= 8) return dense::launch_tc<64, dense::kEpiPartial, dense::kOctet>(g, parts, stream);
    return dense::few_rows(M, K) ? dense::launch_tc<64, dense::kEpiPartial, dense::kFew>(g, parts, stream)
                                 : dense::launch_tc<64, dense::kEpiPartial, dense::kAny>(g, parts, stream);
  }
  const int block_n = dense::pick_block_n(M, N, false);
  if (block_n == 256 && dense::use_pair(M, N)) return dense::launch_tc<256, dense::kEpiAdd, dense::kPair>(g, parts, stream);
  switch (block_n) {
    case 256: return dense::launch_tc<256, dense::kEpiAdd, dense::kAny>(g, parts, stream);
    case 128: return dense::launch_tc<128, dense::kEpiAdd, dense::kAny>(g, parts, stream);
    default: return dense::launch_tc<64, dense::kEpiAdd, dense::kAny>(g, parts, stream);
  }
}
