// bf16 rows of the mixed-map attention (fr_mix_attn_rows in the header): decode steps and short portions, head sizes up to
// 128, in one launch per call.
//
//   flash_rows_kernel  DIFF and PLAIN: a CTA takes one row, one kv head and one share of the visible keys; its warps walk
//                      blocks of 32 keys with running maxima and sums, the shares meet in the cluster's shared memory
//   talk_rows_kernel   TALK: a cluster takes one row, a CTA of it one kv head; the weights of every head stay in shared
//                      memory, where the CTAs of the cluster read each other's to mix them
//
// A row has a few queries per kv head, so nothing here is bound by arithmetic: what counts is the chain of dependent
// loads (position, table row, slots, keys, values) and the instructions per key. The scores of 16 keys and up to 8
// queries are one mma.sync per 16 dimensions, with the keys as its 16-row operand straight from global memory: lane t of
// a quad loads 16 consecutive bytes of a key and the queries are loaded the same way, so both sides see the same
// permutation of the dimensions and the sum is unchanged. Weights stay fp32; weights times values are fp32 FMAs.
// An mma.sync cuts off bits of what it adds up, so each begins at zero and fp32 additions join them, and values are summed per block
// of keys first. With one accumulator throughout a quarter more of the outputs were not the bf16 nearest to the 64-bit result than from
// the general kernels, 3.3e-4 against 2.4e-4 at 800 keys of unit scores; now 2.2e-4 (64 x 2000 PLAIN 90.9 -> 93.7 us, others within 4 %).
// Measured against one kernel that writes all scores to global memory and one that mixes them (caches larger than L2):
//   rows x keys, kv heads          before      here
//   DIFF   1 x  800, 8            18.0 us    9.7 us
//   DIFF  64 x  150, 8            36.4      20.3
//   TALK   1 x  800, 8            23.0      17.5
//   TALK  64 x  150, 8            41.0      20.3
//   PLAIN  1 x   60, 8            13.7       4.8
//   PLAIN  5 x 2000, 8            59.5      24.4
//   PLAIN 64 x 2000, 8           256.0      93.7  (5.6 TB/s)
#include "attn_mix.cuh"

namespace fr {
namespace mix {

// Products of 32 keys of a warp with the queries of one kv head: element (key, source) of `sc` [32][NS]
template <int REP, int MAPS, int NCH>
struct Scores {
  static constexpr int NS = REP * MAPS;
  uint32_t q[MAPS][NCH][4];  // query lane / 4, dimensions 32 j + 8 (lane % 4) ..

  __device__ __forceinline__ void load_queries(const fr_mix_attn& a, int64_t t_row, int g) {
    const int lane = threadIdx.x & 31, n = lane >> 2, t = lane & 3, rep = a.heads / a.kv_heads;
    const __nv_bfloat16* qr = static_cast<const __nv_bfloat16*>(a.q) + t_row * a.ldq;
#pragma unroll
    for (int m = 0; m < MAPS; ++m)
#pragma unroll
      for (int j = 0; j < NCH; ++j) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (n < rep && 32 * j + 8 * t < a.dim) {
          const int src = source_of(a, MAPS * g + m, n);
          v = *reinterpret_cast<const uint4*>(qr + static_cast<int64_t>(src) * a.dim + 32 * j + 8 * t);
        }
        q[m][j][0] = v.x; q[m][j][1] = v.y; q[m][j][2] = v.z; q[m][j][3] = v.w;
      }
  }

  static __device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }

  // of the 32 keys whose slots the lanes hold
  __device__ __forceinline__ void operator()(const fr_mix_attn& a, int g, int slot, float* sc) const {
    const int lane = threadIdx.x & 31, r = lane >> 2, t = lane & 3;
    const __nv_bfloat16* kc = static_cast<const __nv_bfloat16*>(a.k) + static_cast<int64_t>(MAPS * g) * a.dim;
    const __nv_bfloat16* k[4];  // keys r, r + 8, r + 16, r + 24
#pragma unroll
    for (int o = 0; o < 4; ++o) k[o] = kc + static_cast<int64_t>(__shfl_sync(0xffffffffu, slot, o * 8 + r)) * a.ldk;
    constexpr int kMaps = MAPS * NCH <= 4 ? MAPS : 1;  // maps whose loads are in flight before the first product
#pragma unroll
    for (int m0 = 0; m0 < MAPS; m0 += kMaps) {
      uint4 x[4][kMaps][NCH];
#pragma unroll
      for (int o = 0; o < 4; ++o)
#pragma unroll
        for (int m = 0; m < kMaps; ++m)
#pragma unroll
          for (int j = 0; j < NCH; ++j)
            x[o][m][j] = *reinterpret_cast<const uint4*>(k[o] + (m0 + m) * a.dim + (32 * j + 8 * t < a.dim ? 32 * j + 8 * t : 0));
#pragma unroll
      for (int j = 0; j < NCH; ++j)
        if (32 * j + 8 * t >= a.dim) {
#pragma unroll
          for (int o = 0; o < 4; ++o)
#pragma unroll
            for (int m = 0; m < kMaps; ++m) x[o][m][j] = make_uint4(0, 0, 0, 0);
        }
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int m = 0; m < kMaps; ++m) {
          float d[4];
#pragma unroll
          for (int j = 0; j < NCH; ++j) {
            const uint4 &lo = x[2 * half][m][j], &hi = x[2 * half + 1][m][j];
            float e[4] = {0.f, 0.f, 0.f, 0.f}, f[4] = {0.f, 0.f, 0.f, 0.f};
            mma(e, lo.x, hi.x, lo.y, hi.y, q[m0 + m][j][0], q[m0 + m][j][1]);
            mma(f, lo.z, hi.z, lo.w, hi.w, q[m0 + m][j][2], q[m0 + m][j][3]);
#pragma unroll
            for (int y = 0; y < 4; ++y) d[y] = j == 0 ? e[y] + f[y] : d[y] + (e[y] + f[y]);
          }
          float* s0 = sc + (half * 16 + r) * NS + (m0 + m) * REP + 2 * t;
          if (2 * t < REP) {
            s0[0] = d[0];
            s0[8 * NS] = d[2];
          }
          if (2 * t + 1 < REP) {
            s0[1] = d[1];
            s0[8 * NS + 1] = d[3];
          }
        }
    }
  }
};

// acc[n] += sum over the keys of w[key][n] * V[key]; lane vl = lane % VL holds columns 8 vl .., keys 32 / VL at a time.
// Lanes behind vdim repeat the first columns; nobody reads what they hold.
template <int N, int VL>
__device__ __forceinline__ void add_values(const fr_mix_attn& a, int g, int slot, int nk, const float* w, float (&acc)[N][8]) {
  constexpr int kAt = 32 / VL, kFlight = 8;  // loads in flight per lane
  const int lane = threadIdx.x & 31, vl = lane % VL, sub = lane / VL;
  const __nv_bfloat16* vc = static_cast<const __nv_bfloat16*>(a.v) + static_cast<int64_t>(g) * a.vdim + (vl * 8 < a.vdim ? vl * 8 : 0);
#pragma unroll 1
  for (int x0 = 0; x0 * kAt < nk; x0 += kFlight) {
    uint4 raw[kFlight];  // the slot of a key that is not there is the last key's
#pragma unroll
    for (int u = 0; u < kFlight; ++u)
      raw[u] = *reinterpret_cast<const uint4*>(vc + static_cast<int64_t>(__shfl_sync(0xffffffffu, slot, (x0 + u) * kAt + sub)) * a.ldv);
#pragma unroll
    for (int u = 0; u < kFlight; ++u) {
      const int key = (x0 + u) * kAt + sub;
      if (key >= nk) raw[u] = make_uint4(0, 0, 0, 0);  // adds nothing, whatever the last key's values are
      const uint32_t r4[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const float f = w[key * N + n];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc[n][2 * e] = fmaf(f, __uint_as_float(r4[e] << 16), acc[n][2 * e]);
          acc[n][2 * e + 1] = fmaf(f, __uint_as_float(r4[e] & 0xffff0000u), acc[n][2 * e + 1]);
        }
      }
    }
  }
}

// the value row of this lane's key on its way into L2 while the scores are computed
__device__ __forceinline__ void prefetch_value(const fr_mix_attn& a, int g, int slot) {
  const __nv_bfloat16* p = static_cast<const __nv_bfloat16*>(a.v) + static_cast<int64_t>(slot) * a.ldv + static_cast<int64_t>(g) * a.vdim;
  for (int c = 0; c < a.vdim; c += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + c));
}
// and the key row, of the `maps` maps of the kv head
__device__ __forceinline__ void prefetch_key(const fr_mix_attn& a, int maps, int g, int slot) {
  const __nv_bfloat16* p = static_cast<const __nv_bfloat16*>(a.k) + static_cast<int64_t>(slot) * a.ldk + static_cast<int64_t>(maps * g) * a.dim;
  for (int c = 0; c < maps * a.dim; c += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + c));
}

// A row's place and what it sees. Read through L2: with `early` (fr_mix_attn_rows_early) this happens before the launch waits for
// the one that precedes it, and the keys and values of a warp's first blocks are on their way into L2 by then. In steps
// of the 1.7b sizes: one request of 800 keys, DIFF 16.1 -> 15.0 and TALK 18.9 -> 16.6 us behind the projections; 64 requests of 150 keys 26.1
// -> 23.0 and 25.6 -> 20.0 (TALK also has eight CTAs' weights in flight where it mixes them). Running through the instructions once
// before the wait, to have them in the caches, cost what it took (15.0 -> 25.5 us): the launch ahead is nearly over when this begins.
struct Place {
  const int32_t* table;     // slots of the request's positions
  int i, lo, n_first, n;    // own position; the first n_first visible keys lie at 0, the others from lo on
  __device__ __forceinline__ int key(int x) const { return x < n_first ? x : lo + (x - n_first); }
};
__device__ __forceinline__ Place place_of(const fr_mix_attn& a, int64_t t, int max_keys) {
  const int64_t i = __ldcg(a.pos + t);
  const Visible v = visible_keys(a, i, max_keys);
  return Place{a.req_to_token + __ldcg(a.req_rows + __ldcg(a.tok_req + t)) * a.table_stride, static_cast<int>(i), static_cast<int>(v.lo),
               v.n_first, v.n};
}
__device__ __forceinline__ int slot_at(const fr_mix_attn& a, const Place& p, int x) {
  const int s = __ldcg(p.table + p.key(x));
  return s < 0 ? 0 : (s >= a.num_slots ? static_cast<int>(a.num_slots - 1) : s);
}
constexpr int kEarlyBlocks = 2;  // blocks of 32 keys per warp that are brought into L2 before the wait

__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

constexpr int kFlashWarps = 4;

template <int REP, int MAPS, int NCH, int VL>
__global__ void __launch_bounds__(kFlashWarps * 32, REP * MAPS >= 8 ? 2 : (MAPS * NCH > 4 || REP == 4 ? 3 : 4))
flash_rows_kernel(const __grid_constant__ fr_mix_attn a, int row0, int max_keys, int splits, int early) {
  constexpr int NS = REP * MAPS, VP = VL * 8;
  __shared__ __align__(16) float sc[kFlashWarps][32 * NS];
  __shared__ float o_w[kFlashWarps][NS * VP];  // per warp; afterwards the CTA's sum in the first
  __shared__ float m_w[kFlashWarps][NS], l_w[kFlashWarps][NS];
  __shared__ float m_c[NS], l_c[NS], red[kFlashWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int split = blockIdx.x, g = blockIdx.y;
  const int rep = a.heads / a.kv_heads;
  const int64_t t = row0 + static_cast<int64_t>(blockIdx.z);
  Place at;
  int k_lo, k_hi, k0, next;
  auto slot = [&](int base) {  // behind the last key: the last one's, loaded and not used
    return slot_at(a, at, min(base + lane, k_hi - 1));
  };
  auto begin = [&] {
    at = place_of(a, t, max_keys);
    const int per = ((at.n + splits - 1) / splits + 31) / 32 * 32;  // whole blocks per share
    k_lo = min(split * per, at.n);
    k_hi = min(k_lo + per, at.n);
    k0 = k_lo + warp * 32;
    next = k0 < k_hi ? slot(k0) : 0;
  };
  if (early) {
    begin();
    for (int b = 0, k = k0; b < kEarlyBlocks && k < k_hi; ++b, k += kFlashWarps * 32) {
      const int x = b == 0 ? next : slot(k);
      prefetch_key(a, MAPS, g, x);
      prefetch_value(a, g, x);
    }
  }
  ptx::griddep_wait();
  ptx::griddep_launch_dependents();
  if (!early) begin();
  Scores<REP, MAPS, NCH> scores;
  scores.load_queries(a, t, g);
  float m[NS], l[NS], acc[NS][8] = {};
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    m[s] = -INFINITY;
    l[s] = 0.f;
  }
  float* my = sc[warp];
  for (; k0 < k_hi; k0 += kFlashWarps * 32) {
    const int here = next, nk = min(32, k_hi - k0);
    const bool more = k0 + kFlashWarps * 32 < k_hi;
    if (more) next = slot(k0 + kFlashWarps * 32);
    prefetch_value(a, g, here);
    __syncwarp();
    scores(a, g, here, my);
    __syncwarp();
    if (more) prefetch_key(a, MAPS, g, next);
    const float dist = static_cast<float>(at.i - at.key(k0 + min(lane, nk - 1)));
    float p[NS], fade[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      float v = my[lane * NS + s] * a.scale;
      if (a.slopes != nullptr && s % REP < rep) v -= a.slopes[source_of(a, MAPS * g + s / REP, s % REP)] * dist;
      v = lane < nk ? v : -INFINITY;
      const float mn = fmaxf(m[s], warp_max(v));
      // scores of -inf (behind the last key, or an infinite key) weigh nothing, also while no finite one has been seen
      const float corr = m[s] == -INFINITY ? 0.f : expf(m[s] - mn);
      p[s] = v == -INFINITY ? 0.f : expf(v - mn);
      l[s] = l[s] * corr + p[s];
      m[s] = mn;
      fade[s] = corr;
    }
    float blk[NS][8] = {};
#pragma unroll
    for (int s = 0; s < NS; ++s) my[lane * NS + s] = p[s];
    __syncwarp();
    add_values<NS, VL>(a, g, here, nk, my, blk);
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[s][e] = fmaf(acc[s][e], fade[s], blk[s][e]);
  }
  // the warps' shares, then the CTAs'
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const float ls = warp_sum(l[s]);
    if (lane == 0) {
      m_w[warp][s] = m[s];
      l_w[warp][s] = ls;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float v = acc[s][e];
#pragma unroll
      for (int o = VL; o < 32; o *= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane < VL) o_w[warp][s * VP + lane * 8 + e] = v;
    }
  }
  __syncthreads();
  // no key above -inf: no share. Its sums are zero then, or NaN from a NaN score, which has to reach the output.
  auto weight = [](float mw, float mx) { return mw == -INFINITY ? 0.f : expf(mw - mx); };
  if (tid < NS) {
    float mx = m_w[0][tid], ls = 0.f;
    for (int w = 1; w < kFlashWarps; ++w) mx = fmaxf(mx, m_w[w][tid]);
    for (int w = 0; w < kFlashWarps; ++w) {
      const float f = weight(m_w[w][tid], mx);
      ls += l_w[w][tid] * f;
      m_w[w][tid] = f;  // the warp's factor from here on
    }
    m_c[tid] = mx;
    l_c[tid] = ls;
  }
  __syncthreads();
  for (int c = tid; c < NS * VP; c += kFlashWarps * 32) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kFlashWarps; ++w) v += o_w[w][c] * m_w[w][c / VP];
    o_w[0][c] = v;
  }
  if (splits > 1) cluster_sync(); else __syncthreads();
  // output head g * rep + n belongs to CTA n % splits of the cluster; a thread has one column
  for (int n = split; n < rep; n += splits) {
    float f = 0.f;
    const bool col = tid < VP;
    if (splits == 1) {
      if (col) {
        f = o_w[0][n * VP + tid] / l_c[n];
        if (MAPS == 2) f -= a.lambda * (o_w[0][(REP + n) * VP + tid] / l_c[REP + n]);
      }
    } else {
#pragma unroll
      for (int mp = 0; mp < MAPS; ++mp) {
        const int s = mp * REP + n;
        const uint32_t am = ptx::smem_u32(&m_c[s]), al = ptx::smem_u32(&l_c[s]), ao = ptx::smem_u32(&o_w[0][s * VP + (col ? tid : 0)]);
        float mc[8], lc[8], oc[8], mx = -INFINITY;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          mc[c] = -INFINITY;
          lc[c] = oc[c] = 0.f;
          if (c < splits) {
            mc[c] = ld_cluster(ptx::mapa(am, c));
            lc[c] = ld_cluster(ptx::mapa(al, c));
            oc[c] = ld_cluster(ptx::mapa(ao, c));
          }
          mx = fmaxf(mx, mc[c]);
        }
        float ls = 0.f, os = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float w = weight(mc[c], mx);
          ls += lc[c] * w;
          os += oc[c] * w;
        }
        f += (mp == 0 ? 1.0f : -a.lambda) * (os / ls);
      }
    }
    const int head = g * rep + n;
    float r = 1.0f;
    if (MAPS == 2) {
      const float ss = warp_sum(tid < a.vdim ? f * f : 0.f);  // the head's own padding holds zero
      __syncthreads();
      if (lane == 0) red[warp] = ss;
      __syncthreads();
      float tot = 0.f;
#pragma unroll
      for (int w = 0; w < kFlashWarps; ++w) tot += red[w];
      r = a.out_scale / sqrtf(tot / static_cast<float>(a.vdim_true) + a.eps);
    } else if (a.head_gate != nullptr) {
      r = 1.0f / (1.0f + expf(-a.head_gate[t * a.ld_gate + head]));
    }
    if (col && tid < a.vdim) {
      __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out) + t * a.ldo + static_cast<int64_t>(head) * a.vdim;
      out[tid] = __float2bfloat16_rn(f * r);
    }
  }
  if (splits > 1) cluster_sync();  // nobody leaves while its shares are read
}

// ---------------------------------------------------------------------------
// TALK: cluster of kv_heads CTAs
// ---------------------------------------------------------------------------
constexpr int kTalkSmem = 96 * 1024;
constexpr int kTalkWarps = 16;  // of a CTA when there are few rows

static int talk_smem(int rep_p, int heads, int max_keys, int warps, int vp) {
  const int cap = (max_keys + 31) / 32 * 32;
  // [rep_p][cap] weights, [cap][rep_p] mixed, [cap] slots, [heads][rep_p] coefficients, [warps][rep_p][vp] sums
  return (2 * rep_p * cap + cap + heads * rep_p + warps * rep_p * vp) * 4;
}

template <int REP, int NCH, int VL, int W>
__global__ void __launch_bounds__(W * 32, W == 4 ? 4 : 1)
talk_rows_kernel(const __grid_constant__ fr_mix_attn a, int row0, int max_keys, int early) {
  constexpr int VP = VL * 8;
  extern __shared__ __align__(16) float smem[];
  __shared__ __align__(16) float sc[W][32 * REP];
  __shared__ float red[W][REP], il[REP];
  const int cap = (max_keys + 31) / 32 * 32, rep = a.heads / a.kv_heads;
  float* pw = smem;                              // [REP][cap]
  float* mw = pw + REP * cap;                    // [cap][REP]
  int* slots = reinterpret_cast<int*>(mw + REP * cap);
  float* cf = reinterpret_cast<float*>(slots + cap);  // [heads][REP]
  float* o_w = cf + a.heads * REP;               // [W][REP][VP]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int g = blockIdx.x;
  const int64_t t = row0 + static_cast<int64_t>(blockIdx.y);
  Place at;
  auto begin = [&] {
    for (int e = tid; e < a.heads * REP; e += W * 32) {  // coefficient of source s in output o of this kv head
      const int s = e / REP, o = e % REP;
      cf[e] = o < rep ? a.coef[static_cast<int64_t>(g * rep + o) * a.heads + s] : 0.f;
    }
    at = place_of(a, t, max_keys);
    for (int k0 = warp * 32, b = 0; k0 < at.n; k0 += W * 32, ++b) {
      const int x = slot_at(a, at, min(k0 + lane, at.n - 1));
      slots[k0 + lane] = x;
      if (b < kEarlyBlocks) {
        if (early) prefetch_key(a, 1, g, x);
        prefetch_value(a, g, x);
      }
    }
  };
  if (early) begin();
  ptx::griddep_wait();
  ptx::griddep_launch_dependents();
  if (!early) begin();
  const int n = at.n;
  Scores<REP, 1, NCH> scores;
  scores.load_queries(a, t, g);
  float mx[REP];
#pragma unroll
  for (int s = 0; s < REP; ++s) mx[s] = -INFINITY;
  float* my = sc[warp];
  for (int k0 = warp * 32; k0 < n; k0 += W * 32) {
    const int idx = min(k0 + lane, n - 1);
    __syncwarp();
    scores(a, g, slots[k0 + lane], my);
    __syncwarp();
    const float dist = static_cast<float>(at.i - at.key(idx));
#pragma unroll
    for (int s = 0; s < REP; ++s) {
      float v = my[lane * REP + s] * a.scale;
      if (a.slopes != nullptr && s < rep) v -= a.slopes[g * rep + s] * dist;
      if (k0 + lane >= n) v = -INFINITY;
      pw[s * cap + k0 + lane] = v;
      mx[s] = fmaxf(mx[s], v);
    }
  }
#pragma unroll
  for (int s = 0; s < REP; ++s) {
    const float v = warp_max(mx[s]);
    if (lane == 0) red[warp][s] = v;
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < REP; ++s) {
    mx[s] = red[0][s];
#pragma unroll
    for (int w = 1; w < W; ++w) mx[s] = fmaxf(mx[s], red[w][s]);
  }
  __syncthreads();
  const int n32 = (n + 31) / 32 * 32;
#pragma unroll
  for (int s = 0; s < REP; ++s) {
    float l = 0.f;
    for (int k = tid; k < n32; k += W * 32) {
      const float e = k < n ? expf(pw[s * cap + k] - mx[s]) : 0.f;
      pw[s * cap + k] = e;
      l += e;
    }
    l = warp_sum(l);
    if (lane == 0) red[warp][s] = l;
  }
  __syncthreads();
  if (tid < REP) {
    float l = 0.f;
    for (int w = 0; w < W; ++w) l += red[w][tid];
    il[tid] = 1.0f / l;
  }
  cluster_sync();  // every head's weights and sums are there
  for (int e = tid; e < a.heads * REP; e += W * 32) {
    const int s = e / REP;
    cf[e] *= ld_cluster(ptx::mapa(ptx::smem_u32(&il[s % rep]), s / rep));
  }
  __syncthreads();
  for (int k = tid; k < n32; k += W * 32) {
    float w[REP] = {};
    constexpr int kAhead = REP <= 2 ? 8 : (REP == 4 ? 4 : 2);  // CTAs whose weights are in flight; at most 16 registers
    for (int c0 = 0; c0 < a.kv_heads; c0 += kAhead) {
      float e[kAhead][REP];
#pragma unroll
      for (int c = 0; c < kAhead; ++c) {
        if (c0 + c >= a.kv_heads) break;
        const uint32_t base = ptx::mapa(ptx::smem_u32(pw + k), c0 + c);
#pragma unroll
        for (int s = 0; s < REP; ++s)
          if (s < rep) e[c][s] = ld_cluster(base + s * cap * 4);
      }
#pragma unroll
      for (int c = 0; c < kAhead; ++c) {
        if (c0 + c >= a.kv_heads) break;
#pragma unroll
        for (int s = 0; s < REP; ++s) {
          if (s >= rep) break;
          const float* f = cf + ((c0 + c) * rep + s) * REP;
#pragma unroll
          for (int o = 0; o < REP; ++o) w[o] = fmaf(f[o], e[c][s], w[o]);
        }
      }
    }
#pragma unroll
    for (int o = 0; o < REP; ++o) mw[k * REP + o] = w[o];
  }
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // done with the others' memory
  float acc[REP][8] = {};
  for (int k0 = warp * 32; k0 < n; k0 += W * 32) {
    float blk[REP][8] = {};
    add_values<REP, VL>(a, g, slots[k0 + lane], min(32, n - k0), mw + k0 * REP, blk);
#pragma unroll
    for (int o = 0; o < REP; ++o)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[o][e] += blk[o][e];
  }
#pragma unroll
  for (int o = 0; o < REP; ++o)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float v = acc[o][e];
#pragma unroll
      for (int x = VL; x < 32; x *= 2) v += __shfl_xor_sync(0xffffffffu, v, x);
      if (lane < VL) o_w[(warp * REP + o) * VP + lane * 8 + e] = v;
    }
  __syncthreads();
  for (int c = tid; c < rep * VP; c += W * 32) {
    const int o = c / VP, col = c % VP;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) v += o_w[(w * REP + o) * VP + col];
    if (col < a.vdim)
      static_cast<__nv_bfloat16*>(a.out)[t * a.ldo + static_cast<int64_t>(g * rep + o) * a.vdim + col] = __float2bfloat16_rn(v);
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // nobody leaves while its weights are read
}

template <int REP, int MAPS, int NCH, int VL>
static int launch_flash(const fr_mix_attn& a, int row0, int n_rows, int max_keys, bool early, cudaStream_t stream) {
  // shares of the keys while two CTAs per SM are not reached and a share keeps its four warps busy
  int splits = 1;
  const int64_t ctas = static_cast<int64_t>(n_rows) * a.kv_heads;
  while (splits < 8 && ctas * splits * 2 <= 2 * device_sm_count() && max_keys > splits * 32 * kFlashWarps) splits *= 2;
  return launch_cluster(flash_rows_kernel<REP, MAPS, NCH, VL>, dim3(splits, a.kv_heads, n_rows), kFlashWarps * 32, 0, stream, splits,
                        n_rows <= kPdlRows, a, row0, max_keys, splits, early ? 1 : 0);
}

template <int REP, int NCH, int VL, int W>
static int launch_talk(const fr_mix_attn& a, int row0, int n_rows, int max_keys, bool early, cudaStream_t stream) {
  const int smem = talk_smem(REP, a.heads, max_keys, W, VL * 8);
  static PerDeviceFlag f;
  if (ensure_dyn_smem(f, talk_rows_kernel<REP, NCH, VL, W>, kTalkSmem) != FR_OK) return FR_ERR_CUDA;
  return launch_cluster(talk_rows_kernel<REP, NCH, VL, W>, dim3(a.kv_heads, n_rows), W * 32, smem, stream, a.kv_heads, n_rows <= kPdlRows,
                        a, row0, max_keys, early ? 1 : 0);
}

template <int REP, int NCH, int VL>
static int launch_sizes(const fr_mix_attn& a, int row0, int n_rows, int max_keys, bool early, cudaStream_t stream) {
  if (a.mix == FR_MIX_PLAIN) return launch_flash<REP, 1, NCH, VL>(a, row0, n_rows, max_keys, early, stream);
  if (a.mix == FR_MIX_DIFF) {
    if constexpr (REP <= 4) return launch_flash<REP, 2, NCH, VL>(a, row0, n_rows, max_keys, early, stream);
    return FR_ERR_UNSUPPORTED;
  }
  // many rows: small CTAs, so that all of them are resident at once; few: more warps per head
  if (static_cast<int64_t>(n_rows) * a.kv_heads > device_sm_count()) return launch_talk<REP, NCH, VL, 4>(a, row0, n_rows, max_keys, early, stream);
  return launch_talk<REP, NCH, VL, kTalkWarps>(a, row0, n_rows, max_keys, early, stream);
}

template <int REP>
static int launch_rep(const fr_mix_attn& a, int row0, int n_rows, int max_keys, bool early, cudaStream_t stream) {
  if (a.dim <= 64) {
    if (a.vdim <= 64) return launch_sizes<REP, 2, 8>(a, row0, n_rows, max_keys, early, stream);
    return launch_sizes<REP, 2, 16>(a, row0, n_rows, max_keys, early, stream);
  }
  if (a.vdim <= 64) return launch_sizes<REP, 4, 8>(a, row0, n_rows, max_keys, early, stream);
  return launch_sizes<REP, 4, 16>(a, row0, n_rows, max_keys, early, stream);
}

// Whether one launch does it: bf16, heads of at most 128, up to 8 heads per kv head (DIFF 4: two maps each), and for TALK
// a cluster of at most 8 CTAs whose weights fit into shared memory (two heads per kv head: about 4000 keys).
bool fused_rows_fit(const fr_mix_attn& a, int max_keys) {
  const int rep = a.heads / a.kv_heads;
  if (a.dtype != 0 || a.dim > 128 || a.vdim > 128 || rep > (a.mix == FR_MIX_DIFF ? 4 : 8) || a.num_slots > 0x7fffffff) return false;
  if (a.mix != FR_MIX_TALK) return true;
  const int rep_p = rep <= 1 ? 1 : (rep <= 2 ? 2 : (rep <= 4 ? 4 : 8));
  return (a.kv_heads & (a.kv_heads - 1)) == 0 && a.kv_heads <= 8 && a.heads <= 64 && max_keys <= 8192 &&
         talk_smem(rep_p, a.heads, max_keys, kTalkWarps, a.vdim <= 64 ? 64 : 128) <= kTalkSmem;
}

int fused_rows(const fr_mix_attn& a, int row0, int n_rows, int max_keys, bool early, cudaStream_t stream) {
  const int rep = a.heads / a.kv_heads;
  if (rep == 1) return launch_rep<1>(a, row0, n_rows, max_keys, early, stream);
  if (rep == 2) return launch_rep<2>(a, row0, n_rows, max_keys, early, stream);
  if (rep <= 4) return launch_rep<4>(a, row0, n_rows, max_keys, early, stream);
  return launch_rep<8>(a, row0, n_rows, max_keys, early, stream);
}

}  // namespace mix
}  // namespace fr
