// Decode-time attention over the contiguous ring-buffer KV cache, and the cache update kernels.
//
// A decode step has 1 query token per sequence (or 1 + S at a chunk boundary: the last text token of the chunk and
// its S summary tokens).  Every query attends ONE contiguous slice [start, start + len) of its sequence's cache
// (layout [scratch | current chunk | sliding-chunk ring | summaries | headroom], keys cached after RoPE, so physical
// order does not matter and no mask is needed inside the slice).  The work is bound by reading K and V once:
//   * grid (splits, KV heads, batch): a CTA stages 64-key tiles of K and V in shared memory with coalesced 16-byte
//     loads (rows padded by one word -> conflict-free "thread = key" reads) and serves all G * Tq queries that share
//     the KV head from the same tile (GQA heads are never re-read or materialised);
//   * partial (max, sum, out) per split go to a scratch buffer; a second kernel merges the splits.
// Slices, slot indices and enable flags are device tensors, so one captured launch serves every step.
//
// Replaces SDPA over a repeat_kv-expanded slice plus copy_ ops in the reference's HF model
// (examples/pretrain/hf_template/modeling_qwen3sa.py:306-434, :591-612, :816-876).
#include "common.cuh"
#include "host.h"

namespace ksa {

constexpr int kDecThreads = 128;
constexpr int kDecTile = 64;       // keys per shared-memory tile
constexpr int kDecKeys = 16;       // keys per iteration of a warp of the tensor-core variant
constexpr int kDecMaxQ = 16;       // queries (G * Tq) served per CTA
constexpr int kDecMaxSplits = 64;  // splits of the key range when the last split merges them itself

struct DecodeArgs {
  const bf16* q;        // [B, Tq] rows of Hq heads, `q_rs` elements apart
  const bf16* k_cache;  // [B, Hkv, cap, D]
  const bf16* v_cache;
  const int* start;     // [B, Tq]
  const int* len;       // [B, Tq]
  float* part_o;        // [B, Tq, Hq, splits, D]
  float* part_ml;       // [B, Tq, Hq, splits, 2]
  bf16* out;            // [B, Tq, Hq, D]
  int B, Tq, Hq, Hkv, D, cap, splits, keys_per_split;   // keys_per_split 0: an even share of each slice
  float scale;
  long long q_rs;
  int* counters;        // [B * Hkv] zeros, or null: with counters the last split of a KV group to finish merges the
                        // splits itself (and puts the counter back to zero); without, decode_combine_kernel does
};

// Called by every thread of a CTA after it has written its split's partial results.  The CTA that finishes last for
// its (batch, KV head) merges all splits of the group's nq = G * Tq queries into `out`.
__device__ __forceinline__ void combine_if_last(const DecodeArgs& a, int b, int kvh, int nq, int G) {
  if (a.counters == nullptr) return;
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const int prev = atomicAdd(&a.counters[b * a.Hkv + kvh], 1);
    s_last = prev == a.splits - 1;
    if (s_last) a.counters[b * a.Hkv + kvh] = 0;      // ready for the next launch on this stream
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // weights of the splits: stage (max, sum) of every (query, split), then one thread per query turns them into
  // exp(m_split - m) / l; the outputs are then plain weighted sums with independent loads
  __shared__ float s_w[kDecMaxQ][kDecMaxSplits], s_ls[kDecMaxQ][kDecMaxSplits];
  const int D = a.D, S = a.splits;
  for (int i = threadIdx.x; i < nq * S; i += blockDim.x) {
    const int q = i / S, sp = i - q * S;
    const long long row = ((long long)b * a.Tq + q / G) * a.Hq + kvh * G + q % G;
    s_w[q][sp] = __ldcg(a.part_ml + (row * S + sp) * 2);
    s_ls[q][sp] = __ldcg(a.part_ml + (row * S + sp) * 2 + 1);
  }
  __syncthreads();
  if (threadIdx.x < nq) {
    const int q = threadIdx.x;
    float m = -INFINITY, l = 0.f;
    for (int sp = 0; sp < S; ++sp) m = fmaxf(m, s_w[q][sp]);
    for (int sp = 0; sp < S; ++sp) {
      const float f = s_w[q][sp] == -INFINITY ? 0.f : __expf(s_w[q][sp] - m);
      s_w[q][sp] = f;
      l += s_ls[q][sp] * f;
    }
    const float inv = l > 0.f ? 1.f / l : 0.f;
    for (int sp = 0; sp < S; ++sp) s_w[q][sp] *= inv;
  }
  __syncthreads();
  // a thread takes one head dimension of four queries at once and asks for sixteen partial results before it adds any: the merge is a
  // chain of loads from other SMs' writes, and with one query at a time it was half of a short slice's time
  constexpr int QB = 4, SB = 4;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    for (int q0 = 0; q0 < nq; q0 += QB) {
      long long row[QB];
      float o[QB];
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        const int q = min(q0 + u, nq - 1);
        row[u] = ((long long)b * a.Tq + q / G) * a.Hq + kvh * G + q % G;
        o[u] = 0.f;
      }
      for (int sp = 0; sp < S; sp += SB) {
        float v[QB][SB];
#pragma unroll
        for (int u = 0; u < QB; ++u)
#pragma unroll
          for (int w = 0; w < SB; ++w) v[u][w] = sp + w < S ? __ldcg(a.part_o + (row[u] * S + sp + w) * D + d) : 0.f;
#pragma unroll
        for (int u = 0; u < QB; ++u)
#pragma unroll
          for (int w = 0; w < SB; ++w)
            if (sp + w < S) o[u] = fmaf(v[u][w], s_w[min(q0 + u, nq - 1)][sp + w], o[u]);
      }
#pragma unroll
      for (int u = 0; u < QB; ++u)
        if (q0 + u < nq) a.out[row[u] * D + d] = __float2bfloat16(o[u]);
    }
  }
}

template <int D>
__global__ void __launch_bounds__(kDecThreads) decode_attn_kernel(DecodeArgs a) {
  grid_dependency_launch();   // the successor may start now: in a decode step it is a projection that reads its weights first
  grid_dependency_wait();     // the previous kernel's results are complete from here on
  constexpr int ROW_W = D / 2 + 1;  // 32-bit words per padded row
  __shared__ uint32_t k_s[kDecTile * ROW_W];
  __shared__ uint32_t v_s[kDecTile * ROW_W];
  __shared__ float q_s[kDecMaxQ * D];
  __shared__ float p_s[kDecMaxQ * kDecTile];
  __shared__ float m_s[kDecMaxQ], l_s[kDecMaxQ], corr_s[kDecMaxQ];
  __shared__ int s_start[kDecMaxQ], s_end[kDecMaxQ];
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int G = a.Hq / a.Hkv;
  const int nq = G * a.Tq;  // query index qi = t * G + g
  const int tid = threadIdx.x;
  for (int i = tid; i < nq * D; i += kDecThreads) {
    const int qi = i / D, d = i % D, t = qi / G, g = qi % G;
    q_s[i] = __bfloat162float(a.q[((long long)b * a.Tq + t) * a.q_rs + (kvh * G + g) * D + d]) * a.scale;
  }
  if (tid < nq) {
    const int t = tid / G;
    const int st = a.start[b * a.Tq + t];
    s_start[tid] = max(st, 0);
    s_end[tid] = min(st + a.len[b * a.Tq + t], a.cap);     // whatever the device holds as slices: never past the cache
    m_s[tid] = -INFINITY;
    l_s[tid] = 0.f;
  }
  __syncthreads();
  int lo = a.cap, hi = 0;
  for (int qi = 0; qi < nq; ++qi) { lo = min(lo, s_start[qi]); hi = max(hi, s_end[qi]); }
  const int k0 = lo + split * a.keys_per_split;
  const int k1 = min(hi, k0 + a.keys_per_split);
  // output accumulators: thread owns dims d = tid, tid + 128, ... for every query
  constexpr int DPT = (D + kDecThreads - 1) / kDecThreads;
  float acc[kDecMaxQ][DPT];
#pragma unroll
  for (int qi = 0; qi < kDecMaxQ; ++qi)
#pragma unroll
    for (int j = 0; j < DPT; ++j) acc[qi][j] = 0.f;
  const bf16* kb = a.k_cache + ((long long)b * a.Hkv + kvh) * a.cap * D;
  const bf16* vb = a.v_cache + ((long long)b * a.Hkv + kvh) * a.cap * D;
  for (int kt = k0; kt < k1; kt += kDecTile) {
    const int nkeys = min(kDecTile, k1 - kt);
    __syncthreads();
    for (int i = tid; i < nkeys * (D / 8); i += kDecThreads) {
      const int r = i / (D / 8), v = i % (D / 8);
      const uint4 ku = *reinterpret_cast<const uint4*>(kb + (long long)(kt + r) * D + v * 8);
      const uint4 vu = *reinterpret_cast<const uint4*>(vb + (long long)(kt + r) * D + v * 8);
      uint32_t* kd = k_s + r * ROW_W + v * 4;
      uint32_t* vd = v_s + r * ROW_W + v * 4;
      kd[0] = ku.x; kd[1] = ku.y; kd[2] = ku.z; kd[3] = ku.w;
      vd[0] = vu.x; vd[1] = vu.y; vd[2] = vu.z; vd[3] = vu.w;
    }
    __syncthreads();
    // scores: thread -> (key = tid % 64, queries qi = tid / 64, +2, ...)
    {
      const int r = tid % kDecTile;
      for (int qi = tid / kDecTile; qi < nq; qi += kDecThreads / kDecTile) {
        float s = -INFINITY;
        const int key = kt + r;
        if (r < nkeys && key >= s_start[qi] && key < s_end[qi]) {
          s = 0.f;
          const uint32_t* row = k_s + r * ROW_W;
          const float* qv = q_s + qi * D;
#pragma unroll 8
          for (int w = 0; w < D / 2; ++w) {
            const float2 f = unpack_bf16x2(row[w]);
            s += qv[2 * w] * f.x + qv[2 * w + 1] * f.y;
          }
        }
        p_s[qi * kDecTile + r] = s;
      }
    }
    __syncthreads();
    // online softmax state per query: one warp per query (strided)
    for (int qi = tid >> 5; qi < nq; qi += kDecThreads >> 5) {
      const int lane = tid & 31;
      const float s0 = p_s[qi * kDecTile + lane], s1 = p_s[qi * kDecTile + lane + 32];
      const float mx = warp_max(fmaxf(s0, s1));
      const float m_old = m_s[qi];
      const float m_new = fmaxf(m_old, mx);
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float p0 = __expf(s0 - m_use), p1 = __expf(s1 - m_use);
      p_s[qi * kDecTile + lane] = p0;
      p_s[qi * kDecTile + lane + 32] = p1;
      const float sum = warp_sum(p0 + p1);
      if (lane == 0) {
        const float c = m_old == -INFINITY ? 0.f : __expf(m_old - m_use);
        corr_s[qi] = c;
        l_s[qi] = l_s[qi] * c + sum;
        m_s[qi] = m_new;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < DPT; ++j) {
      const int d = tid + j * kDecThreads;
      if (d < D) {
        const bf16* vcol = reinterpret_cast<const bf16*>(v_s) + d;
#pragma unroll
        for (int qi = 0; qi < kDecMaxQ; ++qi) {
          if (qi < nq) {
            float o = acc[qi][j] * corr_s[qi];
            const float* pr = p_s + qi * kDecTile;
            for (int r = 0; r < nkeys; ++r) o += pr[r] * __bfloat162float(vcol[r * ROW_W * 2]);
            acc[qi][j] = o;
          }
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int qi = 0; qi < kDecMaxQ; ++qi) {
    if (qi < nq) {
      const int t = qi / G, g = qi % G;
      const long long base = ((((long long)b * a.Tq + t) * a.Hq + kvh * G + g) * a.splits + split);
#pragma unroll
      for (int j = 0; j < DPT; ++j) {
        const int d = tid + j * kDecThreads;
        if (d < D) a.part_o[base * D + d] = acc[qi][j];
      }
      if (tid == 0) {
        a.part_ml[base * 2] = m_s[qi];
        a.part_ml[base * 2 + 1] = l_s[qi];
      }
    }
  }
  combine_if_last(a, b, kvh, nq, G);
}

// ------------------------------------------------------------------------------------------ tensor-core variant
// Same interface and the same split / combine scheme, but a key is read from global memory exactly once and never
// staged in shared memory.  Scores: warp-level mma.sync m16n8k16 with the (up to 16) queries of the KV group as the
// 16-row operand and 8 keys as the 8-column operand; a lane loads 16 contiguous bytes of a key (and of a query) and
// hands them to two MMAs as k slots {2t, 2t+1, 2t+8, 2t+9}, a permutation of the head dimension that is the same on
// both sides.  Probabilities go through a 1 KB per-warp shared buffer so that the P.V product runs with
// "lane = 4 head dimensions" (V rows are read as 8 bytes per lane, coalesced) on the FMA units.
__device__ __forceinline__ void mma_qk(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One warp's share of a split: sixteen keys at a time, W warps in turn.  Leaves the rows' maxima and sums (rows g and g + 8 of this lane's
// group, log2 units, the sums complete over the four lanes of a row) and the unscaled outputs of its four head dimensions.
template <int NQ, int W>
__device__ __forceinline__ void decode_warp(const DecodeArgs& a, int split, int kvh, int b, int warp, int lane, float (*s_p)[NQ],
                                            float (&acc)[NQ][4], float& m0, float& m1, float& l0, float& l1) {
  constexpr int D = 128, KPI = kDecKeys;
  const int G = a.Hq / a.Hkv;
  const int nq = G * a.Tq;
  const int g = lane >> 2, t = lane & 3;
  // per-row (g and g+8) slice bounds, and the CTA's key range
  int st0 = 0, en0 = 0, st1 = 0, en1 = 0, lo = a.cap, hi = 0;
  for (int qi = 0; qi < nq; ++qi) {
    int s = a.start[b * a.Tq + qi / G];
    const int e = min(s + a.len[b * a.Tq + qi / G], a.cap);      // whatever the device holds as slices: never past the cache
    s = max(s, 0);
    lo = min(lo, s); hi = max(hi, e);
    if (qi == g) { st0 = s; en0 = e; }
    if (qi == g + 8) { st1 = s; en1 = e; }
  }
  const int per = a.keys_per_split > 0 ? a.keys_per_split : (max(hi - lo, 0) + a.splits * KPI - 1) / (a.splits * KPI) * KPI;
  const int k0 = lo + split * per;
  const int k1 = min(hi, k0 + per);
  // query fragments: row g and row g+8, 4 blocks of 32 head dimensions
  uint4 qa[4], qb[4];
#pragma unroll
  for (int blk = 0; blk < 4; ++blk) {
    qa[blk] = make_uint4(0, 0, 0, 0);
    qb[blk] = make_uint4(0, 0, 0, 0);
    if (g < nq) {
      const int tq = g / G, gg = g % G;
      qa[blk] = *reinterpret_cast<const uint4*>(a.q + ((long long)b * a.Tq + tq) * a.q_rs + (kvh * G + gg) * D + blk * 32 + t * 8);
    }
    if (NQ > 8 && g + 8 < nq) {
      const int tq = (g + 8) / G, gg = (g + 8) % G;
      qb[blk] = *reinterpret_cast<const uint4*>(a.q + ((long long)b * a.Tq + tq) * a.q_rs + (kvh * G + gg) * D + blk * 32 + t * 8);
    }
  }
  const bf16* kb = a.k_cache + ((long long)b * a.Hkv + kvh) * a.cap * D;
  const bf16* vb = a.v_cache + ((long long)b * a.Hkv + kvh) * a.cap * D;
  m0 = m1 = -INFINITY;             // running max / partial sums of rows g and g+8
  l0 = l1 = 0.f;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[q][i] = 0.f;
  const float sc = a.scale * 1.4426950408889634f;              // scores in log2 units

  for (int kbase = k0 + warp * KPI; kbase < k1; kbase += W * KPI) {
    // ---- scores of 16 keys
    float s[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int key = min(kbase + j * 8 + g, a.cap - 1);
      const bf16* krow = kb + (long long)key * D + t * 8;
      uint4 kk[4];
#pragma unroll
      for (int blk = 0; blk < 4; ++blk) kk[blk] = *reinterpret_cast<const uint4*>(krow + blk * 32);
#pragma unroll
      for (int i = 0; i < 4; ++i) s[j][i] = 0.f;
#pragma unroll
      for (int blk = 0; blk < 4; ++blk) {
        mma_qk(s[j], qa[blk].x, qb[blk].x, qa[blk].y, qb[blk].y, kk[blk].x, kk[blk].y);
        mma_qk(s[j], qa[blk].z, qb[blk].z, qa[blk].w, qb[blk].w, kk[blk].z, kk[blk].w);
      }
    }
    // ---- V rows of the same keys: lane owns head dimensions 4*lane .. 4*lane+3 (requested before the softmax math)
    uint2 vv[KPI];
#pragma unroll
    for (int k = 0; k < KPI; ++k) {
      const int key = min(kbase + k, a.cap - 1);
      vv[k] = *reinterpret_cast<const uint2*>(vb + (long long)key * D + lane * 4);
    }
    // ---- mask, online softmax (rows g and g+8; this lane's columns are keys j*8 + 2t, 2t+1)
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int key = kbase + j * 8 + 2 * t + e;
        const bool in = key < k1;
        s[j][e] = (in && key >= st0 && key < en0) ? s[j][e] * sc : -INFINITY;
        s[j][2 + e] = (in && key >= st1 && key < en1) ? s[j][2 + e] * sc : -INFINITY;
        mx0 = fmaxf(mx0, s[j][e]);
        mx1 = fmaxf(mx1, s[j][2 + e]);
      }
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
    const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1);
    const float u0 = n0 == -INFINITY ? 0.f : n0, u1 = n1 == -INFINITY ? 0.f : n1;
    const float c0 = m0 == -INFINITY ? 0.f : exp2f(m0 - u0), c1 = m1 == -INFINITY ? 0.f : exp2f(m1 - u1);
    m0 = n0; m1 = n1;
    l0 *= c0; l1 *= c1;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float p0 = exp2f(s[j][e] - u0), p1 = exp2f(s[j][2 + e] - u1);
        l0 += p0; l1 += p1;
        if (g < NQ) s_p[j * 8 + 2 * t + e][g] = p0;
        if (NQ > 8) s_p[j * 8 + 2 * t + e][g + 8] = p1;
      }
    // correction factors of all queries: row q lives in lanes 4*(q%8) .. +3
    float corr[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) corr[q] = __shfl_sync(0xffffffffu, q < 8 ? c0 : c1, (q & 7) * 4);
    __syncwarp();
    // ---- O += P V on the FMA units
#pragma unroll
    for (int q = 0; q < NQ; ++q)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[q][i] *= corr[q];
#pragma unroll
    for (int k = 0; k < KPI; ++k) {
      const float2 v01 = unpack_bf16x2(vv[k].x), v23 = unpack_bf16x2(vv[k].y);
#pragma unroll
      for (int q4 = 0; q4 < NQ / 4; ++q4) {
        const float4 p = *reinterpret_cast<const float4*>(&s_p[k][q4 * 4]);
        const float pq[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[q4 * 4 + i][0] = fmaf(pq[i], v01.x, acc[q4 * 4 + i][0]);
          acc[q4 * 4 + i][1] = fmaf(pq[i], v01.y, acc[q4 * 4 + i][1]);
          acc[q4 * 4 + i][2] = fmaf(pq[i], v23.x, acc[q4 * 4 + i][2]);
          acc[q4 * 4 + i][3] = fmaf(pq[i], v23.y, acc[q4 * 4 + i][3]);
        }
      }
    }
  }
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
}

template <int NQ>   // queries served per CTA, padded: 4, 8 or 16
__global__ void __launch_bounds__(kDecThreads) decode_attn_mma_kernel(DecodeArgs a) {
  grid_dependency_launch();   // the successor may start now: in a decode step it is a projection that reads its weights first
  grid_dependency_wait();     // the previous kernel's results are complete from here on
  constexpr int D = 128;
  __shared__ __align__(16) float s_p[4][kDecKeys][NQ];  // per warp: probabilities, [key][query]
  __shared__ float s_m[4][NQ], s_l[4][NQ];
  __shared__ __align__(16) float s_o[4][NQ][D];
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int G = a.Hq / a.Hkv;
  const int nq = G * a.Tq;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  float acc[NQ][4], m0, m1, l0, l1;
  decode_warp<NQ, 4>(a, split, kvh, b, warp, lane, s_p[warp], acc, m0, m1, l0, l1);
  // ---- merge the four warps, write this split's partial result
  if (t == 0) {
    if (g < NQ) { s_m[warp][g] = m0; s_l[warp][g] = l0; }
    if (NQ > 8) { s_m[warp][g + 8] = m1; s_l[warp][g + 8] = l1; }
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) *reinterpret_cast<float4*>(&s_o[warp][q][lane * 4]) = make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
  __syncthreads();
  for (int i = threadIdx.x; i < nq * D; i += kDecThreads) {
    const int q = i / D, d = i % D;
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) m = fmaxf(m, s_m[w][q]);
    float o = 0.f, l = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = s_m[w][q] == -INFINITY ? 0.f : exp2f(s_m[w][q] - m);
      o += s_o[w][q][d] * f;
      l += s_l[w][q] * f;
    }
    const int tq = q / G, gg = q % G;
    const long long base = ((((long long)b * a.Tq + tq) * a.Hq + kvh * G + gg) * a.splits + split);
    a.part_o[base * D + d] = o;
    if (d == 0) {
      a.part_ml[base * 2] = m == -INFINITY ? -INFINITY : m * 0.6931471805599453f;   // natural-log units for the combine
      a.part_ml[base * 2 + 1] = l;
    }
  }
  combine_if_last(a, b, kvh, nq, G);
}

// Slices of short caches (the ring and summaries of a summary layer, short contexts): the splits of a KV group are a cluster, which shares
// each slice evenly and merges through its shared memory.  What bounds such a slice is the chain of latencies, and the merge by the split
// that finishes last (partial results to global memory, a counter, all of them read back) was half of it: a decode step of four
// sequences of 1030 keys through four layers and the head 424 -> 408 us, of one 367 -> 351, of two of 330 keys 375 -> 356.
// Four to eight warps a CTA are as good as one another; with twelve, which ask for all of a split's keys at once, the next projection finds no
// room beside the CTAs and reads its weights late (448 us).  An L2 prefetch of the keys ahead of the wait changed nothing.
// Where the lines lie, in us of attention (32 heads) and the projection behind it, by the grid of splits and here:
//   * a cluster of every group fits beside the others: of 8 groups a sequence, four sequences of 330 keys 17.9 -> 15.9, of 1130 20.7 -> 21.0, but five
//     18.8 -> 19.2 and 20.8 -> 24.0, eight 19.3 -> 22.0 and 23.7 -> 27.4;
//   * up to 2048 slots: one sequence of 2000 keys 18.9 -> 15.8, two 20.3 -> 17.0, three of 2018 20.7 -> 17.6, eight of four groups 34.5 -> 27.6.  What
//     is in the cache is not known here, and the grid has as many splits as the cache takes: a long cache that is not full
//     would gain as well (8192 slots, 1030 keys, four sequences 38.8 -> 20.4; 8000 keys 57.2 -> 51.8, but one 27.9 -> 30.4);
//   * with more clusters' blocks than SMs and at most four queries a group to 1536, two rounds of a warp's keys: four sequences of 1506 keys 20.8 ->
//     21.8, of 1634 21.5 -> 24.0, of 2018 21.9 -> 24.7.
constexpr int kDecClusterKeys = 2048, kDecClusterKeysCrowded = 1536;
constexpr int kDecCluster = 8;
template <int NQ>
constexpr int dec_cluster_warps() { return NQ <= 8 ? 6 : 4; }      // sixteen queries' outputs of four warps take 32 KB of shared memory

__device__ __forceinline__ float ld_cluster_f32(const float* local, uint32_t rank) {
  float v;
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
               : "=f"(v) : "r"(smem_u32(local)), "r"(rank) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int NQ>
__global__ void __launch_bounds__(dec_cluster_warps<NQ>() * 32) decode_attn_cluster_kernel(DecodeArgs a) {
  constexpr int D = 128, W = dec_cluster_warps<NQ>();
  __shared__ __align__(16) float s_p[W][kDecKeys][NQ];
  __shared__ float s_m[W][NQ], s_l[W][NQ], s_cm[NQ], s_cl[NQ];
  __shared__ __align__(16) float s_o[W][NQ][D];
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int G = a.Hq / a.Hkv, nq = G * a.Tq;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  grid_dependency_launch();   // the successor may start now: in a decode step it is a projection that reads its weights first
  grid_dependency_wait();     // the previous kernel's results are complete from here on
  float acc[NQ][4], m0, m1, l0, l1;
  decode_warp<NQ, W>(a, split, kvh, b, warp, lane, s_p[warp], acc, m0, m1, l0, l1);
  if ((lane & 3) == 0) {
    const int g = lane >> 2;
    if (g < NQ) { s_m[warp][g] = m0; s_l[warp][g] = l0; }
    if (NQ > 8) { s_m[warp][g + 8] = m1; s_l[warp][g + 8] = l1; }
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) *reinterpret_cast<float4*>(&s_o[warp][q][lane * 4]) = make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
  __syncthreads();
  // the warps' parts -> this split's, in the place of the first warp's
  for (int i = threadIdx.x; i < nq * D; i += W * 32) {
    const int q = i / D, d = i % D;
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < W; ++w) m = fmaxf(m, s_m[w][q]);
    float o = 0.f, l = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float f = s_m[w][q] == -INFINITY ? 0.f : exp2f(s_m[w][q] - m);
      o += s_o[w][q][d] * f;
      l += s_l[w][q] * f;
    }
    s_o[0][q][d] = o;
    if (d == 0) { s_cm[q] = m; s_cl[q] = l; }
  }
  cluster_barrier();
  // every split finishes its share of the outputs
  const int share = (nq * D + kDecCluster - 1) / kDecCluster, end = min((split + 1) * share, nq * D);
  for (int i = split * share + (int)threadIdx.x; i < end; i += W * 32) {
    const int q = i / D, d = i % D;
    float ms[kDecCluster], ls[kDecCluster], os[kDecCluster], m = -INFINITY;
#pragma unroll
    for (int r = 0; r < kDecCluster; ++r) {
      ms[r] = ld_cluster_f32(&s_cm[q], r);
      ls[r] = ld_cluster_f32(&s_cl[q], r);
      os[r] = ld_cluster_f32(&s_o[0][q][d], r);
      m = fmaxf(m, ms[r]);
    }
    float o = 0.f, l = 0.f;
#pragma unroll
    for (int r = 0; r < kDecCluster; ++r) {
      const float f = ms[r] == -INFINITY ? 0.f : exp2f(ms[r] - m);
      o = fmaf(os[r], f, o);
      l = fmaf(ls[r], f, l);
    }
    a.out[(((long long)b * a.Tq + q / G) * a.Hq + kvh * G + q % G) * D + d] = __float2bfloat16(l > 0.f ? o / l : 0.f);
  }
  cluster_barrier();          // nobody leaves while its part may still be read
}

template <int NQ>
static int launch_decode_cluster(DecodeArgs a, cudaStream_t st) {
  a.splits = kDecCluster;
  a.keys_per_split = 0;       // of the slice, not of the cache
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.splits, a.Hkv, a.B);
  cfg.blockDim = dim3(dec_cluster_warps<NQ>() * 32);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = a.splits;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent_launches() ? 2 : 1;
  KSA_CHECK_CUDA(cudaLaunchKernelEx(&cfg, decode_attn_cluster_kernel<NQ>, a));
  return 0;
}

// one CTA per (b, t, head): merge the splits
__global__ void __launch_bounds__(128) decode_combine_kernel(DecodeArgs a) {
  grid_dependency_launch();   // the successor may start now: in a decode step it is a projection that reads its weights first
  grid_dependency_wait();     // the previous kernel's results are complete from here on
  const long long row = blockIdx.x;  // (b * Tq + t) * Hq + h
  const float* ml = a.part_ml + row * a.splits * 2;
  float m = -INFINITY;
  for (int s = 0; s < a.splits; ++s) m = fmaxf(m, ml[2 * s]);
  float l = 0.f;
  for (int s = 0; s < a.splits; ++s) l += ml[2 * s] == -INFINITY ? 0.f : ml[2 * s + 1] * __expf(ml[2 * s] - m);
  const float inv = l > 0.f ? 1.f / l : 0.f;
  for (int d = threadIdx.x; d < a.D; d += blockDim.x) {
    float o = 0.f;
    for (int s = 0; s < a.splits; ++s) {
      if (ml[2 * s] == -INFINITY) continue;
      o += a.part_o[(row * a.splits + s) * a.D + d] * __expf(ml[2 * s] - m);
    }
    a.out[row * a.D + d] = __float2bfloat16(o * inv);
  }
}

// cache[b, h, slot[b, t], :] = src[b, t, h, :] for slot >= 0 (K and V together)
__global__ void __launch_bounds__(256)
kv_cache_append_kernel(const bf16* k_new, const bf16* v_new, bf16* k_cache,
                       bf16* v_cache, const int* slots, int B, int T, int H, int D, int cap,
                       long long src_row_stride, long long src_batch_stride) {
  grid_dependency_launch();   // the successor may start now: in a decode step it is a projection that reads its weights first
  grid_dependency_wait();     // the previous kernel's results are complete from here on
  const long long vec = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int per = D / 8;
  if (vec >= (long long)B * T * H * per) return;
  const int v = vec % per;
  const int h = (vec / per) % H;
  const int t = (vec / ((long long)per * H)) % T;
  const int b = vec / ((long long)per * H * T);
  const int slot = slots[b * T + t];
  if (slot < 0 || slot >= cap) return;
  const long long src = (long long)b * src_batch_stride + (long long)t * src_row_stride + (long long)h * D + v * 8;
  const long long dst = (((long long)b * H + h) * cap + slot) * D + v * 8;
  *reinterpret_cast<uint4*>(k_cache + dst) = *reinterpret_cast<const uint4*>(k_new + src);
  *reinterpret_cast<uint4*>(v_cache + dst) = *reinterpret_cast<const uint4*>(v_new + src);
}

// Keys and values of a prompt's packed rows ([B * L] text rows, then [B * Ns] summary rows; heads of a row next to one another) -> the
// cache of one layer, [B, H, cap, D].  A summary layer (chunk > 0) keeps the last `window` complete chunks, chunk c in ring place
// c % window, the rest of the text from right to left in the current chunk, and all summaries; a full layer keeps every row at its index.
// One launch for what were eighteen strided copies a layer, 5.5 us each; it is bound by the memory, 33 MB for four prompts of 1000 tokens.
struct CacheFill {
  const bf16 *k, *v;
  bf16 *k_cache, *v_cache;
  long long rs;
  int B, L, Ns, H, D, cap;
  int chunk, n_sum, window, text0, sum0;
  int first;               // first text row that is kept
};
__global__ void __launch_bounds__(256) kv_cache_fill_kernel(CacheFill a) {
  grid_dependency_enter();
  const int per = a.D / 8, rows = a.L - a.first + a.Ns;
  const long long vec = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (vec >= (long long)a.B * rows * a.H * per) return;
  const int v = (int)(vec % per), h = (int)(vec / per % a.H);
  const long long br = vec / ((long long)per * a.H);
  const int b = (int)(br / rows), t = (int)(br % rows) + a.first;
  long long row;
  int slot;
  if (t >= a.L) {
    row = (long long)a.B * a.L + (long long)b * a.Ns + (t - a.L);
    slot = a.sum0 + t - a.L;
  } else {
    row = (long long)b * a.L + t;
    slot = t;
    if (a.chunk > 0) {
      const int c = t / a.chunk, at = t - c * a.chunk;
      slot = c < a.L / a.chunk ? a.text0 + c % a.window * a.chunk + at : a.n_sum + a.chunk - 1 - at;
    }
  }
  const long long src = row * a.rs + (long long)h * a.D + v * 8;
  const long long dst = (((long long)b * a.H + h) * a.cap + slot) * a.D + v * 8;
  *reinterpret_cast<uint4*>(a.k_cache + dst) = *reinterpret_cast<const uint4*>(a.k + src);
  *reinterpret_cast<uint4*>(a.v_cache + dst) = *reinterpret_cast<const uint4*>(a.v + src);
}

// cache[b, h, dst[b] + r, :] = cache[b, h, src[b] + r, :] for r < rows, for sequences with enable[b] != 0
__global__ void __launch_bounds__(256)
kv_cache_move_kernel(bf16* k_cache, bf16* v_cache, const int* src,
                     const int* dst, const int* enable, int B, int H, int D, int cap,
                     int rows) {
  grid_dependency_launch();   // the successor may start now: in a decode step it is a projection that reads its weights first
  grid_dependency_wait();     // the previous kernel's results are complete from here on
  const long long vec = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int per = D / 8;
  if (vec >= (long long)B * H * rows * per) return;
  const int v = vec % per;
  const int r = (vec / per) % rows;
  const int h = (vec / ((long long)per * rows)) % H;
  const int b = vec / ((long long)per * rows * H);
  if (enable && !enable[b]) return;
  const long long base = ((long long)b * H + h) * cap;
  const long long s = (base + src[b] + r) * D + v * 8, d = (base + dst[b] + r) * D + v * 8;
  *reinterpret_cast<uint4*>(k_cache + d) = *reinterpret_cast<const uint4*>(k_cache + s);
  *reinterpret_cast<uint4*>(v_cache + d) = *reinterpret_cast<const uint4*>(v_cache + s);
}

}  // namespace ksa

using namespace ksa;

// q_rs: elements from one (sequence, query) row of q to the next.  Scratch sizes the caller allocates: part_o [B*Tq*Hq*splits*D] fp32, part_ml [B*Tq*Hq*splits*2] fp32.
// counters: B*Hkv int32 zeros that launches on one stream may share (each launch leaves them zero), or null for a
// separate merge kernel.
KSA_API int ksa_decode_attn(const void* q, const void* k_cache, const void* v_cache, const void* start, const void* len,
                            void* part_o, void* part_ml, void* out, int B, int Tq, int Hq, int Hkv, int D, int cap,
                            int splits, int keys_per_split, long long q_rs, float scale, void* counters, void* stream) {
  KSA_ENTER(q);
  KSA_REQUIRE(D == 128 || D == 64, "decode_attn: head_dim %d unsupported (64 or 128)", D);
  KSA_REQUIRE(Hq % Hkv == 0 && (Hq / Hkv) * Tq <= kDecMaxQ, "decode_attn: (Hq/Hkv) * Tq = %d exceeds %d queries per CTA",
              (Hq / Hkv) * Tq, kDecMaxQ);
  KSA_REQUIRE(q_rs % 8 == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0, "decode_attn: query rows must be 16-byte aligned");
  KSA_REQUIRE(splits >= 1 && keys_per_split >= 1, "decode_attn: bad split configuration");
  KSA_REQUIRE(counters == nullptr || splits <= kDecMaxSplits, "decode_attn: %d splits (at most %d with counters)", splits,
              kDecMaxSplits);
  if (B == 0) return 0;
  DecodeArgs a{(const bf16*)q, (const bf16*)k_cache, (const bf16*)v_cache, (const int*)start, (const int*)len,
               (float*)part_o, (float*)part_ml, (bf16*)out, B, Tq, Hq, Hkv, D, cap, splits, keys_per_split, scale, q_rs,
               (int*)counters};
  dim3 grid(splits, Hkv, B);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int nq = (Hq / Hkv) * Tq;
  const int blocks = kDecCluster * Hkv * B, sms = sm_count();
  const bool crowded = blocks > sms && nq <= 4;
  if (D == 128 && counters != nullptr && blocks <= 2 * sms && cap <= (crowded ? kDecClusterKeysCrowded : kDecClusterKeys)) {
    if (nq <= 4) return launch_decode_cluster<4>(a, st);
    return nq <= 8 ? launch_decode_cluster<8>(a, st) : launch_decode_cluster<16>(a, st);
  }
  if (D == 128 && nq <= 4) KSA_CHECK_CUDA(launch_kernel(decode_attn_mma_kernel<4>, grid, dim3(kDecThreads), 0, st, a));
  else if (D == 128 && nq <= 8) KSA_CHECK_CUDA(launch_kernel(decode_attn_mma_kernel<8>, grid, dim3(kDecThreads), 0, st, a));
  else if (D == 128) KSA_CHECK_CUDA(launch_kernel(decode_attn_mma_kernel<16>, grid, dim3(kDecThreads), 0, st, a));
  else KSA_CHECK_CUDA(launch_kernel(decode_attn_kernel<64>, grid, dim3(kDecThreads), 0, st, a));
  if (counters == nullptr) KSA_CHECK_CUDA(launch_kernel(decode_combine_kernel, dim3(B * Tq * Hq), dim3(128), 0, st, a));
  return 0;
}

KSA_API int ksa_kv_cache_append(const void* k_new, const void* v_new, void* k_cache, void* v_cache, const void* slots,
                                int B, int T, int H, int D, int cap, long long src_row_stride,
                                long long src_batch_stride, void* stream) {
  KSA_ENTER(k_new);
  KSA_REQUIRE(D % 8 == 0, "kv_cache_append: head_dim must be a multiple of 8");
  const long long n = (long long)B * T * H * (D / 8);
  if (n == 0) return 0;
  KSA_CHECK_CUDA(launch_kernel(kv_cache_append_kernel, dim3((unsigned)((n + 255) / 256)),
                              dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), (const bf16*)k_new,
                              (const bf16*)v_new, (bf16*)k_cache, (bf16*)v_cache, (const int*)slots, B, T, H, D, cap,
                              src_row_stride, src_batch_stride));
  return 0;
}

// k, v: first key and first value of the packed rows (row stride rs); k_cache, v_cache: the first of the B sequences' caches.  chunk = 0: a full
// layer, else the geometry of the ring buffer (first slot of the ring, of the summaries).
KSA_API int ksa_kv_cache_fill(const void* k, const void* v, void* k_cache, void* v_cache, int B, int L, int Ns, int H, int D, int cap,
                              long long rs, int chunk, int n_sum, int window, int text0, int sum0, void* stream) {
  KSA_ENTER(k);
  KSA_REQUIRE(D % 8 == 0 && rs % 8 == 0, "kv_cache_fill: head_dim %d and row stride %lld must be multiples of 8", D, rs);
  KSA_REQUIRE(((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(k_cache) |
                reinterpret_cast<uintptr_t>(v_cache)) & 15) == 0, "kv_cache_fill: rows and caches must be 16-byte aligned");
  KSA_REQUIRE(B >= 0 && L >= 0 && Ns >= 0 && H > 0 && chunk >= 0 && window >= 0 && n_sum >= 0, "kv_cache_fill: bad shape");
  CacheFill a{(const bf16*)k, (const bf16*)v, (bf16*)k_cache, (bf16*)v_cache, rs, B, L, Ns, H, D, cap, chunk, n_sum, window, text0, sum0, 0};
  if (chunk > 0) {
    a.first = (L / chunk > window ? L / chunk - window : 0) * chunk;
    KSA_REQUIRE(n_sum + chunk <= cap && text0 + window * chunk <= cap && sum0 + Ns <= cap, "kv_cache_fill: %d slots do not hold the prompt", cap);
  } else {
    KSA_REQUIRE(L <= cap && Ns == 0, "kv_cache_fill: %d slots do not hold %d rows", cap, L);
  }
  const long long n = (long long)B * (L - a.first + Ns) * H * (D / 8);
  if (n == 0) return 0;
  KSA_CHECK_CUDA(launch_stream_kernel(n * 64, kv_cache_fill_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0,
                                      reinterpret_cast<cudaStream_t>(stream), a));
  return 0;
}

KSA_API int ksa_kv_cache_move(void* k_cache, void* v_cache, const void* src, const void* dst, const void* enable, int B,
                              int H, int D, int cap, int rows, void* stream) {
  KSA_ENTER(k_cache);
  const long long n = (long long)B * H * rows * (D / 8);
  if (n == 0) return 0;
  KSA_CHECK_CUDA(launch_kernel(kv_cache_move_kernel, dim3((unsigned)((n + 255) / 256)),
                              dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), (bf16*)k_cache, (bf16*)v_cache,
                              (const int*)src, (const int*)dst, (const int*)enable, B, H, D, cap, rows));
  return 0;
}

namespace ksa {
// The slices of a step's text tokens on a ring-buffer cache (inference/cache.py), one thread per sequence: what PyTorch takes ten
// kernels of a microsecond and a half for, none of which the next one may overlap.
__global__ void decode_step_slices_kernel(const int* cbl, const int* chunks, int* out, int B, int n_sum, int chunk, int window, int text0,
                                          int sum0) {
  grid_dependency_launch();
  grid_dependency_wait();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const int done = chunks[b], slot = n_sum + chunk - 1 - cbl[b];
  const int end = done >= window ? sum0 + (done - window) * n_sum : text0 + done * chunk;
  out[b] = slot;
  out[B + b] = end - slot;
}
// The counters after an ordinary step.
__global__ void decode_advance_kernel(int* text_len, int* cbl, int B) {
  grid_dependency_launch();
  grid_dependency_wait();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  text_len[b] += 1;
  if (cbl != nullptr) cbl[b] += 1;
}
}  // namespace ksa

// out [2, B] int32: write slot (also the start of the slice), slice length.
KSA_API int ksa_decode_step_slices(const void* cbl, const void* chunks, void* out, int B, int n_sum, int chunk, int window, int text0,
                                   int sum0, void* stream) {
  KSA_ENTER(cbl);
  if (B == 0) return 0;
  KSA_CHECK_CUDA(launch_kernel(decode_step_slices_kernel, dim3((B + 127) / 128), dim3(128), 0, reinterpret_cast<cudaStream_t>(stream),
                               (const int*)cbl, (const int*)chunks, (int*)out, B, n_sum, chunk, window, text0, sum0));
  return 0;
}

// text_len += 1, and cbl += 1 unless null.
KSA_API int ksa_decode_advance(void* text_len, void* cbl, int B, void* stream) {
  KSA_ENTER(text_len);
  if (B == 0) return 0;
  KSA_CHECK_CUDA(launch_kernel(decode_advance_kernel, dim3((B + 127) / 128), dim3(128), 0, reinterpret_cast<cudaStream_t>(stream),
                               (int*)text_len, (int*)cbl, B));
  return 0;
}
