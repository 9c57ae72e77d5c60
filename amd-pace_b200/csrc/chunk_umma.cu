// Recurrences with one decay per head and token (lightning attention, state-space recurrence) over prompts, in chunks of 128 tokens on
// tcgen05: what the chunks add to the state (side by side), the states in front of the chunks (a sum over the chunks, elementwise),
// the outputs (side by side).  With l_i the sum of a chunk's log decays up to token i, s_j a token's step (lightning: 1) and S the
// state in front of the chunk:
//     add = sum_j e^(l_n - l_j) s_j k_j v_j^T,   S' = e^(l_n) S + add
//     out_i = e^(l_i) S^T q_i + sum_{j <= i} e^(l_i - l_j) s_j (q_i . k_j) v_j
// Operands as in the chunks of 64 (lightning.cu, ssd_chunk.cu): q, k, v are bf16 values; states and sums stay in fp32, and where an fp32
// quantity enters a bf16 product it is split into two terms (weights, the state that is read) or three (the keys that enter the state).
//
// Why this form: the chunks of 64 walk a sequence one after another on mma.sync, whose rate (one m16n8k16 per 16 cycles and scheduler)
// was two thirds of a chunk's time; tcgen05 does the same products in a tenth of it, and what is left - loads, silu, splits, the waits
// between the products of a chunk - is hidden by two blocks per SM that are at different chunks.
// us with all launches of a call: lightning, one prompt of 4096 tokens, 16 heads of 128 x 128: 147 -> 78 (states 33, prefix 10, outputs 30,
// 270 MB through L2 and HBM), 512 tokens 78 -> 27, 4 prompts of 300 to 2000 tokens, 32 heads 302 -> 138; state space with its convolution,
// 8 prompts of 203 to 733 tokens, 32 heads of 128 x 64: 115 -> 102, one of 4096, 64 heads 310 -> 187.
#include "chunk_umma.cuh"
#include "umma.cuh"

namespace pace {
namespace {

constexpr int kChunk = 128, kThreads = 256;
constexpr int kBlock = kChunk * 128;       // bytes of 64 columns of a tile: 128 rows of 128 bytes, swizzled

// Byte of 8 columns (piece p) of a row in a tile: a block's rows are 128 bytes, 16-byte pieces xor row
__device__ __forceinline__ int tile_at(int row, int p) { return (p >> 3) * kBlock + row * 128 + (((p & 7) ^ (row & 7)) << 4); }
// Element of the states' scratch: rows in groups of eight, so that a warp's rows and a tile's pieces both lie together
template <int VP> __device__ __forceinline__ int add_at(int row, int p) { return (((row >> 3) * (VP / 8) + p) * 8 + (row & 7)) * 8; }

struct Item { int e, c, t0, n, count; };
// The chunk of a place: sequence e has places cu[e] / 128 + e and on (a bound of the chunks in front that needs no sum)
__device__ __forceinline__ bool find_item(const pace_step_t& st, int place, Item* it) {
  const int lane = threadIdx.x & 31;
  for (int e0 = 0; e0 < st.n_entries; e0 += 32) {
    const int e = e0 + lane;
    int at = 0, end = 0, c = -1;
    if (e < st.n_entries) {
      at = st.cu[e], end = st.cu[e + 1];
      c = place - (at / kChunk + e);
      if (c >= (end - at + kChunk - 1) / kChunk) c = -1;
    }
    const unsigned m = __ballot_sync(0xffffffffu, c >= 0);
    if (!m) continue;
    const int from = __ffs(m) - 1;
    it->e = e0 + from;
    it->c = __shfl_sync(0xffffffffu, c, from);
    at = __shfl_sync(0xffffffffu, at, from);
    end = __shfl_sync(0xffffffffu, end, from);
    it->t0 = at + it->c * kChunk;
    it->count = end - at;
    it->n = min(kChunk, end - it->t0);
    return true;
  }
  return false;
}

struct Sync {
  uint64_t mma, values, from_state, kv, s_hi, s_lo;   // products (keys or scores, values, state), copies
  uint32_t tmem_slot;
  int abort_flag;
  float l[kChunk], dt[kChunk], part[4];
};

__device__ __forceinline__ uint32_t start_block(Sync& sy, int cols) {
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sy.tmem_slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 32) {
    sy.abort_flag = 0;
    mbar_init(&sy.mma, 1);
    mbar_init(&sy.values, 1);
    mbar_init(&sy.from_state, 1);
    mbar_init(&sy.kv, 1);
    mbar_init(&sy.s_hi, 1);
    mbar_init(&sy.s_lo, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return *reinterpret_cast<volatile uint32_t*>(&sy.tmem_slot);
}
__device__ __forceinline__ void end_block(uint32_t tmem, int cols) {
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

// l (sums of log decays) and dt of the chunk's tokens, zero steps behind its end; ends with a barrier
template <bool SSD>
__device__ __forceinline__ void token_sums(const ChunkArgs& a, const Item& it, int h, Sync& sy) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if constexpr (SSD) {
    float dt = 0.f, l = 0.f;
    if (tid < kChunk) {
      if (tid < it.n) dt = softplus_fast(__bfloat162float(a.dt_raw[(size_t)(it.t0 + tid) * a.dt_stride + h]) + a.dt_bias[h]);
      l = a.neg_a[h] * dt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float x = __shfl_up_sync(0xffffffffu, l, o);
        if (lane >= o) l += x;
      }
      if (lane == 31) sy.part[warp] = l;
    }
    __syncthreads();
    if (tid < kChunk) {
      for (int w = 0; w < warp; ++w) l += sy.part[w];
      sy.l[tid] = l;
      sy.dt[tid] = dt;
    }
  } else {
    if (tid < kChunk) sy.l[tid] = powf(a.decay[h], (float)tid);      // powers of the decay
  }
  __syncthreads();
}

// eight bf16 of a row of projections; lightning: through silu, rounded
template <bool SSD> __device__ __forceinline__ uint4 activated(uint4 x) {
  if constexpr (SSD) return x;
  uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = bf2_to_f2(w[i]);
    w[i] = f2_to_bf2(silu_t<__nv_bfloat16>(f.x), silu_t<__nv_bfloat16>(f.y));
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// 16-byte pieces of a tile's rows, spread over the threads: COLS / 8 threads per row
template <int COLS> struct Rows {
  static constexpr int kPer = COLS / 8, kStep = kThreads / kPer, kN = kChunk / kStep;
  uint4 x[kN];
  __device__ __forceinline__ int piece() const { return threadIdx.x % kPer; }
  __device__ __forceinline__ int row(int i) const { return threadIdx.x / kPer + i * kStep; }
  __device__ __forceinline__ void load(const __nv_bfloat16* src, int64_t stride, int n, int cols) {
    const int p = piece();
#pragma unroll
    for (int i = 0; i < kN; ++i)
      x[i] = row(i) < n && p * 8 < cols ? __ldg(reinterpret_cast<const uint4*>(src + (size_t)row(i) * stride + p * 8)) : make_uint4(0, 0, 0, 0);
  }
};

__device__ __forceinline__ uint32_t desc_lo(const void* p, uint32_t lbo_bytes) { return ((smem_u32(p) >> 4) & 0x3FFFu) | ((lbo_bytes >> 4) << 16); }

// ------------------------------- what a chunk adds -------------------------------
template <bool SSD, int VP>
__global__ void __launch_bounds__(kThreads, 2) chunk_states_kernel(pace_step_t st, ChunkArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char *hi = smem, *mid = smem + 2 * kBlock, *vt = smem + 4 * kBlock;
  Sync& sy = *reinterpret_cast<Sync*>(smem + 4 * kBlock + VP / 64 * kBlock);
  Item it;
  if (!find_item(st, a.place0 + blockIdx.z, &it)) return;
  const int h = blockIdx.y, vb = blockIdx.x, v0 = vb * VP, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const __nv_bfloat16* rows = a.src + (size_t)it.t0 * a.src_stride;
  Rows<128> k;
  Rows<VP> v;
  k.load(rows + a.k_at + (h / a.per_group) * a.q_step, a.src_stride, it.n, a.dim);
  v.load(rows + a.v_at + (size_t)h * a.vdim + v0, a.src_stride, it.n, a.vdim - v0);
  const uint32_t tmem = start_block(sy, VP);
  token_sums<SSD>(a, it, h, sy);
  const float l_end = SSD ? sy.l[kChunk - 1] : 0.f;
  const size_t place = ((size_t)blockIdx.z * a.heads + h) * a.v_blocks + vb;
  unsigned char* keep = SSD ? nullptr : a.kv + place * (2 * kBlock + VP / 64 * kBlock);   // keys and values behind silu, as tiles

#pragma unroll
  for (int i = 0; i < Rows<128>::kN; ++i) {
    const int r = k.row(i), at = tile_at(r, k.piece());
    const uint4 x = activated<SSD>(k.x[i]);
    if constexpr (!SSD) *reinterpret_cast<uint4*>(keep + at) = x;
    const float w = SSD ? exp_t<__nv_bfloat16>(l_end - sy.l[r]) * sy.dt[r] : r < it.n ? sy.l[it.n - 1 - r] : 0.f;
    const uint32_t in[4] = {x.x, x.y, x.z, x.w};
    uint32_t th[4], tm[4], tl[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = bf2_to_f2(in[j]);
      const float x0 = f.x * w, x1 = f.y * w;
      th[j] = f2_to_bf2(x0, x1);
      const float2 g = bf2_to_f2(th[j]);
      split_bf2(x0 - g.x, x1 - g.y, tm[j], tl[j]);
    }
    *reinterpret_cast<uint4*>(hi + at) = make_uint4(th[0], th[1], th[2], th[3]);
    *reinterpret_cast<uint4*>(mid + at) = make_uint4(tm[0], tm[1], tm[2], tm[3]);
    k.x[i] = make_uint4(tl[0], tl[1], tl[2], tl[3]);       // the third terms wait for the first ones' place
  }
#pragma unroll
  for (int i = 0; i < Rows<VP>::kN; ++i) {
    const int at = tile_at(v.row(i), v.piece());
    const uint4 x = activated<SSD>(v.x[i]);
    *reinterpret_cast<uint4*>(vt + at) = x;
    if constexpr (!SSD) *reinterpret_cast<uint4*>(keep + 2 * kBlock + at) = x;
  }
  fence_proxy_async();
  __syncthreads();
  // both operands are read along the tokens (columns lie together): 64-column blocks kBlock apart, 16 tokens 2048 bytes
  constexpr uint32_t IDESC = umma_idesc(VP, true) | (1u << 15);
  const int steps = (it.n + 15) / 16;
  const uint32_t v_lo = desc_lo(vt, kBlock);
  volatile int* abort = &sy.abort_flag;
  auto product = [&](const unsigned char* t, bool first) {
    const uint32_t t_lo = desc_lo(t, kBlock);
    for (int s = 0; s < steps; ++s)
      umma_bf16(tmem, pack64(t_lo + s * (2048 >> 4), kDescHi), pack64(v_lo + s * (2048 >> 4), kDescHi), IDESC, first && s == 0 ? 0u : 1u);
  };
  const bool leader = warp == 0 && elect_one();
  if (leader) {
    product(hi, true);
    umma_commit(&sy.mma);
    product(mid, false);
  }
  __syncwarp();
  bool ok = umma_wait(&sy.mma, 0, abort);
#pragma unroll
  for (int i = 0; i < Rows<128>::kN; ++i) *reinterpret_cast<uint4*>(hi + tile_at(k.row(i), k.piece())) = k.x[i];
  fence_proxy_async();
  __syncthreads();
  if (leader) {
    product(hi, false);
    umma_commit(&sy.mma);
  }
  __syncwarp();
  ok = umma_wait(&sy.mma, 1, abort) && ok;
  tc_fence_after();
  // a thread has a row of the state and half of its columns
  const int row = (warp & 3) * 32 + lane, c0 = (warp >> 2) * (VP / 2);
  float* add = a.add + place * (kChunk * VP);
#pragma unroll
  for (int b = 0; b < VP / 64; ++b) {
    uint32_t x[32];
    tmem_ld32(tmem + ((uint32_t)(warp & 3) << 21) + c0 + b * 32, x);
    tmem_wait_ld();
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float* to = add + add_at<VP>(row, (c0 + b * 32) / 8 + g);
      if (!ok) for (int j = 0; j < 8; ++j) x[8 * g + j] = 0x7fc00000u;      // (a wait ran out: not a number)
      *reinterpret_cast<uint4*>(to) = make_uint4(x[8 * g], x[8 * g + 1], x[8 * g + 2], x[8 * g + 3]);
      *reinterpret_cast<uint4*>(to + 4) = make_uint4(x[8 * g + 4], x[8 * g + 5], x[8 * g + 6], x[8 * g + 7]);
    }
  }
  if (SSD && tid == 0) a.log_decay[place] = l_end;
  if (*abort && warp == 0)   // products in flight end before the block's memory is given back
    for (int k = 0; k < 4096; ++k) __nanosleep(256);
  end_block(tmem, VP);
}

// ------------------------------- the states in front of the chunks -------------------------------
// A thread has eight columns of a row; states leave as tiles in two bf16 terms.
template <bool SSD, int VP>
__global__ void __launch_bounds__(kThreads) chunk_prefix_kernel(pace_step_t st, ChunkArgs a) {
  const int e = blockIdx.z, h = blockIdx.y / a.v_blocks, vb = blockIdx.y % a.v_blocks;
  const int u = blockIdx.x * kThreads + threadIdx.x, p = (u >> 3) % (VP / 8), row = (u / VP) * 8 + (u & 7), col = vb * VP + p * 8;
  const int cu = st.cu[e], count = st.cu[e + 1] - cu, n = (count + kChunk - 1) / kChunk;
  // this round's chunks [c_a, c_z) of the sequence; the state comes in with its first chunk and between rounds
  const int at = cu / kChunk + e - a.place0, c_a = max(0, -at), c_z = min(n, a.places - at);
  if (c_a >= c_z) return;
  const bool fresh = st.start[e] == 0 && c_a == 0, mine = row < a.dim && col < a.vdim;
  float* state = a.state + (((size_t)st.slot[e] * a.heads + h) * a.dim + row) * a.vdim + col;
  float s[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] = 0.f;
  if (!fresh && mine) Vec<float, 8>::load(state, s);
  const int64_t step = (int64_t)a.heads * a.v_blocks, first = at * step + blockIdx.y;
  const float full = SSD ? 0.f : powf(a.decay[h], (float)kChunk), rest = SSD ? 0.f : powf(a.decay[h], (float)(count - (n - 1) * kChunk));
  constexpr int kBatch = 4;                                // chunks whose loads are in flight together
  for (int c0 = c_a; c0 < c_z; c0 += kBatch) {
    float x[kBatch][8], f[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b)
      if (c0 + b < c_z) {
        const size_t place = first + (c0 + b) * step;
        Vec<float, 8>::load(a.add + place * (kChunk * VP) + add_at<VP>(row, p), x[b]);
        if constexpr (SSD) f[b] = a.log_decay[place];
      }
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int c = c0 + b;
      if (c >= c_z) break;
      if (c > 0 || !fresh) {
        unsigned char* to = a.tiles + (first + c * step) * (4 * kChunk * VP) + tile_at(row, p);
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split_bf2(s[2 * j], s[2 * j + 1], hi[j], lo[j]);
        *reinterpret_cast<uint4*>(to) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(to + 2 * kChunk * VP) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
      const float g = SSD ? exp_t<__nv_bfloat16>(f[b]) : c + 1 < n ? full : rest;
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = fmaf(g, s[j], x[b][j]);
    }
  }
  if (mine) Vec<float, 8>::store(state, s);
}

// ------------------------------- outputs -------------------------------
// Shared memory: q | k, behind the scores the state's first terms (VP = 64: both) | v, behind its product the second terms.  Tensor
// memory: the weighted values in columns 0 .., scores, then weights, then the state's part in columns 128 ..: 256 columns and at most
// 97 KB, so that two blocks share an SM.
template <bool SSD, int VP>
__global__ void __launch_bounds__(kThreads, 2) chunk_out_kernel(pace_step_t st, ChunkArgs a) {
  constexpr int kV = VP / 64 * kBlock;                     // bytes of a tile of value columns
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char *qt = smem, *kt = smem + 2 * kBlock, *vt = smem + 4 * kBlock;
  unsigned char *sh = kt, *sl = VP == 64 ? kt + kV : vt;
  Sync& sy = *reinterpret_cast<Sync*>(smem + 4 * kBlock + kV);
  Item it;
  if (!find_item(st, a.place0 + blockIdx.z, &it)) return;
  const int h = blockIdx.y, vb = blockIdx.x, v0 = vb * VP, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t place = ((size_t)blockIdx.z * a.heads + h) * a.v_blocks + vb;
  const bool state = it.c > 0 || st.start[it.e] != 0;      // (a sequence that begins here begins from zeros)
  const unsigned char *tiles = a.tiles + place * (2 * kV), *keep = SSD ? nullptr : a.kv + place * (2 * kBlock + kV);
  const __nv_bfloat16* rows = a.src + (size_t)it.t0 * a.src_stride;
  const int head_at = (h / a.per_group) * a.q_step;
  Rows<128> q;
  q.load(rows + a.q_at + head_at, a.src_stride, it.n, a.dim);
  const uint32_t tmem = start_block(sy, 256);
  const uint32_t tO = tmem, tS = tmem + 128;
  volatile int* abort = &sy.abort_flag;
  if (tid == 0) {
    if constexpr (!SSD) {
      mbar_arrive_expect_tx(&sy.kv, 2 * kBlock + kV);
      bulk_g2s(kt, keep, 2 * kBlock, &sy.kv);
      bulk_g2s(vt, keep + 2 * kBlock, kV, &sy.kv);
    }
  }
  if constexpr (SSD) {
    Rows<128> k;
    k.load(rows + a.k_at + head_at, a.src_stride, it.n, a.dim);
    Rows<VP> v;
    v.load(rows + a.v_at + (size_t)h * a.vdim + v0, a.src_stride, it.n, a.vdim - v0);
#pragma unroll
    for (int i = 0; i < Rows<128>::kN; ++i) *reinterpret_cast<uint4*>(kt + tile_at(k.row(i), k.piece())) = k.x[i];
#pragma unroll
    for (int i = 0; i < Rows<VP>::kN; ++i) *reinterpret_cast<uint4*>(vt + tile_at(v.row(i), v.piece())) = v.x[i];
  }
#pragma unroll
  for (int i = 0; i < Rows<128>::kN; ++i) *reinterpret_cast<uint4*>(qt + tile_at(q.row(i), q.piece())) = activated<SSD>(q.x[i]);
  token_sums<SSD>(a, it, h, sy);
  fence_proxy_async();
  __syncthreads();

  // scores: q and k along the head dimension
  const int steps = (it.n + 15) / 16;
  const uint32_t q_lo = desc_lo(qt, 16), k_lo = desc_lo(kt, 16);
  if (warp == 0) {
    bool ok = SSD || umma_wait(&sy.kv, 0, abort);
    if (ok && elect_one()) {
      for (int s = 0; s < 8; ++s) {
        const uint32_t at = (s >> 2) * (kBlock >> 4) + (s & 3) * 2;
        umma_bf16(tS, pack64(q_lo + at, kDescHi), pack64(k_lo + at, kDescHi), umma_idesc(kChunk, false), s ? 1u : 0u);
      }
      umma_commit(&sy.mma);
    }
    __syncwarp();
  }
  bool ok = umma_wait(&sy.mma, 0, abort);
  if (state && tid == 0 && ok) {                           // the keys have been read
    mbar_arrive_expect_tx(&sy.s_hi, kV);
    bulk_g2s(sh, tiles, kV, &sy.s_hi);
    if (VP == 64) {
      mbar_arrive_expect_tx(&sy.s_lo, kV);
      bulk_g2s(sl, tiles + kV, kV, &sy.s_lo);
    }
  }
  tc_fence_after();

  // weights: a thread has a row and half of the keys; two bf16 terms take the scores' place
  const int row = (warp & 3) * 32 + lane, half = warp >> 2;
  const uint32_t lanes = (uint32_t)(warp & 3) << 21;
  uint32_t x[2][32];
  tmem_ld32(tS + lanes + half * 64, x[0]);
  tmem_ld32(tS + lanes + half * 64 + 32, x[1]);
  tmem_wait_ld();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const float l_row = SSD ? sy.l[row] : 0.f;
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    uint32_t hi[16], lo[16];
    const bool seen = half * 64 + b * 32 <= (warp & 3) * 32 + 31;     // (uniform: some key is in sight of some row of the warp)
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      float w[2];
      if (!seen) {
        hi[k] = lo[k] = 0u;
        continue;
      }
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const int j = half * 64 + b * 32 + 2 * k + o;
        const float f = SSD ? exp_t<__nv_bfloat16>(l_row - sy.l[j]) * sy.dt[j] : sy.l[max(row - j, 0)];
        w[o] = j <= row ? __uint_as_float(x[b][2 * k + o]) * f : 0.f;
      }
      split_bf2(w[0], w[1], hi[k], lo[k]);
    }
    tmem_st16(tS + lanes + half * 32 + b * 16, hi);
    tmem_st16(tS + lanes + 64 + half * 32 + b * 16, lo);
  }
  tmem_wait_st();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    const bool leader = elect_one();
    const uint32_t v_lo = desc_lo(vt, kBlock);
    constexpr uint32_t IDESC = umma_idesc(VP, true);
    if (ok && leader) {
      // (rows in front of a step's 16 tokens stay out of it: zero weights would hand on an infinity or NaN among later values)
      for (int t = 0; t < 2; ++t)
        for (int s = 0; s < steps; ++s)
          umma_bf16_ts(tO, tS + t * 64 + s * 8, pack64(v_lo + s * (2048 >> 4), kDescHi), IDESC, t | s ? 1u : 0u, s * 16);
      umma_commit(&sy.values);
    }
    __syncwarp();
    if (ok && state) {
      // the state's part, in the weights' place
      ok = umma_wait(&sy.values, 0, abort);
      if (VP != 64 && ok && leader) {
        mbar_arrive_expect_tx(&sy.s_lo, kV);
        bulk_g2s(sl, tiles + kV, kV, &sy.s_lo);
      }
      __syncwarp();
      for (int t = 0; t < 2 && ok; ++t) {
        ok = umma_wait(t ? &sy.s_lo : &sy.s_hi, 0, abort);
        const uint32_t s_lo = desc_lo(t ? sl : sh, kBlock);
        if (ok && leader)
          for (int s = 0; s < 8; ++s) {
            const uint32_t at = (s >> 2) * (kBlock >> 4) + (s & 3) * 2;
            umma_bf16(tS, pack64(q_lo + at, kDescHi), pack64(s_lo + s * (2048 >> 4), kDescHi), IDESC, t | s ? 1u : 0u);
          }
        __syncwarp();
      }
      if (ok && leader) umma_commit(&sy.from_state);
      __syncwarp();
    }
  }
  ok = umma_wait(&sy.values, 0, abort) && ok;
  if (state && ok) ok = umma_wait(&sy.from_state, 0, abort);
  tc_fence_after();
  const float f = SSD ? exp_t<__nv_bfloat16>(l_row) : powf(a.decay[h], (float)(row + 1));
  const float skip = SSD ? a.d_skip[h] : 0.f;
  __nv_bfloat16* out = a.out + (size_t)(it.t0 + row) * a.out_stride + (size_t)h * a.vdim;
  const __nv_bfloat16* vr = rows + (size_t)row * a.src_stride + a.v_at + (size_t)h * a.vdim;
#pragma unroll
  for (int b = 0; b < VP / 64; ++b) {
    const int c0 = half * (VP / 2) + b * 32;
    uint32_t o[32], s[32];
    tmem_ld32(tO + lanes + c0, o);
    if (state) tmem_ld32(tS + lanes + c0, s);
    tmem_wait_ld();
    if (row >= it.n) continue;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int c = v0 + c0 + g * 8;
      if (c >= a.vdim) break;
      float y[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        y[j] = __uint_as_float(o[8 * g + j]);
        if (state) y[j] = fmaf(f, __uint_as_float(s[8 * g + j]), y[j]);
        if (!ok) y[j] = __uint_as_float(0x7fc00000u);      // (a wait ran out: not a number)
      }
      if constexpr (SSD) {
        float xv[8];
        Vec<__nv_bfloat16, 8>::load(vr + c, xv);
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = fmaf(skip, xv[j], y[j]);
      }
      Vec<__nv_bfloat16, 8>::store(out + c, y);
    }
  }
  if (*abort && warp == 0)   // copies and products in flight end before the block's memory is given back
    for (int k = 0; k < 4096; ++k) __nanosleep(256);
  end_block(tmem, 256);
}

template <bool SSD, int VP>
int launch(const pace_step_t& st, ChunkArgs a, int places, cudaStream_t s) {
  constexpr int kV = VP / 64 * kBlock, smem = 4 * kBlock + kV + (int)sizeof(Sync);
  static bool configured[16] = {};
  int dev = 0;
  PACE_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 16 || !configured[dev]) {
    PACE_CUDA_TRY(cudaFuncSetAttribute(chunk_states_kernel<SSD, VP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    PACE_CUDA_TRY(cudaFuncSetAttribute(chunk_out_kernel<SSD, VP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (dev < 16) configured[dev] = true;
  }
  for (const int per = a.places; a.place0 < places; a.place0 += per) {
    a.places = places - a.place0 < per ? places - a.place0 : per;
    const dim3 grid((unsigned)a.v_blocks, (unsigned)a.heads, (unsigned)a.places);
    chunk_states_kernel<SSD, VP><<<grid, kThreads, smem, s>>>(st, a);
    PACE_LAUNCH_CHECK("chunk_states_kernel");
    chunk_prefix_kernel<SSD, VP><<<dim3(kChunk * VP / 8 / kThreads, (unsigned)(a.heads * a.v_blocks), (unsigned)st.n_entries), kThreads, 0, s>>>(st, a);
    PACE_LAUNCH_CHECK("chunk_prefix_kernel");
    chunk_out_kernel<SSD, VP><<<grid, kThreads, smem, s>>>(st, a);
    PACE_LAUNCH_CHECK("chunk_out_kernel");
  }
  return PACE_OK;
}

// Scratch of a round of launches; all places of a step together, or as many as the budget holds: a step of many tokens goes through in
// rounds, the states of the sequences that a round leaves in the middle wait where they belong.  4096 tokens of 32 lightning heads take
// 198 MB and one round; 16384 of 64 heads 1.5 GB at once 988 us, in rounds of 512 MB 1074, 256 MB 1157, 128 MB 1274, 32 MB 2157.
constexpr uint64_t kBudget = 512ull << 20;
struct Parts { uint64_t add, tiles, kv, log_decay, total; int places, per_round, v_blocks; };
Parts parts_of(const pace_step_t& st, int heads, int vdim, bool lightning) {
  Parts p;
  const int vp = vdim <= 64 ? 64 : 128;
  p.places = st.n_tokens / kChunk + st.n_entries;
  p.v_blocks = (vdim + vp - 1) / vp;
  const uint64_t items = (uint64_t)heads * p.v_blocks, add = (uint64_t)kChunk * vp * 4, kv = lightning ? 2 * kBlock + (uint64_t)kChunk * vp * 2 : 0;
  const uint64_t fit = kBudget / (items * (2 * add + kv + 4));
  p.per_round = fit < 1 ? 1 : fit < (uint64_t)p.places ? (int)fit : p.places;
  const uint64_t n = (uint64_t)p.per_round * items;
  p.add = p.tiles = n * add;
  p.kv = n * kv;
  p.log_decay = lightning ? 0 : (n * 4 + 255) / 256 * 256;
  p.total = p.add + p.tiles + p.kv + p.log_decay;
  return p;
}

}  // namespace

// Which of the two forms a step takes.  The chunks of 64 are one launch in which every sequence walks its chunks one after another (a
// block per SM), the chunks of 128 three launches over all chunks side by side (two blocks per SM), whose last chunks are half empty.
// Both are estimated, in us on the device, from what they showed over steps of 130 to 1024 tokens, 1 to 16 sequences and 16 to 64 heads
// (state space of 64 / 128 values, lightning of 128), and with them a call: two launches and an allocation more cost the host 10 us
// where nothing else is in flight.  Calls of the chunks of 64 and of 128, us: state space, 32 heads of 64, one prompt of 300 tokens 43.1 and
// 49.2, of 400 53.7 and 50.1; 4 of 300 45.3 and 57.1, 8 of 500 117 and 113, 16 of 200 118 and 109; of 128 values, 4 of 600 106 and 121, one
// of 300 56.0 and 50.9; lightning, 32 heads, one of 130 34.8 and 30.9, 4 of 300 54.1 and 64.2, 8 of 500 160 and 143.
bool chunk_umma_pays(const pace_step_t& st, int heads, int vdim, bool lightning, int segments) {
  if (st.max_count < kChunk + 1 || st.n_entries < 1) return false;
  if (segments > 1) return true;        // (long sequences that leave SMs idle: the chunks of 64 go through twice)
  const int vp = vdim <= 64 ? 64 : 128, n = st.n_entries, wide = vp / 64 - 1;
  const float items = (float)heads * ((vdim + vp - 1) / vp);
  const int waves = (int)((n * items + 147.f) / 148.f);
  const float longest = (float)((st.max_count + 63) / 64), mean = fminf(longest, ceilf((float)st.n_tokens / (64.f * n)));
  const float walk = waves <= 1 ? longest : fmaxf(longest, mean * waves + 0.5f * (longest - mean));
  const float old_us = 3.5f + (wide ? 8.2f : 5.6f) * (lightning ? 1.11f : 1.f) * walk;
  const float places = fminf((float)(st.n_tokens / kChunk + n), (float)n * ((st.max_count + kChunk - 1) / kChunk));
  const float new_us = fmaxf(wide ? 24.f : 18.f, 8.f + (wide ? 0.126f : 0.073f) * places * items);
  return lightning ? fmaxf(30.f, new_us + 9.f) < fmaxf(30.f, old_us + 4.5f) : fmaxf(50.f, new_us + 21.f) < fmaxf(40.f, old_us + 15.f);
}

uint64_t chunk_umma_bytes(const pace_step_t& st, int heads, int dim, int vdim, bool lightning) {
  if (dim <= 64 || dim > 128 || dim % 8 || vdim % 8 || heads > 65535 || st.n_entries > 65535 || st.max_count < kChunk + 1) return 0;
  const Parts p = parts_of(st, heads, vdim, lightning);
  if (p.per_round > 65535 || (int64_t)heads * p.v_blocks > 65535) return 0;
  return p.total <= kBudget + 256 ? p.total : 0;
}

bool chunk_umma_fits(const pace_step_t& st, const ChunkArgs& a, const void* workspace, uint64_t workspace_bytes) {
  const uint64_t need = chunk_umma_bytes(st, a.heads, a.dim, a.vdim, a.decay != nullptr);
  return need && workspace && workspace_bytes >= need && aligned16(workspace) && aligned16(a.src) && aligned16(a.out) && aligned16(a.state) &&
         a.src_stride % 8 == 0 && a.out_stride % 8 == 0 && a.q_at % 8 == 0 && a.k_at % 8 == 0 && a.v_at % 8 == 0 && a.q_step % 8 == 0;
}

int chunk_umma(const pace_step_t& st, ChunkArgs a, void* workspace, cudaStream_t s) {
  const bool lightning = a.decay != nullptr;
  const Parts p = parts_of(st, a.heads, a.vdim, lightning);
  unsigned char* w = static_cast<unsigned char*>(workspace);
  a.place0 = 0, a.places = p.per_round, a.v_blocks = p.v_blocks;
  a.add = reinterpret_cast<float*>(w);
  a.tiles = w + p.add;
  a.kv = a.tiles + p.tiles;
  a.log_decay = reinterpret_cast<float*>(a.kv + p.kv);
  if (lightning) return a.vdim <= 64 ? launch<false, 64>(st, a, p.places, s) : launch<false, 128>(st, a, p.places, s);
  return a.vdim <= 64 ? launch<true, 64>(st, a, p.places, s) : launch<true, 128>(st, a, p.places, s);
}

}  // namespace pace
