// Causal softmax attention over the paged pool on the CUDA cores, for rows the tensor-core kernels do not
// take: fp32 caches, head sizes beyond 128, any pair of key and value sizes up to 640 and 512; with or without a span,
// a distance bias and a sink.  Two kernels: register tiles for fp32 rows of up to 128 elements (second half of the file), and one
// for everything else.
//
// Everything else: a thread block owns 32 query rows (token, grouped head) of one (sequence, KV head); its eight warps hold
// four rows each.  Keys and values pass through shared memory 32 at a time: a lane scores one key for its
// warp's rows, then owns value columns while the weights are passed round by shuffles.  Online softmax,
// everything in fp32.
#include <type_traits>

#include "span.cuh"

namespace pace {
namespace {

struct GeneralArgs {
  const void* q;
  void* out;
  const int32_t* rows;   // row of q and out of a token, nullptr: the token itself
  const float* slopes;
  const float* sinks;
  int H, d, vd, q_row, o_row, row;   // elements of a row of q, out and the pool
  int entry0, span, span_size;
  float scale, softcap;
  int64_t o_tok;         // elements between the rows of out
};

constexpr int kRows = 32, kKeys = 32, kRowsPerWarp = 4, kThreads = 256;

template <typename T, int VI>  // VI: value columns per lane
__global__ void __launch_bounds__(kThreads)
    attn_general_kernel(KVView kv, pace_step_t st, GeneralArgs a) {
  extern __shared__ float smem[];
  const T* __restrict__ q = static_cast<const T*>(a.q);
  T* __restrict__ out = static_cast<T*>(a.out);
  const int H = a.H, d = a.d, vd = a.vd, row = a.row;
  const int e = a.entry0 + blockIdx.z, g = blockIdx.y;
  const int Gq = H / kv.n_kv_heads;
  const int t0 = st.cu[e], count = st.cu[e + 1] - t0, start = st.start[e];
  const int r0 = blockIdx.x * kRows;
  if (r0 >= count * Gq) return;
  const int slot = st.slot[e];
  if (slot < 0 || slot >= kv.max_seqs) {
    if (threadIdx.x == 0) raise_status(kv.status, PACE_DEV_BAD_INDEX);
    return;
  }
  const int ks_ld = d | 1;
  float* qs = smem;                      // [kRows][d]
  float* ks = qs + kRows * d;            // [kKeys][ks_ld]
  float* vs = ks + kKeys * ks_ld;        // [kKeys][vd]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  for (int i = tid; i < kRows * d; i += kThreads) {
    const int r = i / d, c = i - r * d;
    float v = 0.f;
    if (r0 + r < count * Gq) {
      const int tok = (r0 + r) / Gq, hh = g * Gq + (r0 + r) % Gq;
      v = to_f<T>(q[((size_t)(a.rows ? a.rows[t0 + tok] : t0 + tok) * H + hh) * a.q_row + c]);
    }
    qs[i] = v;
  }
  int last[kRowsPerWarp];   // last visible position of the warp's rows, -1 for rows that do not exist
  int first[kRowsPerWarp];  // first one
  float slope[kRowsPerWarp];
  float m[kRowsPerWarp], l[kRowsPerWarp], acc[kRowsPerWarp][VI];
#pragma unroll
  for (int r = 0; r < kRowsPerWarp; ++r) {
    const int rr = r0 + warp * kRowsPerWarp + r;
    last[r] = rr < count * Gq ? start + rr / Gq : -1;
    first[r] = last[r] < 0 ? 0 : span_first(a.span, a.span_size, last[r]);
    slope[r] = (a.slopes && last[r] >= 0) ? a.slopes[g * Gq + rr % Gq] : 0.f;
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int i = 0; i < VI; ++i) acc[r][i] = 0.f;
  }
  const int r_end = min(r0 + kRows, count * Gq) - 1;
  const int n_keys = start + r_end / Gq + 1;
  for (int k0 = span_first(a.span, a.span_size, start + r0 / Gq) / kKeys * kKeys; k0 < n_keys; k0 += kKeys) {
    __syncthreads();
    for (int i = tid; i < kKeys * (d + vd); i += kThreads) {
      const bool is_v = i >= kKeys * d;
      const int w = is_v ? vd : d, o = is_v ? i - kKeys * d : i;
      const int j = o / w, c = o - j * w, pos = k0 + j;
      float v = 0.f;
      if (pos < n_keys) {
        const int lp = pos / kv.page_tokens;
        const int pg = view_page(kv, slot, lp);
        if (pg >= 0)
          v = to_f<T>((reinterpret_cast<const T*>(is_v ? kv.v : kv.k))[(((size_t)pg * kv.n_kv_heads + g) * kv.page_tokens +
                                                                       (pos - lp * kv.page_tokens)) * row + c]);
        else
          raise_status(kv.status, PACE_DEV_BAD_INDEX);
      }
      if (is_v) vs[j * vd + c] = v; else ks[j * ks_ld + c] = v;
    }
    __syncthreads();
    float s[kRowsPerWarp] = {0.f, 0.f, 0.f, 0.f};
    const float* kr = ks + lane * ks_ld;
    const float* qr = qs + warp * kRowsPerWarp * d;
    for (int c = 0; c < d; ++c) {
      const float x = kr[c];
#pragma unroll
      for (int r = 0; r < kRowsPerWarp; ++r) s[r] = fmaf(qr[r * d + c], x, s[r]);
    }
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) {
      if (last[r] < k0 || first[r] >= k0 + kKeys) continue;  // (the warp's rows agree: lanes differ in the key only)
      const int pos = k0 + lane;
      float x = -INFINITY;
      if (pos <= last[r] && pos >= first[r]) {
        x = s[r] * a.scale;
        if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
        x += slope[r] * (float)(pos - last[r]);
      }
      float mx = x;
#pragma unroll
      for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      mx = fmaxf(mx, m[r]);
      const float p = expf(x - mx);
      float sum = p;
#pragma unroll
      for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      const float f = expf(m[r] - mx);
      m[r] = mx;
      l[r] = l[r] * f + sum;
#pragma unroll
      for (int i = 0; i < VI; ++i) acc[r][i] *= f;
      for (int j = 0; j < kKeys; ++j) {
        const float pj = __shfl_sync(0xffffffffu, p, j);
#pragma unroll
        for (int i = 0; i < VI; ++i) {
          const int c = lane + 32 * i;
          if (c < vd) acc[r][i] = fmaf(pj, vs[j * vd + c], acc[r][i]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kRowsPerWarp; ++r) {
    const int rr = r0 + warp * kRowsPerWarp + r;
    if (last[r] < 0) continue;
    const int tok = rr / Gq, hh = g * Gq + rr % Gq;
    if (a.sinks) {  // one more term of the denominator
      const float sink = a.sinks[hh], mx = fmaxf(m[r], sink), f = expf(m[r] - mx);
      l[r] = l[r] * f + expf(sink - mx);
#pragma unroll
      for (int i = 0; i < VI; ++i) acc[r][i] *= f;
    }
    T* o = out + (a.rows ? a.rows[t0 + tok] : t0 + tok) * a.o_tok + (int64_t)hh * a.o_row;
#pragma unroll
    for (int i = 0; i < VI; ++i) {
      const int c = lane + 32 * i;
      if (c < vd) o[c] = from_f<T>(acc[r][i] / l[r]);
    }
  }
}

template <typename T, int VI>
int launch_general(const KVView& kv, const pace_step_t& st, const GeneralArgs& a, int entries, int max_tokens, cudaStream_t s) {
  const size_t smem = sizeof(float) * ((size_t)kRows * a.d + (size_t)kKeys * (a.d | 1) + (size_t)kKeys * a.vd);
  if (smem > 227 * 1024) return PACE_ERR_UNSUPPORTED;
  PACE_CUDA_TRY(cudaFuncSetAttribute(attn_general_kernel<T, VI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int Gq = a.H / kv.n_kv_heads;
  const dim3 grid((unsigned)(((size_t)max_tokens * Gq + kRows - 1) / kRows), (unsigned)kv.n_kv_heads, (unsigned)entries);
  attn_general_kernel<T, VI><<<grid, kThreads, smem, s>>>(kv, st, a);
  PACE_LAUNCH_CHECK("attn_general_kernel");
  return PACE_OK;
}

// ---- 32-bit rows ---------------------------------------------------------------------------------------------------------------
// The kernel above issues a shared-memory load per 4 multiply-adds of a lane and a shuffle per 4 of the second product: 3.3 TFLOP/s of
// the 74 that the FMA units have (two prompts of 701 and 1100 tokens, 16/4 heads of 128: 2102 us).  Register tiles instead: a block of four warps owns 64 rows, a
// thread 8 of them with 4 of a tile's 64 keys, then with 4 or 8 value columns, so that a 16-byte shared-memory load feeds 11 (scores,
// values of up to 64 elements) to 16 multiply-adds.  The rows' operands are the same for 16 lanes (one shared-memory pass), keys and values pass by cp.async while the other
// product runs, and two blocks fit an SM, so that one's barriers and exponentials run beside the other's products.  The same prompts:
// 240 us with the append, 30 TFLOP/s, bound by FMA issue and, in blocks of few keys, by the latency of a tile's chain.  fp32 throughout; a
// score is the sum of two chains (even and odd elements, the halves of a two-wide FMA), which makes neither sum longer: against 64 bits
// 3.0e-7, before 3.9e-7.
constexpr int kTileRows = 64, kTileKeys = 64, kTileThreads = 128;

template <int DP>  // keys' and values' elements in shared memory
struct TileShape {
  static constexpr int kLd = DP + 4;                    // rows 4 banks apart
  static constexpr int kPLd = kTileKeys / 2 + 4;        // weights of half the keys at a time
  static constexpr int kFloats = kTileRows * kLd + kTileKeys * kLd + kTileKeys * DP + kTileRows * kPLd;
  static constexpr size_t kSmem = sizeof(float) * (kFloats + 3 * kTileRows) + sizeof(int64_t) * 2 * kTileKeys;
};

__device__ __forceinline__ void copy16_zfill(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void fma2(float2& c, float2 a, float2 b) {
  asm("{.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%0, %1};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;}"
      : "+f"(c.x), "+f"(c.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
}

template <int DP>
__global__ void __launch_bounds__(kTileThreads, 2) attn_tile_kernel(KVView kv, pace_step_t st, GeneralArgs a) {
  using S = TileShape<DP>;
  constexpr int kHalves = DP / 64;                      // 64 value columns: four per lane of a row's sixteen
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;                                     // [rows][kLd]
  float* ks = qs + kTileRows * S::kLd;                  // [keys][kLd]
  float* vs = ks + kTileKeys * S::kLd;                  // [keys][DP]
  float* ps = vs + kTileKeys * DP;                      // [rows][kPLd]
  int64_t* off = reinterpret_cast<int64_t*>(ps + kTileRows * S::kPLd);   // [2][keys] element offset of a key's row, -1: none
  int* row_last = reinterpret_cast<int*>(off + 2 * kTileKeys);           // last position a row sees, -1: no such row
  int* row_first = row_last + kTileRows;
  float* row_slope = reinterpret_cast<float*>(row_first + kTileRows);

  const int H = a.H, d = a.d, vd = a.vd;
  const int g = blockIdx.x, e = a.entry0 + blockIdx.y;
  const int Gq = H / kv.n_kv_heads;
  const int t0 = st.cu[e], rows = (st.cu[e + 1] - t0) * Gq, start = st.start[e];
  const int r0 = (gridDim.z - 1 - blockIdx.z) * kTileRows;               // the last rows see the most keys: they begin first
  if (r0 >= rows) return;
  const int slot = st.slot[e];
  if (slot < 0 || slot >= kv.max_seqs) {
    if (threadIdx.x == 0) raise_status(kv.status, PACE_DEV_BAD_INDEX);
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int half = lane >> 4, cl = lane & 15;           // my rows: 16 warp + 2 i + half; my keys cl + 16 c, my columns 64 h + 4 cl

  const float* __restrict__ q = static_cast<const float*>(a.q);
  for (int i = tid; i < kTileRows * (DP / 4); i += kTileThreads) {
    const int r = i / (DP / 4), c = (i % (DP / 4)) * 4;
    const int rr = r0 + r, n = rr < rows ? min(max(d - c, 0), 4) : 0;
    const int tok = n ? rr / Gq : 0, hh = g * Gq + (n ? rr % Gq : 0);
    copy16_zfill(qs + r * S::kLd + c, q + ((size_t)(a.rows ? a.rows[t0 + tok] : t0 + tok) * H + hh) * a.q_row + (n ? c : 0), 4 * n);
  }
  if (tid < kTileRows) {
    const int rr = r0 + tid, last = rr < rows ? start + rr / Gq : -1;
    row_last[tid] = last;
    row_first[tid] = last < 0 ? 0 : span_first(a.span, a.span_size, last);
    row_slope[tid] = a.slopes && last >= 0 ? a.slopes[g * Gq + rr % Gq] : 0.f;
  }
  // the tiles' keys, what every row of the block sees of them
  const int last_lo = start + r0 / Gq, last_hi = start + (min(r0 + kTileRows, rows) - 1) / Gq;
  const int n_keys = last_hi + 1, first_hi = span_first(a.span, a.span_size, last_hi);
  const int k_begin = span_first(a.span, a.span_size, last_lo) / kTileKeys * kTileKeys;
  const bool full = r0 + kTileRows <= rows;
  // ... and the rows of the warp: values that a row does not see (later tokens, tokens in front of a span) stay out of its sums, where a
  // weight of zero would still hand on an infinity or NaN
  const int wr = r0 + 16 * (threadIdx.x >> 5);
  const int w_lo = wr < rows ? start + wr / Gq : -1, w_hi = wr < rows ? start + (min(wr + 16, rows) - 1) / Gq : -1;
  const int w_first = span_first(a.span, a.span_size, max(w_lo, 0)), w_all = span_first(a.span, a.span_size, max(w_hi, 0));
  const float* kp = static_cast<const float*>(static_cast<const void*>(kv.k));
  const float* vp = static_cast<const float*>(static_cast<const void*>(kv.v));

  auto find = [&](int k0, int64_t* to) {                // where the rows of 64 keys lie
    if (tid < kTileKeys) {
      const int pos = k0 + tid;
      int64_t o = -1;
      if (pos < n_keys) {
        const int lp = pos / kv.page_tokens, pg = view_page(kv, slot, lp);
        if (pg >= 0)
          o = (((int64_t)pg * kv.n_kv_heads + g) * kv.page_tokens + (pos - lp * kv.page_tokens)) * a.row;
        else
          raise_status(kv.status, PACE_DEV_BAD_INDEX);
      }
      to[tid] = o;
    }
  };
  auto fetch = [&](const float* src, int width, float* dst, int ld, const int64_t* at) {
#pragma unroll 4
    for (int i = tid; i < kTileKeys * (DP / 4); i += kTileThreads) {
      const int j = i / (DP / 4), c = (i % (DP / 4)) * 4;
      const int64_t o = at[j];
      const int n = o >= 0 ? min(max(width - c, 0), 4) : 0;
      copy16_zfill(dst + j * ld + c, src + (n ? o + c : 0), 4 * n);
    }
    copies_commit();
  };

  float m[8], l[8];
  float2 acc[8][2 * kHalves];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < 2 * kHalves; ++c) acc[i][c] = make_float2(0.f, 0.f);
  }
  const int my_row = 16 * warp + half;
  find(k_begin, off);
  __syncthreads();
  fetch(kp, d, ks, S::kLd, off);                        // (with the queries)
  fetch(vp, vd, vs, DP, off);
  int buf = 0;
  for (int k0 = k_begin; k0 < n_keys; k0 += kTileKeys, buf ^= 1) {
    const bool more = k0 + kTileKeys < n_keys;
    copies_wait<1>();
    __syncthreads();
    if (more) find(k0 + kTileKeys, off + (buf ^ 1) * kTileKeys);
    float2 s2[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) s2[i][c] = make_float2(0.f, 0.f);
    const float* qr = qs + my_row * S::kLd;
    const float* kr = ks + cl * S::kLd;
#pragma unroll 2
    for (int x = 0; x < d; x += 4) {
      float4 kk[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) kk[c] = *reinterpret_cast<const float4*>(kr + 16 * c * S::kLd + x);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 qq = *reinterpret_cast<const float4*>(qr + 2 * i * S::kLd + x);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          fma2(s2[i][c], make_float2(qq.x, qq.y), make_float2(kk[c].x, kk[c].y));
          fma2(s2[i][c], make_float2(qq.z, qq.w), make_float2(kk[c].z, kk[c].w));
        }
      }
    }
    __syncthreads();                                    // the keys are read, the next tile's rows are found
    if (more) fetch(kp, d, ks, S::kLd, off + (buf ^ 1) * kTileKeys);
    const bool edge = !full || k0 + kTileKeys - 1 > last_lo || k0 < first_hi;
    float p[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int last = row_last[my_row + 2 * i], first = edge ? row_first[my_row + 2 * i] : 0;
      const float slope = a.slopes ? row_slope[my_row + 2 * i] : 0.f;
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int pos = k0 + cl + 16 * c;
        float x = (s2[i][c].x + s2[i][c].y) * a.scale;
        if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
        x += slope * (float)(pos - last);
        if (edge && (pos > last || pos < first)) x = -INFINITY;
        p[i][c] = x;
        mx = fmaxf(mx, x);
      }
#pragma unroll
      for (int o = 8; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      mx = fmaxf(mx, m[i]);
      const float base = mx == -INFINITY ? 0.f : mx;    // (a row that has seen no key yet)
      const float f = expf(m[i] - base);
      m[i] = mx;
      l[i] *= f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        p[i][c] = expf(p[i][c] - base);
        l[i] += p[i][c];
      }
#pragma unroll
      for (int c = 0; c < 2 * kHalves; ++c) {
        acc[i][c].x *= f;
        acc[i][c].y *= f;
      }
    }
    if (more) copies_wait<1>(); else copies_wait<0>();
    __syncthreads();                                    // the values are there
#pragma unroll
    for (int kh = 0; kh < 2; ++kh) {
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        ps[(my_row + 2 * i) * S::kPLd + cl] = p[i][2 * kh];
        ps[(my_row + 2 * i) * S::kPLd + 16 + cl] = p[i][2 * kh + 1];
      }
      __syncwarp();                                     // a warp reads the weights it wrote itself
      const float* pr = ps + my_row * S::kPLd;
      const float* vr = vs + kh * 32 * DP + 4 * cl;
      const int p0 = k0 + 32 * kh, j_a = max(0, w_first - p0), j_z = min(32, w_hi + 1 - p0);   // (the same for the warp)
      auto add_values = [&](auto ragged) {
        constexpr bool some = decltype(ragged)::value;
#pragma unroll 2
        for (int j = some ? j_a & ~3 : 0; j < (some ? j_z : 32); j += 4) {
          float4 pp[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) pp[i] = *reinterpret_cast<const float4*>(pr + 2 * i * S::kPLd + j);
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            if (some && (j + y < j_a || j + y >= j_z)) continue;
            float4 v[kHalves];
#pragma unroll
            for (int h = 0; h < kHalves; ++h) v[h] = *reinterpret_cast<const float4*>(vr + (j + y) * DP + 64 * h);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float w = y == 0 ? pp[i].x : y == 1 ? pp[i].y : y == 2 ? pp[i].z : pp[i].w;
              if (some && w == 0.f) continue;
#pragma unroll
              for (int h = 0; h < kHalves; ++h) {
                fma2(acc[i][2 * h], make_float2(w, w), make_float2(v[h].x, v[h].y));
                fma2(acc[i][2 * h + 1], make_float2(w, w), make_float2(v[h].z, v[h].w));
              }
            }
          }
        }
      };
      if (p0 >= w_all && p0 + 31 <= w_lo) add_values(std::false_type{});   // (every row sees all of them)
      else add_values(std::true_type{});
    }
    __syncthreads();
    if (more) fetch(vp, vd, vs, DP, off + (buf ^ 1) * kTileKeys);
  }

  const bool wide = ((a.o_row | a.o_tok | vd) & 3) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int rr = r0 + my_row + 2 * i;
    float sum = l[i];
#pragma unroll
    for (int o = 8; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (rr >= rows) continue;
    const int tok = rr / Gq, hh = g * Gq + rr % Gq;
    float f = 1.f;
    if (a.sinks) {  // one more term of the denominator
      const float sink = a.sinks[hh], mx = fmaxf(m[i], sink);
      f = expf(m[i] - mx);
      sum = sum * f + expf(sink - mx);
    }
    float* o = static_cast<float*>(a.out) + (a.rows ? a.rows[t0 + tok] : t0 + tok) * a.o_tok + (int64_t)hh * a.o_row;
#pragma unroll
    for (int h = 0; h < kHalves; ++h) {
      const float y[4] = {acc[i][2 * h].x * f / sum, acc[i][2 * h].y * f / sum, acc[i][2 * h + 1].x * f / sum, acc[i][2 * h + 1].y * f / sum};
      const int c = 64 * h + 4 * cl;
      if (wide) {
        if (c < vd) Vec<float, 4>::store(o + c, y);
      } else {
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (c + x < vd) o[c + x] = y[x];
      }
    }
  }
}

template <int DP>
int launch_tiles(const KVView& kv, const pace_step_t& st, const GeneralArgs& a, int entries, int tiles, cudaStream_t s) {
  PACE_CUDA_TRY(cudaFuncSetAttribute(attn_tile_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TileShape<DP>::kSmem));
  attn_tile_kernel<DP><<<dim3((unsigned)kv.n_kv_heads, (unsigned)entries, (unsigned)tiles), kTileThreads, TileShape<DP>::kSmem, s>>>(kv, st, a);
  PACE_LAUNCH_CHECK("attn_tile_kernel");
  return PACE_OK;
}

// Which launches take tiles: fp32 rows of up to 128 elements (a wider head's queries and keys leave no room for a second block) that
// 16-byte copies can read, however few query rows there are.  One entry of 4, 8 or 64 query rows over 1000 keys, heads of 128: 863, 885 and
// 893 us by the kernel above, 177 to 181 us by tiles; 32 entries over 500 keys 455 and 101 us; heads of 64: 337 and 115 us.
bool tiles_fit(const KVView& kv, const GeneralArgs& a, int max_tokens) {
  const int64_t rows = (int64_t)max_tokens * (a.H / kv.n_kv_heads);
  return a.d <= 128 && a.vd <= 128 && rows >= 1 && (rows + kTileRows - 1) / kTileRows <= 65535 &&
         ((a.q_row | a.row) & 3) == 0 && ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(kv.k) | reinterpret_cast<uintptr_t>(kv.v)) & 15) == 0;
}

template <typename T>
int general_t(const KVView& kv, const pace_step_t& st, const GeneralArgs& a, int entries, int max_tokens, cudaStream_t s) {
  if (a.vd <= 32) return launch_general<T, 1>(kv, st, a, entries, max_tokens, s);
  if (a.vd <= 64) return launch_general<T, 2>(kv, st, a, entries, max_tokens, s);
  if (a.vd <= 128) return launch_general<T, 4>(kv, st, a, entries, max_tokens, s);
  if (a.vd <= 256) return launch_general<T, 8>(kv, st, a, entries, max_tokens, s);
  return launch_general<T, 16>(kv, st, a, entries, max_tokens, s);
}

int general(const KVView& kv, const pace_step_t& st, const GeneralArgs& a, int entries, int max_tokens, int dtype, cudaStream_t s) {
  if (a.d > 640 || a.vd > 512 || kv.n_kv_heads > 65535 || entries > 65535) return PACE_ERR_UNSUPPORTED;
  if (dtype == PACE_DTYPE_FP32 && tiles_fit(kv, a, max_tokens)) {
    const int tiles = (int)(((int64_t)max_tokens * (a.H / kv.n_kv_heads) + kTileRows - 1) / kTileRows);
    return a.d <= 64 && a.vd <= 64 ? launch_tiles<64>(kv, st, a, entries, tiles, s) : launch_tiles<128>(kv, st, a, entries, tiles, s);
  }
  return dtype == PACE_DTYPE_BF16 ? general_t<__nv_bfloat16>(kv, st, a, entries, max_tokens, s)
                                  : general_t<float>(kv, st, a, entries, max_tokens, s);
}

}  // namespace

int attn_general_span(const pace_kv_pool_t* p, int layer, const pace_step_t& st, const pace_attn_span_args_t& a,
                      cudaStream_t s) {
  GeneralArgs ga;
  ga.q = a.q;
  ga.out = a.out;
  ga.rows = nullptr;
  ga.slopes = a.slopes;
  ga.sinks = a.sinks;
  ga.H = a.n_q_heads;
  ga.d = a.dim;
  ga.vd = a.vdim;
  ga.q_row = a.q_elems;
  ga.o_row = a.out_elems;
  ga.row = a.dtype == PACE_DTYPE_BF16 ? p->head_dim : p->head_dim / 2;
  ga.entry0 = a.entry_begin;
  ga.span = a.span;
  ga.span_size = a.span_size;
  ga.scale = a.scale;
  ga.softcap = a.softcap;
  ga.o_tok = span_out_row(a);
  return general(make_view(p, layer, nullptr), st, ga, a.entry_end - a.entry_begin, a.max_tokens, a.dtype, s);
}

}  // namespace pace

using namespace pace;

extern "C" int pace_attn_general(const pace_kv_pool_t* p, int32_t layer, const pace_step_t* st, const void* q, void* out,
                                 int32_t H, int32_t d, int32_t vd, float scale, int32_t dtype, void* stream) {
  if (!p || !p->pages || !step_ok(st) || !q || !out || layer < 0 || layer >= p->n_layers) return PACE_ERR_INVALID;
  if (H < 1 || H % p->n_kv_heads || d < 1 || vd < 1 || st->max_count < 0) return PACE_ERR_INVALID;
  if (dtype != PACE_DTYPE_BF16 && dtype != PACE_DTYPE_FP32) return PACE_ERR_INVALID;
  if (p->row_format == PACE_ROWS_BF16 && dtype != PACE_DTYPE_BF16) return PACE_ERR_INVALID;
  GeneralArgs ga;
  ga.row = ga.q_row = ga.o_row = dtype == PACE_DTYPE_BF16 ? p->head_dim : p->head_dim / 2;
  if (d > ga.row || vd > ga.row) return PACE_ERR_INVALID;
  if (st->n_tokens == 0) return PACE_OK;
  PACE_PROFILE("attn_general", stream, "layer=%d entries=%d tokens=%d", layer, st->n_entries, st->n_tokens);
  ga.q = q;
  ga.out = out;
  ga.rows = st->q_row;
  ga.slopes = ga.sinks = nullptr;
  ga.H = H;
  ga.d = d;
  ga.vd = vd;
  ga.entry0 = 0;
  ga.span = PACE_SPAN_ALL;
  ga.span_size = 0;
  ga.scale = scale;
  ga.softcap = 0.f;
  ga.o_tok = (int64_t)H * ga.o_row;
  return general(make_view(p, layer, nullptr), *st, ga, st->n_entries, st->max_count, dtype, (cudaStream_t)stream);
}
