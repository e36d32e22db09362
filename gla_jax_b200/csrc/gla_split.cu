// Chunked GLA in float32 precision on the tensor cores: forward and backward for float32 callers, for head sizes
// that the 128-wide kernels do not serve, and for recurrent_gla over any number of tokens.
//
// Reference algorithm: gla.py:483-625 (chunk forward / backward), gla.py:26-47 and 172-269 (the recurrence, which the
// chunked form equals for any chunk length).
//
// Why split operands.  These paths used to run on float32 FMAs (one SGEMM launch per product, or one FMA chain per
// token), which the CUDA cores bound.  A float32 number is the sum of three bf16 numbers (8 + 8 + 8 significant
// bits), so a float32 product is six bf16 products (the terms below 2^-24 dropped), three when the other side is
// bf16 data already, one when both are; the accumulation is float32 throughout.  That is the precision of the FMA
// form at 1/6 to 1/1 of the tensor rate, several times the FMA rate.  The instruction is the register-operand
// mma.sync: chunks of 64 rows with every operand three planes deep leave room for two blocks per SM at head size 64
// (tcgen05's 128-row tiles of three planes leave it for one, with nothing to run beside its serial phases), and the
// planes need no canonical layout, so that rows, columns and lengths come in any multiple of 16.
//
// One anchor per chunk.  lam = running sum of the log gates inside the chunk, G = its total.  With m = G / 2 per
// feature, q~ = q exp(lam - m) and k~ = k exp(m - lam) give every product of the chunk:
//   P = tril(q~ k~^T)                      O  = P V + q~ (e^m S)
//   dq = exp(lam - m) (dP k~ + dO (e^m S)^T)   dk = exp(m - lam) (dP^T q~ + V (e^(G - m) dS)^T)
//   dV = P^T dO + k~ (e^(G - m) dS)        dP = tril(dO V^T)
// (S: the state entering the chunk, dS: the gradient of the state leaving it; the factors e^m ride on the rows of
// the states while they are split.)  The weights stay within exp(+-LIMIT / 2) as long as sum |g| <= LIMIT over the
// chunk, no single |g| exceeds ONE_GATE and no thread's rows exceed GROUP together (the weights are products of exp(g),
// which must not vanish); chunks beyond that ("sharp") are walked token by token from the state that enters them, in
// float32 FMAs.
//
// Three launches forward, three backward: per-chunk state products (k^^T V, resp. q^^T dO), a scan over the chunks
// in place, and the chunk kernel.  States are float32, N of them per head (slot n: the state that enters chunk n, resp.
// the gradient of the one that leaves it); for a backward the final state follows as slot N, so that
//   dG_n[d] = <S_{n+1}[d,:], dS_n[d,:]>
// is a dot product of two stored rows and dlam = q dq - k dk needs no other inter-chunk term.
#include "gla_common.cuh"
#include "tc_ptx.cuh"
#include "tma_maps.cuh"

namespace gla {

using namespace tc;

namespace {

// A weight of exp(-50) leaves the third plane of a value above the denormals as long as the value itself is above 4e-12
// (2^-126 2^16 exp(50)).  At 140 keys or state gradients below 2e-3 began to lose it: 1e-4 of dk and dv with output
// gradients of 1e-8 and a decay of 134, which the walk by token (2.5 to 2.8 times the time of a mild bf16 chunk, 1.9 of a float32 one) does not touch.
constexpr float PX_LIMIT = 100.f;
constexpr float PX_ONE_GATE = 60.f, PX_GROUP = 80.f;      // of a thread's rows together

// D features, chunks of L rows.  Element-wise stages: a thread owns a column pair and RPT consecutive rows.  Products:
// warps in WR row groups of 16 x WC column groups.
template <int D_, int L_>
struct Px {
  static constexpr int D = D_, L = L_;
  static constexpr int NT = D >= 128 && L == 64 ? 512 : D >= 64 ? 256 : 128;
  static constexpr int CP = D / 2, RG = NT / CP, RPT = L / RG;
  static constexpr int WR = L / 16, WC = (NT / 32) / WR, CW = D / WC;
  static constexpr int NB = (WR + WC - 1) / WC;  // 16 x 16 score blocks per warp, at most
  static constexpr int LD = 2 * D + 16;          // row pitch in bytes: the 16-byte pad spreads ldmatrix rows over the banks
  static constexpr int PLANE = L * LD;
  static constexpr int PW = D < 64 ? D : 64, NP = D / PW, PC = PW / WC;   // state pieces of PW value columns, PC per warp
  static constexpr int LDS = 2 * PW + 16, SPLANE = D * LDS;
  static constexpr int LDT = 2 * L + 16, TPLANE = L * LDT;                // score tile
  static constexpr int SREG = D * PW / 4 / NT;   // float4 loads per thread and state piece
  static constexpr int AP = D + 8;               // row pitch (floats) of the float32 tiles of the closing pass
  static constexpr int TP = 4 * NT / D, TE = D / TP;   // walk by token: threads per four rows or columns of the state, elements of each
  static_assert(PC % 16 == 0 && CW % 16 == 0, "a warp's columns come in pairs of 8-wide tiles");
};

struct PxParams {
  int64_t B, T, H, N;
  int trev;                     // tokens in reverse order (recurrent_gla(reverse=True))
  int out_bf, in_bf;
  const float* g;
  const void *v, *k, *q, *dout;
  int64_t NS;                   // slots of S per head: N, or N + 1 with the final state
  float *S, *dS;                // (B H, NS, D, D), (B H, N, D, D)
  float* eG;                    // (B H, N, D): exp of every chunk's total log decay
  void *out, *dq, *dk, *dv;
  float* dg;
};

// ---- operands --------------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void hmma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// x = hi + mid + lo, eight significant bits each (two values side by side)
__device__ __forceinline__ void split3(float x, float y, uint32_t (&s)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    s[i] = pack_bf16x2(x, y);
    if (i < 2) {
      x -= __uint_as_float(s[i] << 16);
      y -= __uint_as_float(s[i] & 0xffff0000u);
    }
  }
}
__device__ __forceinline__ void st_split3(uint8_t* p, uint32_t plane, float x, float y) {
  uint32_t s[3];
  split3(x, y, s);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(p + i * plane) = s[i];
}
__device__ __forceinline__ void st_split3(uint8_t* p, uint32_t plane, float4 v) {
  uint32_t a[3], b[3];
  split3(v.x, v.y, a);
  split3(v.z, v.w, b);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(p + i * plane) = make_uint2(a[i], b[i]);
}
// A operand (16 rows x 16 of K) of NS planes, stored row-major [m][k] ...
template <int NS>
__device__ __forceinline__ void ld_a(uint32_t (&a)[NS][4], uint32_t base, uint32_t plane, uint32_t ld, int m0, int k0, int lane) {
  const uint32_t addr = base + (uint32_t)(m0 + (lane & 15)) * ld + (uint32_t)(k0 + (lane >> 4) * 8) * 2;
#pragma unroll
  for (int s = 0; s < NS; ++s) ldsm4(a[s], addr + s * plane);
}
// ... or [k][m]
template <int NS>
__device__ __forceinline__ void ld_a_t(uint32_t (&a)[NS][4], uint32_t base, uint32_t plane, uint32_t ld, int m0, int k0, int lane) {
  const uint32_t addr = base + (uint32_t)(k0 + (lane & 7) + ((lane >> 4) & 1) * 8) * ld + (uint32_t)(m0 + ((lane >> 3) & 1) * 8) * 2;
#pragma unroll
  for (int s = 0; s < NS; ++s) ldsm4t(a[s], addr + s * plane);
}
// c[2 NQ tiles of 8 columns] += A B over 16 of K.  B is stored [n][k] (BT = false) or [k][n] (BT = true).  Products of
// planes sa and sb with sa + sb > 2 lie below 2^-24 of the result and are left out; the small ones come first.
// EX (what leaves in float32, or makes what does): the tensor cores cut off what an addition shifts out, which over the
// length of a product adds up to 0.7e-6 (head size 32) to 1.7e-6 (128) of a float32 result; so 16 of K are summed from
// zero and added in float32: 1.8e-7, and 2.5e-7 for the recurrence in FMAs.  It costs 4 % of a float32 call (587 -> 608 us
// for 4 x 2048 tokens of 6 heads of 128, forward and backward) and 1 to 3 % of a bf16 one, whose dlog_fgate is float32.
template <int NSA, int NSB, int NQ, bool BT, bool EX>
__device__ __forceinline__ void mma_step(float (*c)[4], const uint32_t (&a)[NSA][4], uint32_t base, uint32_t plane,
                                         uint32_t ld, int n0, int k0, int lane) {
  const int r8 = lane & 7, h3 = (lane >> 3) & 1, h4 = (lane >> 4) & 1;
#pragma unroll
  for (int j = 0; j < NQ; ++j) {
    const int n = n0 + 16 * j;
    const uint32_t addr = BT ? base + (uint32_t)(k0 + r8 + 8 * h3) * ld + (uint32_t)(n + 8 * h4) * 2
                             : base + (uint32_t)(n + r8 + 8 * h4) * ld + (uint32_t)(k0 + 8 * h3) * 2;
    uint32_t b[NSB][4];
#pragma unroll
    for (int s = 0; s < NSB; ++s) {
      if (BT) ldsm4t(b[s], addr + s * plane); else ldsm4(b[s], addr + s * plane);
    }
    float y[2][4] = {};
    float (&c0)[4] = EX ? y[0] : c[2 * j], (&c1)[4] = EX ? y[1] : c[2 * j + 1];
#pragma unroll
    for (int t = 2; t >= 0; --t)
#pragma unroll
      for (int sa = 0; sa < NSA; ++sa) {
        const int sb = t - sa;
        if (sb >= 0 && sb < NSB) {
          hmma(c0, a[sa], b[sb][0], b[sb][1]);
          hmma(c1, a[sa], b[sb][2], b[sb][3]);
        }
      }
    if (EX)
#pragma unroll
      for (int e = 0; e < 4; ++e) { c[2 * j][e] += y[0][e]; c[2 * j + 1][e] += y[1][e]; }
  }
}
template <typename TI> struct Pair;
template <> struct Pair<bf16> {
  uint32_t u;
  __device__ __forceinline__ void load(const void* p, int64_t e) { u = __ldg(reinterpret_cast<const unsigned int*>((const bf16*)p + e)); }
  __device__ __forceinline__ void zero() { u = 0u; }
  __device__ __forceinline__ float2 get() const { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
};
template <> struct Pair<float> {
  float2 u;
  __device__ __forceinline__ void load(const void* p, int64_t e) { u = __ldg(reinterpret_cast<const float2*>((const float*)p + e)); }
  __device__ __forceinline__ void zero() { u = make_float2(0.f, 0.f); }
  __device__ __forceinline__ float2 get() const { return u; }
};
template <typename TI> constexpr int planes_of() { return sizeof(TI) == 2 ? 1 : 3; }

// Where a chunk's rows lie.
template <class C>
struct ChunkAt {
  int64_t n, bh, row0;
  int step, nv;                 // elements from row to row (negative in reverse), rows inside the sequence
  __device__ __forceinline__ ChunkAt(const PxParams& p, int64_t blk) {
    n = blk % p.N; bh = blk / p.N;
    const int64_t b = bh / p.H, h = bh % p.H;
    const int64_t t0 = n * C::L, left = p.T - t0;
    step = (int)(p.H * C::D);
    row0 = ((b * p.T + (p.trev ? p.T - 1 - t0 : t0)) * p.H + h) * C::D;
    if (p.trev) step = -step;
    nv = left < C::L ? (int)left : C::L;
  }
  __device__ __forceinline__ int64_t row(int r) const { return row0 + (int64_t)r * step; }
};
template <class C>
__device__ __forceinline__ void load_gates(float2 (&g)[C::RPT], const float* gp, const ChunkAt<C>& at, int r0, int cp) {
#pragma unroll
  for (int i = 0; i < C::RPT; ++i)
    g[i] = r0 + i < at.nv ? __ldg(reinterpret_cast<const float2*>(gp + at.row(r0 + i) + 2 * cp)) : make_float2(0.f, 0.f);
}
template <class C, typename TI>
__device__ __forceinline__ void load_pairs(Pair<TI> (&x)[C::RPT], const void* xp, const ChunkAt<C>& at, int r0, int cp) {
#pragma unroll
  for (int i = 0; i < C::RPT; ++i)
    if (r0 + i < at.nv) x[i].load(xp, at.row(r0 + i) + 2 * cp); else x[i].zero();
}
// A chunk of v or dO into planes (row-major, pitch LD)
template <class C, typename TI>
__device__ __forceinline__ void copy_rows(uint8_t* dst, const void* src, const ChunkAt<C>& at) {
  if constexpr (sizeof(TI) == 2) {
#pragma unroll
    for (int j = 0; j < C::L * C::D / 8 / C::NT; ++j) {
      const int id = threadIdx.x + C::NT * j, r = id / (C::D / 8), c = id % (C::D / 8);
      uint4 u = make_uint4(0u, 0u, 0u, 0u);
      if (r < at.nv) u = __ldg(reinterpret_cast<const uint4*>((const bf16*)src + at.row(r) + c * 8));
      *reinterpret_cast<uint4*>(dst + r * C::LD + c * 16) = u;
    }
  } else {
#pragma unroll
    for (int j = 0; j < C::L * C::D / 4 / C::NT; ++j) {
      const int id = threadIdx.x + C::NT * j, r = id / (C::D / 4), c = id % (C::D / 4);
      float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < at.nv) u = __ldg(reinterpret_cast<const float4*>((const float*)src + at.row(r) + c * 4));
      st_split3(dst + r * C::LD + c * 8, C::PLANE, u);
    }
  }
}
// From the log gates of the thread's rows (exp of them on return), exchanged between the row groups: half of the chunk's
// total, exp(lam - half) before the thread's rows, and whether the chunk is sharp.  The weight is a product from the
// anchor on, not the exponential of a sum: with gates of -30 to -55 a sum of that size left 0.5e-6 to 1.1e-6 in a float32
// result, the products 2e-7.  seg: [3][RG][D] floats.
template <class C>
__device__ __forceinline__ bool gate_weights(float2 (&g)[C::RPT], float* seg, int rg, int cp, float2& half, float2& start) {
  float* sab = seg + C::RG * C::D;
  float* prod = sab + C::RG * C::D;
  float2 s = make_float2(0.f, 0.f), a = s, f = make_float2(1.f, 1.f);
  bool big = false;
#pragma unroll
  for (int i = 0; i < C::RPT; ++i) {
    s.x += g[i].x; s.y += g[i].y;
    a.x += fabsf(g[i].x); a.y += fabsf(g[i].y);
    big = big || !(fabsf(g[i].x) <= PX_ONE_GATE) || !(fabsf(g[i].y) <= PX_ONE_GATE);
    g[i] = make_float2(expf(g[i].x), expf(g[i].y));
    f.x *= g[i].x; f.y *= g[i].y;
  }
  big = big || a.x > PX_GROUP || a.y > PX_GROUP;
  *reinterpret_cast<float2*>(seg + rg * C::D + 2 * cp) = s;
  *reinterpret_cast<float2*>(sab + rg * C::D + 2 * cp) = a;
  *reinterpret_cast<float2*>(prod + rg * C::D + 2 * cp) = f;
  __syncthreads();
  s = make_float2(0.f, 0.f); a = s;
#pragma unroll
  for (int r = 0; r < C::RG; ++r) {
    const float2 t = *reinterpret_cast<const float2*>(seg + r * C::D + 2 * cp);
    const float2 u = *reinterpret_cast<const float2*>(sab + r * C::D + 2 * cp);
    s.x += t.x; s.y += t.y;
    a.x += u.x; a.y += u.y;
  }
  half = make_float2(0.5f * s.x, 0.5f * s.y);
  start = make_float2(expf(-half.x), expf(-half.y));
#pragma unroll
  for (int r = 0; r < C::RG - 1; ++r)
    if (r < rg) {
      const float2 t = *reinterpret_cast<const float2*>(prod + r * C::D + 2 * cp);
      start.x *= t.x; start.y *= t.y;
    }
  return __syncthreads_or(big || !(a.x <= PX_LIMIT) || !(a.y <= PX_LIMIT)) != 0;
}

// ---- a chunk token by token -----------------------------------------------------------------------------------------------
// The recurrence itself, from the state that enters the chunk: every weight is a product of exp(g), so that a gate that
// resets the state costs the later tokens nothing.  (Weights exp(lam_i - lam_j) from running sums, which stood here
// before, lost what the sums had grown to: 4e-5 of out after one gate of -1e4, 1.1e-4 after eight, against 2e-7.)
// A thread holds TE elements of each of four rows (COL = false) or columns (COL = true) of the state, so that a value it
// reads from shared memory, which bounds the walk, serves four sums; TP consecutive threads share the four.  What a
// token adds is w[element] scalar(token)[row or column], and out(token, row or column, sum_e z[e] state[e]) leaves
// through lanes 0 to 3 of the TP.  f, w, z: float32 [L][D].
//   REV = false: state = f state + w scalar, then the sum;   REV = true: state += w scalar, then the sum, then state *= f
// Measured, bf16 4 x 2048 tokens, 6 heads, every chunk sharp, forward and with the backward: head size 128 1288, 3322 us
// (pair by pair) -> 333, 1063; head size 64 579, 1567 -> 110, 375 (mild chunks: 126, 389 and 44, 150).
// It also serves a chunk in which the tensor cores leave something that is not finite.  Their products meet the zeros
// above the diagonal, so a not-a-number or an infinity reached up to 15 earlier tokens, an infinity became
// not-a-number in the split, and a weighted q or k beyond 1e38 overflowed: the recurrence does none of that.
// What they leave shows every case (0 x inf and inf - inf included), so nothing but the sums needs looking at.
template <int N>
__device__ __forceinline__ float not_finite(const float (&c)[N][4], float z) {       // 0 as long as everything is finite
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) z = fmaf(c[j][e], 0.f, z);
  return z;
}
template <int VW> __device__ __forceinline__ void ld_vec(float (&x)[VW], const float* p) {
  if constexpr (VW == 2) { const float2 v = *reinterpret_cast<const float2*>(p); x[0] = v.x; x[1] = v.y; }
  else { const float4 v = *reinterpret_cast<const float4*>(p); x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w; }
}
// The four sums over TP lanes: lane lp of the TP is left with x[quarter(lp)].
__device__ __forceinline__ int quarter(int lp) { return 2 * (lp & 1) + ((lp >> 1) & 1); }
template <int TP>
__device__ __forceinline__ float sum_quarters(const float (&x)[4], int lp) {
  const bool o1 = (lp & 1) != 0, o2 = (lp & 2) != 0;
  const float a = (o1 ? x[2] : x[0]) + __shfl_xor_sync(0xffffffffu, o1 ? x[0] : x[2], 1);
  const float b = (o1 ? x[3] : x[1]) + __shfl_xor_sync(0xffffffffu, o1 ? x[1] : x[3], 1);
  float c = (o2 ? b : a) + __shfl_xor_sync(0xffffffffu, o2 ? a : b, 2);
#pragma unroll
  for (int d = 4; d < TP; d <<= 1) c += __shfl_xor_sync(0xffffffffu, c, d);
  return c;
}
template <class C, bool COL, bool REV, class Scalar, class Out>
__device__ __forceinline__ void walk(float (&m)[4][C::TE], const float* f, const float* w, const float* z, int nv, int own, int part,
                                     Scalar scalar, Out out) {
  constexpr int VW = C::TE < 4 ? C::TE : 4;
  float s[4], next[4];
  scalar(REV ? nv - 1 : 0, s);
#pragma unroll 1
  for (int i = 0; i < nv; ++i) {
    const int t = REV ? nv - 1 - i : i;
    if (i + 1 < nv) scalar(REV ? t - 1 : t + 1, next);
    float o[4] = {0.f, 0.f, 0.f, 0.f}, fr[4];
    if (!COL) ld_vec<4>(fr, f + t * C::D + own);
#pragma unroll
    for (int j = 0; j < C::TE / VW; ++j) {
      const int e = t * C::D + VW * (part + C::TP * j);
      float we[VW], ze[VW], fe[VW];
      ld_vec<VW>(we, w + e);
      ld_vec<VW>(ze, z + e);
      if (COL) ld_vec<VW>(fe, f + e);
#pragma unroll
      for (int u = 0; u < VW; ++u)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          float& x = m[r][VW * j + u];
          const float ft = COL ? fe[u] : fr[r];
          x = REV ? fmaf(we[u], s[r], x) : fmaf(ft, x, we[u] * s[r]);
          o[r] = fmaf(ze[u], x, o[r]);
          if (REV) x *= ft;
        }
    }
    const float c = sum_quarters<C::TP>(o, part);
    if (part < 4) out(t, own + quarter(part), c);
#pragma unroll
    for (int r = 0; r < 4; ++r) s[r] = next[r];
  }
}
template <class C, bool COL>
__device__ __forceinline__ void load_state(float (&m)[4][C::TE], const float* st, int own, int part) {
  constexpr int VW = C::TE < 4 ? C::TE : 4;
#pragma unroll
  for (int j = 0; j < C::TE / VW; ++j) {
    const int e = VW * (part + C::TP * j);
    float x[4];
    if (COL) {
#pragma unroll
      for (int u = 0; u < VW; ++u) {
        ld_vec<4>(x, st + (e + u) * C::D + own);
#pragma unroll
        for (int r = 0; r < 4; ++r) m[r][VW * j + u] = x[r];
      }
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float y[VW];
        ld_vec<VW>(y, st + (own + r) * C::D + e);
#pragma unroll
        for (int u = 0; u < VW; ++u) m[r][VW * j + u] = y[u];
      }
    }
  }
}
// a chunk of an array, or exp of it, as float32 [L][D]
template <class C, typename TI, bool EXP = false>
__device__ __forceinline__ void stage(float* dst, const void* src, const ChunkAt<C>& at) {
#pragma unroll 4
  for (int id = threadIdx.x; id < at.nv * C::CP; id += C::NT) {
    const int r = id / C::CP, c = id % C::CP;
    Pair<TI> x;
    x.load(src, at.row(r) + 2 * c);
    const float2 y = x.get();
    *reinterpret_cast<float2*>(dst + r * C::D + 2 * c) = EXP ? make_float2(expf(y.x), expf(y.y)) : y;
  }
}
template <class C, typename TI>
__device__ __noinline__ void fwd_by_token(float* f, const float* Sn, const PxParams& p) {
  const ChunkAt<C> at(p, blockIdx.x);
  float *k = f + C::L * C::D, *q = k + C::L * C::D;
  stage<C, float, true>(f, p.g, at);
  stage<C, TI>(k, p.k, at);
  stage<C, TI>(q, p.q, at);
  __syncthreads();
  const int own = threadIdx.x / C::TP * 4, part = threadIdx.x % C::TP;
  float m[4][C::TE];
  load_state<C, true>(m, Sn, own, part);
  walk<C, true, false>(m, f, k, q, at.nv, own, part, [&](int t, float (&s)[4]) {
    Pair<TI> a, b;
    a.load(p.v, at.row(t) + own);
    b.load(p.v, at.row(t) + own + 2);
    s[0] = a.get().x; s[1] = a.get().y; s[2] = b.get().x; s[3] = b.get().y;
  }, [&](int t, int c, float o) { st_any(p.out, p.out_bf, at.row(t) + c, o); });
}
// dq forwards and dk backwards by rows of the states, dv backwards by columns; dg collects q dq, then the sums
template <class C, typename TI, typename TY>
__device__ __noinline__ void bwd_by_token(float* f, const float* Sn, const float* dSn, const PxParams& p) {
  const ChunkAt<C> at(p, blockIdx.x);
  float *k = f + C::L * C::D, *q = k + C::L * C::D, *v = q + C::L * C::D, *dout = v + C::L * C::D;
  stage<C, float, true>(f, p.g, at);
  stage<C, TI>(k, p.k, at);
  stage<C, TI>(q, p.q, at);
  stage<C, TI>(v, p.v, at);
  stage<C, TY>(dout, p.dout, at);
  __syncthreads();
  const int own = threadIdx.x / C::TP * 4, part = threadIdx.x % C::TP;
  auto from = [&](const float* x) { return [=](int t, float (&s)[4]) { ld_vec<4>(s, x + t * C::D + own); }; };
  float m[4][C::TE];
  load_state<C, false>(m, Sn, own, part);
  walk<C, false, false>(m, f, v, dout, at.nv, own, part, from(k), [&](int t, int d, float o) {
    st_f((TI*)p.dq, at.row(t) + d, o);
    p.dg[at.row(t) + d] = q[t * C::D + d] * o;
  });
  float dots[4] = {0.f, 0.f, 0.f, 0.f};
  load_state<C, false>(m, dSn, own, part);
  constexpr int VW = C::TE < 4 ? C::TE : 4;
#pragma unroll
  for (int j = 0; j < C::TE / VW; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float y[VW];                              // of the state that leaves the chunk
      ld_vec<VW>(y, Sn + (C::D + own + r) * C::D + VW * (part + C::TP * j));
#pragma unroll
      for (int u = 0; u < VW; ++u) dots[r] = fmaf(y[u], m[r][VW * j + u], dots[r]);
    }
  float sum = sum_quarters<C::TP>(dots, part);
  walk<C, false, true>(m, f, dout, v, at.nv, own, part, from(q), [&](int t, int d, float o) {
    st_f((TI*)p.dk, at.row(t) + d, o);
    sum += p.dg[at.row(t) + d] - k[t * C::D + d] * o;
    p.dg[at.row(t) + d] = sum;
  });
  load_state<C, true>(m, dSn, own, part);
  walk<C, true, true>(m, f, q, k, at.nv, own, part, from(dout), [&](int t, int c, float o) { st_f((TI*)p.dv, at.row(t) + c, o); });
}

// MODE 0: S = f S + k v;  MODE 1, backwards: dS = f (dS + q dO); both from zero
template <class C, typename TI, typename TY, int MODE>
__device__ __noinline__ void product_by_token(float* f, float* st, const PxParams& p) {
  constexpr int VW = C::TE < 4 ? C::TE : 4;
  const ChunkAt<C> at(p, blockIdx.x);
  float* x = f + C::L * C::D;
  stage<C, float, true>(f, p.g, at);
  stage<C, TI>(x, MODE == 0 ? p.k : p.q, at);
  __syncthreads();
  const int own = threadIdx.x / C::TP * 4, part = threadIdx.x % C::TP;
  float m[4][C::TE] = {};
#pragma unroll 1
  for (int i = 0; i < at.nv; ++i) {
    const int t = MODE == 0 ? i : at.nv - 1 - i;
    Pair<TY> a, b;
    a.load(MODE == 0 ? p.v : p.dout, at.row(t) + own);
    b.load(MODE == 0 ? p.v : p.dout, at.row(t) + own + 2);
    const float s[4] = {a.get().x, a.get().y, b.get().x, b.get().y};
#pragma unroll
    for (int j = 0; j < C::TE / VW; ++j) {
      float fe[VW], xe[VW];
      ld_vec<VW>(fe, f + t * C::D + VW * (part + C::TP * j));
      ld_vec<VW>(xe, x + t * C::D + VW * (part + C::TP * j));
#pragma unroll
      for (int u = 0; u < VW; ++u)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          float& y = m[r][VW * j + u];
          y = MODE == 0 ? fmaf(fe[u], y, xe[u] * s[r]) : fe[u] * fmaf(xe[u], s[r], y);
        }
    }
  }
#pragma unroll
  for (int j = 0; j < C::TE / VW; ++j)
#pragma unroll
    for (int u = 0; u < VW; ++u)
      *reinterpret_cast<float4*>(st + (VW * (part + C::TP * j) + u) * C::D + own) =
          make_float4(m[0][VW * j + u], m[1][VW * j + u], m[2][VW * j + u], m[3][VW * j + u]);
}

// ---- per-chunk state products ----------------------------------------------------------------------------------------
// MODE 0: S slot n = k^^T V, k^ = k exp(G - lam);  MODE 1: dS slot n = q^^T dO, q^ = q exp(lam).  The weights are
// anchored at the chunk's ends here and never exceed one for log gates <= 0.  Also leaves exp(G).
template <class C, typename TI, typename TY, int MODE>
__global__ void __launch_bounds__(C::NT, sizeof(TI) + sizeof(TY) == 4 && C::L == 64 ? 1024 / C::NT : 512 / C::NT) px_product_kernel(const __grid_constant__ PxParams p) {
  constexpr int NSY = planes_of<TY>();
  extern __shared__ __align__(16) uint8_t sm[];
  uint8_t* sX = sm;
  uint8_t* sY = sm + 3 * C::PLANE;
  float* seg = reinterpret_cast<float*>(sY + NSY * C::PLANE);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cp = tid % C::CP, rg = tid / C::CP, r0 = rg * C::RPT;
  const ChunkAt<C> at(p, blockIdx.x);
  float2 g[C::RPT];
  Pair<TI> x[C::RPT];
  grid_dep_wait();
  grid_dep_launch();
  load_gates<C>(g, p.g, at, r0, cp);
  load_pairs<C, TI>(x, MODE == 0 ? p.k : p.q, at, r0, cp);
  copy_rows<C, TY>(sY, MODE == 0 ? p.v : p.dout, at);
  float2 s = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < C::RPT; ++i) { s.x += g[i].x; s.y += g[i].y; }
  *reinterpret_cast<float2*>(seg + rg * C::D + 2 * cp) = s;
  __syncthreads();
  float2 side = make_float2(0.f, 0.f), total = side;        // gates after (MODE 0) or before (MODE 1) the thread's rows
#pragma unroll
  for (int r = 0; r < C::RG; ++r) {
    const float2 t = *reinterpret_cast<const float2*>(seg + r * C::D + 2 * cp);
    if (MODE == 0 ? r > rg : r < rg) { side.x += t.x; side.y += t.y; }
    total.x += t.x; total.y += t.y;
  }
  float2 run = make_float2(expf(side.x), expf(side.y));
  if (rg == 0) *reinterpret_cast<float2*>(p.eG + (at.bh * p.N + at.n) * C::D + 2 * cp) = make_float2(expf(total.x), expf(total.y));
  if (MODE == 0) {
#pragma unroll
    for (int i = C::RPT - 1; i >= 0; --i) {
      const float2 v = x[i].get();
      st_split3(sX + (r0 + i) * C::LD + cp * 4, C::PLANE, v.x * run.x, v.y * run.y);
      run.x *= expf(g[i].x); run.y *= expf(g[i].y);
    }
  } else {
#pragma unroll
    for (int i = 0; i < C::RPT; ++i) {
      const float2 v = x[i].get();
      run.x *= expf(g[i].x); run.y *= expf(g[i].y);
      st_split3(sX + (r0 + i) * C::LD + cp * 4, C::PLANE, v.x * run.x, v.y * run.y);
    }
  }
  __syncthreads();
  constexpr int WM = C::D / 16, WN = (C::NT / 32) / WM, NW = C::D / WN;       // warps over key rows, value columns per warp
  static_assert(WM * WN == C::NT / 32, "warps must tile the state");
  const int m0 = 16 * (warp % WM), c0 = NW * (warp / WM);
  float acc[NW / 8][4];
#pragma unroll
  for (int j = 0; j < NW / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
  const uint32_t aX = smem_u32(sX), aY = smem_u32(sY);
#pragma unroll 2
  for (int ks = 0; ks < C::L / 16; ++ks) {
    uint32_t a[3][4];
    ld_a_t<3>(a, aX, C::PLANE, C::LD, m0, 16 * ks, lane);
    mma_step<3, NSY, NW / 16, true, (sizeof(TI) + sizeof(TY) > 4)>(acc, a, aY, C::PLANE, C::LD, c0, 16 * ks, lane);
  }
  float* o = (MODE == 0 ? p.S + (at.bh * p.NS + at.n) * C::D * C::D : p.dS + (at.bh * p.N + at.n) * C::D * C::D);
#pragma unroll
  for (int j = 0; j < NW / 8; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<float2*>(o + (m0 + (lane >> 2) + 8 * h) * C::D + c0 + 8 * j + 2 * (lane & 3)) =
          make_float2(acc[j][2 * h], acc[j][2 * h + 1]);
  if (__syncthreads_or(!(not_finite(acc, 0.f) == 0.f))) {
    static_assert(2 * C::L * C::D * 4 <= (3 + NSY) * C::PLANE, "the walk by token keeps exp(g) and k or q over the operands");
    product_by_token<C, TI, TY, MODE>(reinterpret_cast<float*>(sm), o, p);
  }
}

// ---- scan over the chunks, in place --------------------------------------------------------------------------------------
// s = init; over the chunks (mode 1: backwards): x = slot n, slot n = s, s = eG_n s + x; s goes to `fin` and to slot N if
// there is one.
// One thread per four value columns; eight chunks' loads in flight (the chain itself is one FMA per chunk).
template <typename TS>
__global__ void __launch_bounds__(128) px_scan_kernel(int64_t total, int64_t D, int64_t N, int64_t NS, const float* __restrict__ eG,
                                                      const TS* __restrict__ init, float* S, TS* __restrict__ fin, int mode) {
  constexpr int AHEAD = 8;
  const int64_t e4 = (int64_t)blockIdx.x * 128 + threadIdx.x, DD = D * D;
  if (e4 * 4 >= total) return;
  const int64_t bh = e4 * 4 / DD, e = e4 * 4 % DD, dk = e / D;
  float* sp = S + bh * NS * DD + e;
  const float* gp = eG + bh * N * D + dk;
  grid_dep_wait();
  grid_dep_launch();
  float4 s;
  s.x = ld_f(init, bh * DD + e); s.y = ld_f(init, bh * DD + e + 1); s.z = ld_f(init, bh * DD + e + 2); s.w = ld_f(init, bh * DD + e + 3);
  float4 x[AHEAD];
  float f[AHEAD];
  auto fetch = [&](int64_t i, int u) {
    const int64_t n = mode ? N - 1 - i : i;
    x[u] = *reinterpret_cast<const float4*>(sp + n * DD);
    f[u] = __ldg(gp + n * D);
  };
#pragma unroll
  for (int u = 0; u < AHEAD; ++u) if (u < N) fetch(u, u);
  for (int64_t i0 = 0; i0 < N; i0 += AHEAD) {
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int64_t i = i0 + u;
      if (i < N) {
        const int64_t n = mode ? N - 1 - i : i;
        *reinterpret_cast<float4*>(sp + n * DD) = s;
        s = make_float4(fmaf(f[u], s.x, x[u].x), fmaf(f[u], s.y, x[u].y), fmaf(f[u], s.z, x[u].z), fmaf(f[u], s.w, x[u].w));
        if (i + AHEAD < N) fetch(i + AHEAD, u);
      }
    }
  }
  if (NS > N) *reinterpret_cast<float4*>(sp + N * DD) = s;
  if (fin != nullptr) {
    st_f(fin, bh * DD + e, s.x); st_f(fin, bh * DD + e + 1, s.y); st_f(fin, bh * DD + e + 2, s.z); st_f(fin, bh * DD + e + 3, s.w);
  }
}

// ---- pieces of the chunk kernels -------------------------------------------------------------------------------------------
// q~ and k~ as split planes; em[d] = e^m, which the rows of S take, and ed[d] = exp(G - m), from the same products as the
// weights, which those of dS take.
template <class C, typename TI>
__device__ __forceinline__ void build_qk(uint8_t* sQ, uint8_t* sK, float* em, float* ed, const float2 (&f)[C::RPT], const Pair<TI> (&q)[C::RPT],
                                         const Pair<TI> (&k)[C::RPT], float2 half, float2 start, int rg, int cp) {
  const int r0 = rg * C::RPT;
  if (rg == 0) *reinterpret_cast<float2*>(em + 2 * cp) = make_float2(expf(half.x), expf(half.y));
  float2 run = start;
#pragma unroll
  for (int i = 0; i < C::RPT; ++i) {
    run.x *= f[i].x; run.y *= f[i].y;
    const float2 x = q[i].get();
    st_split3(sQ + (r0 + i) * C::LD + cp * 4, C::PLANE, x.x * run.x, x.y * run.y);
  }
  if (ed != nullptr && rg == C::RG - 1) *reinterpret_cast<float2*>(ed + 2 * cp) = run;
  run = make_float2(1.f / run.x, 1.f / run.y);
#pragma unroll
  for (int i = C::RPT - 1; i >= 0; --i) {
    const float2 x = k[i].get();
    st_split3(sK + (r0 + i) * C::LD + cp * 4, C::PLANE, x.x * run.x, x.y * run.y);
    run.x *= f[i].x; run.y *= f[i].y;
  }
}
// Value columns [PW pc, PW pc + PW) of a state (float32, D x D), rows scaled by em, as split planes.
template <class C>
__device__ __forceinline__ void fetch_piece(float4 (&x)[C::SREG], const float* st, int pc) {
#pragma unroll
  for (int j = 0; j < C::SREG; ++j) {
    const int id = threadIdx.x + C::NT * j, r = id / (C::PW / 4), c = id % (C::PW / 4);
    x[j] = *reinterpret_cast<const float4*>(st + r * C::D + pc * C::PW + c * 4);
  }
}
template <class C>
__device__ __forceinline__ void store_piece(uint8_t* dst, const float4 (&x)[C::SREG], const float* em) {
#pragma unroll
  for (int j = 0; j < C::SREG; ++j) {
    const int id = threadIdx.x + C::NT * j, r = id / (C::PW / 4), c = id % (C::PW / 4);
    const float w = em[r];
    st_split3(dst + r * C::LDS + c * 8, C::SPLANE, make_float4(x[j].x * w, x[j].y * w, x[j].z * w, x[j].w * w));
  }
}
// The warp's score blocks (row block wr, column blocks wc, wc + WC, ... up to the diagonal): A B^T over D.
template <class C, int NSA, int NSB, bool EX>
__device__ __forceinline__ void score_blocks(float (&x)[C::NB][2][4], uint32_t aA, uint32_t aB, int wr, int wc, int lane) {
#pragma unroll
  for (int i = 0; i < C::NB; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) x[i][j][e] = 0.f;
  if (wc <= wr) {
#pragma unroll 2
    for (int ks = 0; ks < C::D / 16; ++ks) {
      uint32_t a[NSA][4];
      ld_a<NSA>(a, aA, C::PLANE, C::LD, 16 * wr, 16 * ks, lane);
#pragma unroll
      for (int i = 0; i < C::NB; ++i)
        if (wc + C::WC * i <= wr) mma_step<NSA, NSB, 1, false, EX>(x[i], a, aB, C::PLANE, C::LD, 16 * (wc + C::WC * i), 16 * ks, lane);
    }
  }
}
// ... as split planes of the score tile [i][j], entries above the diagonal zero
template <class C>
__device__ __forceinline__ void store_scores(uint8_t* t, const float (&x)[C::NB][2][4], int wr, int wc, int lane) {
#pragma unroll
  for (int i = 0; i < C::NB; ++i) {
    const int cb = wc + C::WC * i;
    if (cb <= wr) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = 16 * wr + (lane >> 2) + 8 * h, c = 16 * cb + 8 * j + 2 * (lane & 3);
          st_split3(t + r * C::LDT + c * 2, C::TPLANE, c <= r ? x[i][j][2 * h] : 0.f, c + 1 <= r ? x[i][j][2 * h + 1] : 0.f);
        }
    }
  }
}
template <typename TI>
__device__ __forceinline__ void st_pair(void* p, int64_t e, float x, float y) {
  if constexpr (sizeof(TI) == 2) *reinterpret_cast<uint32_t*>((bf16*)p + e) = pack_bf16x2(x, y);
  else *reinterpret_cast<float2*>((float*)p + e) = make_float2(x, y);
}
template <int N>
__device__ __forceinline__ void zero_acc(float (&c)[N][4]) {
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[j][e] = 0.f;
}

// ---- forward chunk kernel ---------------------------------------------------------------------------------------------
template <class C, typename TI>
struct FwdLay {
  static constexpr int NSV = planes_of<TI>();
  static constexpr uint32_t most(uint32_t a, uint32_t b) { return a > b ? a : b; }
  // The region of k~ takes the scores once they are formed and, with one piece of the state (D <= 64), that piece once
  // the scores are consumed: three blocks per SM at head size 64 in bf16 instead of two (419 instead of 437 us for a
  // whole forward + backward of 202752 token-heads, with the overlapped launches).  Two pieces: the first has a region of its own, the second follows k~.
  static constexpr uint32_t KREG = most(C::NP > 1 ? 0 : 3 * C::TPLANE, most(3 * C::SPLANE, 3 * C::PLANE));
  static constexpr uint32_t Q = 0, K = Q + 3 * C::PLANE, V = K + KREG, S = C::NP > 1 ? V + NSV * C::PLANE : K;
  static constexpr uint32_t T = C::NP > 1 ? S + 3 * C::SPLANE : K, SEG = C::NP > 1 ? T + 3 * C::TPLANE : V + NSV * C::PLANE;
  static constexpr uint32_t EM = SEG + 3 * C::RG * C::D * 4, END = EM + C::D * 4;
  static constexpr int BLOCKS = C::NP > 1 ? 1 : sizeof(TI) == 2 ? 3 : 2;
  static_assert(3 * C::L * C::D * 4 <= V, "the walk by token keeps exp(g), k and q over q~ and k~");
};
template <class C, typename TI, bool EX>
__global__ void __launch_bounds__(C::NT, FwdLay<C, TI>::BLOCKS) px_fwd_kernel(const __grid_constant__ PxParams p) {
  using Lay = FwdLay<C, TI>;
  extern __shared__ __align__(16) uint8_t sm[];
  float* seg = reinterpret_cast<float*>(sm + Lay::SEG);
  float* em = reinterpret_cast<float*>(sm + Lay::EM);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cp = tid % C::CP, rg = tid / C::CP, r0 = rg * C::RPT;
  const ChunkAt<C> at(p, blockIdx.x);
  const float* Sn = p.S + (at.bh * p.NS + at.n) * C::D * C::D;
  float4 sx[C::SREG];
  {
    float2 g[C::RPT];
    Pair<TI> q[C::RPT], k[C::RPT];
    // the inputs were complete before the state product, which waited for everything before it, could start
    load_gates<C>(g, p.g, at, r0, cp);
    load_pairs<C, TI>(q, p.q, at, r0, cp);
    load_pairs<C, TI>(k, p.k, at, r0, cp);
    copy_rows<C, TI>(sm + Lay::V, p.v, at);
    float2 half, start;
    if (gate_weights<C>(g, seg, rg, cp, half, start)) {
      grid_dep_wait();
      grid_dep_launch();
      fwd_by_token<C, TI>(reinterpret_cast<float*>(sm), Sn, p);
      return;
    }
    build_qk<C, TI>(sm + Lay::Q, sm + Lay::K, em, nullptr, g, q, k, half, start, rg, cp);
    __syncthreads();
  }
  const int wr = warp % C::WR, wc = warp / C::WR, m0 = 16 * wr;
  const uint32_t aQ = smem_u32(sm + Lay::Q), aK = smem_u32(sm + Lay::K), aV = smem_u32(sm + Lay::V), aS = smem_u32(sm + Lay::S);
  const uint32_t aT = smem_u32(sm + Lay::T);
  float o[C::NP][C::PC / 8][4];
#pragma unroll
  for (int pc = 0; pc < C::NP; ++pc) zero_acc(o[pc]);
  {
    float x[C::NB][2][4];
    score_blocks<C, 3, 3, EX>(x, aQ, aK, wr, wc, lane);
    __syncthreads();                      // the scores are formed: the region of k~ is free
    store_scores<C>(sm + Lay::T, x, wr, wc, lane);
  }
  grid_dep_wait();                        // the states of the scan before this kernel
  grid_dep_launch();
  fetch_piece<C>(sx, Sn, 0);
  if (C::NP > 1) {
    float4 s1[C::SREG];
    fetch_piece<C>(s1, Sn, 1);
    store_piece<C>(sm + Lay::S, sx, em);
    store_piece<C>(sm + Lay::K, s1, em);
  }
  __syncthreads();
#pragma unroll 1
  for (int kk = 0; kk <= wr; ++kk) {
    uint32_t a[3][4];
    ld_a<3>(a, aT, C::TPLANE, C::LDT, m0, 16 * kk, lane);
#pragma unroll
    for (int pc = 0; pc < C::NP; ++pc)
      mma_step<3, Lay::NSV, C::PC / 16, true, EX>(o[pc], a, aV, C::PLANE, C::LD, pc * C::PW + wc * C::PC, 16 * kk, lane);
  }
  if (C::NP == 1) {
    __syncthreads();                      // the scores are consumed
    store_piece<C>(sm + Lay::S, sx, em);
    __syncthreads();
  }
#pragma unroll 2
  for (int ks = 0; ks < C::D / 16; ++ks) {
    uint32_t a[3][4];
    ld_a<3>(a, aQ, C::PLANE, C::LD, m0, 16 * ks, lane);
#pragma unroll
    for (int pc = 0; pc < C::NP; ++pc)
      mma_step<3, 3, C::PC / 16, true, EX>(o[pc], a, pc == 0 ? aS : aK, C::SPLANE, C::LDS, wc * C::PC, 16 * ks, lane);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = m0 + (lane >> 2) + 8 * h;
    if (r < at.nv) {
      const int64_t e = at.row(r) + wc * C::PC + 2 * (lane & 3);
#pragma unroll
      for (int pc = 0; pc < C::NP; ++pc)
#pragma unroll
        for (int j = 0; j < C::PC / 8; ++j) {
          const int64_t c = e + pc * C::PW + 8 * j;
          if (p.out_bf) st_pair<bf16>(p.out, c, o[pc][j][2 * h], o[pc][j][2 * h + 1]);
          else st_pair<float>(p.out, c, o[pc][j][2 * h], o[pc][j][2 * h + 1]);
        }
    }
  }
  float z = 0.f;
#pragma unroll
  for (int pc = 0; pc < C::NP; ++pc) z = not_finite(o[pc], z);
  if (__syncthreads_or(!(z == 0.f))) fwd_by_token<C, TI>(reinterpret_cast<float*>(sm), Sn, p);      // writes all of it again
}

// ---- backward chunk kernel --------------------------------------------------------------------------------------------
// A warp's 16 rows serve twice: as rows i for dq = dP k~ + dO S^T, and as rows j for dk = dP^T q~ + V dS^T and
// dV = P^T dO + k~ dS.  dP and then P pass through one score tile (read transposed for the second role), which shares
// its place with the states' pieces of 64 value columns.
template <class C, typename TI, typename TY>
struct BwdLay {
  static constexpr int NSV = planes_of<TI>(), NSD = planes_of<TY>();
  static constexpr uint32_t most(uint32_t a, uint32_t b) { return a > b ? a : b; }
  static constexpr uint32_t SREGION = most(3 * C::SPLANE, 3 * C::TPLANE);      // score tile, state pieces
  static constexpr uint32_t Q = 0, K = Q + 3 * C::PLANE, V = K + 3 * C::PLANE, DO = V + NSV * C::PLANE, S = DO + NSD * C::PLANE;
  static constexpr uint32_t SEG = S + SREGION, EM = SEG + 3 * C::RG * C::D * 4, ED = EM + C::D * 4, DG = ED + C::D * 4, END = DG + C::D * 4;
  static constexpr int BLOCKS = 232448 / (END + 1024);      // per SM, what shared memory holds (registers must not hold fewer)
  static_assert(C::L * C::AP * 4 <= 3 * C::PLANE, "dq and dk are staged in float32 over q~ and k~");
  static_assert(5 * C::L * C::D * 4 <= SEG, "the walk by token keeps exp(g), k, q, v and dO over the operands");
};
// dG[d] += <S_{n+1}[d, piece], dS_n[d, piece]>: PW / 4 consecutive threads hold a row of the piece
template <class C>
__device__ __forceinline__ void dot_piece(float* dG, const float4 (&x)[C::SREG], const float* Snext, int pc) {
  float4 y[C::SREG];
  fetch_piece<C>(y, Snext, pc);
#pragma unroll
  for (int j = 0; j < C::SREG; ++j) {
    float s = x[j].x * y[j].x + x[j].y * y[j].y + x[j].z * y[j].z + x[j].w * y[j].w;
#pragma unroll
    for (int o = C::PW / 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const int id = threadIdx.x + C::NT * j, r = id / (C::PW / 4);
    if (id % (C::PW / 4) == 0) dG[r] = pc == 0 ? s : dG[r] + s;
  }
}
template <class C, typename TI, typename TY>
__global__ void __launch_bounds__(C::NT, BwdLay<C, TI, TY>::BLOCKS) px_bwd_kernel(const __grid_constant__ PxParams p) {
  using Lay = BwdLay<C, TI, TY>;
  constexpr int NSV = Lay::NSV, NSD = Lay::NSD, L = C::L, D = C::D;
  constexpr bool EX = sizeof(TI) == 4;    // dv; dq and dk make dg, which is float32 always
  extern __shared__ __align__(16) uint8_t sm[];
  float* seg = reinterpret_cast<float*>(sm + Lay::SEG);
  float* em = reinterpret_cast<float*>(sm + Lay::EM);
  float* ed = reinterpret_cast<float*>(sm + Lay::ED);
  float* dG = reinterpret_cast<float*>(sm + Lay::DG);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cp = tid % C::CP, rg = tid / C::CP, r0 = rg * C::RPT;
  const ChunkAt<C> at(p, blockIdx.x);
  const float* Sn = p.S + (at.bh * p.NS + at.n) * D * D;
  const float* dSn = p.dS + (at.bh * p.N + at.n) * D * D;
  float4 sx[C::SREG];
  float2 start;
  {
    float2 g[C::RPT];
    Pair<TI> q[C::RPT], k[C::RPT];
    load_gates<C>(g, p.g, at, r0, cp);
    load_pairs<C, TI>(q, p.q, at, r0, cp);
    load_pairs<C, TI>(k, p.k, at, r0, cp);
    copy_rows<C, TI>(sm + Lay::V, p.v, at);
    copy_rows<C, TY>(sm + Lay::DO, p.dout, at);
    float2 half;
    if (gate_weights<C>(g, seg, rg, cp, half, start)) {
      grid_dep_wait();
      grid_dep_launch();
      bwd_by_token<C, TI, TY>(reinterpret_cast<float*>(sm), Sn, dSn, p);
      return;
    }
    build_qk<C, TI>(sm + Lay::Q, sm + Lay::K, em, ed, g, q, k, half, start, rg, cp);
  }
  grid_dep_wait();                        // the gradient states of the scan before this kernel
  grid_dep_launch();
  fetch_piece<C>(sx, Sn, 0);
  __syncthreads();

  const int wr = warp % C::WR, wc = warp / C::WR, m0 = 16 * wr;
  const uint32_t aQ = smem_u32(sm + Lay::Q), aK = smem_u32(sm + Lay::K), aV = smem_u32(sm + Lay::V);
  const uint32_t aD = smem_u32(sm + Lay::DO), aS = smem_u32(sm + Lay::S);
  const float* Snext = Sn + D * D;
  float dq[C::CW / 8][4], dk[C::CW / 8][4], dv[C::NP][C::PC / 8][4];
  zero_acc(dq);
  zero_acc(dk);
#pragma unroll
  for (int pc = 0; pc < C::NP; ++pc) zero_acc(dv[pc]);
  float x[C::NB][2][4];
  score_blocks<C, NSD, NSV, true>(x, aD, aV, wr, wc, lane);               // dP = tril(dO V^T)
  store_scores<C>(sm + Lay::S, x, wr, wc, lane);
  __syncthreads();
#pragma unroll 1
  for (int kk = 0; kk <= wr; ++kk) {                                // dq += dP k~
    uint32_t a[3][4];
    ld_a<3>(a, aS, C::TPLANE, C::LDT, m0, 16 * kk, lane);
    mma_step<3, 3, C::CW / 16, true, true>(dq, a, aK, C::PLANE, C::LD, wc * C::CW, 16 * kk, lane);
  }
#pragma unroll 1
  for (int kk = wr; kk < L / 16; ++kk) {                            // dk += dP^T q~
    uint32_t a[3][4];
    ld_a_t<3>(a, aS, C::TPLANE, C::LDT, m0, 16 * kk, lane);
    mma_step<3, 3, C::CW / 16, true, true>(dk, a, aQ, C::PLANE, C::LD, wc * C::CW, 16 * kk, lane);
  }
  score_blocks<C, 3, 3, EX>(x, aQ, aK, wr, wc, lane);                   // P = tril(q~ k~^T)
  __syncthreads();
  store_scores<C>(sm + Lay::S, x, wr, wc, lane);
  __syncthreads();
#pragma unroll 1
  for (int kk = wr; kk < L / 16; ++kk) {                              // dV = P^T dO
    uint32_t a[3][4];
    ld_a_t<3>(a, aS, C::TPLANE, C::LDT, m0, 16 * kk, lane);
#pragma unroll
    for (int pc = 0; pc < C::NP; ++pc)
      mma_step<3, NSD, C::PC / 16, true, EX>(dv[pc], a, aD, C::PLANE, C::LD, pc * C::PW + wc * C::PC, 16 * kk, lane);
  }
#pragma unroll
  for (int i = 0; i < 2 * C::NP; ++i) {       // the pieces of S_n (dq += dO S^T), then those of dS_n (dk += V dS^T, dV += k~ dS)
    const int pc = i % C::NP;
    __syncthreads();                          // what the buffer held is consumed
    if (i >= C::NP) dot_piece<C>(dG, sx, Snext, pc);
    store_piece<C>(sm + Lay::S, sx, i < C::NP ? em : ed);
    if (i + 1 < 2 * C::NP) fetch_piece<C>(sx, i + 1 < C::NP ? Sn : dSn, (i + 1) % C::NP);
    __syncthreads();
    if (i < C::NP) {
#pragma unroll 1
      for (int ks = 0; ks < C::PW / 16; ++ks) {
        uint32_t a[NSD][4];
        ld_a<NSD>(a, aD, C::PLANE, C::LD, m0, pc * C::PW + 16 * ks, lane);
        mma_step<NSD, 3, C::CW / 16, false, true>(dq, a, aS, C::SPLANE, C::LDS, wc * C::CW, 16 * ks, lane);
      }
    } else {
#pragma unroll 1
      for (int ks = 0; ks < C::PW / 16; ++ks) {
        uint32_t a[NSV][4];
        ld_a<NSV>(a, aV, C::PLANE, C::LD, m0, pc * C::PW + 16 * ks, lane);
        mma_step<NSV, 3, C::CW / 16, false, true>(dk, a, aS, C::SPLANE, C::LDS, wc * C::CW, 16 * ks, lane);
      }
#pragma unroll 1
      for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t a[3][4];
        ld_a<3>(a, aK, C::PLANE, C::LD, m0, 16 * ks, lane);
        mma_step<3, 3, C::PC / 16, true, EX>(dv[pc], a, aS, C::SPLANE, C::LDS, wc * C::PC, 16 * ks, lane);
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = m0 + (lane >> 2) + 8 * h;
    if (r < at.nv) {
      const int64_t e = at.row(r) + wc * C::PC + 2 * (lane & 3);
#pragma unroll
      for (int pc = 0; pc < C::NP; ++pc)
#pragma unroll
        for (int j = 0; j < C::PC / 8; ++j) st_pair<TI>(p.dv, e + pc * C::PW + 8 * j, dv[pc][j][2 * h], dv[pc][j][2 * h + 1]);
    }
  }
  float z = not_finite(dk, not_finite(dq, 0.f));
#pragma unroll
  for (int pc = 0; pc < C::NP; ++pc) z = not_finite(dv[pc], z);
  if (__syncthreads_or(!(z == 0.f))) {                    // (every operand is dead)
    bwd_by_token<C, TI, TY>(reinterpret_cast<float*>(sm), Sn, dSn, p);
    return;
  }
  float* tq = reinterpret_cast<float*>(sm + Lay::Q);
  float* tk = reinterpret_cast<float*>(sm + Lay::K);
#pragma unroll
  for (int j = 0; j < C::CW / 8; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = (m0 + (lane >> 2) + 8 * h) * C::AP + wc * C::CW + 8 * j + 2 * (lane & 3);
      *reinterpret_cast<float2*>(tq + e) = make_float2(dq[j][2 * h], dq[j][2 * h + 1]);
      *reinterpret_cast<float2*>(tk + e) = make_float2(dk[j][2 * h], dk[j][2 * h + 1]);
    }
  __syncthreads();

  // ---- closing pass: a thread finishes RPT rows of two features ------------------------------------------------------
  float2 g[C::RPT];
  Pair<TI> q[C::RPT], k[C::RPT];
  load_gates<C>(g, p.g, at, r0, cp);
  load_pairs<C, TI>(q, p.q, at, r0, cp);
  load_pairs<C, TI>(k, p.k, at, r0, cp);
  float2 run = start;
  float2 dl[C::RPT];
#pragma unroll
  for (int i = 0; i < C::RPT; ++i) {
    const int r = r0 + i;
    g[i] = make_float2(expf(g[i].x), expf(g[i].y));
    run.x *= g[i].x; run.y *= g[i].y;
    float2 y = *reinterpret_cast<const float2*>(tq + r * C::AP + 2 * cp);
    y.x *= run.x; y.y *= run.y;
    const float2 qf = q[i].get();
    dl[i] = make_float2(qf.x * y.x, qf.y * y.y);
    if (r < at.nv) st_pair<TI>(p.dq, at.row(r) + 2 * cp, y.x, y.y);
  }
  run = make_float2(1.f / run.x, 1.f / run.y);
#pragma unroll
  for (int i = C::RPT - 1; i >= 0; --i) {
    const int r = r0 + i;
    float2 y = *reinterpret_cast<const float2*>(tk + r * C::AP + 2 * cp);
    y.x *= run.x; y.y *= run.y;
    run.x *= g[i].x; run.y *= g[i].y;
    const float2 kf = k[i].get();
    dl[i].x -= kf.x * y.x; dl[i].y -= kf.y * y.y;
    if (r < at.nv) st_pair<TI>(p.dk, at.row(r) + 2 * cp, y.x, y.y);
  }
#pragma unroll
  for (int i = C::RPT - 2; i >= 0; --i) { dl[i].x += dl[i + 1].x; dl[i].y += dl[i + 1].y; }
  *reinterpret_cast<float2*>(seg + rg * D + 2 * cp) = dl[0];
  __syncthreads();
  float2 off = *reinterpret_cast<const float2*>(dG + 2 * cp);
#pragma unroll
  for (int r = C::RG - 1; r > 0; --r)
    if (r > rg) {
      const float2 t = *reinterpret_cast<const float2*>(seg + r * D + 2 * cp);
      off.x += t.x; off.y += t.y;
    }
#pragma unroll
  for (int i = 0; i < C::RPT; ++i)
    if (r0 + i < at.nv) *reinterpret_cast<float2*>(p.dg + at.row(r0 + i) + 2 * cp) = make_float2(dl[i].x + off.x, dl[i].y + off.y);
}

// ---- host side ----------------------------------------------------------------------------------------------------------
template <class C, typename TI, typename TY, int MODE>
int launch_product(cudaStream_t st, const PxParams& p, int64_t chunks) {
  constexpr size_t smem = (3 + planes_of<TY>()) * C::PLANE + C::RG * C::D * 4;
  static SmemAttrOnce attr;
  GLA_TRY(attr.ensure(px_product_kernel<C, TI, TY, MODE>, smem));
  ProfScope ps(MODE == 0 ? "px_state_product" : "px_dstate_product", st);
  GLA_LAUNCHED(launch_overlapped(px_product_kernel<C, TI, TY, MODE>, dim3((unsigned)chunks), dim3(C::NT), smem, st, p));
  return GLA_OK;
}
template <typename TS>
int launch_scan(cudaStream_t st, int64_t BH, int64_t D, int64_t N, int64_t NS, const float* eG, const void* init, float* S, void* fin, int mode) {
  const int64_t total = BH * D * D;
  ProfScope ps("px_scan_kernel", st);
  GLA_LAUNCHED(launch_overlapped(px_scan_kernel<TS>, dim3((unsigned)((total / 4 + 127) / 128)), dim3(128), 0, st, total, D, N, NS, eG,
                                 (const TS*)init, S, (TS*)fin, mode));
  return GLA_OK;
}
template <class C, typename TI, bool EX>
int launch_fwd(cudaStream_t st, const PxParams& p, int64_t chunks) {
  static SmemAttrOnce attr;
  GLA_TRY(attr.ensure(px_fwd_kernel<C, TI, EX>, FwdLay<C, TI>::END));
  ProfScope ps("px_fwd_kernel", st);
  GLA_LAUNCHED(launch_overlapped(px_fwd_kernel<C, TI, EX>, dim3((unsigned)chunks), dim3(C::NT), FwdLay<C, TI>::END, st, p));
  return GLA_OK;
}
template <class C, typename TI>
int run_fwd(cudaStream_t st, const PxParams& p, const void* init, void* fin) {
  const int64_t BH = p.B * p.H, chunks = BH * p.N;
  GLA_TRY((launch_product<C, TI, TI, 0>(st, p, chunks)));
  GLA_TRY(launch_scan<TI>(st, BH, C::D, p.N, p.NS, p.eG, init, p.S, fin, 0));
  if constexpr (sizeof(TI) == 2)
    if (p.out_bf) return launch_fwd<C, TI, false>(st, p, chunks);
  return launch_fwd<C, TI, true>(st, p, chunks);
}
// states != 0: the states are in p.S and p.eG already (a forward's residuals); otherwise they are formed here first
template <class C, typename TI, typename TY>
int run_bwd(cudaStream_t st, const PxParams& p, int states, const void* init, const void* dfin, void* dinit) {
  const int64_t BH = p.B * p.H, chunks = BH * p.N;
  if (!states) {
    GLA_TRY((launch_product<C, TI, TI, 0>(st, p, chunks)));
    GLA_TRY(launch_scan<TI>(st, BH, C::D, p.N, p.NS, p.eG, init, p.S, nullptr, 0));
  }
  GLA_TRY((launch_product<C, TI, TY, 1>(st, p, chunks)));
  GLA_TRY(launch_scan<TI>(st, BH, C::D, p.N, p.N, p.eG, dfin, p.dS, dinit, 1));
  static SmemAttrOnce attr;
  GLA_TRY(attr.ensure(px_bwd_kernel<C, TI, TY>, BwdLay<C, TI, TY>::END));
  ProfScope ps("px_bwd_kernel", st);
  GLA_LAUNCHED(launch_overlapped(px_bwd_kernel<C, TI, TY>, dim3((unsigned)chunks), dim3(C::NT), BwdLay<C, TI, TY>::END, st, p));
  return GLA_OK;
}
template <int D, int L>
int dispatch_fwd(cudaStream_t st, const PxParams& p, const void* init, void* fin) {
  return p.in_bf ? run_fwd<Px<D, L>, bf16>(st, p, init, fin) : run_fwd<Px<D, (D >= 128 ? 32 : L)>, float>(st, p, init, fin);
}
size_t f32b(int64_t n) { return align_up((size_t)n * 4, 256); }

}  // namespace

// Rows of a chunk: 64, or 32 where three planes of every operand at head size 128 leave no room for more.
static int64_t px_rows(int64_t D, int narrow) { return D >= 128 && narrow ? 32 : 64; }
bool px_supported(int64_t D) { return D == 32 || D == 64 || D == 128; }
// states: (B H, N, D, D) float32, N + 1 of them with the final one | exp(G): (B H, N, D) float32.  bf: every array in bf16
size_t px_state_bytes(int64_t B, int64_t T, int64_t H, int64_t D, int bf, int final_state) {
  const int64_t n = (T + px_rows(D, !bf) - 1) / px_rows(D, !bf);
  return f32b(B * H * (n + (final_state ? 1 : 0)) * D * D) + f32b(B * H * n * D);
}
int px_fwd(cudaStream_t st, int64_t B, int64_t T, int64_t H, int64_t D, int bf, const void* hidden_init, const float* g,
           const void* v, const void* k, const void* q, void* hidden_final, void* out, int out_bf, void* states, int final_state, int reverse) {
  const int64_t N = (T + px_rows(D, !bf) - 1) / px_rows(D, !bf);
  if (B * H * N > 2147483647LL || B * H * D * D / 512 > 2147483647LL) return GLA_ERR_TOO_LARGE;
  PxParams p{};
  p.B = B; p.T = T; p.H = H; p.N = N; p.NS = N + (final_state ? 1 : 0); p.trev = reverse; p.in_bf = bf; p.out_bf = out_bf;
  p.g = g; p.v = v; p.k = k; p.q = q; p.out = out;
  p.S = (float*)states;
  p.eG = (float*)((char*)states + f32b(B * H * p.NS * D * D));
  switch (D) {
    case 32: return dispatch_fwd<32, 64>(st, p, hidden_init, hidden_final);
    case 64: return dispatch_fwd<64, 64>(st, p, hidden_init, hidden_final);
    case 128: return dispatch_fwd<128, 64>(st, p, hidden_init, hidden_final);
    default: return GLA_ERR_UNSUPPORTED;
  }
}
template <int D>
static int dispatch_bwd(cudaStream_t st, const PxParams& p, int do_bf, int states, const void* init, const void* dfin, void* dinit) {
  constexpr int LN = D >= 128 ? 32 : 64;
  if (p.in_bf && do_bf) return run_bwd<Px<D, 64>, bf16, bf16>(st, p, states, init, dfin, dinit);
  if (p.in_bf) return run_bwd<Px<D, LN>, bf16, float>(st, p, states, init, dfin, dinit);
  return do_bf ? run_bwd<Px<D, LN>, float, bf16>(st, p, states, init, dfin, dinit)
               : run_bwd<Px<D, LN>, float, float>(st, p, states, init, dfin, dinit);
}
// states: a forward's (px_fwd) with the final one when have_states, else scratch for as much; ws: scratch for the gradient
// states, px_state_bytes without a final one
int px_bwd(cudaStream_t st, int64_t B, int64_t T, int64_t H, int64_t D, int bf, const void* hidden_init, const float* g,
           const void* v, const void* k, const void* q, const void* dhidden_final, const void* dout, int do_bf,
           void* dhidden_init, float* dg, void* dv, void* dk, void* dq, void* states, int have_states, void* ws, int reverse) {
  const int64_t L = px_rows(D, !(bf && do_bf)), N = (T + L - 1) / L;
  if (have_states && L != px_rows(D, !bf)) return GLA_ERR_UNSUPPORTED;
  if (B * H * N > 2147483647LL || B * H * D * D / 512 > 2147483647LL) return GLA_ERR_TOO_LARGE;
  PxParams p{};
  p.B = B; p.T = T; p.H = H; p.N = N; p.NS = N + 1; p.trev = reverse; p.in_bf = bf;
  p.g = g; p.v = v; p.k = k; p.q = q; p.dout = dout;
  p.dq = dq; p.dk = dk; p.dv = dv; p.dg = dg;
  p.S = (float*)states;
  p.eG = (float*)((char*)states + f32b(B * H * p.NS * D * D));
  p.dS = (float*)ws;
  if (have_states == 0) {
    switch (D) {
      case 32: return dispatch_bwd<32>(st, p, do_bf, 0, hidden_init, dhidden_final, dhidden_init);
      case 64: return dispatch_bwd<64>(st, p, do_bf, 0, hidden_init, dhidden_final, dhidden_init);
      case 128: return dispatch_bwd<128>(st, p, do_bf, 0, hidden_init, dhidden_final, dhidden_init);
      default: return GLA_ERR_UNSUPPORTED;
    }
  }
  switch (D) {
    case 32: return dispatch_bwd<32>(st, p, do_bf, 1, hidden_init, dhidden_final, dhidden_init);
    case 64: return dispatch_bwd<64>(st, p, do_bf, 1, hidden_init, dhidden_final, dhidden_init);
    case 128: return dispatch_bwd<128>(st, p, do_bf, 1, hidden_init, dhidden_final, dhidden_init);
    default: return GLA_ERR_UNSUPPORTED;
  }
}

}  // namespace gla
