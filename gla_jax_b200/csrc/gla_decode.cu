// Single-token step of gated linear attention with a persistent state (serving / decode path).
//
// One step of the reference's definitional recurrence (gla.py:26-47) for a batch of requests:
//     S <- exp(g) (.) S + k (x) v         (the decay multiplies along the key axis)
//     o  = q S
// with the state (B, H, D, D) kept in float32 in device memory between calls and updated in place;
// hidden_init -> hidden_final chaining of recurrent_gla is exact (gla.py:720-723), so T calls of this
// step equal one recurrent_gla call over T tokens.  The reference has no such entry point: its callers
// would run recurrent_gla with T = 1.
//
// The step is pure HBM streaming: 2 * 4 * D * D bytes of state per (request, head) against 5 D bytes of
// everything else.  A block owns 32 value columns of one head's state: 8 lanes of four columns x 16 row lanes, every
// 16-byte load of its rows issued before one is used (16 KB per block at D = 128, sixteen blocks per SM), partial sums
// of o combined through shared memory.  Steps of one model follow each other back to back, so the launch overlaps the
// kernel before it.  Measured, 32 requests x 16 heads, D = 128: 14.3 us (scalar loads, plain launch) -> 12.0 us (the bytes at the copy
// rate: 10.4).
#include "gla_common.cuh"

namespace gla {

constexpr int DC = 32;       // value columns per block
constexpr int DL = DC / 4;   // column lanes
constexpr int DR = 16;       // row lanes

// a state whose base is not 16-byte aligned (a view) takes four scalar accesses instead
template <bool AL> __device__ __forceinline__ float4 ld_state(const float* p) {
  if constexpr (AL) return *reinterpret_cast<const float4*>(p);
  else return make_float4(p[0], p[1], p[2], p[3]);
}
template <bool AL> __device__ __forceinline__ void st_state(float* p, float4 x) {
  if constexpr (AL) *reinterpret_cast<float4*>(p) = x;
  else { p[0] = x.x; p[1] = x.y; p[2] = x.z; p[3] = x.w; }
}
template <int D, bool AL>
__global__ void __launch_bounds__(DL * DR) decode_step_kernel(float* __restrict__ S, const float* __restrict__ g,
                                                              const void* __restrict__ v, const void* __restrict__ k,
                                                              const void* __restrict__ q, void* __restrict__ out,
                                                              int bf, int out_bf) {
  constexpr int RPT = D / DR;                   // key rows per thread
  __shared__ float red[DR][DC];
  __shared__ float fk[3][D];                    // exp(g), k, q of this (request, head)
  const int cl = threadIdx.x % DL, rl = threadIdx.x / DL;
  const int64_t bh = blockIdx.y;
  const int c0 = blockIdx.x * DC + 4 * cl;
  float* Sp = S + (bh * D + rl) * (int64_t)D + c0;     // rows rl, rl + 16, ...
  grid_dep_wait();
  grid_dep_launch();
  float4 s[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) s[i] = ld_state<AL>(Sp + (int64_t)i * DR * D);
  for (int i = threadIdx.x; i < D; i += DL * DR) {
    fk[0][i] = expf(g[bh * D + i]);
    fk[1][i] = ld_any(k, bf, bh * D + i);
    fk[2][i] = ld_any(q, bf, bh * D + i);
  }
  float4 vv;
  vv.x = ld_any(v, bf, bh * D + c0); vv.y = ld_any(v, bf, bh * D + c0 + 1);
  vv.z = ld_any(v, bf, bh * D + c0 + 2); vv.w = ld_any(v, bf, bh * D + c0 + 3);
  __syncthreads();
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = rl + i * DR;
    const float f = fk[0][r], kr = fk[1][r], qr = fk[2][r];
    float4 n;
    n.x = fmaf(f, s[i].x, kr * vv.x); n.y = fmaf(f, s[i].y, kr * vv.y);
    n.z = fmaf(f, s[i].z, kr * vv.z); n.w = fmaf(f, s[i].w, kr * vv.w);
    st_state<AL>(Sp + (int64_t)i * DR * D, n);
    acc.x = fmaf(qr, n.x, acc.x); acc.y = fmaf(qr, n.y, acc.y); acc.z = fmaf(qr, n.z, acc.z); acc.w = fmaf(qr, n.w, acc.w);
  }
  *reinterpret_cast<float4*>(&red[rl][4 * cl]) = acc;
  __syncthreads();
  if (threadIdx.x < DC) {
    float o = 0.f;
#pragma unroll
    for (int j = 0; j < DR; ++j) o += red[j][threadIdx.x];
    st_any(out, out_bf, bh * D + blockIdx.x * DC + threadIdx.x, o);
  }
}

template <int D>
static int launch_decode(cudaStream_t st, int64_t BH, float* S, const float* g, const void* v, const void* k,
                         const void* q, void* out, int bf, int out_bf) {
  if (BH > 65535) return GLA_ERR_TOO_LARGE;
  ProfScope ps("decode_step_kernel", st);
  GLA_LAUNCHED(launch_overlapped(aligned16(S) ? decode_step_kernel<D, true> : decode_step_kernel<D, false>, dim3(D / DC, (unsigned)BH), dim3(DL * DR), 0, st, S, g, v, k, q, out, bf, out_bf));
  return GLA_OK;
}

int decode_step(cudaStream_t st, int64_t B, int64_t H, int64_t D, int bf, float* state, const float* g, const void* v,
                const void* k, const void* q, void* out, int out_bf) {
  const int64_t BH = B * H;
  switch (D) {
    case 32: return launch_decode<32>(st, BH, state, g, v, k, q, out, bf, out_bf);
    case 64: return launch_decode<64>(st, BH, state, g, v, k, q, out, bf, out_bf);
    case 128: return launch_decode<128>(st, BH, state, g, v, k, q, out, bf, out_bf);
    case 256: return launch_decode<256>(st, BH, state, g, v, k, q, out, bf, out_bf);
    default: return GLA_ERR_UNSUPPORTED;
  }
}

}  // namespace gla
