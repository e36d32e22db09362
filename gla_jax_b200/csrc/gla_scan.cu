// Memory-bound scan kernels: cumsum along time, the log-space linear-RNN scan, the D x D
// state scan over chunks and the cross-rank state combine.  All math in float32.
//
// Reference operators restated here: ops.py:152-284 (cumsum), ops.py:286-456 (linear-RNN
// scan).  The reference lowers these to a generic Triton `tt.scan` (ops.py:18-104) and
// needs a host-side hierarchy for long axes; here a thread block walks the time axis in
// tiles, scanning within a tile in registers and carrying the running total, so any length
// is one launch with fully coalesced 128-byte row segments.
#include "gla_common.cuh"
#include "tc_ptx.cuh"
#include "tma_maps.cuh"
#include <cmath>

namespace gla {

// ---------------------------------------------------------------------------------------
// cumsum: src (N, T, D) -> dst (N, T, D), inclusive along T, + init (N, D).
// ---------------------------------------------------------------------------------------

// The combine rules of the scan library (gla_scan_op): each is associative with an identity element, which is what
// the tiled scan needs (padding, carries, segment totals).  ops.py:82-104 scans with an arbitrary traced function;
// here the function is one of these, picked by the caller.
struct OpAdd { static __device__ __forceinline__ float id() { return 0.f; }
               static __device__ __forceinline__ float f(float a, float b) { return a + b; } };
struct OpMul { static __device__ __forceinline__ float id() { return 1.f; }
               static __device__ __forceinline__ float f(float a, float b) { return a * b; } };
struct OpMax { static __device__ __forceinline__ float id() { return -INFINITY; }
               static __device__ __forceinline__ float f(float a, float b) { return fmaxf(a, b); } };
struct OpMin { static __device__ __forceinline__ float id() { return INFINITY; }
               static __device__ __forceinline__ float f(float a, float b) { return fminf(a, b); } };
struct OpLogAddExp {      // log(exp(a) + exp(b)), evaluated around the larger argument
  static __device__ __forceinline__ float id() { return -INFINITY; }
  static __device__ __forceinline__ float f(float a, float b) {
    const float m = fmaxf(a, b), n = fminf(a, b);
    return m == -INFINITY ? m : m + log1pf(__expf(n - m));
  }
};

// One scan kernel for every layout.  What bounds it is HBM, so what counts is how many bytes are in flight and that
// every byte moves once, also when the array has few rows and a long axis: a block of 32 column lanes x 8 row lanes
// holds 8 RPT rows of 32 VEC columns in registers, and up to sixteen blocks of a thread-block cluster take consecutive
// pieces of the axis and exchange their totals through distributed shared memory, so that the axis is cut over
// blocks without a second pass over the data.  A row segment is one coalesced access per warp (128 to 512 bytes) at
// any width and alignment.  A thread holds 32 values, so that four blocks fit an SM and 128 KB of loads are in flight
// there; other blocks' loads cover a block's combine phase (prefetching the next tile in registers instead halves
// the blocks: measured slower).  Longer axes are walked in steps of a cluster's rows with the carry in registers.
// Measured, float32 (N, T, D) unless marked, us before (a ring of TMA tiles, one block per 128 columns) -> now, and the
// time of the bytes at the copy rate: (24, 4096, 136) 70 -> 27, 16; (96, 4096, 128) 72 -> 74, 62; (512, 128, 768)
// 75 -> 66, 62; (1, 16384, 96) 385 -> 12, 2; (2, 16384, 1024) 263 -> 56, 41; bf16 (9, 1342, 808) 37 -> 16, 6.
constexpr int SK_RL = 8;      // row lanes
constexpr int SK_MAXCL = 16;  // blocks of a cluster, at most (above 8: opt-in)
template <typename T, int VEC> __device__ __forceinline__ void sk_load(const T* p, float (&y)[VEC]) {
  if constexpr (VEC == 1) y[0] = ld_f(p, 0);
  else if constexpr (sizeof(T) == 4 && VEC == 2) { const float2 u = __ldg(reinterpret_cast<const float2*>(p)); y[0] = u.x; y[1] = u.y; }
  else if constexpr (sizeof(T) == 4) { const float4 u = __ldg(reinterpret_cast<const float4*>(p)); y[0] = u.x; y[1] = u.y; y[2] = u.z; y[3] = u.w; }
  else {
#pragma unroll
    for (int i = 0; i < VEC; i += 2) {
      const uint32_t u = __ldg(reinterpret_cast<const unsigned int*>(p) + i / 2);
      y[i] = __uint_as_float(u << 16); y[i + 1] = __uint_as_float(u & 0xffff0000u);
    }
  }
}
template <typename T, int VEC> __device__ __forceinline__ void sk_store(T* p, const float (&y)[VEC]) {
  if constexpr (VEC == 1) st_f(p, 0, y[0]);
  else if constexpr (sizeof(T) == 4 && VEC == 2) *reinterpret_cast<float2*>(p) = make_float2(y[0], y[1]);
  else if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(p) = make_float4(y[0], y[1], y[2], y[3]);
  else {
#pragma unroll
    for (int i = 0; i < VEC; i += 2) *(reinterpret_cast<uint32_t*>(p) + i / 2) = tc::pack_bf16x2(y[i], y[i + 1]);
  }
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <typename TI, typename TO, typename OP, int VEC, int RPT>
__global__ void __launch_bounds__(32 * SK_RL, 4) scan_kernel(const TI* __restrict__ src, const TI* __restrict__ sub,
                                                          const TI* __restrict__ init, TO* __restrict__ dst, int64_t T,
                                                          int64_t D, int gy, int cl, int reverse) {
  __shared__ float tot[2][SK_RL][32 * VEC];        // totals of the row lanes, double-buffered by tile parity
  __shared__ float peer[2][SK_MAXCL][32 * VEC];         // totals of the cluster's blocks; every block writes its own into all
  const int tx = threadIdx.x, rl = threadIdx.y;
  const int rank = (int)(blockIdx.x % cl);
  const int64_t item = blockIdx.x / cl, n = item / gy;
  const int64_t c = (item % gy) * (32 * VEC) + tx * VEC;
  const bool cvalid = c < D;                        // VEC divides D
  constexpr int ROWS = SK_RL * RPT;
  float carry[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) carry[v] = OP::id();
  grid_dep_wait();
  grid_dep_launch();
  if (init != nullptr && cvalid) sk_load<TI, VEC>(init + n * D + c, carry);
  // scan position p lies at row p (forward) or T - 1 - p (reversed); a thread's rows are `rs` elements apart
  const int64_t rs = reverse ? -D : D, p0 = (int64_t)rank * ROWS + rl * RPT;
  const int64_t off0 = n * T * D + c + (reverse ? T - 1 - p0 : p0) * D, step = (int64_t)cl * ROWS;
  const TI* ps = src + off0;
  const TI* ps2 = sub ? sub + off0 : nullptr;
  TO* po = dst + off0;
  auto rows_in = [&](int64_t t0) -> int {           // this thread's rows inside the axis for the step at t0
    const int64_t left = T - (t0 + p0);
    return !cvalid || left <= 0 ? 0 : left < RPT ? (int)left : RPT;
  };
  auto fetch = [&](int nr, float (&y)[RPT][VEC]) {
    if (nr == RPT) {                                // whole tiles: nothing between the loads
#pragma unroll
      for (int r = 0; r < RPT; ++r) sk_load<TI, VEC>(ps + r * rs, y[r]);
    } else {
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
#pragma unroll
        for (int v = 0; v < VEC; ++v) y[r][v] = OP::id();
        if (r < nr) sk_load<TI, VEC>(ps + r * rs, y[r]);
      }
    }
    if (ps2) {
#pragma unroll
      for (int r = 0; r < RPT; ++r)
        if (r < nr) {
          float z[VEC];
          sk_load<TI, VEC>(ps2 + r * rs, z);
#pragma unroll
          for (int v = 0; v < VEC; ++v) y[r][v] -= z[v];
        }
      ps2 += step * rs;
    }
    ps += step * rs;
  };
  if (cl > 1) cluster_barrier();                    // every block of the cluster runs before one writes to another
  int par = 0;
  for (int64_t t0 = 0; t0 < T; t0 += step, par ^= 1) {
    float x[RPT][VEC];
    const int nr = rows_in(t0);
    fetch(nr, x);
#pragma unroll
    for (int r = 1; r < RPT; ++r)
#pragma unroll
      for (int v = 0; v < VEC; ++v) x[r][v] = OP::f(x[r - 1][v], x[r][v]);
#pragma unroll
    for (int v = 0; v < VEC; ++v) tot[par][rl][v * 32 + tx] = x[RPT - 1][v];
    __syncthreads();
    float off[VEC], all[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) {
      float lower = OP::id(), sum = OP::id();
#pragma unroll
      for (int r = 0; r < SK_RL; ++r) {
        const float y = tot[par][r][v * 32 + tx];
        if (r < rl) lower = OP::f(lower, y);
        sum = OP::f(sum, y);
      }
      off[v] = lower;
      all[v] = sum;
    }
    if (cl > 1) {
      for (int to = rl; to < cl; to += SK_RL) {     // row lane r hands the block's totals to blocks r, r + 8 of the cluster
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
          uint32_t a = tc::smem_u32(&peer[par][rank][v * 32 + tx]);
          asm volatile("{\n\t.reg .u32 ra;\n\tmapa.shared::cluster.u32 ra, %0, %1;\n\tst.shared::cluster.f32 [ra], %2;\n\t}"
                       :: "r"(a), "r"(to), "f"(all[v]) : "memory");
        }
      }
      // a buffer is rewritten two steps later, past a barrier that every reader of it has arrived at
      cluster_barrier();
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        float before = carry[v];
        for (int k = 0; k < cl; ++k) {
          if (k == rank) off[v] = OP::f(before, off[v]);
          before = OP::f(before, peer[par][k][v * 32 + tx]);
        }
        carry[v] = before;
      }
    } else {
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        off[v] = OP::f(carry[v], off[v]);
        carry[v] = OP::f(carry[v], all[v]);
      }
    }
#pragma unroll
    for (int r = 0; r < RPT; ++r)
      if (r < nr) {
        float y[VEC];
#pragma unroll
        for (int v = 0; v < VEC; ++v) y[v] = OP::f(off[v], x[r][v]);
        sk_store<TO, VEC>(po + r * rs, y);
      }
    po += step * rs;
  }
}

__device__ __forceinline__ float4 ld4_f(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 ld4_f(const bf16* p) {
  const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x), b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
  const float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
  return make_float4(fa.x, fa.y, fb.x, fb.y);
}
__device__ __forceinline__ void st4_f(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st4_f(bf16* p, float4 v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&a); u.y = *reinterpret_cast<uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = u;
}

template <typename OP> __device__ __forceinline__ float4 op4(float4 a, float4 b) {
  return make_float4(OP::f(a.x, b.x), OP::f(a.y, b.y), OP::f(a.z, b.z), OP::f(a.w, b.w));
}
// ---------------------------------------------------------------------------------------
// The float32 scan of wide rows as a TMA pipeline.  Serves the shapes whose column blocks
// nearly fill the device once but not evenly with smaller blocks (see scan_ring_us).  A 64-row x 128-column tile travels
// as ONE tensor copy
// (cp.async.bulk.tensor over a 3-d map (column, row, n): rows past the end of the axis and columns past D are
// zero-filled on the way in and skipped on the way out) into a ring of NST shared-memory stages, the threads scan
// a landed tile out of shared memory, write the result into one of two staging tiles, and a tensor store takes it
// back.  Up to NST tiles (32 KB each) are in flight per block at no register cost.  (One bulk copy per ROW was
// measured first: 128 copy instructions per tile made the kernel twice as slow as the load/store one.)
//   thread 0       issues the copy of tile i + NST once tile i has been read
//   thread 32      issues the store of tile i and waits for the store of tile i - 2 to have read its stage
//   all 8 warps    thread = four columns x eight consecutive scan positions; row lanes combine through shared memory
// A reversed scan walks the tiles from the end of the axis; its tiles are laid out so that every one but the FIRST
// in scan order starts on a multiple of 64 rows from the end (no store ever starts at a negative row), and a
// thread's scan position p sits in stage row nr - 1 - p.
// Every mbarrier wait is bounded; a block whose wait expires stops, waits (bounded) for the copies it still has
// in flight and counts itself in g_scan_wait_timeouts.
// ---------------------------------------------------------------------------------------
namespace {
using namespace tc;
__device__ unsigned int g_scan_wait_timeouts = 0;
constexpr int BK_RPT = 8;                      // rows per thread
constexpr int BK_RL = 8;                       // row lanes
constexpr int BK_ROWS = BK_RPT * BK_RL;        // rows of a tile (64)
constexpr int BK_NST = 4;                      // input stages
constexpr int BK_TILE = BK_ROWS * 128 * 4;     // bytes of a tile (32 KB)
constexpr int BK_SMEM = (BK_NST + 2) * BK_TILE + 1024;

__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int PENDING> __device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" :: "n"(PENDING) : "memory");
}
template <int PENDING> __device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group %0;" :: "n"(PENDING) : "memory");
}

struct ScanMaps { CUtensorMap in, out; };

template <typename OP, bool MULTI>
__global__ void __launch_bounds__(32 * BK_RL, 1) cumsum_tma_kernel(const __grid_constant__ ScanMaps maps, const float* __restrict__ init,
                                                                   int64_t N, int64_t T, int64_t D, int reverse) {
  extern __shared__ uint8_t bk_raw[];
  uint8_t* sm = (uint8_t*)(((uintptr_t)bk_raw + 1023) & ~(uintptr_t)1023);
  __shared__ float4 tot[2][BK_RL][32];
  __shared__ float4 car[2][32];
  __shared__ uint64_t full[BK_NST];
  const int tx = threadIdx.x, rl = threadIdx.y, tid = rl * 32 + tx;
  // Work items are (row n, block of 128 columns); a block takes items blockIdx.x, + gridDim.x, ... and streams their
  // tiles back to back through the same ring, so that short axes (a chunk of 128 positions is two tiles) do not pay
  // a block start-up each.
  const int64_t gy = (D + 127) / 128, items = N * gy;
  // MULTI == false is the same kernel for grids with one item per block: the walk over items folds away
  const int64_t my_items = MULTI ? (items - blockIdx.x + gridDim.x - 1) / gridDim.x : 1;
  // tiles of an item in scan order: forward tile i starts at row 64 i; reversed, tile 0 holds the last `rem` rows of
  // the axis and tile i >= 1 the 64 rows before those of tile i - 1
  const int rem = (int)(T % BK_ROWS ? T % BK_ROWS : BK_ROWS);
  const int64_t ntiles = (T + BK_ROWS - 1) / BK_ROWS, total = my_items * ntiles;
  const int Ti = (int)T;
  auto rows_of = [&](int i) {
    if (reverse) return i == 0 ? rem : BK_ROWS;
    const int left = Ti - i * BK_ROWS;
    return left < BK_ROWS ? left : BK_ROWS;
  };
  auto start_of = [&](int i) { return reverse ? Ti - rem - i * BK_ROWS : i * BK_ROWS; };
  const uint32_t in0 = smem_u32(sm), out0 = in0 + BK_NST * BK_TILE, full0 = smem_u32(full);
  const float4 ident = make_float4(OP::id(), OP::id(), OP::id(), OP::id());

  if (tid == 0) {
    for (int s2 = 0; s2 < BK_NST; ++s2) mbar_init(full0 + 8 * s2, 1);
    mbar_fence_init();
  }
  __syncthreads();
  static_assert((BK_NST & (BK_NST - 1)) == 0, "the ring index is kept with a mask");
  // the producer's own walk over (item, tile), NST tiles ahead of the consumers'; all walks keep their place with
  // counters (no division per tile)
  int64_t p_item = blockIdx.x, p_g = 0;
  int p_i = 0, p_n = (int)(p_item / gy), p_c0 = (int)(p_item % gy) * 128;
  auto issue_load = [&]() {                   // one thread
    const uint32_t sidx = (uint32_t)p_g & (BK_NST - 1), bar = full0 + 8 * sidx;
    mbar_arrive_expect_tx(bar, BK_TILE);      // the box counts in full, zero-filled parts included
    tma_load_3d(in0 + sidx * BK_TILE, &maps.in, p_c0, start_of(p_i), p_n, bar);
    ++p_g;
    ++p_i;
    if (MULTI && p_i == (int)ntiles) {
      p_i = 0; p_item += gridDim.x;
      p_n = (int)(p_item / gy); p_c0 = (int)(p_item % gy) * 128;
    }
  };
  if (tid == 0)
    for (int a = 0; a < BK_NST && p_g < total; ++a) issue_load();
  auto init_of = [&](int nn, int cc) {
    const int64_t c = (int64_t)cc + tx * 4;
    return (init != nullptr && c < D) ? ld4_f(init + (int64_t)nn * D + c) : ident;
  };
  int64_t item = blockIdx.x, g = 0;
  int i = 0, n = (int)(item / gy), c0 = (int)(item % gy) * 128;
  if (rl == BK_RL - 1 && total > 0) car[0][tx] = init_of(n, c0);
  bool ok = true;
  int par = 0, st = 0;
  uint32_t phase = 0;
  for (; g < total; ++g, par ^= 1) {
    const bool cvalid = (int64_t)c0 + tx * 4 < D;
    ok = mbar_wait(full0 + 8 * st, phase);       // on expiry the tile is garbage: voted on below
    const int nrt = rows_of(i);
    const int nr = nrt - rl * BK_RPT;                 // this thread's scan positions inside the tile (<= 0: none)
    // scan position p = 8 rl + r of the tile sits in stage row p (forward) or nrt - 1 - p (reversed)
    const int row0 = reverse ? nrt - 1 - rl * BK_RPT : rl * BK_RPT, rstep = reverse ? -32 : 32;
    const float4* in = reinterpret_cast<const float4*>(sm + st * BK_TILE) + row0 * 32 + tx;
    float4 x[BK_RPT];
#pragma unroll
    for (int r = 0; r < BK_RPT; ++r) x[r] = (cvalid && r < nr) ? in[r * rstep] : ident;
#pragma unroll
    for (int r = 1; r < BK_RPT; ++r) x[r] = op4<OP>(x[r - 1], x[r]);
    tot[par][rl][tx] = x[BK_RPT - 1];
    // the staging tile that this tile is about to write was last read by the store of two tiles ago: all but the
    // newest store group must have read their stage
    if (tid == 32) bulk_wait_read<1>();
    // stage st has been read by everyone and the totals are visible; the same barrier takes the vote on the waits,
    // so that the whole block leaves together if any thread's wait expired
    if (!__syncthreads_and(ok)) { ok = false; break; }
    if (tid == 0 && p_g < total) issue_load();
    float4 off = car[par][tx];
    for (int r2 = 0; r2 < rl; ++r2) off = op4<OP>(off, tot[par][r2][tx]);
    const bool last_tile = MULTI && i + 1 == (int)ntiles;
    int n2 = n, c2 = c0;
    if (last_tile) { const int64_t nx = item + gridDim.x; n2 = (int)(nx / gy); c2 = (int)(nx % gy) * 128; }
    // the carry into the next tile: this item's running value, or the next item's initial value
    if (rl == BK_RL - 1)
      car[par ^ 1][tx] = !last_tile ? op4<OP>(off, x[BK_RPT - 1]) : item + gridDim.x < items ? init_of(n2, c2) : ident;
    float4* o = reinterpret_cast<float4*>(sm + (BK_NST + par) * BK_TILE) + row0 * 32 + tx;
#pragma unroll
    for (int r = 0; r < BK_RPT; ++r)
      if (r < nr) o[r * rstep] = op4<OP>(off, x[r]);
    fence_async_smem();                                // the staging tile is read by the async proxy
    __syncthreads();
    if (tid == 32) {
      tma_store_3d(&maps.out, c0, start_of(i), n, out0 + (uint32_t)par * BK_TILE);
      bulk_commit();
    }
    if (last_tile) { i = 0; item += gridDim.x; n = n2; c0 = c2; } else ++i;
    if (++st == BK_NST) { st = 0; phase ^= 1u; }
  }
  if (tid == 32) bulk_wait_all<0>();                    // the block's stores have completed before it leaves
  if (!ok) {
    // copies already requested land in this block's shared memory: give them their (bounded) time before leaving
    if (tid == 0)
      for (int64_t j = g; j < p_g; ++j) mbar_wait(full0 + 8 * ((uint32_t)j & (BK_NST - 1)), (uint32_t)((j / BK_NST) & 1));
    if (tid == 0) atomicAdd(&g_scan_wait_timeouts, 1u);
  }
}
}  // namespace

unsigned int scan_read_wait_timeouts() {
  unsigned int v = 0;
  cudaMemcpyFromSymbol(&v, g_scan_wait_timeouts, sizeof(v));
  return v;
}

template <typename OP>
static int launch_cumsum_tma_op(cudaStream_t st, int64_t N, int64_t T, int64_t D, const float* src, const float* init, float* dst,
                                int reverse) {
  ProfScope ps("cumsum_kernel", st);
  static SmemAttrOnce attr[2];
  GLA_TRY(attr[0].ensure(cumsum_tma_kernel<OP, false>, BK_SMEM));
  GLA_TRY(attr[1].ensure(cumsum_tma_kernel<OP, true>, BK_SMEM));
  ScanMaps maps;
  GLA_TRY(make_map_ntd_f32(&maps.in, src, N, T, D, BK_ROWS));
  GLA_TRY(make_map_ntd_f32(&maps.out, dst, N, T, D, BK_ROWS));
  // one block per SM (the ring takes most of its shared memory), fewer when there are fewer (row, column block) items
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t items = N * ((D + 127) / 128);
  dim3 block(32, BK_RL);
  if (items <= sms) cumsum_tma_kernel<OP, false><<<dim3((unsigned)items), block, BK_SMEM, st>>>(maps, init, N, T, D, reverse);
  else              cumsum_tma_kernel<OP, true><<<dim3((unsigned)sms), block, BK_SMEM, st>>>(maps, init, N, T, D, reverse);
  GLA_CHECK_LAUNCH();
  return GLA_OK;
}

// Blocks per cluster: the time of a grid is its waves over the SMs (four blocks each) times a block's steps; a step costs
// the larger of its latency (about 2.5 us, 2 us more with the exchange) and of its SM's share of HBM.  The count that
// minimises that by a clear margin is taken: 1 where rows and columns alone fill the device, up to 16 for a few rows with a long axis.
// (148 SMs: latency and share were measured there, and the model holds for that number.)
static int scan_cluster(int64_t items, int64_t T, int rows, double tile_bytes, double* us = nullptr) {
  constexpr int SMS = 148, PER_SM = 4;
  int best = 1;
  double best_t = 0;
  for (int cl = 1; cl <= SK_MAXCL; cl *= 2) {
    if (cl > 1 && (int64_t)(cl / 2) * rows >= T) break;
    const double total = (double)items * cl, full = floor(total / (SMS * PER_SM)), rest = total - full * SMS * PER_SM;
    const double lat = cl > 1 ? 4.5 : 2.5, share = tile_bytes / 44e3;       // us; 44 KB/us per SM
    const double steps = (double)((T + (int64_t)cl * rows - 1) / ((int64_t)cl * rows));
    const double t = steps * (full * fmax(lat, PER_SM * share) + (rest > 0 ? fmax(lat, ceil(rest / SMS) * share) : 0.0));
    if (cl == 1 || t < 0.85 * best_t) { best = cl; best_t = t; }
  }
  if (us != nullptr) *us = best_t;
  return best;
}
// The ring's time (us): a block streams its item's rows at about 58 GB/s, read and write, one block per SM, all of them
// at 5.9 TB/s at most (measured at N = 96, D = 128 and N = 90, D = 132, T = 4096: 72 and 144 us).
static double scan_ring_us(int64_t N, int64_t T, int64_t D) {
  const double items = (double)N * ((D + 127) / 128), bytes = (double)T * 128 * 8;
  return fmax(ceil(items / 148) * bytes / 58e3, items * bytes / 5.9e6);
}
template <typename TI, typename TO, typename OP, int VEC, int RPT>
static int launch_scan_rows(cudaStream_t st, int64_t N, int64_t T, int64_t D, const void* src, const void* sub, const void* init,
                            void* dst, int reverse) {
  const int64_t gy = (D + 32 * VEC - 1) / (32 * VEC), items = N * gy;
  const int cl = scan_cluster(items, T, SK_RL * RPT, (double)SK_RL * RPT * 32 * VEC * (sizeof(TI) + sizeof(TO)));
  if (items * cl > 2147483647LL || gy > 2147483647LL) return GLA_ERR_TOO_LARGE;
  static SmemAttrOnce attr16;
  if (cl > 8) GLA_TRY(attr16.allow_large_clusters(scan_kernel<TI, TO, OP, VEC, RPT>));
  ProfScope ps("cumsum_kernel", st);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(items * cl));
  cfg.blockDim = dim3(32, SK_RL);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;        // see launch_overlapped
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cl; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cl > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, scan_kernel<TI, TO, OP, VEC, RPT>, (const TI*)src, (const TI*)sub, (const TI*)init,
                                           (TO*)dst, T, D, (int)gy, cl, reverse);
  if (e != cudaSuccess) return record_cuda_error(e);
  GLA_CHECK_LAUNCH();
  return GLA_OK;
}
// Columns per lane and rows per lane (32 values together): a block's 8 row lanes should not outrun a short axis, and on
// a long one narrow blocks give more of them.  bf16 keeps two columns per lane, which fill a 128-byte line of a row.
template <typename TI, typename TO, typename OP>
static int launch_scan_op(cudaStream_t st, int64_t N, int64_t T, int64_t D, const void* src, const void* sub, const void* init,
                          void* dst, int reverse) {
  auto vec = [&](int v) {
    auto on = [](const void* p, size_t a) { return ((uintptr_t)p % a) == 0; };
    return D % v == 0 && on(src, v * sizeof(TI)) && on(sub, v * sizeof(TI)) && on(init, v * sizeof(TI)) && on(dst, v * sizeof(TO));
  };
  auto fits = [&](int v) { return vec(v) && (D + 32 * v - 1) / (32 * v) * (32 * v) * 4 <= D * 5; };      // idle columns
  if (sizeof(TI) == 4 && T <= 8 * SK_RL && fits(4)) return launch_scan_rows<TI, TO, OP, 4, 8>(st, N, T, D, src, sub, init, dst, reverse);
  if (T <= 16 * SK_RL && fits(2)) return launch_scan_rows<TI, TO, OP, 2, 16>(st, N, T, D, src, sub, init, dst, reverse);
  if (sizeof(TI) == 2 && vec(2)) return launch_scan_rows<TI, TO, OP, 2, 16>(st, N, T, D, src, sub, init, dst, reverse);
  if constexpr (sizeof(TI) == 4 && sizeof(TO) == 4) {
    // (12 %: what the model of the register kernel leaves out where two or three blocks share an SM, 83 us at N = 50,
    // T = 4096, D = 256 against 72 with the ring)
    if (sub == nullptr && T >= 1024 && vec(4) && (D + 127) / 128 <= 65535 && N <= 2147483647LL && T <= 2147483647LL) {
      double us;
      scan_cluster(N * ((D + 31) / 32), T, SK_RL * 32, SK_RL * 32 * 32 * 8.0, &us);
      if (scan_ring_us(N, T, D) < 1.12 * us) return launch_cumsum_tma_op<OP>(st, N, T, D, (const float*)src, (const float*)init, (float*)dst, reverse);
    }
  }
  return T <= 8 * SK_RL ? launch_scan_rows<TI, TO, OP, 1, 8>(st, N, T, D, src, sub, init, dst, reverse)
                        : launch_scan_rows<TI, TO, OP, 1, 32>(st, N, T, D, src, sub, init, dst, reverse);
}
template <typename TI, typename TO>
static int launch_scan_types(cudaStream_t st, int64_t N, int64_t T, int64_t D, const void* src, const void* sub, const void* init,
                             void* dst, int reverse, int op) {
  switch (op) {
    case GLA_SCAN_MUL: return launch_scan_op<TI, TO, OpMul>(st, N, T, D, src, sub, init, dst, reverse);
    case GLA_SCAN_MAX: return launch_scan_op<TI, TO, OpMax>(st, N, T, D, src, sub, init, dst, reverse);
    case GLA_SCAN_MIN: return launch_scan_op<TI, TO, OpMin>(st, N, T, D, src, sub, init, dst, reverse);
    case GLA_SCAN_LOGADDEXP: return launch_scan_op<TI, TO, OpLogAddExp>(st, N, T, D, src, sub, init, dst, reverse);
    default: return launch_scan_op<TI, TO, OpAdd>(st, N, T, D, src, sub, init, dst, reverse);
  }
}

int launch_cumsum(cudaStream_t st, int64_t N, int64_t T, int64_t D, const void* src, const void* init,
                  void* dst, int reverse, int in_bf16, int out_bf16, const void* sub, int op) {
  if (N <= 0 || T <= 0 || D <= 0) return GLA_ERR_BAD_DIMS;
  if (op < GLA_SCAN_ADD || op > GLA_SCAN_LOGADDEXP || (sub != nullptr && op != GLA_SCAN_ADD)) return GLA_ERR_UNSUPPORTED;
  if (in_bf16) return out_bf16 ? launch_scan_types<bf16, bf16>(st, N, T, D, src, sub, init, dst, reverse, op)
                               : launch_scan_types<bf16, float>(st, N, T, D, src, sub, init, dst, reverse, op);
  return out_bf16 ? launch_scan_types<float, bf16>(st, N, T, D, src, sub, init, dst, reverse, op)
                  : launch_scan_types<float, float>(st, N, T, D, src, sub, init, dst, reverse, op);
}




// ---------------------------------------------------------------------------------------
// rnn_scan: sequential over T, parallel over the elements of the state.  A thread owns FOUR consecutive value
// columns of one key row (one 16- or 8-byte access per step instead of four scalar ones, and one exp() of the
// gate per step for the four), and keeps the loads of the next UNR steps in flight while it combines the
// current ones: the recurrence is a chain, so what the kernel can overlap is the memory latency of later steps.
// The scalar form below serves value widths that are not multiples of four.
// ---------------------------------------------------------------------------------------
template <typename TKV, bool RUNS>
__global__ void __launch_bounds__(128) rnn_scan_vec4_kernel(int64_t T, int64_t K, int64_t V, int64_t nblk,
                                                            const float* __restrict__ g, const TKV* __restrict__ kv,
                                                            const float* __restrict__ ig, const TKV* __restrict__ ikv,
                                                            float* __restrict__ out_log, TKV* __restrict__ out_state,
                                                            int reverse, int last_only, int nseg, int64_t L) {
  constexpr int UNR = 4;
  // nseg > 1: the axis is cut into runs of L scan positions that separate blocks scan, every run but the first from
  // the identity; rnn_carry_kernel / rnn_fix_kernel below then put the runs together (long axes with few rows)
  // (RUNS == false is the plain scan: the run arithmetic folds away)
  const int64_t prob2 = blockIdx.x / nblk, prob = RUNS ? prob2 / nseg : prob2, seg = RUNS ? prob2 % nseg : 0;
  const int64_t e4 = (blockIdx.x % nblk) * 128 + threadIdx.x;      // group of four value columns
  const int64_t KV = K * V, V4 = V / 4;
  if (e4 >= K * V4) return;
  const int64_t kk = e4 / V4, e = e4 * 4;
  const bool writes_log = (e4 % V4) == 0;
  grid_dep_wait();
  grid_dep_launch();
  float A = (ig && seg == 0) ? ig[prob * K + kk] : 0.f;
  float4 b = (ikv && seg == 0) ? ld4_f(ikv + prob * KV + e) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float* gp = g + prob * T * K + kk;
  const TKV* xp = kv + prob * T * KV + e;
  TKV* op = out_state + prob * T * KV + e;
  float* lp = out_log + prob * T * K + kk;
  const int64_t s_beg = RUNS ? seg * L : 0;
  const int64_t Tfull = T;
  if (RUNS) T = Tfull - s_beg < L ? Tfull - s_beg : L;             // scan positions of this run (T below: the run's)
  auto tix = [&](int64_t s) { return reverse ? (Tfull - 1 - (s_beg + s)) : s_beg + s; };
  float gn[UNR];
  float4 xn[UNR];
#pragma unroll
  for (int u = 0; u < UNR; ++u) {
    const int64_t t = tix(u < T ? u : T - 1);
    gn[u] = gp[t * K];
    xn[u] = ld4_f(xp + t * KV);
  }
  for (int64_t s0 = 0; s0 < T; s0 += UNR) {
    float gc[UNR];
    float4 xc[UNR];
#pragma unroll
    for (int u = 0; u < UNR; ++u) { gc[u] = gn[u]; xc[u] = xn[u]; }
#pragma unroll
    for (int u = 0; u < UNR; ++u) {           // the next group's loads, issued before this group is combined
      const int64_t sn = s0 + UNR + u;
      const int64_t t = tix(sn < T ? sn : T - 1);
      gn[u] = gp[t * K];
      xn[u] = ld4_f(xp + t * KV);
    }
#pragma unroll
    for (int u = 0; u < UNR; ++u) {
      const int64_t sc = s0 + u;
      if (sc < T) {
        const float f = expf(gc[u]);
        b.x = fmaf(f, b.x, xc[u].x); b.y = fmaf(f, b.y, xc[u].y);
        b.z = fmaf(f, b.z, xc[u].z); b.w = fmaf(f, b.w, xc[u].w);
        A += gc[u];
        if (!last_only || sc == T - 1) {
          const int64_t t = tix(sc);
          st4_f(op + t * KV, b);
          if (writes_log) lp[t * K] = A;
        }
      }
    }
  }
}

// The runs of a segmented scan put together.  carry (one thread per four value columns, sequential over the runs):
// the true pair at the end of run s - 1, C_s = (CL_s, CS_s), from the runs' local last rows
//   C_1 = local last row of run 0 (which started from the caller's initial pair),
//   CL_{s+1} = CL_s + l_s,   CS_{s+1} = exp(l_s) CS_s + x_s        (l_s, x_s: local last row of run s),
// into wsL (batch, nseg, K) and wsS (batch, nseg, K, V), float32.
template <typename TKV>
__global__ void __launch_bounds__(128) rnn_carry_kernel(int64_t T, int64_t K, int64_t V, int64_t nblk, int nseg, int64_t L,
                                                        const float* __restrict__ out_log, const TKV* __restrict__ out_state,
                                                        float* __restrict__ wsL, float* __restrict__ wsS, int reverse) {
  const int64_t prob = blockIdx.x / nblk;
  const int64_t e4 = (blockIdx.x % nblk) * 128 + threadIdx.x;
  const int64_t KV = K * V, V4 = V / 4;
  if (e4 >= K * V4) return;
  const int64_t kk = e4 / V4, e = e4 * 4;
  const bool writes_log = (e4 % V4) == 0;
  float CL = 0.f;
  float4 CS = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int sg = 0; sg < nseg; ++sg) {
    if (sg > 0) {
      if (writes_log) wsL[(prob * nseg + sg) * K + kk] = CL;
      *reinterpret_cast<float4*>(wsS + (prob * nseg + sg) * KV + e) = CS;
    }
    const int64_t last = (sg + 1) * L < T ? (sg + 1) * L - 1 : T - 1;      // scan position of the run's last row
    const int64_t row = reverse ? T - 1 - last : last;
    const float l = out_log[(prob * T + row) * K + kk];
    const float4 x = ld4_f(out_state + (prob * T + row) * KV + e);
    const float f = expf(l);
    CS = make_float4(fmaf(f, CS.x, x.x), fmaf(f, CS.y, x.y), fmaf(f, CS.z, x.z), fmaf(f, CS.w, x.w));
    CL += l;
  }
}
// fix (one thread per row and four value columns, rows of the runs after the first): state = exp(local log) C_S + local
// state.  The logs are corrected by rnn_fix_log_kernel afterwards (this kernel reads the local ones).
template <typename TKV>
__global__ void __launch_bounds__(256) rnn_fix_kernel(int64_t batch, int64_t T, int64_t K, int64_t V, int nseg, int64_t L,
                                                      const float* __restrict__ out_log, TKV* __restrict__ out_state,
                                                      const float* __restrict__ wsS, int reverse) {
  const int64_t KV4 = K * (V / 4), rows = T - L;
  const int64_t id = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (id >= batch * rows * KV4) return;
  const int64_t e4 = id % KV4, pos = L + (id / KV4) % rows, prob = id / KV4 / rows;
  const int64_t kk = e4 / (V / 4), e = e4 * 4, sg = pos / L;
  const int64_t row = reverse ? T - 1 - pos : pos;
  const float f = expf(out_log[(prob * T + row) * K + kk]);
  const float4 c = *reinterpret_cast<const float4*>(wsS + (prob * nseg + sg) * K * V + e);
  TKV* p = out_state + (prob * T + row) * K * V + e;
  const float4 x = ld4_f(p);
  st4_f(p, make_float4(fmaf(f, c.x, x.x), fmaf(f, c.y, x.y), fmaf(f, c.z, x.z), fmaf(f, c.w, x.w)));
}
__global__ void __launch_bounds__(256) rnn_fix_log_kernel(int64_t batch, int64_t T, int64_t K, int nseg, int64_t L,
                                                          float* __restrict__ out_log, const float* __restrict__ wsL,
                                                          int reverse) {
  const int64_t rows = T - L;
  const int64_t id = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (id >= batch * rows * K) return;
  const int64_t kk = id % K, pos = L + (id / K) % rows, prob = id / K / rows;
  const int64_t row = reverse ? T - 1 - pos : pos;
  out_log[(prob * T + row) * K + kk] += wsL[(prob * nseg + pos / L) * K + kk];
}

template <typename TKV>
__global__ void __launch_bounds__(256) rnn_scan_kernel(int64_t T, int64_t K, int64_t V, int64_t nblk,
                                                       const float* __restrict__ g, const TKV* __restrict__ kv,
                                                       const float* __restrict__ ig, const TKV* __restrict__ ikv,
                                                       float* __restrict__ out_log, TKV* __restrict__ out_state,
                                                       int reverse, int last_only) {
  const int64_t prob = blockIdx.x / nblk;
  const int64_t e = (blockIdx.x % nblk) * 256 + threadIdx.x;
  const int64_t KV = K * V;
  if (e >= KV) return;
  const int64_t kk = e / V, vv = e % V;
  float A = ig ? ig[prob * K + kk] : 0.f;
  float b = ikv ? ld_f(ikv, prob * KV + e) : 0.f;
  const float* gp = g + prob * T * K + kk;
  const TKV* xp = kv + prob * T * KV + e;
  TKV* op = out_state + prob * T * KV + e;
  float* lp = out_log + prob * T * K + kk;
#pragma unroll 4
  for (int64_t s = 0; s < T; ++s) {
    const int64_t t = reverse ? (T - 1 - s) : s;
    const float gt = gp[t * K];
    b = expf(gt) * b + ld_f(xp, t * KV);
    A += gt;
    if (!last_only || s == T - 1) {
      st_f(op, t * KV, b);
      if (vv == 0) lp[t * K] = A;
    }
  }
}

// Runs for a long axis with few rows: enough blocks for the device, runs of at least 128 positions.
static void rnn_scan_runs(int64_t batch, int64_t T, int64_t K, int64_t V, int* nseg, int64_t* L) {
  *nseg = 1; *L = T;
  if (V % 4 != 0 || T < 512) return;
  const int64_t blocks = batch * ((K * (V / 4) + 127) / 128);
  if (blocks >= 2 * 148) return;
  int64_t want = (4 * 148 + blocks - 1) / blocks;
  if (want > T / 128) want = T / 128;
  if (want < 2) return;
  *L = (T + want - 1) / want;
  *nseg = (int)((T + *L - 1) / *L);
}
size_t rnn_scan_ws_bytes(int64_t batch, int64_t T, int64_t K, int64_t V) {
  int nseg; int64_t L;
  rnn_scan_runs(batch, T, K, V, &nseg, &L);
  return nseg > 1 ? (size_t)(batch * nseg * (K + K * V)) * sizeof(float) + 16 : 0;
}

int launch_rnn_scan(cudaStream_t st, int64_t batch, int64_t T, int64_t K, int64_t V, const float* g,
                    const void* kv, const float* ig, const void* ikv, float* out_log, void* out_state,
                    int reverse, int last_only, int kv_bf16, float* ws, size_t ws_bytes) {
  ProfScope ps("rnn_scan_kernel", st);
  const bool al = (((uintptr_t)kv | (uintptr_t)out_state | (uintptr_t)ikv) & 15) == 0;
  if (V % 4 == 0 && al) {
    int64_t nblk = (K * (V / 4) + 127) / 128;
    int nseg = 1; int64_t L = T;
    if (ws != nullptr && !last_only && ((uintptr_t)ws & 15) == 0) {
      rnn_scan_runs(batch, T, K, V, &nseg, &L);
      if (ws_bytes < (size_t)(batch * nseg * (K + K * V)) * sizeof(float) + 16) { nseg = 1; L = T; }
    }
    if (nblk * batch * nseg > 2147483647LL) return GLA_ERR_TOO_LARGE;
    dim3 grid((unsigned)(nblk * batch * nseg)), block(128);
    auto run = [&](auto kern, auto t) {
      using TKV = decltype(t);
      return launch_overlapped(kern, grid, block, 0, st, T, K, V, nblk, g, (const TKV*)kv, ig, (const TKV*)ikv, out_log, (TKV*)out_state,
                               reverse, last_only, nseg, nseg > 1 ? L : T);
    };
    if (kv_bf16) GLA_LAUNCHED(run(nseg > 1 ? rnn_scan_vec4_kernel<bf16, true> : rnn_scan_vec4_kernel<bf16, false>, bf16()));
    else GLA_LAUNCHED(run(nseg > 1 ? rnn_scan_vec4_kernel<float, true> : rnn_scan_vec4_kernel<float, false>, 0.f));
    if (nseg > 1) {
      float* wsL = ws;
      float* wsS = ws + batch * nseg * K;      // batch * nseg * K floats: a multiple of 16 bytes when K % 4 == 0
      if ((batch * nseg * K) % 4 != 0) wsS += 4 - (batch * nseg * K) % 4;
      const int64_t nfix = batch * (T - L) * K * (V / 4), nlog = batch * (T - L) * K;
      if ((nfix + 255) / 256 > 2147483647LL) return GLA_ERR_TOO_LARGE;
      if (kv_bf16) {
        rnn_carry_kernel<bf16><<<(unsigned)(nblk * batch), 128, 0, st>>>(T, K, V, nblk, nseg, L, out_log, (const bf16*)out_state, wsL, wsS, reverse);
        rnn_fix_kernel<bf16><<<(unsigned)((nfix + 255) / 256), 256, 0, st>>>(batch, T, K, V, nseg, L, out_log, (bf16*)out_state, wsS, reverse);
      } else {
        rnn_carry_kernel<float><<<(unsigned)(nblk * batch), 128, 0, st>>>(T, K, V, nblk, nseg, L, out_log, (const float*)out_state, wsL, wsS, reverse);
        rnn_fix_kernel<float><<<(unsigned)((nfix + 255) / 256), 256, 0, st>>>(batch, T, K, V, nseg, L, out_log, (float*)out_state, wsS, reverse);
      }
      rnn_fix_log_kernel<<<(unsigned)((nlog + 255) / 256), 256, 0, st>>>(batch, T, K, nseg, L, out_log, wsL, reverse);
      GLA_CHECK_LAUNCH();
    }
    return GLA_OK;
  }
  int64_t nblk = (K * V + 255) / 256;
  if (nblk * batch > 2147483647LL) return GLA_ERR_TOO_LARGE;
  dim3 grid((unsigned)(nblk * batch)), block(256);
  if (kv_bf16)
    rnn_scan_kernel<bf16><<<grid, block, 0, st>>>(T, K, V, nblk, g, (const bf16*)kv, ig, (const bf16*)ikv,
                                                  out_log, (bf16*)out_state, reverse, last_only);
  else
    rnn_scan_kernel<float><<<grid, block, 0, st>>>(T, K, V, nblk, g, (const float*)kv, ig, (const float*)ikv,
                                                   out_log, (float*)out_state, reverse, last_only);
  GLA_CHECK_LAUNCH();
  return GLA_OK;
}

// ---------------------------------------------------------------------------------------
// State scan over chunks (the D x D recurrence of the chunk algorithm, gla.py:711-723 and
// its mirror gla.py:759-771).  Four consecutive value-columns per thread; sequential over
// the N chunks; writes the state BEFORE each update ("exclusive") and the final state.
// ---------------------------------------------------------------------------------------
template <typename TX, typename TI, typename TB, typename TF>
__global__ void __launch_bounds__(256) state_scan_kernel(int64_t N, int64_t D, int64_t nblk,
                                                         const float* __restrict__ G, const TX* X,
                                                         const TI* __restrict__ init, TB* before,
                                                         TF* __restrict__ final_state, int reverse) {
  const int64_t bh = blockIdx.x / nblk;
  const int64_t e = ((blockIdx.x % nblk) * 256 + threadIdx.x) * 4;
  const int64_t DD = D * D;
  if (e >= DD) return;
  const int64_t dk = e / D;
  float s[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i] = init ? ld_f(init, bh * DD + e + i) : 0.f;
  const float* gp = G + bh * N * D + dk;
  const TX* xp = X + bh * N * DD + e;
  TB* bp = before ? before + bh * N * DD + e : nullptr;
#pragma unroll 2
  for (int64_t i = 0; i < N; ++i) {
    const int64_t n = reverse ? (N - 1 - i) : i;
    const float f = expf(gp[n * D]);
    float x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = ld_f(xp, n * DD + j);
    if (bp) {
#pragma unroll
      for (int j = 0; j < 4; ++j) st_f(bp, n * DD + j, s[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = f * s[j] + x[j];
  }
  if (final_state) {
#pragma unroll
    for (int j = 0; j < 4; ++j) st_f(final_state, bh * DD + e + j, s[j]);
  }
}

template <typename TX, typename TI, typename TB>
static int state_scan_dispatch_final(cudaStream_t st, dim3 grid, int64_t N, int64_t D, int64_t nblk, const float* G,
                                     const void* X, const void* init, void* before, void* fin, int final_bf16,
                                     int reverse) {
  if (final_bf16)
    state_scan_kernel<TX, TI, TB, bf16><<<grid, 256, 0, st>>>(N, D, nblk, G, (const TX*)X, (const TI*)init,
                                                              (TB*)before, (bf16*)fin, reverse);
  else
    state_scan_kernel<TX, TI, TB, float><<<grid, 256, 0, st>>>(N, D, nblk, G, (const TX*)X, (const TI*)init,
                                                               (TB*)before, (float*)fin, reverse);
  GLA_CHECK_LAUNCH();
  return GLA_OK;
}

int launch_state_scan(cudaStream_t st, int64_t BH, int64_t N, int64_t D, const float* G, const void* X,
                      int x_bf16, const void* init, int init_bf16, void* before, int before_bf16,
                      void* final_state, int final_bf16, int reverse) {
  if (x_bf16) return GLA_ERR_UNSUPPORTED;   // chunk products are always kept in float32
  int64_t nblk = (D * D / 4 + 255) / 256;
  dim3 grid((unsigned)(nblk * BH));
  ProfScope ps("state_scan_kernel", st);
  if (init_bf16) {
    if (before_bf16)
      return state_scan_dispatch_final<float, bf16, bf16>(st, grid, N, D, nblk, G, X, init, before, final_state, final_bf16, reverse);
    return state_scan_dispatch_final<float, bf16, float>(st, grid, N, D, nblk, G, X, init, before, final_state, final_bf16, reverse);
  }
  if (before_bf16)
    return state_scan_dispatch_final<float, float, bf16>(st, grid, N, D, nblk, G, X, init, before, final_state, final_bf16, reverse);
  return state_scan_dispatch_final<float, float, float>(st, grid, N, D, nblk, G, X, init, before, final_state, final_bf16, reverse);
}

// ---------------------------------------------------------------------------------------
// Cross-rank combine for sequence parallelism: an exclusive decayed scan over ranks of the
// per-rank (total log decay, local state) pairs, evaluated for one rank.
// ---------------------------------------------------------------------------------------
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) sp_combine_kernel(int64_t R, int64_t rank, int64_t BH, int64_t D,
                                                         const float* __restrict__ all_G,
                                                         const float* __restrict__ all_S,
                                                         const TI* __restrict__ init, TO* __restrict__ result,
                                                         int reverse) {
  const int64_t DD = D * D;
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (e >= BH * DD) return;
  const int64_t bh = e / DD, dk = (e % DD) / D;
  float acc = init ? ld_f(init, e) : 0.f;
  if (!reverse) {
    for (int64_t s = 0; s < rank; ++s)
      acc = expf(all_G[(s * BH + bh) * D + dk]) * acc + all_S[s * BH * DD + e];
  } else {
    for (int64_t s = R - 1; s > rank; --s)
      acc = expf(all_G[(s * BH + bh) * D + dk]) * acc + all_S[s * BH * DD + e];
  }
  st_f(result, e, acc);
}

// Both results a rank needs from the gathered pairs in one launch: the state entering its slice (float32, for the
// correction of its stored states) and the state leaving the last slice in scan order (the whole sequence's
// hidden_final, or dhidden_init in the reverse direction).  The pairs may sit in one packed record per rank (what
// a single all-gather of [G | S] gives): gstride / sstride are the distances between ranks in floats.
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) sp_combine2_kernel(int64_t R, int64_t rank, int64_t BH, int64_t D,
                                                          const float* __restrict__ all_G, int64_t gstride,
                                                          const float* __restrict__ all_S, int64_t sstride,
                                                          const TI* __restrict__ init, float* __restrict__ entering,
                                                          TO* __restrict__ total, int reverse) {
  const int64_t DD = D * D;
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (e >= BH * DD) return;
  const int64_t bh = e / DD, dk = (e % DD) / D;
  float acc = init ? ld_f(init, e) : 0.f;
  for (int64_t i = 0; i < R; ++i) {
    const int64_t s = reverse ? R - 1 - i : i;
    if (s == rank && entering != nullptr) entering[e] = acc;
    acc = expf(all_G[s * gstride + bh * D + dk]) * acc + all_S[s * sstride + e];
  }
  if (total != nullptr) st_f(total, e, acc);
}

int launch_sp_combine2(cudaStream_t st, int64_t R, int64_t rank, int64_t BH, int64_t D, const float* all_G, int64_t gstride,
                       const float* all_S, int64_t sstride, const void* init, int init_bf16, float* entering, void* total,
                       int total_bf16, int reverse) {
  const int64_t n = BH * D * D;
  dim3 grid((unsigned)((n + 255) / 256));
  ProfScope ps("sp_combine_kernel", st);
  if (init_bf16 && total_bf16)
    sp_combine2_kernel<bf16, bf16><<<grid, 256, 0, st>>>(R, rank, BH, D, all_G, gstride, all_S, sstride, (const bf16*)init, entering, (bf16*)total, reverse);
  else if (init_bf16 && !total_bf16)
    sp_combine2_kernel<bf16, float><<<grid, 256, 0, st>>>(R, rank, BH, D, all_G, gstride, all_S, sstride, (const bf16*)init, entering, (float*)total, reverse);
  else if (!init_bf16 && total_bf16)
    sp_combine2_kernel<float, bf16><<<grid, 256, 0, st>>>(R, rank, BH, D, all_G, gstride, all_S, sstride, (const float*)init, entering, (bf16*)total, reverse);
  else
    sp_combine2_kernel<float, float><<<grid, 256, 0, st>>>(R, rank, BH, D, all_G, gstride, all_S, sstride, (const float*)init, entering, (float*)total, reverse);
  GLA_CHECK_LAUNCH();
  return GLA_OK;
}

int launch_sp_combine(cudaStream_t st, int64_t R, int64_t rank, int64_t BH, int64_t D, const float* all_G,
                      const float* all_S, const void* init, int init_bf16, void* result, int result_bf16,
                      int reverse) {
  int64_t n = BH * D * D;
  dim3 grid((unsigned)((n + 255) / 256));
  ProfScope ps("sp_combine_kernel", st);
  if (init_bf16 && result_bf16)
    sp_combine_kernel<bf16, bf16><<<grid, 256, 0, st>>>(R, rank, BH, D, all_G, all_S, (const bf16*)init, (bf16*)result, reverse);
  else if (init_bf16 && !result_bf16)
    sp_combine_kernel<bf16, float><<<grid, 256, 0, st>>>(R, rank, BH, D, all_G, all_S, (const bf16*)init, (float*)result, reverse);
  else if (!init_bf16 && result_bf16)
    sp_combine_kernel<float, bf16><<<grid, 256, 0, st>>>(R, rank, BH, D, all_G, all_S, (const float*)init, (bf16*)result, reverse);
  else
    sp_combine_kernel<float, float><<<grid, 256, 0, st>>>(R, rank, BH, D, all_G, all_S, (const float*)init, (float*)result, reverse);
  GLA_CHECK_LAUNCH();
  return GLA_OK;
}

}  // namespace gla
