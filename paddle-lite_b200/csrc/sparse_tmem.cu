// fp32 sparse_conv2d (1x1) with the activations in tensor memory.
//
// Per non-zero and pixel the walk reads one activation and does one multiply-add.  Out of shared memory that read is the
// bound: 4 bytes per multiply-add against 128 bytes per clock and SM keep the FMA pipes a quarter busy.  Tensor memory
// delivers 43 to 85 bytes per clock to each of the four schedulers (loads of four and eight columns, as measured below),
// 170 to 340 to the SM, so the activations live there: lane = pixel, column =
// (input channel, pixel group).  One tcgen05.ld of four (eight) columns gives every lane of a warp four (eight) pixels of one
// channel -- the column address is the non-zero's channel -- and feeds as many multiply-adds per lane.
//
// A CTA owns all 512 columns of its SM.  The four lane quadrants are independent teams of four warps: a team takes a group
// of 128 (256) pixels of the flattened batch, so images of any size fill it, loads 128 (64) input channels of it, and its
// warps walk the output channels in turn.  Layers of more channels go through in chunks; the partial sums wait in y as the
// fp32 values they are, so the sum of an output is formed exactly as the reference does: bias first, then one fused
// multiply-add per non-zero in ascending channel order.  While a team walks, half of the next group's channels are on their
// way into shared memory.
//
// Measured, 256 images: 128 -> 128 on 56 x 56 697 us out of shared memory, 376 here (12.7 instructions per non-zero and 128
// pixels, half of the issue slots; the HBM floor is 126 us); 32 -> 64 on 112 x 112 316 / 231 (floor 189).  Loads of four
// columns take 8 to 12 cycles per scheduler, of eight 12 to 16, which is why few channels (up to 64) go eight pixels a lane;
// above that the second chunk's round trip of the partial sums costs what the saved instructions give (385 / 387 us).
#include "sparse_tmem.cuh"

#include <algorithm>

#include "tc_device.cuh"

namespace plb {

namespace {

using namespace tc;

constexpr int kTeamWarps = 4;
constexpr int kThreads = 4 * kTeamWarps * 32;
constexpr int kAheadBytes = 16 * 512;  // per warp: what is prefetched of its channels through shared memory
template <int P>
constexpr int kBatchEntries = P == 8 ? 4 : 8;  // entries of a batch: 32 registers of activations
constexpr int kStageBytes = 4 * kTeamWarps * kAheadBytes;

struct Args {
  const float* x;
  const int4* rows;
  const int4* batches;
  float* y;
  long pixels;  // batch * hw
  int hw, cin, cout, chunks, slices, items;
  float alpha;
};

template <int P>
__device__ __forceinline__ void tm_ld(uint32_t addr, uint32_t* r) {
  if (P == 8)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4 % P]), "=r"(r[5 % P]), "=r"(r[6 % P]), "=r"(r[7 % P])
                 : "r"(addr)
                 : "memory");
  else
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void tm_st4(uint32_t addr, float4 v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(__float_as_uint(v.x)),
               "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w))
               : "memory");
}
// The wait names the registers the loads fill, so that nothing that reads them can be moved in front of it.
template <int N>
__device__ __forceinline__ void tm_wait(uint32_t (&r)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}
__device__ __forceinline__ void team_barrier(int quad) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + quad), "n"(32 * kTeamWarps) : "memory");
}

// The lists of non-zeros are read by every team for every group; activations and results pass through once.  Left alone,
// the stream of results evicts the lists from L1 (hit rate 20 %, the walk then waits for L2).
__device__ __forceinline__ int4 ld_list(const int4* p) {
  int4 v;
  asm volatile("ld.global.nc.L1::evict_last.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_stream4(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_stream(const float* p) {
  float v;
  asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void st_stream4(float* p, float4 v) {
  asm volatile("st.global.L1::no_allocate.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_stream(float* p, float v) {
  asm volatile("st.global.L1::no_allocate.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// A batch of R entries as it lies in memory: R columns, then every weight twice (the operand pairs of the packed
// multiply-add, ready in aligned registers).
template <int R>
__device__ __forceinline__ void load_columns(const int4* p, uint32_t (&col)[R]) {
#pragma unroll
  for (int i = 0; i < R / 4; ++i) {
    const int4 q = ld_list(p + i);
    col[4 * i] = q.x; col[4 * i + 1] = q.y; col[4 * i + 2] = q.z; col[4 * i + 3] = q.w;
  }
}

// The first N entries of a batch: N loads in flight, then the multiply-adds in order.  The columns were loaded ahead; once
// the loads are issued their registers take the columns of the batch at `next`.
template <int N, int P, int R>
__device__ __forceinline__ void walk(uint32_t taddr, uint32_t (&col)[R], const int4* batch, const int4* next, float2 (&acc)[P / 2]) {
  uint32_t v[P * N];
#pragma unroll
  for (int i = 0; i < N; ++i) tm_ld<P>(taddr + col[i], v + P * i);
  int4 w[(N + 1) / 2];
#pragma unroll
  for (int i = 0; i < (N + 1) / 2; ++i) w[i] = ld_list(batch + R / 4 + i);
  load_columns<R>(next, col);
  tm_wait(v);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float2 ww = i & 1 ? make_float2(__int_as_float(w[i >> 1].z), __int_as_float(w[i >> 1].w))
                            : make_float2(__int_as_float(w[i >> 1].x), __int_as_float(w[i >> 1].y));
#pragma unroll
    for (int k = 0; k < P / 2; ++k)
      acc[k] = __ffma2_rn(ww, make_float2(__uint_as_float(v[P * i + 2 * k]), __uint_as_float(v[P * i + 2 * k + 1])), acc[k]);
  }
}

// The P pixels of a lane.  VEC (planes of whole 16-byte groups): fours of consecutive ones; else 32 apart, so that a warp's
// accesses are whole 128-byte rows wherever an image starts.  Offsets are relative to the image of the group's first pixel
// (a group spans few images).  Pixels past the end read the last one and are not stored.
template <int P, bool VEC>
struct Pixels {
  static constexpr int kN = VEC ? P / 4 : P;
  const float* x0;
  float* y0;
  int x[kN], y[kN];
  uint32_t valid;
  __device__ __forceinline__ void set(const Args& a, int item, int lane) {
    const long base = static_cast<long>(item / a.slices) * (32 * P);
    const long n0 = base / a.hw;
    const int p0 = static_cast<int>(base - n0 * a.hw);
    x0 = a.x + n0 * a.cin * a.hw;
    y0 = a.y + n0 * a.cout * a.hw;
    const long left = a.pixels - base;
    valid = 0;
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      int g = VEC ? 4 * (lane + 32 * j) : lane + 32 * j;
      if (g < left) valid |= 1u << j;
      else g = static_cast<int>(left) - (VEC ? 4 : 1);
      const int n = (p0 + g) / a.hw, p = p0 + g - n * a.hw;
      x[j] = n * a.cin * a.hw + p;
      y[j] = n * a.cout * a.hw + p;
    }
  }
  __device__ __forceinline__ float4 load_x(long plane, int k) const {
    const float* src = x0 + plane;
    if (VEC) return ld_stream4(src + x[k % kN]);
    return make_float4(ld_stream(src + x[4 * k % kN]), ld_stream(src + x[(4 * k + 1) % kN]), ld_stream(src + x[(4 * k + 2) % kN]),
                       ld_stream(src + x[(4 * k + 3) % kN]));
  }
  __device__ __forceinline__ void prefetch_x(long plane, int k, uint32_t dst) const {
    const float* src = x0 + plane;
    if (VEC) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + x[k % kN]) : "memory");
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * j), "l"(src + x[(4 * k + j) % kN]) : "memory");
    }
  }
  __device__ __forceinline__ float4 load_y(long plane, int k) const {
    const float* src = y0 + plane;
    if (VEC) return __ldcg(reinterpret_cast<const float4*>(src + y[k % kN]));
    return make_float4(__ldcg(src + y[4 * k % kN]), __ldcg(src + y[(4 * k + 1) % kN]), __ldcg(src + y[(4 * k + 2) % kN]),
                       __ldcg(src + y[(4 * k + 3) % kN]));
  }
  __device__ __forceinline__ void store_y(long plane, int k, float4 v) const {
    float* dst = y0 + plane;
    if (VEC) {
      if (valid >> k & 1) st_stream4(dst + y[k % kN], v);
      return;
    }
    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (valid >> (4 * k + j) & 1) st_stream(dst + y[(4 * k + j) % kN], e[j]);
  }
};

// P pixels per lane: 512 / P channels at a time.
template <int P, bool VEC, int ACT>
__global__ void __launch_bounds__(kThreads, 1) sparse_f32_tmem_kernel(const Args a) {
  constexpr int kChannels = 512 / P;
  constexpr int kWarpChannels = kChannels / kTeamWarps;     // channels of a chunk that one warp loads
  constexpr int kAhead = kAheadBytes / (32 * 4 * P);        // of those, how many are prefetched
  constexpr int R = kBatchEntries<P>;
  constexpr int kBatchWords = 3 * R / 4;                    // 16-byte words of a batch
  extern __shared__ __align__(128) uint8_t stage_mem[];
  __shared__ uint32_t tmem_slot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quad = warp & 3, member = warp >> 2;  // (a warp reaches the tensor-memory lanes of its quadrant only)
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
  const uint32_t stage = smem_u32(stage_mem) + warp * kAheadBytes + lane * 16;  // this lane's bytes: nobody else touches them
  pdl_sync_with_previous_kernel();

  const int stride = 4 * gridDim.x;
  int item = quad * gridDim.x + blockIdx.x, chunk = 0;
  Pixels<P, VEC> px;
  auto prefetch = [&](const Pixels<P, VEC>& of, int of_chunk) {
    const int c0 = of_chunk * kChannels + member;
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int c = c0 + kTeamWarps * j;
      if (c >= a.cin) break;
#pragma unroll
      for (int k = 0; k < P / 4; ++k) of.prefetch_x(static_cast<long>(c) * a.hw, k, stage + (j * (P / 4) + k) * 512);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (item < a.items) {
    px.set(a, item, lane);
    prefetch(px, 0);
  }
  while (item < a.items) {
    // every walk of the previous chunk has read what it needs
    tc_fence_before();
    team_barrier(quad);
    tc_fence_after();
    {
      const int c0 = chunk * kChannels + member;
      constexpr int kBatch = 32 / P;
#pragma unroll 1
      for (int j0 = kAhead; j0 < kWarpChannels && c0 + kTeamWarps * j0 < a.cin; j0 += kBatch) {
        float4 v[kBatch][P / 4];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
          const int c = c0 + kTeamWarps * (j0 + j);
#pragma unroll
          for (int k = 0; k < P / 4; ++k) v[j][k] = px.load_x(static_cast<long>(c < a.cin ? c : a.cin - 1) * a.hw, k);
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j)
#pragma unroll
          for (int k = 0; k < P / 4; ++k) tm_st4(taddr + P * (member + kTeamWarps * (j0 + j)) + 4 * k, v[j][k]);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        if (c0 + kTeamWarps * j >= a.cin) break;
#pragma unroll
        for (int k = 0; k < P / 4; ++k)
          tm_st4(taddr + P * (member + kTeamWarps * j) + 4 * k, lds128f(stage + (j * (P / 4) + k) * 512));
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    team_barrier(quad);
    tc_fence_after();
    // the next chunk's first channels travel while this one is walked
    const bool last_chunk = chunk + 1 == a.chunks;
    const int next_item = last_chunk ? item + stride : item, next_chunk = last_chunk ? 0 : chunk + 1;
    Pixels<P, VEC> next = px;
    if (next_item < a.items) {
      if (last_chunk) next.set(a, next_item, lane);
      prefetch(next, next_chunk);
    }
    const int slice = item % a.slices;
    const int oc1 = static_cast<int>(static_cast<long>(a.cout) * (slice + 1) / a.slices);
    int oc = static_cast<int>(static_cast<long>(a.cout) * slice / a.slices) + member;
    const int4* rows = a.rows + static_cast<long>(chunk) * a.cout;
    const int4 none = make_int4(0, 0, 0, 0);
    int4 row = oc < oc1 ? ld_list(rows + oc) : none;
    uint32_t col[R];
    load_columns<R>(a.batches + row.x, col);
    for (; oc < oc1; oc += kTeamWarps) {
      const int4 row_next = oc + kTeamWarps < oc1 ? ld_list(rows + oc + kTeamWarps) : none;
      const long plane = static_cast<long>(oc) * a.hw;
      float2 acc[P / 2];
      if (chunk == 0) {
        const float b = __int_as_float(row.z);
#pragma unroll
        for (int k = 0; k < P / 2; ++k) acc[k] = make_float2(b, b);
      } else {
#pragma unroll
        for (int k = 0; k < P / 4; ++k) {
          const float4 s = px.load_y(plane, k);
          acc[2 * k] = make_float2(s.x, s.y);
          acc[2 * k + 1] = make_float2(s.z, s.w);
        }
      }
      const int4* p = a.batches + row.x;
      const int4* p_next = a.batches + row_next.x;
      int n = row.y;
      for (; n > R; n -= R, p += kBatchWords) walk<R, P, R>(taddr, col, p, p + kBatchWords, acc);
      switch (n) {
        case 0: load_columns<R>(p_next, col); break;
        case 1: walk<1, P, R>(taddr, col, p, p_next, acc); break;
        case 2: walk<2, P, R>(taddr, col, p, p_next, acc); break;
        case 3: walk<3, P, R>(taddr, col, p, p_next, acc); break;
        case 4: walk<4, P, R>(taddr, col, p, p_next, acc); break;
        case 5: walk<R == 8 ? 5 : R, P, R>(taddr, col, p, p_next, acc); break;  // (5 to 8: batches of eight only)
        case 6: walk<R == 8 ? 6 : R, P, R>(taddr, col, p, p_next, acc); break;
        case 7: walk<R == 8 ? 7 : R, P, R>(taddr, col, p, p_next, acc); break;
        default: walk<R, P, R>(taddr, col, p, p_next, acc); break;
      }
      row = row_next;
#pragma unroll
      for (int k = 0; k < P / 4; ++k) {
        float4 s = make_float4(acc[2 * k].x, acc[2 * k].y, acc[2 * k + 1].x, acc[2 * k + 1].y);
        if (last_chunk) {
          s.x = act_apply(s.x, ACT, a.alpha);
          s.y = act_apply(s.y, ACT, a.alpha);
          s.z = act_apply(s.z, ACT, a.alpha);
          s.w = act_apply(s.w, ACT, a.alpha);
        }
        px.store_y(plane, k, s);
      }
    }
    px = next;
    item = next_item;
    chunk = next_chunk;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
}

typedef void (*Kernel)(const Args);
template <int P, bool VEC>
Kernel pick(int act) {
  switch (act) {
    case PLB_ACT_RELU: return sparse_f32_tmem_kernel<P, VEC, PLB_ACT_RELU>;
    case PLB_ACT_RELU6: return sparse_f32_tmem_kernel<P, VEC, PLB_ACT_RELU6>;
    case PLB_ACT_LEAKY: return sparse_f32_tmem_kernel<P, VEC, PLB_ACT_LEAKY>;
    default: return sparse_f32_tmem_kernel<P, VEC, PLB_ACT_NONE>;
  }
}

}  // namespace

bool sparse_tmem_build(int cin, int cout, long hw, const std::vector<int>& row_ptr, const std::vector<int>& col,
                       const std::vector<float>& val, const float* bias, SparseTmemLists* out) {
  if (hw > (1L << 30) / std::max(cin, cout)) return false;
  out->pixels = cin <= 64 ? 8 : 4;
  const int channels = 512 / out->pixels, chunks = (cin + channels - 1) / channels;
  out->rows.assign(static_cast<size_t>(chunks) * cout, make_int4(0, 0, 0, 0));
  out->batches.clear();
  const int entries = out->pixels == 8 ? kBatchEntries<8> : kBatchEntries<4>;
  std::vector<int> at(row_ptr.begin(), row_ptr.end() - 1);  // next entry of each row
  for (int k = 0; k < chunks; ++k)
    for (int oc = 0; oc < cout; ++oc) {
      int4& row = out->rows[static_cast<size_t>(k) * cout + oc];
      row.x = static_cast<int>(out->batches.size() / 4);
      if (bias) memcpy(&row.z, &bias[oc], 4);
      for (int& t = at[oc]; t < row_ptr[oc + 1] && col[t] < (k + 1) * channels; ++t) {
        if (t > row_ptr[oc] && col[t] < col[t - 1]) return false;
        int bits;
        memcpy(&bits, &val[t], 4);
        const int i = row.y % entries;
        if (i == 0) out->batches.resize(out->batches.size() + 3 * entries, 0);
        int* batch = &out->batches[out->batches.size() - 3 * entries];
        batch[i] = out->pixels * (col[t] - k * channels);
        batch[entries + 2 * i] = batch[entries + 2 * i + 1] = bits;
        ++row.y;
      }
    }
  for (int oc = 0; oc < cout; ++oc)
    if (at[oc] != row_ptr[oc + 1]) return false;
  out->batches.resize(out->batches.size() + 3 * entries, 0);
  return true;
}

namespace {

bool aligned16(const SparseTmemProblem& p) {
  return p.hw % 4 == 0 && ((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.y)) & 15) == 0;
}

// Few pixel groups: several teams share one, each with a slice of the output channels (and its own copy of the activations).
// The number of slices that finishes first by the cycles of a load, a non-zero and a row.
struct Split {
  int slices;
  long waves;  // items per team, rounded up
};
Split split(const SparseTmemProblem& p, int sm_count) {
  const int chunks = (p.cin + 512 / p.pixels - 1) / (512 / p.pixels);
  const long groups = (static_cast<long>(p.batch) * p.hw + 32 * p.pixels - 1) / (32 * p.pixels), teams = 4L * sm_count;
  Split best = {1, 1};
  double best_cost = 0;
  for (int s = 1; s <= 64 && (s == 1 || s * kTeamWarps <= p.cout); ++s) {
    const long waves = (groups * s + teams - 1) / teams;
    const double cost = waves * (5.0 * p.pixels * p.cin + 3.0 * p.pixels * p.nnz / s + 60.0 * chunks * ((p.cout + s - 1) / s));
    if (s == 1 || cost < best_cost) {
      best_cost = cost;
      best = {s, waves};
    }
  }
  return best;
}

}  // namespace

// Costs in us, fitted to 500 layers (32 to 1024 channels, 4 to 112 pixels a side, 1 to 256 images, densities 0.05 to 0.35); the
// choice is 0.2 % from the faster kernel over all of them.  Measured, here / the other one: 137 -> 288 on 98 x 98, 47 images
// 885 / 838; 160 -> 220 on 16 x 16, 164 images 59 / 47, but 159 -> 160 on 9520 pixels, 2 images 26 / 34; 329 -> 43 on 16 x 16,
// 7 images 12.9 / 8.8; 192 -> 82 on 5 x 5, 12 images 16 / 4.9; 448 -> 150 on 4225 pixels, 4 images 100 / 196.
bool sparse_tmem_better(const SparseTmemProblem& p, int sm_count) {
  const bool vec = aligned16(p), tiles = vec && p.cin <= 512;
  if (p.batch > 65535 || (!tiles && p.cout > 65535)) return true;  // beyond the other kernels' grids
  // against whole channels of a few pixels per thread: 130 -> 70 on 19 x 23, 64 images 41 / 135; faster on all 115 measured
  if (!tiles && p.cin <= 160) return true;
  const int chunks = (p.cin + 512 / p.pixels - 1) / (512 / p.pixels);
  const Split sp = split(p, sm_count);
  const double w = static_cast<double>(sp.waves), nnz = static_cast<double>(p.nnz);
  const double load = w * p.pixels * p.cin, walk = w * p.pixels * nnz / sp.slices;
  const double rows = w * chunks * ((p.cout + sp.slices * kTeamWarps - 1) / (sp.slices * kTeamWarps));
  const double partial = (chunks - 1.0) * p.batch * p.hw * p.cout;  // sums that wait in y
  const double here = vec ? 3.0 + 4.8e-3 * load + 2.0e-3 * walk + 0.36 * rows + 0.54 * chunks + 5.8e-7 * partial
                          : 3.8 + 1.01e-2 * load + 1.9e-3 * walk + 0.52 * rows + 0.79 * chunks + 3.3e-7 * partial + 0.38 * w;
  double there;
  if (tiles) {  // tiles of 4 * pg pixels in shared memory, two blocks per SM: every block walks all non-zeros
    const int pg = p.cin <= 128 ? 32 : p.cin <= 256 ? 16 : 8;
    const long blocks = static_cast<long>(p.batch) * ((p.hw + 4 * pg - 1) / (4 * pg)), slots = 2L * sm_count;
    const double walks = static_cast<double>((blocks + slots - 1) / slots) * nnz;
    there = 0.95 * (pg == 32 ? 5.1 + 1.06e-2 * walks : pg == 16 ? 5.6 + 5.5e-3 * walks : 8.5 + 3.0e-3 * walks);
  } else {  // one thread per output
    there = 2.6 + 0.067 * nnz / p.cout + 4.75e-7 * nnz * p.batch * ((p.hw + 31) / 32 * 32) +
            4.7e-4 * p.cout * p.batch * ((p.hw + 255) / 256);
  }
  return here < there;
}

int sparse_tmem_launch(plb_ctx* ctx, const SparseTmemProblem& p) {
  Args a;
  a.x = p.x; a.rows = static_cast<const int4*>(p.rows); a.batches = static_cast<const int4*>(p.batches); a.y = p.y;
  a.pixels = static_cast<long>(p.batch) * p.hw;
  a.hw = p.hw; a.cin = p.cin; a.cout = p.cout; a.alpha = p.alpha;
  const int channels = 512 / p.pixels;
  a.chunks = (p.cin + channels - 1) / channels;
  if (a.pixels == 0) return PLB_OK;
  const long groups = (a.pixels + 32 * p.pixels - 1) / (32 * p.pixels), teams = 4L * ctx->sm_count;
  a.slices = split(p, ctx->sm_count).slices;
  if (groups * a.slices + teams > 0x7fffffffL) return fail(PLB_E_UNSUPPORTED, "sparse grid too large");
  a.items = static_cast<int>(groups * a.slices);
  const bool vec = aligned16(p);
  Kernel kern = p.pixels == 8 ? (vec ? pick<8, true>(p.act) : pick<8, false>(p.act))
                              : (vec ? pick<4, true>(p.act) : pick<4, false>(p.act));
  PLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kStageBytes));
  PLB_CUDA(launch_kernel(kern, dim3(std::min<long>(a.items, ctx->sm_count)), dim3(kThreads), kStageBytes, ctx->stream, a));
  ctx->launches++;
  ctx->sparse_tmem_launches++;
  return PLB_OK;
}

}  // namespace plb
