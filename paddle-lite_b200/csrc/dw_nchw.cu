// Depthwise convolution on NCHW tensors as they are.
//
// By bytes the layer is one read of x and one write of y; staged channels-last (transposing pass, channels-last kernel,
// transposing pass back) it is three of each.  Here a block takes whole consecutive planes of the tensor, which is one
// contiguous piece of memory whatever the image size: it is copied into shared memory with 16-byte loads, computed there,
// and the results, staged the same way, leave with 16-byte stores.  Neither image rows nor planes need any alignment.
// In this layout four neighbouring pixels of a channel are one word, so the windows of the dp4a need no transposes: a
// thread owns four output columns of one plane and slides down a strip of its rows; an input row is two to four words,
// shifted into place once, and meets all filter rows it belongs to; accumulator rows rotate through registers.
// Measured against the staged passes: 5x5, 736 channels on 49 x 49, 9 images: 251 -> 41 us (16 MB in, 16 MB out); 3x3,
// 28 channels on 13 x 13, one image: 8.6 -> 4.2 us.
#include "dw_nchw.cuh"

#include <algorithm>

#include "dw_device.cuh"
#include "igemm_tc.cuh"
#include "tc_device.cuh"

namespace plb {

namespace {

using namespace dw;

constexpr int kThreads = 256;
constexpr int kSlack = 32;              // bytes in front of and behind the staged input that a row's word loads may touch
constexpr int kBlockBytes = 36 * 1024;  // shared memory a block aims at: five or six blocks per SM hide each other's copies
constexpr int kMaxBytes = 110 * 1024;   // ... and the most one may take (two blocks per SM)

struct Args {
  const int8_t* x;
  const int8_t* w;
  const float* scale;
  const float* bias;
  void* y;
  long planes;
  float alpha;
  int c, h, w_px, ho, wo, pad_t, pad_l, cg_pad;
  int per_block;              // planes of a block
  int strip, strips, quads;   // output rows per strip, strips of a plane, groups of four columns of a row
  int par_off, out_off;       // shared memory: parameters of the block's planes, staged results
};

template <int K>
struct PlaneParams {
  uint32_t lo[K], hi[K];  // filter rows: taps 0..3 and tap 4
  float scale, bias;
};

// A strip of four output columns.  K x K filter, stride S.  `row` = byte offset (shared memory) of input row `ih`, first
// column of the first window; rows outside the image and columns outside it (masks) read as zero.
template <int K, int S, int MODE, int ACT, bool SMALL>
__device__ __forceinline__ void strip4(const Args& a, const PlaneParams<K>& pp, const uint8_t* smem, int row, int ih, int iw,
                                       int rows, uint8_t* out, int ncols) {
  constexpr int kBytes = 3 * S + K;           // input bytes under four windows
  constexpr int kWords = (kBytes + 3) / 4;
  constexpr int kLive = (K + S - 1) / S;      // output rows under accumulation at a time
  constexpr int kPeriod = kLive * S;
  uint32_t wlo[K], whi[K];
#pragma unroll
  for (int r = 0; r < K; ++r) {
    wlo[r] = pp.lo[r];
    if (K > 4) whi[r] = pp.hi[r];
  }
  const float scale = pp.scale, bias = pp.bias;
  const float ub = MODE == OUT_I8 ? tc::quant_upper_bound<ACT>(a.alpha) : 0.f;
  uint32_t mask[kWords];
#pragma unroll
  for (int i = 0; i < kWords; ++i) {
    mask[i] = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
      if (iw + 4 * i + b >= 0 && iw + 4 * i + b < a.w_px) mask[i] |= 0xffu << (8 * b);
  }
  int acc[kLive][4];
#pragma unroll
  for (int l = 0; l < kLive; ++l)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[l][j] = kDwMagic;
  const int in_rows = (rows - 1) * S + K;
  const int out_row = a.wo * (MODE == OUT_I8 ? 1 : 4);
  for (int base = 0; base < in_rows; base += kPeriod) {
#pragma unroll
    for (int p = 0; p < kPeriod; ++p) {
      const int i = base + p;
      uint32_t t[kWords + 1];
      const bool live = i < in_rows && static_cast<unsigned>(ih + i) < static_cast<unsigned>(a.h);
      const uint32_t* src = reinterpret_cast<const uint32_t*>(smem + (row & ~3));
#pragma unroll
      for (int v = 0; v <= kWords; ++v) t[v] = live ? src[v] : 0u;
      uint32_t d[kWords];
#pragma unroll
      for (int v = 0; v < kWords; ++v) d[v] = __funnelshift_r(t[v], t[v + 1], 8 * (row & 3)) & mask[v];
      row += a.w_px;
      uint32_t win[4], fifth[4];
      if (S == 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          win[j] = __funnelshift_r(d[0], d[1], 8 * j);
          fifth[j] = d[1] >> (8 * j);
        }
      } else {
        win[0] = d[0]; win[1] = __funnelshift_r(d[0], d[1], 16); win[2] = d[1]; win[3] = __funnelshift_r(d[1], d[kWords - 1], 16);
        fifth[0] = d[1]; fifth[1] = d[1] >> 16; fifth[2] = d[kWords - 1]; fifth[3] = d[kWords - 1] >> 16;
      }
#pragma unroll
      for (int r = 0; r < K; ++r) {
        if ((p + kPeriod * K - r) % S != 0) continue;
        const int l = (p + kPeriod * K - r) / S % kLive;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[l][j] = __dp4a(static_cast<int>(win[j]), static_cast<int>(wlo[r]), r == 0 ? kDwMagic : acc[l][j]);
          if (K > 4) acc[l][j] = __dp4a(static_cast<int>(fifth[j]), static_cast<int>(whi[r]), acc[l][j]);
        }
      }
      if ((p + kPeriod * K - (K - 1)) % S != 0) continue;
      // filter row K - 1 was the last one of this output row
      const int l = (p + kPeriod * K - (K - 1)) / S % kLive;
      const int num = i - (K - 1);
      if (num >= 0 && i < in_rows) {
        if (MODE == OUT_ACC) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < ncols) reinterpret_cast<int*>(out)[j] = acc[l][j] - kDwMagic;
        } else {
          float v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = fmaf(__int_as_float(acc[l][j]) - tc::kRoundMagic, scale, bias);
          if (MODE == OUT_I8) {
            const uint32_t q = tc::requant_pack4<ACT, SMALL>(make_float2(v[0], v[1]), make_float2(v[2], v[3]), a.alpha, ub);
            if (ncols >= 4 && (reinterpret_cast<uintptr_t>(out) & 3) == 0) {
              *reinterpret_cast<uint32_t*>(out) = q;
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (j < ncols) out[j] = static_cast<uint8_t>(q >> (8 * j));
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = tc::act_f32<ACT>(v[j], a.alpha);
            if (ncols >= 4 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
              *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (j < ncols) reinterpret_cast<float*>(out)[j] = v[j];
            }
          }
        }
        out += out_row;
      }
    }
  }
}

template <int K, int S, int MODE, int ACT, bool SMALL>
__global__ void __launch_bounds__(kThreads) dw_nchw_kernel(const Args a) {
  extern __shared__ __align__(16) uint8_t smem[];
  pdl_sync_with_previous_kernel();
  constexpr int EB = MODE == OUT_I8 ? 1 : 4;
  const long p0 = static_cast<long>(blockIdx.x) * a.per_block;
  const int planes = static_cast<int>(min(static_cast<long>(a.per_block), a.planes - p0));
  const int hw = a.h * a.w_px, howo = a.ho * a.wo;
  // copy in: 16-byte pieces of global memory, at the same offset from a 16-byte boundary in shared memory
  const uintptr_t x_first = reinterpret_cast<uintptr_t>(a.x), x_end = x_first + a.planes * static_cast<long>(hw);
  const uintptr_t src = x_first + p0 * hw;
  const int lead = static_cast<int>(src & 15);
  const int pieces = (lead + planes * hw + 15) / 16;
  uint8_t* in = smem + kSlack;
  for (int i = threadIdx.x; i < pieces; i += kThreads) {
    const uintptr_t at = src - lead + 16l * i;
    if (at >= x_first && at + 16 <= x_end) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(in + 16 * i)), "l"(at) : "memory");
    } else {  // a piece that reaches past the tensor
      for (int b = 0; b < 16; ++b)
        if (at + b >= x_first && at + b < x_end) in[16 * i + b] = *reinterpret_cast<const uint8_t*>(at + b);
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  PlaneParams<K>* params = reinterpret_cast<PlaneParams<K>*>(smem + a.par_off);
  for (int i = threadIdx.x; i < planes; i += kThreads) {
    const int ch = static_cast<int>((p0 + i) % a.c);
    PlaneParams<K> pp;
#pragma unroll
    for (int r = 0; r < K; ++r) {
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int s = 0; s < K; ++s) {
        const uint32_t tap = static_cast<uint8_t>(__ldg(a.w + static_cast<long>(r * K + s) * a.cg_pad + ch));
        if (s < 4) lo |= tap << (8 * s);
        else hi = tap;
      }
      pp.lo[r] = lo;
      pp.hi[r] = hi;
    }
    pp.scale = MODE == OUT_ACC ? 0.f : __ldg(a.scale + ch);
    pp.bias = MODE == OUT_ACC ? 0.f : __ldg(a.bias + ch);
    params[i] = pp;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // results go to the same offset from a 16-byte boundary as their place in global memory
  const uintptr_t dst = reinterpret_cast<uintptr_t>(a.y) + p0 * howo * EB;
  const int out_lead = static_cast<int>(dst & 15);
  uint8_t* out = smem + a.out_off + out_lead;
  const int per_plane = a.strips * a.quads;
  for (int u = threadIdx.x; u < planes * per_plane; u += kThreads) {
    const int plane = u / per_plane, in_plane = u - plane * per_plane;
    const int strip = in_plane / a.quads, quad = in_plane - strip * a.quads;
    const int oh = strip * a.strip, ow = quad * 4;
    const int ih = oh * S - a.pad_t, iw = ow * S - a.pad_l;
    strip4<K, S, MODE, ACT, SMALL>(a, params[plane], smem, kSlack + lead + plane * hw + ih * a.w_px + iw, ih, iw, min(a.strip, a.ho - oh),
                            out + (static_cast<long>(plane) * howo + oh * a.wo + ow) * EB, a.wo - ow);
  }
  __syncthreads();
  const int bytes = planes * howo * EB;
  for (int i = threadIdx.x; i < (out_lead + bytes + 15) / 16; i += kThreads) {
    const uint8_t* from = smem + a.out_off + 16 * i;
    uint8_t* to = reinterpret_cast<uint8_t*>(dst - out_lead + 16l * i);
    if (16 * i >= out_lead && 16 * i + 16 <= out_lead + bytes) {
      *reinterpret_cast<uint4*>(to) = *reinterpret_cast<const uint4*>(from);
    } else {  // shared with the neighbouring block
      for (int b = 0; b < 16; ++b)
        if (16 * i + b >= out_lead && 16 * i + b < out_lead + bytes) to[b] = from[b];
    }
  }
}

typedef void (*Kernel)(const Args);
template <int K, int S, int MODE, bool SMALL>
Kernel pick_act(int act) {
  switch (act) {
    case PLB_ACT_RELU: return dw_nchw_kernel<K, S, MODE, PLB_ACT_RELU, SMALL>;
    case PLB_ACT_RELU6: return dw_nchw_kernel<K, S, MODE, PLB_ACT_RELU6, SMALL>;
    case PLB_ACT_LEAKY: return dw_nchw_kernel<K, S, MODE, PLB_ACT_LEAKY, SMALL>;
    default: return dw_nchw_kernel<K, S, MODE, PLB_ACT_NONE, SMALL>;
  }
}
template <int K, int S>
Kernel pick(int mode, bool small, int act) {
  if (mode == OUT_ACC) return dw_nchw_kernel<K, S, OUT_ACC, PLB_ACT_NONE, false>;
  if (mode == OUT_F32) return pick_act<K, S, OUT_F32, false>(act);
  return small ? pick_act<K, S, OUT_I8, true>(act) : pick_act<K, S, OUT_I8, false>(act);
}

// Shared memory of a block of n planes: {slack, input, slack} {parameters} {output}.
struct Layout {
  long par_off, out_off, bytes;
};
Layout layout(const ConvGeom& g, int mode, long n) {
  Layout l;
  const long params = g.kh == 3 ? sizeof(PlaneParams<3>) : sizeof(PlaneParams<5>);
  l.par_off = (kSlack + 16 + n * g.h * g.w + kSlack + 15) / 16 * 16;
  l.out_off = (l.par_off + n * params + 15) / 16 * 16;
  l.bytes = l.out_off + 16 + (n * g.ho * g.wo * (mode == OUT_I8 ? 1 : 4) + 15) / 16 * 16;
  return l;
}

}  // namespace

bool dw_nchw_supported(const ConvGeom& g, int mode) {
  if (mode != OUT_I8 && mode != OUT_F32 && mode != OUT_ACC) return false;
  if (g.kh != g.kw || (g.kh != 3 && g.kh != 5) || g.stride_h != g.stride_w || g.stride_h < 1 || g.stride_h > 2) return false;
  if (g.dil_h != 1 || g.dil_w != 1) return false;
  // a row's words start at most pad_l bytes in front of its plane (rows above the image are not read) and end within the
  // slack behind it for the columns that four-column groups add to a row
  if (g.pad_l > kSlack - 8) return false;
  const long last = static_cast<long>((g.wo + 3) / 4 * 4 - 1) * g.stride_w - g.pad_l + g.kw;
  if (last - g.w > kSlack - 12) return false;
  return static_cast<long>(g.h) * g.w <= kMaxBytes && static_cast<long>(g.ho) * g.wo <= kMaxBytes &&
         layout(g, mode, 1).bytes <= kMaxBytes;
}

int dw_nchw_launch(plb_ctx* ctx, const ConvGeom& g, const int8_t* x, const int8_t* w_tc, const OutSpec& out) {
  Args a;
  a.x = x; a.w = w_tc; a.scale = out.epi.scale; a.bias = out.epi.bias; a.y = out.y; a.alpha = out.epi.alpha;
  a.planes = static_cast<long>(g.batch) * g.cout;
  a.c = g.cout; a.h = g.h; a.w_px = g.w; a.ho = g.ho; a.wo = g.wo; a.pad_t = g.pad_t; a.pad_l = g.pad_l; a.cg_pad = g.cg_pad;
  // planes per block: up to the shared memory it aims at, fewer while there are not four blocks per SM
  long n = std::max<long>(1, (a.planes + 4L * ctx->sm_count - 1) / (4L * ctx->sm_count));
  while (n > 1 && layout(g, out.mode, n).bytes > kBlockBytes) n = n > 8 ? n * 7 / 8 : n - 1;
  a.per_block = static_cast<int>(n);
  a.quads = (g.wo + 3) / 4;
  a.strip = g.ho;
  while (a.strip > 4 && n * a.quads * ((g.ho + a.strip - 1) / a.strip) < kThreads) a.strip = (a.strip + 1) / 2;
  a.strips = (g.ho + a.strip - 1) / a.strip;
  const Layout l = layout(g, out.mode, n);
  a.par_off = static_cast<int>(l.par_off);
  a.out_off = static_cast<int>(l.out_off);
  const long blocks = (a.planes + n - 1) / n;
  if (blocks > 0x7fffffffL) return fail(PLB_E_UNSUPPORTED, "depthwise: too many blocks");
  const bool small = out.epi.acc_small != 0;
  Kernel k = g.kh == 3 ? (g.stride_h == 1 ? pick<3, 1>(out.mode, small, out.epi.act) : pick<3, 2>(out.mode, small, out.epi.act))
                       : (g.stride_h == 1 ? pick<5, 1>(out.mode, small, out.epi.act) : pick<5, 2>(out.mode, small, out.epi.act));
  PLB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBytes));
  PLB_CUDA(launch_kernel(k, dim3(static_cast<unsigned>(blocks)), dim3(kThreads), static_cast<size_t>(l.bytes), ctx->stream, a));
  ctx->launches++;
  return PLB_OK;
}

}  // namespace plb
