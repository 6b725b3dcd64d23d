// Learned initial guess for the per-kx Poisson problems: a small U-Net on
// the problems' right-hand sides, trained on (rhs, solution) pairs that the
// solver itself produced, and its kernels.
//
// Network (per problem, one image): 4 levels of two 3x3 convolutions with
// ReLU and C channels at every level, 2x2 average pooling down,
// nearest-neighbour upsampling up, the skip tensor joined as channels
// C..2C-1 of the first decoder convolution, and a final 3x3 convolution to
// one channel.  Activations are BF16 (NHWC, a one-pixel zero border around
// every image so that a shifted read never needs a bounds check); weights
// are kept in FP32 (master copy, Adam moments) and rounded to BF16 when a
// tile is staged; gradients are FP32.
//
// The three convolution passes are the GEMMs
//   forward     M = pixels, N = Cout,  K = 9 Cin     A = shifted input, B = W
//   input grad  M = pixels, N = Cin,   K = 9 Cout    A = shifted dZ,    B = W^T
//   weight grad M = Cout,   N = 9 Cin, K = pixels    A = dZ^T,          B = shifted input
// (the weight gradient is split over pixels and summed with FP32 atomics).
// With channel counts that are multiples of 16 the first two run on tcgen05
// (k_conv_tc) and the third on k_conv_dw; the first and the last layer have
// kernels of their own; k_conv_gemm (mma.sync, element-wise operand loaders)
// takes every other channel count, and every layer with set_tcgen05(0).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "ek_internal.h"
#include "ek_unet.h"

namespace ek {
namespace unet {

constexpr int BM = 64, BN = 64, BK = 32, PAD = 8, NT = 128;

__device__ __forceinline__ unsigned short f2bf(float f) {
  // round to nearest even; NaN kept quiet
  unsigned u = __float_as_uint(f);
  if ((u & 0x7f800000u) == 0x7f800000u && (u & 0x7fffffu)) return (unsigned short)((u >> 16) | 0x40u);
  u += 0x7fffu + ((u >> 16) & 1u);
  return (unsigned short)(u >> 16);
}
__device__ __forceinline__ float bf2f(unsigned short h) { return __uint_as_float((unsigned)h << 16); }

// Image geometry: N images of H x W interior pixels, stored (H+2) x (W+2)
// with a zero border, C channels innermost.
struct Img {
  int N, H, W;
  __device__ __forceinline__ size_t at(int n, int y, int x, int C) const {
    return (((size_t)n * (H + 2) + (y + 1)) * (W + 2) + (x + 1)) * C;
  }
};

// One convolution's operands.  The input is the channel concatenation of
// x1 (c1 channels) and x2 (c2 channels, may be 0); activations BF16.
struct ConvArgs {
  Img g;
  const unsigned short *x1, *x2;
  int c1, c2, cin, cout;
  const float *w;       // [cout][9][cin]
  const float *bias;    // [cout]
  // forward output
  unsigned short *y;    // BF16 [.. cout], or
  float *y32;           // FP32 one channel (the last layer), no border
  int relu;
  // input-gradient pass
  const float *dz;      // FP32 [.. cout] with border
  float *dx1, *dx2;     // FP32 [.. c1], [.. c2] with border
  const unsigned short *m1, *m2;  // ReLU masks (the activations x1, x2), or null
  // weight-gradient pass
  const unsigned short *dzb;  // dZ rounded to BF16, bordered (the tensor-core passes' operand)
  unsigned short *dxb1, *dxb2;  // BF16 copies of dx1 / dx2 (null: none)
  float *dw;            // [cout][9][cin] accumulated
  int kchunk;           // pixels per block along K
};

__device__ __forceinline__ void pix(const Img &g, long m, int &n, int &y, int &x) {
  // 32-bit divisions while the pixel count allows (a 64-bit one is a long
  // integer sequence, a few times the cost of these kernels' own work)
  const long hw = (long)g.H * g.W;
  n = ((m | hw) >> 32) ? (int)(m / hw) : (int)((unsigned)m / (unsigned)hw);
  const int r = (int)(m - (long)n * hw);
  y = r / g.W;
  x = r - y * g.W;
}

__device__ __forceinline__ float act_in(const ConvArgs &a, int n, int y, int x, int ci) {
  if (ci < a.c1) return bf2f(a.x1[a.g.at(n, y, x, a.c1) + ci]);
  return bf2f(a.x2[a.g.at(n, y, x, a.c2) + (ci - a.c1)]);
}

enum { PASS_FWD = 0, PASS_DX = 1, PASS_DW = 2 };

template <int PASS>
struct Ops;

// forward: A(m = pixel, k = tap*cin + ci) = x[pixel + offset(tap)][ci]
template <>
struct Ops<PASS_FWD> {
  static __device__ long M(const ConvArgs &a) { return (long)a.g.N * a.g.H * a.g.W; }
  static __device__ int N(const ConvArgs &a) { return a.cout; }
  static __device__ long K(const ConvArgs &a) { return 9L * a.cin; }
  static __device__ float A(const ConvArgs &a, long m, long k) {
    int n, y, x;
    pix(a.g, m, n, y, x);
    const int tap = (int)(k / a.cin), ci = (int)(k - (long)tap * a.cin);
    return act_in(a, n, y + tap / 3 - 1, x + tap % 3 - 1, ci);
  }
  static __device__ float B(const ConvArgs &a, int nn, long k) { return a.w[(size_t)nn * 9 * a.cin + k]; }
};

// input gradient: dX[p][ci] = sum_{tap,co} W[co][tap][ci] dZ[p - offset(tap)][co]
template <>
struct Ops<PASS_DX> {
  static __device__ long M(const ConvArgs &a) { return (long)a.g.N * a.g.H * a.g.W; }
  static __device__ int N(const ConvArgs &a) { return a.cin; }
  static __device__ long K(const ConvArgs &a) { return 9L * a.cout; }
  static __device__ float A(const ConvArgs &a, long m, long k) {
    int n, y, x;
    pix(a.g, m, n, y, x);
    const int tap = (int)(k / a.cout), co = (int)(k - (long)tap * a.cout);
    return a.dz[a.g.at(n, y - (tap / 3 - 1), x - (tap % 3 - 1), a.cout) + co];
  }
  static __device__ float B(const ConvArgs &a, int ci, long k) {
    const int tap = (int)(k / a.cout), co = (int)(k - (long)tap * a.cout);
    return a.w[((size_t)co * 9 + tap) * a.cin + ci];
  }
};

// weight gradient: dW[co][tap*cin + ci] = sum_p dZ[p][co] x[p + offset(tap)][ci]
template <>
struct Ops<PASS_DW> {
  static __device__ long M(const ConvArgs &a) { return a.cout; }
  static __device__ int N(const ConvArgs &a) { return 9 * a.cin; }
  static __device__ long K(const ConvArgs &a) { return (long)a.g.N * a.g.H * a.g.W; }
  static __device__ float A(const ConvArgs &a, long co, long p) {
    int n, y, x;
    pix(a.g, p, n, y, x);
    return a.dz[a.g.at(n, y, x, a.cout) + co];
  }
  static __device__ float B(const ConvArgs &a, int nn, long p) {
    int n, y, x;
    pix(a.g, p, n, y, x);
    const int tap = nn / a.cin, ci = nn - tap * a.cin;
    return act_in(a, n, y + tap / 3 - 1, x + tap % 3 - 1, ci);
  }
};

__device__ __forceinline__ void mma_bf16(float *d, const unsigned *a, const unsigned *b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <int PASS>
__device__ __forceinline__ void epilogue(const ConvArgs &a, long m, int nn, float v) {
  if (PASS == PASS_FWD) {
    v += a.bias[nn];
    if (a.relu) v = fmaxf(v, 0.f);
    if (a.y32) {
      a.y32[m] = v;
    } else {
      int n, y, x;
      pix(a.g, m, n, y, x);
      a.y[a.g.at(n, y, x, a.cout) + nn] = f2bf(v);
    }
  } else if (PASS == PASS_DX) {
    int n, y, x;
    pix(a.g, m, n, y, x);
    if (nn < a.c1) {
      const size_t q = a.g.at(n, y, x, a.c1) + nn;
      if (a.m1 && !(bf2f(a.m1[q]) > 0.f)) v = 0.f;
      a.dx1[q] = v;
    } else {
      const size_t q = a.g.at(n, y, x, a.c2) + (nn - a.c1);
      if (a.m2 && !(bf2f(a.m2[q]) > 0.f)) v = 0.f;
      a.dx2[q] = v;
    }
  } else {
    atomicAdd(&a.dw[(size_t)m * 9 * a.cin + nn], v);
  }
}

// The GEMM: a 64 x 64 tile per block of 4 warps (2 x 2, 32 x 32 each),
// K in steps of 32 staged through shared memory as BF16 with the K index
// contiguous (rows padded by 8 elements: the fragment loads of a warp hit
// 32 distinct banks).
template <int PASS>
__global__ void __launch_bounds__(NT) k_conv_gemm(ConvArgs a) {
  __shared__ __align__(16) unsigned short As[BM][BK + PAD];
  __shared__ __align__(16) unsigned short Bs[BN][BK + PAD];
  const long M = Ops<PASS>::M(a);
  const int Nn = Ops<PASS>::N(a);
  const long K = Ops<PASS>::K(a);
  const long m0 = (long)blockIdx.x * BM;
  const int n0 = (int)blockIdx.y * BN;
  long k0 = 0, k1 = K;
  if (PASS == PASS_DW) {
    k0 = (long)blockIdx.z * a.kchunk;
    k1 = min(K, k0 + (long)a.kchunk);
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int gq = lane >> 2, tq = lane & 3;
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
  for (long kb = k0; kb < k1; kb += BK) {
    // stage A and B; the weight-gradient pass walks pixels (its K) fastest
#pragma unroll 4
    for (int e = 0; e < BM * BK / NT; ++e) {
      const int idx = e * NT + tid;
      const int r = (PASS == PASS_DW) ? idx % BM : idx / BK;
      const int kk = (PASS == PASS_DW) ? idx / BM : idx % BK;
      const long m = m0 + r, k = kb + kk;
      const float v = (m < M && k < k1) ? Ops<PASS>::A(a, m, k) : 0.f;
      As[r][kk] = f2bf(v);
    }
#pragma unroll 4
    for (int e = 0; e < BN * BK / NT; ++e) {
      const int idx = e * NT + tid;
      const int r = (PASS == PASS_DW) ? idx % BN : idx / BK;
      const int kk = (PASS == PASS_DW) ? idx / BN : idx % BK;
      const int nn = n0 + r;
      const long k = kb + kk;
      const float v = (nn < Nn && k < k1) ? Ops<PASS>::B(a, nn, k) : 0.f;
      Bs[r][kk] = f2bf(v);
    }
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < BK; ks += 16) {
      unsigned af[2][4], bq[4][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wm + i * 16 + gq;
        af[i][0] = *reinterpret_cast<const unsigned *>(&As[r][ks + 2 * tq]);
        af[i][1] = *reinterpret_cast<const unsigned *>(&As[r + 8][ks + 2 * tq]);
        af[i][2] = *reinterpret_cast<const unsigned *>(&As[r][ks + 2 * tq + 8]);
        af[i][3] = *reinterpret_cast<const unsigned *>(&As[r + 8][ks + 2 * tq + 8]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = wn + j * 8 + gq;
        bq[j][0] = *reinterpret_cast<const unsigned *>(&Bs[r][ks + 2 * tq]);
        bq[j][1] = *reinterpret_cast<const unsigned *>(&Bs[r][ks + 2 * tq + 8]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], af[i], bq[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long m = m0 + wm + i * 16 + gq + ((q & 2) ? 8 : 0);
        const int nn = n0 + wn + j * 8 + 2 * tq + (q & 1);
        if (m < M && nn < Nn) epilogue<PASS>(a, m, nn, acc[i][j][q]);
      }
}

// ---------------------------------------------------------------------------
// Convolution on the 5th-generation tensor cores (tcgen05), for the layers
// with cin and cout multiples of 16: the forward pass, and with DX the input
// gradient (A = the BF16 dZ shifted the other way, K = 9 cout, N = cin, B =
// the weights with cin and cout swapped, ReLU mask in the epilogue, FP32
// result with a BF16 copy for the layer below).
//
// The GEMM runs over the stored pixels of the bordered images as one linear
// index p (border outputs are computed and dropped: 5% of 72 x 104), so a
// tap is a constant offset and no im2col is needed.  A tile is 256 pixels,
// two M = 128 accumulators of N = cout in TMEM.  Its input pixels with their
// halo sit in shared memory once, as planes of 8 channels, 16 bytes a pixel:
// eight consecutive pixels of a plane are one no-swizzle K-major core matrix
// wherever they start, so tap (dy, dx) only moves the descriptor's start
// address (leading byte offset = the plane, stride byte offset = 128).  An
// im2col tile staged per tap, as this kernel did before, moved 9 x 128
// pixels per 128 outputs where this moves 470 per 256 (W = 104).  The halo
// is the contiguous range of pixels while W < 256, else the three rows
// apart.  With room for two stages the next tile's copies run under this
// one's MMAs and epilogue.  One thread issues the 2 x 9 cin / 16
// tcgen05.mma (kind::f16, BF16 x BF16 -> FP32) and commits them to an
// mbarrier.  The K order is k_conv_gemm's and the results equal its bit for
// bit (a backward pass carries any other rounding through every BF16 operand
// below it).
// Measured on 16 images of 72 x 104, 32 channels, GB300: the 13 such layers
// of a forward pass 298 -> 206 us (the im2col tile), of a backward pass
// 2,466 -> 228 us (k_conv_gemm); the batch's whole gradient 9.37 -> 1.09 ms.
// The waits are bounded: if one runs out the kernel flags the error, waits
// once more (bounded) for the MMAs it issued, frees its TMEM and leaves.
namespace tc {

constexpr int kM = 128;
constexpr long kWaitLimit = 1L << 24;

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
// shared memory matrix descriptor: start, leading and stride byte offsets
// (>> 4), version 1, no swizzle
__device__ __forceinline__ unsigned long long sdesc(unsigned addr, unsigned lbo, unsigned sbo) {
  return (unsigned long long)((addr >> 4) & 0x3fffu) | ((unsigned long long)((lbo >> 4) & 0x3fffu) << 16) |
         ((unsigned long long)((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}
// instruction descriptor of kind::f16: FP32 accumulator, A and B BF16 and
// K-major, N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr unsigned idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned phase, long limit) {
  for (long it = 0; it < limit; ++it) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

}  // namespace tc

// Shared-memory geometry of a k_conv_tc launch, the same on host and device.
struct TcShape {
  int cin, cout;  // operand channels of the GEMM: K = 9 cin, N = cout
  int rows;       // pixels of a stage (tile and halo)
  int seg;        // rows apart of the three dy segments
  int plane;      // bytes of a plane of 8 channels
  int stages, ncols;
  __host__ __device__ size_t stage_bytes() const { return (size_t)(cin / 8) * plane; }
  __host__ __device__ size_t b_bytes() const { return (size_t)cout * 9 * cin * 2; }
  __host__ __device__ size_t smem() const { return stage_bytes() * stages + b_bytes() + 32; }
};

namespace tc {

constexpr int kTile = 256;  // pixels

// N accumulator columns of one thread's row, 8 at a time
__device__ __forceinline__ void ld8(unsigned *r, unsigned addr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ unsigned pack2(float a, float b) { return (unsigned)f2bf(a) | ((unsigned)f2bf(b) << 16); }

}  // namespace tc

template <bool DX>
__global__ void __launch_bounds__(256) k_conv_tc(ConvArgs a, TcShape sh, int *err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int cin = sh.cin, cout = sh.cout;
  const int K = 9 * cin, KC = K / 8;
  unsigned char *Bs = smem + sh.stage_bytes() * sh.stages;
  unsigned long long *bar = reinterpret_cast<unsigned long long *>(Bs + sh.b_bytes());
  unsigned *tslot = reinterpret_cast<unsigned *>(bar + 1);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int w2 = a.g.W + 2, hw2 = (a.g.H + 2) * w2;
  const long P = (long)a.g.N * hw2;
  const long plo = w2 + 1, phi = P - w2 - 1;  // holds every interior pixel
  const int ntile = (int)((phi - plo + tc::kTile - 1) / tc::kTile);
  const unsigned sbase = tc::smem_u32(smem);

  // TMEM: one warp allocates the columns, kept for every tile of this CTA
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc::smem_u32(tslot)),
                 "r"(sh.ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(tc::smem_u32(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // a tile's pixels and halo: C8 16-byte chunks a pixel, chunk innermost over
  // the threads (coalesced), zero outside the buffer
  const int C8 = cin / 8;
  const int c18 = (DX ? cin : a.c1) / 8;
  auto stage = [&](int tile, int slot) {
    const long p0 = plo + (long)tile * tc::kTile - 1;
    const unsigned sz = sbase + (unsigned)slot * (unsigned)sh.stage_bytes();
    for (int q = tid; q < sh.rows * C8; q += 256) {
      const int r = q / C8, c8 = q - r * C8;
      const int sg = (sh.seg == w2) ? 0 : r / sh.seg;
      const long p = p0 - w2 + r + (long)sg * (w2 - sh.seg);
      const bool in = p < P;
      const size_t pp = in ? (size_t)p : 0;
      const unsigned short *src = (c8 < c18) ? (DX ? a.dzb : a.x1) + (pp * c18 + c8) * 8
                                             : a.x2 + (pp * (C8 - c18) + (c8 - c18)) * 8;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sz + (unsigned)c8 * (unsigned)sh.plane +
                                                                          (unsigned)r * 16u),
                   "l"(src), "r"(in ? 16 : 0)
                   : "memory");
    }
  };
  if (sh.stages == 2 && (int)blockIdx.x < ntile) stage((int)blockIdx.x, 0);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  // B once per CTA: row co = the weights W[co][tap][ci] rounded to BF16; the
  // input gradient's row n holds W[k][tap][n] (n runs over the threads, so
  // that the strided reads coalesce).  8-row x 16-byte core matrices, the
  // K-adjacent ones 128 bytes apart, the next 8 rows K*16 bytes apart.
  for (int q = tid; q < cout * KC; q += 256) {
    int nn, kc;
    float v[8];
    if (DX) {
      kc = q / cout;
      nn = q - kc * cout;
      const int tap = (kc * 8) / cin, kk = kc * 8 - tap * cin;
      const float *w = a.w + ((size_t)kk * 9 + tap) * cout + nn;
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = w[(size_t)e * 9 * cout];
    } else {
      nn = q / KC;
      kc = q - nn * KC;
      const float4 *w = reinterpret_cast<const float4 *>(a.w + (size_t)nn * K + (size_t)kc * 8);
      const float4 w0 = w[0], w1 = w[1];
      v[0] = w0.x, v[1] = w0.y, v[2] = w0.z, v[3] = w0.w, v[4] = w1.x, v[5] = w1.y, v[6] = w1.z, v[7] = w1.w;
    }
    const unsigned off = (unsigned)(nn >> 3) * (unsigned)KC * 128u + (unsigned)kc * 128u + (unsigned)(nn & 7) * 16u;
    *reinterpret_cast<uint4 *>(Bs + off) =
        make_uint4(tc::pack2(v[0], v[1]), tc::pack2(v[2], v[3]), tc::pack2(v[4], v[5]), tc::pack2(v[6], v[7]));
  }
  const unsigned barad = tc::smem_u32(bar);
  unsigned phase = 0;
  int slot = 0;
  for (int tile = (int)blockIdx.x; tile < ntile; tile += (int)gridDim.x) {
    if (sh.stages == 2) {
      // the other stage's MMAs ended before the last epilogue
      if (tile + (int)gridDim.x < ntile) stage(tile + (int)gridDim.x, slot ^ 1);
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      stage(tile, 0);
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    // the copies must be visible to the tensor cores' async proxy
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem = *tslot;
    if (tid == 0) {
      const unsigned idesc = tc::idesc_bf16(tc::kM, cout);
      const unsigned a0 = sbase + (unsigned)slot * (unsigned)sh.stage_bytes(), b0 = tc::smem_u32(Bs);
      const unsigned sbo = (unsigned)KC * 128u;
      for (int h = 0; h < 2; ++h) {
        unsigned ks = 0;
        for (int tap = 0; tap < 9; ++tap) {
          const int dy = DX ? 2 - tap / 3 : tap / 3, dx = DX ? 2 - tap % 3 : tap % 3;
          const unsigned at = a0 + (unsigned)(h * tc::kM + dy * sh.seg + dx) * 16u;
          for (int kk = 0; kk < cin / 16; ++kk, ++ks) {
            const unsigned long long da = tc::sdesc(at + (unsigned)(2 * kk) * (unsigned)sh.plane, (unsigned)sh.plane, 128u);
            const unsigned long long db = tc::sdesc(b0 + ks * 256u, 128u, sbo);
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem + (unsigned)(h * cout)),
                "l"(da), "l"(db), "r"(idesc), "r"(ks > 0 ? 1u : 0u)
                : "memory");
          }
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(barad)
                   : "memory");
    }
    bool done = tc::mbar_wait(barad, phase, tc::kWaitLimit);
    if (!done) {
      atomicExch(err, 1);
      done = tc::mbar_wait(barad, phase, tc::kWaitLimit);
    }
    phase ^= 1u;
    // every warp of the CTA takes the same branch (tcgen05.ld is .aligned)
    const bool ok = __syncthreads_and(done) != 0;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (!ok) break;
    // thread tid holds pixel p: warps 0-3 the first accumulator's 128 rows,
    // warps 4-7 the second's; every lane loads, interior pixels store
    const long p = plo + (long)tile * tc::kTile + tid;
    const int r = (int)(p % hw2), yb = r / w2, xb = r - yb * w2;
    const bool inner = p < phi && yb >= 1 && yb <= a.g.H && xb >= 1 && xb <= a.g.W;
    const unsigned tw = tmem + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)((warp >> 2) * cout);
    for (int c0 = 0; c0 < cout; c0 += 16) {
      unsigned u[16];
      tc::ld8(u, tw + (unsigned)c0);
      tc::ld8(u + 8, tw + (unsigned)c0 + 8u);
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      if (inner) {
#pragma unroll
        for (int j = 0; j < 16; j += 8) {
          const int c = c0 + j;
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(u[j + e]);
          if (DX) {
            // columns 0..c1-1 belong to x1, the rest to x2 (multiples of 8)
            const bool one = c < a.c1;
            const size_t q = one ? (size_t)p * a.c1 + c : (size_t)p * a.c2 + (c - a.c1);
            const unsigned short *mk = one ? a.m1 : a.m2;
            if (mk) {
              const uint4 mv = *reinterpret_cast<const uint4 *>(mk + q);
              const unsigned mw[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (!(bf2f((unsigned short)(mw[e >> 1] >> (16 * (e & 1)))) > 0.f)) v[e] = 0.f;
            }
            float4 *o = reinterpret_cast<float4 *>((one ? a.dx1 : a.dx2) + q);
            o[0] = make_float4(v[0], v[1], v[2], v[3]);
            o[1] = make_float4(v[4], v[5], v[6], v[7]);
            unsigned short *ob = one ? a.dxb1 : a.dxb2;
            if (ob)
              *reinterpret_cast<uint4 *>(ob + q) = make_uint4(tc::pack2(v[0], v[1]), tc::pack2(v[2], v[3]),
                                                              tc::pack2(v[4], v[5]), tc::pack2(v[6], v[7]));
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              v[e] += a.bias[c + e];
              if (a.relu) v[e] = fmaxf(v[e], 0.f);
            }
            *reinterpret_cast<uint4 *>(a.y + (size_t)p * cout + c) =
                make_uint4(tc::pack2(v[0], v[1]), tc::pack2(v[2], v[3]), tc::pack2(v[4], v[5]), tc::pack2(v[6], v[7]));
          }
        }
      }
      __syncwarp();
    }
    // the next tile's MMAs overwrite the accumulators
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (sh.stages == 2) slot ^= 1;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(*tslot), "r"(sh.ncols) : "memory");
  }
}

// The two thin convolutions of the network, on the CUDA cores with the same
// arithmetic as the tensor-core GEMMs (weights rounded to BF16, BF16
// activations, FP32 accumulation): the first (cin = cin of the network, a
// 9 cin-long K) and the last (cout = 1).  As GEMMs their K or N fills a
// small part of a tensor-core tile.
// first layer: one thread per pixel, all cout outputs (cin <= 4).  CO: cout
// when it is 16, 32 or 64 (sums and stores sized to it), 0 for any cout <= 64
template <int CO>
__global__ void k_conv_first(ConvArgs a) {
  constexpr int CM = CO ? CO : 64;
  extern __shared__ float wsh[];  // [9 cin][cout] rounded weights, then bias
  const int cin = a.cin, cout = CO ? CO : a.cout, K = 9 * cin;
  for (int q = threadIdx.x; q < K * cout; q += blockDim.x) {
    const int co = q % cout, k = q / cout;
    wsh[q] = bf2f(f2bf(a.w[(size_t)co * K + k]));
  }
  for (int q = threadIdx.x; q < cout; q += blockDim.x) wsh[K * cout + q] = a.bias[q];
  __syncthreads();
  const long M = (long)a.g.N * a.g.H * a.g.W;
  for (long m = (long)blockIdx.x * blockDim.x + threadIdx.x; m < M; m += (long)gridDim.x * blockDim.x) {
    int n, y, x;
    pix(a.g, m, n, y, x);
    float acc[CM];
#pragma unroll
    for (int co = 0; co < CM; ++co) acc[co] = 0.f;
    for (int tap = 0; tap < 9; ++tap) {
      const unsigned short *src = a.x1 + a.g.at(n, y + tap / 3 - 1, x + tap % 3 - 1, cin);
      for (int ci = 0; ci < cin; ++ci) {
        const float v = bf2f(src[ci]);
        const float *wr = wsh + (tap * cin + ci) * cout;
#pragma unroll
        for (int co = 0; co < CM; ++co)
          if (CO || co < cout) acc[co] = fmaf(v, wr[co], acc[co]);
      }
    }
    unsigned short *out = a.y + a.g.at(n, y, x, cout);
#pragma unroll
    for (int co = 0; co < CM; ++co) {
      if (!CO && co >= cout) break;
      acc[co] += wsh[K * cout + co];
      if (a.relu) acc[co] = fmaxf(acc[co], 0.f);
      if (!CO) out[co] = f2bf(acc[co]);
    }
    if (CO) {
#pragma unroll
      for (int co = 0; co < CM; co += 8)
        *reinterpret_cast<uint4 *>(out + co) = make_uint4(tc::pack2(acc[co], acc[co + 1]), tc::pack2(acc[co + 2], acc[co + 3]),
                                                          tc::pack2(acc[co + 4], acc[co + 5]), tc::pack2(acc[co + 6], acc[co + 7]));
    }
  }
}

// last layer: one output channel in FP32, one thread per pixel
__global__ void k_conv_last(ConvArgs a) {
  extern __shared__ float wsh[];  // [9 cin] rounded weights
  const int cin = a.cin, K = 9 * cin;
  for (int q = threadIdx.x; q < K; q += blockDim.x) wsh[q] = bf2f(f2bf(a.w[q]));
  __syncthreads();
  const float b = a.bias[0];
  const long M = (long)a.g.N * a.g.H * a.g.W;
  for (long m = (long)blockIdx.x * blockDim.x + threadIdx.x; m < M; m += (long)gridDim.x * blockDim.x) {
    int n, y, x;
    pix(a.g, m, n, y, x);
    float acc = 0.f;
    for (int tap = 0; tap < 9; ++tap) {
      const int yy = y + tap / 3 - 1, xx = x + tap % 3 - 1;
      const float *wr = wsh + tap * cin;
      const unsigned short *src = a.x1 + a.g.at(n, yy, xx, cin);
      int ci = 0;
      if (cin % 8 == 0)
        for (; ci < cin; ci += 8) {
          // 8 channels a load, in the order of the scalar loop
          const uint4 q = *reinterpret_cast<const uint4 *>(src + ci);
          const unsigned u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int e = 0; e < 8; ++e)
            acc = fmaf(bf2f((unsigned short)(u[e >> 1] >> (16 * (e & 1)))), wr[ci + e], acc);
        }
      for (; ci < cin; ++ci) acc = fmaf(bf2f(src[ci]), wr[ci], acc);
    }
    float v = acc + b;
    if (a.relu) v = fmaxf(v, 0.f);
    a.y32[m] = v;
  }
}

// ---------------------------------------------------------------------------
// Weight gradient of the layers with channel counts that are multiples of 16.
//
// dW[co][tap][ci] = sum over pixels p of dZ[p][co] x[p + off(tap)][ci].  The
// bordered images make p a plain linear index: dZ is zero on the border, so
// the sum may run over every stored pixel, and a tap is a constant offset.
// A block walks chunks of 128 pixels; per chunk it copies the chunk of dZ and
// the three rows of x it meets (130 pixels each) to shared memory once, with
// cp.async, kStages chunks in flight, where the element-wise staging of
// k_conv_gemm<PASS_DW> read every x nine times and divided every index.
// Warp (dy, group) does the three taps of one dy on 32 pixels of the chunk
// with mma.sync m16n8k16, both operands through ldmatrix.trans (channels are
// innermost in memory, pixels are the K index); 16-byte chunks of a row are
// swizzled so that eight rows fall in distinct banks.  M = cout = 16..64 is
// below the 64-row minimum that a tcgen05 tile would fill, and the copies,
// not the MMAs, bound this kernel.  Partial sums of the four pixel groups
// meet in shared memory; each block adds its tile to dW with one FP32 atomic
// a weight, as before.
// Measured on 16 images of 72 x 104, 32 channels, GB300: the 13 such layers of
// a backward pass 6.0 ms -> 0.23 ms (k_conv_gemm's one thread block a 64 x 64
// tile and chunk, 425 us a layer, to 18 us).
constexpr int kDwPx = 128, kDwStages = 3, kDwThreads = 384;

template <int CH>
__device__ __forceinline__ unsigned dw_slot(int row, int ch8) {
  // byte offset of 16-byte chunk ch8 of a row of CH BF16 channels
  const int sw = (CH == 32) ? (row >> 1) & 3 : (row >> 2) & 1;
  return (unsigned)(row * CH * 2 + ((ch8 ^ sw) << 4));
}
__device__ __forceinline__ void ldsm_x4_t(unsigned *r, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

// CT: channels of a tile of cout and of cin (16 or 32)
template <int CT>
__global__ void __launch_bounds__(kDwThreads, 1) k_conv_dw(ConvArgs a, int nco, int nchunk) {
  constexpr int MT = CT / 16, RB = CT * 2;
  constexpr int kX = kDwPx + 2;
  constexpr int kStage = (kDwPx + 3 * kX) * RB;
  extern __shared__ __align__(1024) unsigned char smem[];
  const int co0 = ((int)blockIdx.y % nco) * CT, ci0 = ((int)blockIdx.y / nco) * CT;
  const bool one = ci0 < a.c1;
  const unsigned short *x = one ? a.x1 + ci0 : a.x2 + (ci0 - a.c1);
  const int xc = one ? a.c1 : a.c2;
  const long w2 = a.g.W + 2;
  const long P = (long)a.g.N * (a.g.H + 2) * w2;
  const long plo = w2 + 1, phi = P - w2 - 1;  // every interior pixel; p + off stays in [0, P)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dy = warp % 3, pg = warp / 3;
  const unsigned sbase = tc::smem_u32(smem);
  float acc[3][MT][2 * MT][4];
#pragma unroll
  for (int t = 0; t < 3; ++t)
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < 2 * MT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[t][i][j][q] = 0.f;

  auto stage = [&](int chunk, int slot) {
    const long p0 = plo + (long)chunk * kDwPx;
    const unsigned sz = sbase + (unsigned)(slot * kStage);
    constexpr int C8 = CT / 8;
    for (int q = tid; q < (kDwPx + 3 * kX) * C8; q += kDwThreads) {
      const int row = q / C8, c8 = q % C8;
      const unsigned short *src;
      bool in;
      unsigned dst;
      if (row < kDwPx) {
        const long p = p0 + row;
        in = p < phi;
        src = a.dzb + (in ? p : 0) * a.cout + co0 + 8 * c8;
        dst = sz + dw_slot<CT>(row, c8);
      } else {
        const int s = (row - kDwPx) / kX, r = (row - kDwPx) - s * kX;
        const long p = p0 - 1 + r + (s - 1) * w2;
        in = p < P;
        src = x + (in ? p : 0) * xc + 8 * c8;
        dst = sz + (unsigned)((kDwPx + s * kX) * RB) + dw_slot<CT>(r, c8);
      }
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  const int first = (int)blockIdx.x, step = (int)gridDim.x;
  int next = first;
  for (int s = 0; s < kDwStages - 1; ++s, next += step) {
    if (next < nchunk) stage(next, s);
    else asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  int slot = 0;
  for (int c = first; c < nchunk; c += step) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kDwStages - 2) : "memory");
    __syncthreads();  // chunk c is in; every warp is done with the slot refilled next
    const int ns = (slot + kDwStages - 1) % kDwStages;
    if (next < nchunk) stage(next, ns);
    else asm volatile("cp.async.commit_group;\n" ::: "memory");
    next += step;
    const unsigned sz = sbase + (unsigned)(slot * kStage);
    const unsigned sx = sz + (unsigned)((kDwPx + dy * kX) * RB);
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      const int px = pg * 32 + ks * 16;
      unsigned af[MT][4];
#pragma unroll
      for (int i = 0; i < MT; ++i)
        ldsm_x4_t(af[i], sz + dw_slot<CT>(px + (lane & 7) + ((lane >> 4) & 1) * 8, 2 * i + ((lane >> 3) & 1)));
#pragma unroll
      for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int jj = 0; jj < MT; ++jj) {
          unsigned bf[4];
          ldsm_x4_t(bf, sx + dw_slot<CT>(px + t + (lane & 7) + ((lane >> 3) & 1) * 8, 2 * jj + ((lane >> 4) & 1)));
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            mma_bf16(acc[t][i][2 * jj], af[i], bf);
            mma_bf16(acc[t][i][2 * jj + 1], af[i], bf + 2);
          }
        }
    }
    slot = (slot + 1) % kDwStages;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  // the pixel groups' sums in shared memory, [tap][co][ci]
  float *red = reinterpret_cast<float *>(smem);
  for (int g = 0; g < 4; ++g) {
    __syncthreads();
    if (pg != g) continue;
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 2 * MT; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int co = i * 16 + (lane >> 2) + ((q & 2) ? 8 : 0), ci = j * 8 + 2 * (lane & 3) + (q & 1);
            float *d = red + ((dy * 3 + t) * CT + co) * CT + ci;
            *d = (g == 0) ? acc[t][i][j][q] : *d + acc[t][i][j][q];
          }
  }
  __syncthreads();
  for (int q = tid; q < 9 * CT * CT; q += kDwThreads) {
    const int ci = q % CT, co = (q / CT) % CT, tap = q / (CT * CT);
    atomicAdd(&a.dw[((size_t)(co0 + co) * 9 + tap) * a.cin + ci0 + ci], red[q]);
  }
}

// The thin layers' weight gradients: one block of 16 warps an SM, because
// every block adds to the same few hundred weights (6 blocks of 8 warps an SM
// spent most of the first layer's 87 us on those atomics).
constexpr int kThinWarps = 16;

// Weight gradient of the first layer (CI = cin <= 4 input channels): one lane
// per output channel, 9 CI sums in registers, the x values broadcast.
template <int CI>
__global__ void __launch_bounds__(32 * kThinWarps) k_dw_first(ConvArgs a) {
  __shared__ float red[kThinWarps][32];
  const long w2 = a.g.W + 2;
  const long P = (long)a.g.N * (a.g.H + 2) * w2;
  const long plo = w2 + 1, phi = P - w2 - 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int co = (int)blockIdx.y * 32 + lane;
  const bool on = co < a.cout;
  float acc[9 * CI];
#pragma unroll
  for (int k = 0; k < 9 * CI; ++k) acc[k] = 0.f;
  const long nw = (long)gridDim.x * kThinWarps;
  for (long p = plo + (long)blockIdx.x * kThinWarps + warp; p < phi; p += nw) {
    const float z = on ? bf2f(f2bf(a.dz[p * a.cout + co])) : 0.f;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      const unsigned short *xp = a.x1 + (p + (tap / 3 - 1) * w2 + tap % 3 - 1) * CI;
      if (CI == 2) {
        const unsigned u = *reinterpret_cast<const unsigned *>(xp);  // both channels in one load
        acc[tap * CI] = fmaf(z, bf2f((unsigned short)u), acc[tap * CI]);
        acc[tap * CI + 1] = fmaf(z, bf2f((unsigned short)(u >> 16)), acc[tap * CI + 1]);
      } else {
#pragma unroll
        for (int ci = 0; ci < CI; ++ci) acc[tap * CI + ci] = fmaf(z, bf2f(xp[ci]), acc[tap * CI + ci]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 9 * CI; ++k) {
    __syncthreads();
    red[warp][lane] = acc[k];
    __syncthreads();
    if (warp == 0 && on) {
      float s = red[0][lane];
#pragma unroll
      for (int w = 1; w < kThinWarps; ++w) s += red[w][lane];
      atomicAdd(&a.dw[(size_t)co * 9 * CI + k], s);
    }
  }
}

// Weight gradient of the last layer (one output channel): one lane per input
// channel, the nine dZ values of a pixel's neighbours broadcast.
__global__ void __launch_bounds__(32 * kThinWarps) k_dw_last(ConvArgs a) {
  __shared__ float red[kThinWarps][32];
  const long w2 = a.g.W + 2;
  const long P = (long)a.g.N * (a.g.H + 2) * w2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ci = (int)blockIdx.y * 32 + lane;
  const bool on = ci < a.cin;
  float acc[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) acc[k] = 0.f;
  const long nw = (long)gridDim.x * kThinWarps;
  // x pixel q meets dZ at q - off(tap); x is zero on the border, so interior
  // q suffice and q - off stays in [0, P)
#pragma unroll 4
  for (long q = w2 + 1 + (long)blockIdx.x * kThinWarps + warp; q < P - w2 - 1; q += nw) {
    const float xv = on ? bf2f(a.x1[q * a.cin + ci]) : 0.f;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap)
      acc[tap] = fmaf(bf2f(f2bf(a.dz[q - (tap / 3 - 1) * w2 - (tap % 3 - 1)])), xv, acc[tap]);
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    __syncthreads();
    red[warp][lane] = acc[k];
    __syncthreads();
    if (warp == 0 && on) {
      float s = red[0][lane];
#pragma unroll
      for (int w = 1; w < kThinWarps; ++w) s += red[w][lane];
      atomicAdd(&a.dw[(size_t)k * a.cin + ci], s);
    }
  }
}

// Input gradient of the last layer (one dZ channel, K = 9 in one k16 step):
// a warp builds the fragments of 16 pixels in registers and issues the same
// mma.sync as k_conv_gemm<PASS_DX> (bit-equal results), cin / 8 of them.
// cin a multiple of 8, at most 64.
__global__ void __launch_bounds__(128) k_dx_last(ConvArgs a) {
  __shared__ unsigned wsh[64][8];  // [ci][k pair], BF16 pairs, taps 9..15 zero
  const int cin = a.cin;
  for (int q = threadIdx.x; q < cin * 8; q += 128) {
    const int ci = q >> 3, k = 2 * (q & 7);
    const unsigned lo = (k < 9) ? f2bf(a.w[(size_t)k * cin + ci]) : 0u;
    const unsigned hi = (k + 1 < 9) ? f2bf(a.w[(size_t)(k + 1) * cin + ci]) : 0u;
    wsh[ci][k >> 1] = lo | (hi << 16);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const long M = (long)a.g.N * a.g.H * a.g.W;
  for (long m0 = ((long)blockIdx.x * 4 + warp) * 16; m0 < M; m0 += (long)gridDim.x * 64) {
    unsigned af[4];
    size_t row[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long m = m0 + gq + 8 * h;
      int n = 0, y = 0, x = 0;
      if (m < M) pix(a.g, m, n, y, x);
      row[h] = a.g.at(n, y, x, 1);
      auto tap = [&](int k) {
        return (k < 9 && m < M) ? (unsigned)f2bf(a.dz[a.g.at(n, y - (k / 3 - 1), x - (k % 3 - 1), 1)]) : 0u;
      };
      af[h] = tap(2 * tq) | (tap(2 * tq + 1) << 16);
      af[2 + h] = tap(2 * tq + 8) | (tap(2 * tq + 9) << 16);
    }
    for (int c0 = 0; c0 < cin; c0 += 8) {
      const unsigned bf[2] = {wsh[c0 + gq][tq], wsh[c0 + gq][tq + 4]};
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      mma_bf16(d, af, bf);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (m0 + gq + 8 * h >= M) continue;
        const size_t q = row[h] * cin + c0 + 2 * tq;
        float v0 = d[2 * h], v1 = d[2 * h + 1];
        if (a.m1) {
          const unsigned mk = *reinterpret_cast<const unsigned *>(a.m1 + q);
          if (!(bf2f((unsigned short)mk) > 0.f)) v0 = 0.f;
          if (!(bf2f((unsigned short)(mk >> 16)) > 0.f)) v1 = 0.f;
        }
        *reinterpret_cast<float2 *>(a.dx1 + q) = make_float2(v0, v1);
        if (a.dxb1) *reinterpret_cast<unsigned *>(a.dxb1 + q) = (unsigned)f2bf(v0) | ((unsigned)f2bf(v1) << 16);
      }
    }
  }
}

// Bias gradient for cout a multiple of 4 that divides 1024, or 1 (c4 = 0): dZ
// is zero on the border, so the sum runs over the stored pixels (a multiple
// of 4 of them, the image sides being even) as a plain float4 stream.
__global__ void __launch_bounds__(256) k_bias_grad4(const float4 *dz, long n4, int c4, float *db) {
  __shared__ float4 red[256];
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  // 256 is a multiple of c4 = cout / 4: a thread meets one channel quad only
#pragma unroll 4
  for (long t = (long)blockIdx.x * 256 + threadIdx.x; t < n4; t += (long)gridDim.x * 256) {
    const float4 v = dz[t];
    s.x += v.x;
    s.y += v.y;
    s.z += v.z;
    s.w += v.w;
  }
  red[threadIdx.x] = s;
  for (int h = 128; h >= max(c4, 1); h >>= 1) {
    __syncthreads();
    if (threadIdx.x < h) {
      const float4 o = red[threadIdx.x + h];
      s.x += o.x;
      s.y += o.y;
      s.z += o.z;
      s.w += o.w;
      red[threadIdx.x] = s;
    }
  }
  if (c4 == 0) {
    if (threadIdx.x == 0) atomicAdd(db, (s.x + s.y) + (s.z + s.w));
  } else if (threadIdx.x < c4) {
    float *d = db + 4 * threadIdx.x;
    atomicAdd(d, s.x);
    atomicAdd(d + 1, s.y);
    atomicAdd(d + 2, s.z);
    atomicAdd(d + 3, s.w);
  }
}

// bias gradient: db[co] += sum over pixels of dZ[p][co]
__global__ void k_bias_grad(Img g, const float *dz, int cout, float *db) {
  const long npx = (long)g.N * g.H * g.W;
  const int co = threadIdx.x % cout;
  const int lanes = blockDim.x / cout;  // pixel lanes per block
  const int pl = threadIdx.x / cout;
  if (pl >= lanes) return;
  float s = 0.f;
  for (long m = (long)blockIdx.x * lanes + pl; m < npx; m += (long)gridDim.x * lanes) {
    int n, y, x;
    pix(g, m, n, y, x);
    s += dz[g.at(n, y, x, cout) + co];
  }
  atomicAdd(&db[co], s);
}

// The four resampling kernels take V channels a thread: 8 when the channel
// count allows (one 16-byte BF16 access), else 1.
template <int V>
__device__ __forceinline__ void ld_bf(const unsigned short *p, float *v) {
  if constexpr (V == 8) {
    const uint4 q = *reinterpret_cast<const uint4 *>(p);
    const unsigned u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = bf2f((unsigned short)(u[e >> 1] >> (16 * (e & 1))));
  } else {
    v[0] = bf2f(p[0]);
  }
}
template <int V>
__device__ __forceinline__ void st_bf(unsigned short *p, const float *v) {
  if constexpr (V == 8)
    *reinterpret_cast<uint4 *>(p) =
        make_uint4(tc::pack2(v[0], v[1]), tc::pack2(v[2], v[3]), tc::pack2(v[4], v[5]), tc::pack2(v[6], v[7]));
  else
    p[0] = f2bf(v[0]);
}
template <int V>
__device__ __forceinline__ void ld_f(const float *p, float *v) {
  if constexpr (V == 8) {
    const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  } else {
    v[0] = p[0];
  }
}
template <int V>
__device__ __forceinline__ void st_f(float *p, const float *v) {
  if constexpr (V == 8) {
    reinterpret_cast<float4 *>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4 *>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    p[0] = v[0];
  }
}
// item t of C / V channel groups a pixel: its pixel and first channel
template <int V>
__device__ __forceinline__ int item(const Img &g, long t, int C, int &im, int &y, int &x) {
  const int cg = C / V;
  const long m = (t >> 31) ? t / cg : (long)((unsigned)t / (unsigned)cg);
  pix(g, m, im, y, x);
  return (int)(t - m * cg) * V;
}

// 2 x 2 average pooling of s (H x W) into p (H/2 x W/2), BF16
template <int V>
__global__ void k_pool_fwd(Img gc, const unsigned short *s, unsigned short *p, int C) {
  const long n = (long)gc.N * gc.H * gc.W * (C / V);
  Img gf{gc.N, gc.H * 2, gc.W * 2};
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    int im, y, x;
    const int c = item<V>(gc, t, C, im, y, x);
    float v00[V], v01[V], v10[V], v11[V];
    ld_bf<V>(s + gf.at(im, 2 * y, 2 * x, C) + c, v00);
    ld_bf<V>(s + gf.at(im, 2 * y, 2 * x + 1, C) + c, v01);
    ld_bf<V>(s + gf.at(im, 2 * y + 1, 2 * x, C) + c, v10);
    ld_bf<V>(s + gf.at(im, 2 * y + 1, 2 * x + 1, C) + c, v11);
#pragma unroll
    for (int e = 0; e < V; ++e) v00[e] = 0.25f * (v00[e] + v01[e] + v10[e] + v11[e]);
    st_bf<V>(p + gc.at(im, y, x, C) + c, v00);
  }
}

// pooling backward: ds += dp[parent] / 4 masked by s > 0; dsb its BF16 copy
template <int V>
__global__ void k_pool_bwd(Img gf, const float *dp, const unsigned short *s, float *ds, unsigned short *dsb, int C) {
  const long n = (long)gf.N * gf.H * gf.W * (C / V);
  Img gc{gf.N, gf.H / 2, gf.W / 2};
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    int im, y, x;
    const int c = item<V>(gf, t, C, im, y, x);
    const size_t q = gf.at(im, y, x, C) + c;
    float v[V], m[V], o[V];
    ld_f<V>(dp + gc.at(im, y / 2, x / 2, C) + c, v);
    ld_bf<V>(s + q, m);
    ld_f<V>(ds + q, o);
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = o[e] + ((m[e] > 0.f) ? 0.25f * v[e] : 0.f);
    st_f<V>(ds + q, v);
    st_bf<V>(dsb + q, v);
  }
}

// nearest upsampling of d (H/2 x W/2) into u (H x W)
template <int V>
__global__ void k_up_fwd(Img gf, const unsigned short *d, unsigned short *u, int C) {
  const long n = (long)gf.N * gf.H * gf.W * (C / V);
  Img gc{gf.N, gf.H / 2, gf.W / 2};
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    int im, y, x;
    const int c = item<V>(gf, t, C, im, y, x);
    const unsigned short *src = d + gc.at(im, y / 2, x / 2, C) + c;
    unsigned short *dst = u + gf.at(im, y, x, C) + c;
    if constexpr (V == 8) *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(src);
    else *dst = *src;
  }
}

// upsampling backward: dd = sum of the four children's du, masked by d > 0;
// ddb its BF16 copy
template <int V>
__global__ void k_up_bwd(Img gc, const float *du, const unsigned short *d, float *dd, unsigned short *ddb, int C) {
  const long n = (long)gc.N * gc.H * gc.W * (C / V);
  Img gf{gc.N, gc.H * 2, gc.W * 2};
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    int im, y, x;
    const int c = item<V>(gc, t, C, im, y, x);
    const size_t q = gc.at(im, y, x, C) + c;
    float v00[V], v01[V], v10[V], v11[V], m[V];
    ld_f<V>(du + gf.at(im, 2 * y, 2 * x, C) + c, v00);
    ld_f<V>(du + gf.at(im, 2 * y, 2 * x + 1, C) + c, v01);
    ld_f<V>(du + gf.at(im, 2 * y + 1, 2 * x, C) + c, v10);
    ld_f<V>(du + gf.at(im, 2 * y + 1, 2 * x + 1, C) + c, v11);
    ld_bf<V>(d + q, m);
#pragma unroll
    for (int e = 0; e < V; ++e) v00[e] = (m[e] > 0.f) ? v00[e] + v01[e] + v10[e] + v11[e] : 0.f;
    st_f<V>(dd + q, v00);
    st_bf<V>(ddb + q, v00);
  }
}

// network input: FP32 [n][h][w][cin] (no border) -> BF16 bordered image
__global__ void k_load_input(Img g, const float *x, unsigned short *xb, int C) {
  const long n = (long)g.N * g.H * g.W * C;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    const int c = (int)(t % C);
    int im, y, xx;
    pix(g, t / C, im, y, xx);
    xb[g.at(im, y, xx, C) + c] = f2bf(x[t]);
  }
}

// mean-square error over the valid hv x wv corner of each image and its
// gradient (bordered, one channel)
__global__ void k_mse(Img g, const float *y, const float *t, int hv, int wv, float *dy, double *loss) {
  const long n = (long)g.N * g.H * g.W;
  const double inv = 1.0 / ((double)g.N * hv * wv);
  double s = 0.0;
  for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < n; m += (long)gridDim.x * blockDim.x) {
    int im, yy, xx;
    pix(g, m, im, yy, xx);
    float d = 0.f;
    if (yy < hv && xx < wv) {
      d = y[m] - t[m];
      s += (double)d * d;
    }
    dy[g.at(im, yy, xx, 1)] = (float)(2.0 * inv) * d;
  }
  s *= inv;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, s);
}

// Adam (Kingma & Ba), bias-corrected step size computed on the host
__global__ void k_adam(float *w, const float *g, float *m, float *v, long n, float lr_t, float b1, float b2,
                       float eps) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr_t * mi / (sqrtf(vi) + eps);
  }
}

}  // namespace unet
}  // namespace ek

// ---------------------------------------------------------------------------
namespace ek {
using namespace unet;

namespace {
unsigned gsz(long n, int bs) {
  long b = (n + bs - 1) / bs;
  if (b < 1) b = 1;
  if (b > 152L * 64) b = 152L * 64;
  return (unsigned)b;
}
size_t img_bytes(int n, int h, int w, int c, size_t es) { return (size_t)n * (h + 2) * (w + 2) * c * es; }

constexpr size_t kTcSmem = 220 * 1024;
// Shared-memory limits, once a device (the same constants whichever thread is first)
void kernel_limits() {
  static OncePerDevice once;
  once(current_device(), [] {
    EK_CUDA(cudaFuncSetAttribute(k_conv_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
    EK_CUDA(cudaFuncSetAttribute(k_conv_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
    EK_CUDA(cudaFuncSetAttribute(k_conv_dw<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
    EK_CUDA(cudaFuncSetAttribute(k_conv_dw<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
  });
}
int sm_count() {
  int v = 0;
  EK_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, current_device()));
  return v;
}
// The stage layout of k_conv_tc for a GEMM of K = 9 cin, N = cout on images g:
// two stages when they fit, one otherwise.  plane: 16 bytes a pixel, 32 bytes
// off a multiple of 128 so that a warp's copies fall in distinct banks.
TcShape tc_shape(const Img &g, int cin, int cout) {
  TcShape t{};
  t.cin = cin;
  t.cout = cout;
  const int w2 = g.W + 2;
  t.seg = (w2 <= tc::kTile + 2) ? w2 : tc::kTile + 2;
  t.rows = tc::kTile + 2 + 2 * t.seg;
  t.plane = (t.rows + (10 - t.rows % 8) % 8) * 16;
  t.stages = 2;
  if (t.smem() > kTcSmem) t.stages = 1;
  t.ncols = 32;
  while (t.ncols < 2 * cout) t.ncols *= 2;
  return t;
}
// Whether a layer runs on the tensor-core kernels, forward, input gradient and
// weight gradient alike: the weight gradient and the input gradient below read
// the BF16 copy that the input gradient above has written, so a network's
// passes must not mix k_conv_tc with k_conv_gemm, which writes FP32 alone.
bool tc_channels(int cin, int cout, int c1) { return cin % 16 == 0 && cout % 16 == 0 && c1 % 16 == 0; }
// Such a layer must fit k_conv_tc in both directions, and is refused beyond 220
// KB for 128 + cout rows of 9 cin BF16 values: networks of 16 and 32 channels run
// (one stage takes at most 170 KB, whatever the image), 48 and 64 need
// set_tcgen05(0).
void tc_require(const Img &g, int cin, int cout) {
  if ((size_t)(tc::kM + cout) * 9 * cin * 2 + 16 > kTcSmem || tc_shape(g, cin, cout).smem() > kTcSmem ||
      tc_shape(g, cout, cin).smem() > kTcSmem)
    throw CudaError("unet: tcgen05 tile does not fit in shared memory");
}
template <bool DX>
void launch_tc(const ConvArgs &a, const TcShape &t, int *err, cudaStream_t s) {
  kernel_limits();
  const long P = (long)a.g.N * (a.g.H + 2) * (a.g.W + 2);
  const long ntile = (P - 2 * (a.g.W + 2) - 2 + tc::kTile - 1) / tc::kTile;
  // persistent CTAs: as many as fit on the SMs by shared memory and TMEM
  const long per_sm = std::max<long>(1, std::min<long>(kTcSmem / (long)t.smem(), 512 / t.ncols));
  k_conv_tc<DX><<<(unsigned)std::min<long>(ntile, (long)sm_count() * per_sm), 256, t.smem(), s>>>(a, t, err);
}
size_t dw_smem(int ct) {
  const size_t stage = (size_t)(kDwPx + 3 * (kDwPx + 2)) * ct * 2;
  return std::max(stage * kDwStages, sizeof(float) * 9 * ct * ct);
}

struct Launcher {
  long &count;
  void check() {
    ++count;
    const cudaError_t e = cudaPeekAtLastError();
    if (e != cudaSuccess) throw CudaError(std::string("unet launch: ") + cudaGetErrorString(e));
  }
};
}  // namespace

void *UNet::alloc(size_t bytes, std::vector<void *> &list) {
  void *p = nullptr;
  EK_CUDA(cudaMalloc(&p, bytes));
  list.push_back(p);
  EK_CUDA(cudaMemset(p, 0, bytes));
  return p;
}

UNet::UNet(int cin_, int C_, int max_n_, int h_, int w_) : cin(cin_), C(C_), max_n(max_n_), h(h_), w(w_) {
  if (h < 8 || w < 8 || h % 8 || w % 8 || cin < 1 || C < 1 || C > 64 || max_n < 1)
    throw CudaError("unet: h and w must be multiples of 8, 1 <= C <= 64");
  const int spec[kLayers][4] = {{cin, C, cin, 0},  {C, C, C, 0}, {C, C, C, 0},     {C, C, C, 0}, {C, C, C, 0},
                                {C, C, C, 0},      {C, C, C, 0}, {C, C, C, 0},     {2 * C, C, C, C}, {C, C, C, 0},
                                {2 * C, C, C, C},  {C, C, C, 0}, {2 * C, C, C, C}, {C, C, C, 0}, {C, 1, C, 0}};
  long off = 0;
  for (int l = 0; l < kLayers; ++l) {
    Layer &L = L_[l];
    L.cin = spec[l][0];
    L.cout = spec[l][1];
    L.c1 = spec[l][2];
    L.c2 = spec[l][3];
    L.woff = off;
    L.boff = off + (long)L.cout * 9 * L.cin;
    L.relu = l < kLayers - 1;
    off = L.boff + L.cout;
  }
  nparam_ = off;
  try {
    param_ = (float *)alloc(sizeof(float) * nparam_, bufs_);
    grad_ = (float *)alloc(sizeof(float) * nparam_, bufs_);
    m_ = (float *)alloc(sizeof(float) * nparam_, bufs_);
    v_ = (float *)alloc(sizeof(float) * nparam_, bufs_);
    loss_ = (double *)alloc(2 * sizeof(double), bufs_);
    tc_err_ = (int *)(loss_ + 1);
    xin_ = (unsigned short *)alloc(img_bytes(max_n, h, w, cin, 2), bufs_);
    for (int l = 0; l < kLevels; ++l) {
      const int hl = h >> l, wl = w >> l;
      t_[l] = (unsigned short *)alloc(img_bytes(max_n, hl, wl, C, 2), bufs_);
      s_[l] = (unsigned short *)alloc(img_bytes(max_n, hl, wl, C, 2), bufs_);
      if (l >= 1) p_[l] = (unsigned short *)alloc(img_bytes(max_n, hl, wl, C, 2), bufs_);
      if (l <= kLevels - 2) {
        u_[l] = (unsigned short *)alloc(img_bytes(max_n, hl, wl, C, 2), bufs_);
        vv_[l] = (unsigned short *)alloc(img_bytes(max_n, hl, wl, C, 2), bufs_);
        d_[l] = (unsigned short *)alloc(img_bytes(max_n, hl, wl, C, 2), bufs_);
      }
    }
    y_ = (float *)alloc(sizeof(float) * (size_t)max_n * h * w, bufs_);
  } catch (...) {
    for (void *p : bufs_) cudaFree(p);
    bufs_.clear();
    throw;
  }
}

UNet::~UNet() {
  for (void *p : gbufs_) cudaFree(p);
  for (void *p : bufs_) cudaFree(p);
}

void UNet::alloc_grads(int n) {
  if (n <= gn_) return;
  for (void *p : gbufs_) cudaFree(p);
  gbufs_.clear();
  gn_ = 0;
  gy_ = (float *)alloc(img_bytes(n, h, w, 1, 4), gbufs_);
  for (int l = 0; l < kLevels; ++l) {
    const int hl = h >> l, wl = w >> l;
    gt_[l] = (float *)alloc(img_bytes(n, hl, wl, C, 4), gbufs_);
    gs_[l] = (float *)alloc(img_bytes(n, hl, wl, C, 4), gbufs_);
    gtb_[l] = (unsigned short *)alloc(img_bytes(n, hl, wl, C, 2), gbufs_);
    gsb_[l] = (unsigned short *)alloc(img_bytes(n, hl, wl, C, 2), gbufs_);
    if (l >= 1) gp_[l] = (float *)alloc(img_bytes(n, hl, wl, C, 4), gbufs_);
    if (l <= kLevels - 2) {
      gu_[l] = (float *)alloc(img_bytes(n, hl, wl, C, 4), gbufs_);
      gv_[l] = (float *)alloc(img_bytes(n, hl, wl, C, 4), gbufs_);
      gd_[l] = (float *)alloc(img_bytes(n, hl, wl, C, 4), gbufs_);
      gvb_[l] = (unsigned short *)alloc(img_bytes(n, hl, wl, C, 2), gbufs_);
      gdb_[l] = (unsigned short *)alloc(img_bytes(n, hl, wl, C, 2), gbufs_);
    }
  }
  gn_ = n;
}

void UNet::set_params(const float *host) {
  EK_CUDA(cudaMemcpy(param_, host, sizeof(float) * nparam_, cudaMemcpyHostToDevice));
  EK_CUDA(cudaMemset(m_, 0, sizeof(float) * nparam_));
  EK_CUDA(cudaMemset(v_, 0, sizeof(float) * nparam_));
  step_ = 0;
}

void UNet::get_params(float *host) const {
  EK_CUDA(cudaMemcpy(host, param_, sizeof(float) * nparam_, cudaMemcpyDeviceToHost));
}

void UNet::layer_shape(int l, int *ci, int *co) const {
  *ci = L_[l].cin;
  *co = L_[l].cout;
}

double UNet::forward_flops(int n) const {
  double f = 0.0;
  const int lev[kLayers] = {0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0};
  for (int l = 0; l < kLayers; ++l)
    f += 2.0 * 9.0 * L_[l].cin * L_[l].cout * (double)n * (h >> lev[l]) * (w >> lev[l]);
  return f;
}

void UNet::run_forward(const float *x, int n, float *y, cudaStream_t s) {
  if (n < 1 || n > max_n) throw CudaError("unet: batch outside 1..max_n");
  Launcher K{launches_};
  Img g[kLevels];
  for (int l = 0; l < kLevels; ++l) g[l] = Img{n, h >> l, w >> l};
  auto conv = [&](int l, int lev, const unsigned short *x1, const unsigned short *x2, unsigned short *out,
                  float *out32) {
    const Layer &Ly = L_[l];
    ConvArgs a{};
    a.g = g[lev];
    a.x1 = x1;
    a.x2 = x2;
    a.c1 = Ly.c1;
    a.c2 = Ly.c2;
    a.cin = Ly.cin;
    a.cout = Ly.cout;
    a.w = param_ + Ly.woff;
    a.bias = param_ + Ly.boff;
    a.y = out;
    a.y32 = out32;
    a.relu = Ly.relu;
    const long M = (long)n * a.g.H * a.g.W;
    if (tc_ && tc_channels(Ly.cin, Ly.cout, Ly.c1)) {
      tc_require(a.g, Ly.cin, Ly.cout);
      launch_tc<false>(a, tc_shape(a.g, Ly.cin, Ly.cout), tc_err_, s);
    } else if (tc_ && out32 && Ly.cout == 1 && !Ly.c2) {
      k_conv_last<<<gsz(M, 256), 256, sizeof(float) * 9 * Ly.cin, s>>>(a);
    } else if (tc_ && !out32 && Ly.cin <= 4 && Ly.cout <= 64 && !Ly.c2) {
      const size_t sm = sizeof(float) * (9 * Ly.cin + 1) * Ly.cout;
      if (Ly.cout == 16) k_conv_first<16><<<gsz(M, 128), 128, sm, s>>>(a);
      else if (Ly.cout == 32) k_conv_first<32><<<gsz(M, 128), 128, sm, s>>>(a);
      else if (Ly.cout == 64) k_conv_first<64><<<gsz(M, 128), 128, sm, s>>>(a);
      else k_conv_first<0><<<gsz(M, 128), 128, sm, s>>>(a);
    } else {
      k_conv_gemm<PASS_FWD><<<dim3((unsigned)((M + BM - 1) / BM), (unsigned)((Ly.cout + BN - 1) / BN)), NT, 0, s>>>(a);
    }
    K.check();
  };
  auto pool = [&](int lev, const unsigned short *src, unsigned short *dst) {
    const long items = (long)n * g[lev].H * g[lev].W * C;
    if (C % 8 == 0) k_pool_fwd<8><<<gsz(items / 8, 256), 256, 0, s>>>(g[lev], src, dst, C);
    else k_pool_fwd<1><<<gsz(items, 256), 256, 0, s>>>(g[lev], src, dst, C);
    K.check();
  };
  auto up = [&](int lev, const unsigned short *src, unsigned short *dst) {
    const long items = (long)n * g[lev].H * g[lev].W * C;
    if (C % 8 == 0) k_up_fwd<8><<<gsz(items / 8, 256), 256, 0, s>>>(g[lev], src, dst, C);
    else k_up_fwd<1><<<gsz(items, 256), 256, 0, s>>>(g[lev], src, dst, C);
    K.check();
  };
  k_load_input<<<gsz((long)n * h * w * cin, 256), 256, 0, s>>>(g[0], x, xin_, cin);
  K.check();
  conv(0, 0, xin_, nullptr, t_[0], nullptr);
  conv(1, 0, t_[0], nullptr, s_[0], nullptr);
  for (int l = 1; l < kLevels; ++l) {
    pool(l, s_[l - 1], p_[l]);
    conv(2 * l, l, p_[l], nullptr, t_[l], nullptr);
    conv(2 * l + 1, l, t_[l], nullptr, s_[l], nullptr);
  }
  const unsigned short *below = s_[kLevels - 1];
  for (int l = kLevels - 2; l >= 0; --l) {
    const int li = 8 + 2 * (kLevels - 2 - l);  // 8, 10, 12
    up(l, below, u_[l]);
    conv(li, l, u_[l], s_[l], vv_[l], nullptr);
    conv(li + 1, l, vv_[l], nullptr, d_[l], nullptr);
    below = d_[l];
  }
  conv(kLayers - 1, 0, d_[0], nullptr, nullptr, y);
}

void UNet::forward(const float *x, int n, float *y, cudaStream_t s) { run_forward(x, n, y, s); }

int UNet::tc_error(cudaStream_t s) {
  int v = 0;
  EK_CUDA(cudaMemcpyAsync(&v, tc_err_, sizeof(int), cudaMemcpyDeviceToHost, s));
  EK_CUDA(cudaStreamSynchronize(s));
  return v;
}

bool UNet::forward_backward(const float *x, const float *t, int n, int hv, int wv, float *y, double &loss,
                            cudaStream_t s) {
  if (!y) y = y_;
  run_forward(x, n, y, s);
  alloc_grads(n);
  Launcher K{launches_};
  Img g[kLevels];
  for (int l = 0; l < kLevels; ++l) g[l] = Img{n, h >> l, w >> l};
  EK_CUDA(cudaMemsetAsync(grad_, 0, sizeof(float) * nparam_, s));
  EK_CUDA(cudaMemsetAsync(loss_, 0, sizeof(double), s));
  k_mse<<<gsz((long)n * h * w, 256), 256, 0, s>>>(g[0], y, t, hv, wv, gy_, loss_);
  K.check();
  // dW, db and (when dx1 is given) dX of layer l at level lev.  dzb is the
  // BF16 copy of dz, dxb1 / dxb2 those of the dX that are a layer's dZ in
  // turn; with set_tcgen05 off, or at other channel counts, the element-wise
  // GEMM does all three from the FP32 arrays.
  auto back = [&](int l, int lev, const unsigned short *x1, const unsigned short *x2, const float *dz,
                  const unsigned short *dzb, float *dx1, unsigned short *dxb1, const unsigned short *m1, float *dx2,
                  const unsigned short *m2) {
    const Layer &Ly = L_[l];
    ConvArgs a{};
    a.g = g[lev];
    a.x1 = x1;
    a.x2 = x2;
    a.c1 = Ly.c1;
    a.c2 = Ly.c2;
    a.cin = Ly.cin;
    a.cout = Ly.cout;
    a.w = param_ + Ly.woff;
    a.dz = dz;
    a.dzb = dzb;
    a.dw = grad_ + Ly.woff;
    a.dx1 = dx1;
    a.dxb1 = dxb1;
    a.dx2 = dx2;
    a.m1 = m1;
    a.m2 = m2;
    const long npx = (long)n * a.g.H * a.g.W;
    const long stored = (long)n * (a.g.H + 2) * (a.g.W + 2);
    const bool mult16 = tc_ && tc_channels(Ly.cin, Ly.cout, Ly.c1);
    const bool last = tc_ && Ly.cout == 1 && !Ly.c2 && Ly.cin % 8 == 0;
    if (mult16) {
      kernel_limits();
      const int ct = (Ly.cout % 32 == 0 && Ly.c1 % 32 == 0 && Ly.cin % 32 == 0) ? 32 : 16;
      const int nco = Ly.cout / ct, ntile = nco * (Ly.cin / ct);
      const int nchunk = (int)((stored - 2 * (a.g.W + 2) - 2 + kDwPx - 1) / kDwPx);
      // one resident block an SM over the tiles; a block takes at least two
      // chunks, so that its atomics are shared by them
      const int nb = std::max(1, std::min((nchunk + 1) / 2, std::max(1, sm_count() / ntile)));
      if (ct == 32)
        k_conv_dw<32><<<dim3((unsigned)nb, (unsigned)ntile), kDwThreads, dw_smem(32), s>>>(a, nco, nchunk);
      else
        k_conv_dw<16><<<dim3((unsigned)nb, (unsigned)ntile), kDwThreads, dw_smem(16), s>>>(a, nco, nchunk);
    } else if (last) {
      k_dw_last<<<dim3((unsigned)sm_count(), (unsigned)(Ly.cin + 31) / 32), 32 * kThinWarps, 0, s>>>(a);
    } else if (tc_ && Ly.cin <= 4 && !Ly.c2) {
      const dim3 gr((unsigned)sm_count(), (unsigned)(Ly.cout + 31) / 32);
      if (Ly.cin == 1) k_dw_first<1><<<gr, 32 * kThinWarps, 0, s>>>(a);
      else if (Ly.cin == 2) k_dw_first<2><<<gr, 32 * kThinWarps, 0, s>>>(a);
      else if (Ly.cin == 3) k_dw_first<3><<<gr, 32 * kThinWarps, 0, s>>>(a);
      else k_dw_first<4><<<gr, 32 * kThinWarps, 0, s>>>(a);
    } else {
      // pixels per block of the weight gradient: about 64 partial sums per
      // weight, each added with one FP32 atomic
      long kc = (npx + 63) / 64;
      kc = ((kc + BK - 1) / BK) * BK;
      if (kc < 4 * BK) kc = 4 * BK;
      a.kchunk = (int)kc;
      k_conv_gemm<PASS_DW><<<dim3(1, (unsigned)((9 * Ly.cin + BN - 1) / BN), (unsigned)((npx + kc - 1) / kc)), NT, 0,
                             s>>>(a);
    }
    K.check();
    if (Ly.cout == 1 || (Ly.cout % 4 == 0 && 1024 % Ly.cout == 0)) {
      const long n4 = stored * Ly.cout / 4;
      k_bias_grad4<<<(unsigned)std::min((n4 + 1023) / 1024, 2L * sm_count()), 256, 0, s>>>(
          reinterpret_cast<const float4 *>(dz), n4, Ly.cout / 4, grad_ + Ly.boff);
    } else {
      const int lanes = 256 / Ly.cout;
      const long nbg = std::min((npx + lanes - 1) / lanes, 4L * 152);
      k_bias_grad<<<(unsigned)nbg, 256, 0, s>>>(a.g, dz, Ly.cout, grad_ + Ly.boff);
    }
    K.check();
    if (!dx1) return;
    if (mult16) {
      launch_tc<true>(a, tc_shape(a.g, Ly.cout, Ly.cin), tc_err_, s);
    } else if (last) {
      k_dx_last<<<(unsigned)std::min((npx + 63) / 64, 8L * sm_count()), 128, 0, s>>>(a);
    } else {
      k_conv_gemm<PASS_DX><<<dim3((unsigned)((npx + BM - 1) / BM), (unsigned)((Ly.cin + BN - 1) / BN)), NT, 0, s>>>(a);
    }
    K.check();
  };
  back(kLayers - 1, 0, d_[0], nullptr, gy_, nullptr, gd_[0], gdb_[0], d_[0], nullptr, nullptr);
  for (int l = 0; l <= kLevels - 2; ++l) {
    const int li = 8 + 2 * (kLevels - 2 - l);
    back(li + 1, l, vv_[l], nullptr, gd_[l], gdb_[l], gv_[l], gvb_[l], vv_[l], nullptr, nullptr);
    back(li, l, u_[l], s_[l], gv_[l], gvb_[l], gu_[l], nullptr, nullptr, gs_[l], s_[l]);
    // the upsampling's gradient into the level below (d of the decoder
    // below, or s of the bottleneck)
    const bool dec = l + 1 <= kLevels - 2;
    float *dst = dec ? gd_[l + 1] : gs_[kLevels - 1];
    unsigned short *dstb = dec ? gdb_[l + 1] : gsb_[kLevels - 1];
    const unsigned short *msk = dec ? d_[l + 1] : s_[kLevels - 1];
    const long items = (long)n * g[l + 1].H * g[l + 1].W * C;
    if (C % 8 == 0) k_up_bwd<8><<<gsz(items / 8, 256), 256, 0, s>>>(g[l + 1], gu_[l], msk, dst, dstb, C);
    else k_up_bwd<1><<<gsz(items, 256), 256, 0, s>>>(g[l + 1], gu_[l], msk, dst, dstb, C);
    K.check();
  }
  for (int l = kLevels - 1; l >= 1; --l) {
    back(2 * l + 1, l, t_[l], nullptr, gs_[l], gsb_[l], gt_[l], gtb_[l], t_[l], nullptr, nullptr);
    back(2 * l, l, p_[l], nullptr, gt_[l], gtb_[l], gp_[l], nullptr, nullptr, nullptr, nullptr);
    const long items = (long)n * g[l - 1].H * g[l - 1].W * C;
    if (C % 8 == 0)
      k_pool_bwd<8><<<gsz(items / 8, 256), 256, 0, s>>>(g[l - 1], gp_[l], s_[l - 1], gs_[l - 1], gsb_[l - 1], C);
    else
      k_pool_bwd<1><<<gsz(items, 256), 256, 0, s>>>(g[l - 1], gp_[l], s_[l - 1], gs_[l - 1], gsb_[l - 1], C);
    K.check();
  }
  back(1, 0, t_[0], nullptr, gs_[0], gsb_[0], gt_[0], gtb_[0], t_[0], nullptr, nullptr);
  back(0, 0, xin_, nullptr, gt_[0], gtb_[0], nullptr, nullptr, nullptr, nullptr, nullptr);
  struct {
    double loss;
    int err;
  } res = {};
  EK_CUDA(cudaMemcpyAsync(&res, loss_, sizeof(res), cudaMemcpyDeviceToHost, s));
  EK_CUDA(cudaStreamSynchronize(s));
  loss = res.loss;
  return !(tc_ && res.err);
}

bool UNet::train_step(const float *x, const float *t, int n, int hv, int wv, double lr, double &loss, cudaStream_t s) {
  if (!forward_backward(x, t, n, hv, wv, nullptr, loss, s)) return false;
  ++step_;
  const double b1 = 0.9, b2 = 0.999;
  const double lr_t = lr * std::sqrt(1.0 - std::pow(b2, (double)step_)) / (1.0 - std::pow(b1, (double)step_));
  k_adam<<<gsz(nparam_, 256), 256, 0, s>>>(param_, grad_, m_, v_, nparam_, (float)lr_t, (float)b1, (float)b2, 1e-8f);
  ++launches_;
  const cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) throw CudaError(std::string("unet adam: ") + cudaGetErrorString(e));
  return true;
}

}  // namespace ek
