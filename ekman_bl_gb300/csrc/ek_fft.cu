// Batched x-direction real FFTs of the duct substep, FP64.
//
// The reference transforms every field line along x through
// REAL_FOURIER_TRANS_* (src/mpi_duct.F90:271-717) and the missing
// FFT_X_TO_FOURIER_OP / FFT_X_TO_PHYSICAL_OP (FFTW 2 rfftw).  Here one warp
// owns one x-line: a length-NX real transform is done as a length-NX/2
// complex radix-2 DIF FFT in shared memory plus the split/merge twiddle
// step.  Forward transforms keep modes 0..NX/3 and scale by 1/NX; the
// inverse reads modes 0..NX/3 (imaginary part of mode 0 ignored) and zeroes
// the two padding points x = NX, NX+1, as the reference's copy loops do.
//
// The forward kernel fuses its producer and consumer:
//   prologue PRO_LOAD  x = a
//            PRO_PROD  x = J a b            (duct.F90:685-691 products)
//            PRO_FLUX  x = flux stencil of a (duct.F90:735-761 form)
//            (with LES, + J tau or + the eddy-viscosity terms: ek_les.cu)
//   epilogue EPI_STORE dst  = X            (modes > NX/3 set to 0)
//            EPI_ADD   dst += X            (duct.F90:779-785)
//            EPI_SUB_IK dst -= i kx X      (duct.F90:712-718)
// so no product or transform temporary ever reaches HBM.
#include <map>
#include <type_traits>
#include <mutex>
#include <utility>

#include "ek_internal.h"

namespace ek {

namespace {

constexpr int kWarpsPerBlock = 4;

struct FftConst {
  Dims d;
  int M, logM;
  const double2 *tw_m, *tw_n;
  const float2 *tw_mf, *tw_nf;  // the same tables rounded to FP32
  const float4 *tw_mff, *tw_nff;  // and split into float-float (re.hi, re.lo, im.hi, im.lo)
  const double *kx;
  Metrics m;
  double inv_nx;  // 1/NX, divided once on the host
  int orth;       // GMAT_12 is zero
};

// T: the arithmetic type of a transform (double; float with the fields still
// stored in FP64; or FF); V: its complex pair.
template <typename T> struct Cx;
template <> struct Cx<double> {
  using V = double2;
  __device__ static V make(double x, double y) { return make_double2(x, y); }
};
template <> struct Cx<float> {
  using V = float2;
  __device__ static V make(float x, float y) { return make_float2(x, y); }
};
struct FF2 {
  FF x, y;
};
template <> struct Cx<FF> {
  using V = FF2;
  __device__ static V make(FF x, FF y) { return FF2{x, y}; }
};
template <typename T> __device__ __forceinline__ const typename Cx<T>::V *tw_m(const FftConst &f);
template <> __device__ __forceinline__ const double2 *tw_m<double>(const FftConst &f) { return f.tw_m; }
template <> __device__ __forceinline__ const float2 *tw_m<float>(const FftConst &f) { return f.tw_mf; }
template <> __device__ __forceinline__ const FF2 *tw_m<FF>(const FftConst &f) {
  return reinterpret_cast<const FF2 *>(f.tw_mff);
}
template <typename T> __device__ __forceinline__ const typename Cx<T>::V *tw_n(const FftConst &f);
template <> __device__ __forceinline__ const double2 *tw_n<double>(const FftConst &f) { return f.tw_n; }
template <> __device__ __forceinline__ const float2 *tw_n<float>(const FftConst &f) { return f.tw_nf; }
template <> __device__ __forceinline__ const FF2 *tw_n<FF>(const FftConst &f) {
  return reinterpret_cast<const FF2 *>(f.tw_nff);
}

// an FP64 value in the arithmetic type T; to float on the integer pipe
// (a plain cast is an F2F on the narrow FP64 pipe)
template <typename T> __device__ __forceinline__ T from_f64(double x) { return (T)x; }
template <> __device__ __forceinline__ float from_f64<float>(double x) { return d2f_bits(x); }

template <typename V>
__device__ __forceinline__ V cmul(V a, V b) {
  V r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}

__device__ __forceinline__ unsigned brev(unsigned v, int logM) { return __brev(v) >> (32 - logM); }

// In-place radix-2 DIF over z[0..M), bit-reversed output.  conj_tw selects
// the inverse transform.
template <typename V>
__device__ __forceinline__ void dif_fft(V *z, int M, const V *tw, bool conj_tw, int lane) {
  for (int s = M >> 1; s >= 1; s >>= 1) {
    const int stride = (M >> 1) / s;  // twiddle step M/(2s)
    for (int q = lane; q < (M >> 1); q += 32) {
      const int t = q & (s - 1);
      const int a = ((q - t) << 1) + t;
      const int b = a + s;
      const V u = z[a], v = z[b];
      V sum, dlt;
      sum.x = u.x + v.x;
      sum.y = u.y + v.y;
      dlt.x = u.x - v.x;
      dlt.y = u.y - v.y;
      z[a] = sum;
      if (t != 0) {
        V w = tw[t * stride];
        if (conj_tw) w.y = -w.y;
        dlt = cmul(dlt, w);
      }
      z[b] = dlt;
    }
    __syncwarp();
  }
}

// One value exchanged with the lane whose index differs in the bits of m.
__device__ __forceinline__ float2 shfl_x(float2 v, int m) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}
template <typename V>
__device__ __forceinline__ V csub(V a, V b) {
  V r;
  r.x = a.x - b.x;
  r.y = a.y - b.y;
  return r;
}
template <typename V>
__device__ __forceinline__ V caddv(V a, V b) {
  V r;
  r.x = a.x + b.x;
  r.y = a.y + b.y;
  return r;
}

// The same radix-2 DIF (same butterflies, same twiddles, bit-reversed
// output in z) with the warp's M = 32 E points held in registers: lane l
// keeps points l + 32 t, t < E.  The log2(E) stages whose pairs are 32 or
// more apart run between a lane's own registers; the five stages below run
// between lanes through shuffles, where a lane's twiddle depends only on the
// lane.  Shared memory is touched once to load and once to store, instead
// of twice per stage.
template <int E, typename V>
__device__ __forceinline__ void dif_fft_reg(V *z, const V *tw, bool conj_tw, int lane) {
  constexpr int M = 32 * E;
  V v[E];
#pragma unroll
  for (int t = 0; t < E; ++t) v[t] = z[lane + 32 * t];
#pragma unroll
  for (int h = E / 2; h >= 1; h >>= 1) {
    // span s = 32 h: pairs (t, t + h) within each block of 2h registers
    const int stride = M / (64 * h);  // M / (2 s)
#pragma unroll
    for (int t = 0; t < E; ++t) {
      if (t & h) continue;
      const V a = v[t], b = v[t + h];
      v[t] = caddv(a, b);
      const int tt = lane + 32 * (t & (h - 1));  // n mod s
      V dlt = csub(a, b);
      if (tt != 0) {
        V w = tw[tt * stride];
        if (conj_tw) w.y = -w.y;
        dlt = cmul(dlt, w);
      }
      v[t + h] = dlt;
    }
  }
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const bool upper = (lane & s) != 0;
    const int tt = lane & (s - 1);
    V w = tw[tt * (M / (2 * s))];
    if (conj_tw) w.y = -w.y;
#pragma unroll
    for (int t = 0; t < E; ++t) {
      const V p = shfl_x(v[t], s);
      if (!upper) {
        v[t] = caddv(v[t], p);
      } else {
        V dlt = csub(p, v[t]);
        if (tt != 0) dlt = cmul(dlt, w);
        v[t] = dlt;
      }
    }
  }
  // v[t] holds DIF position p = lane + 32 t, i.e. frequency brev(p) =
  // rev5(lane) E + revE(t); it goes to its natural-order slot with one pad
  // element every E (fslot), so that this store and the readers' runs of
  // consecutive frequencies fall in distinct banks (the bit-reversed order
  // puts a warp's 32 frequencies E elements apart)
  const int r5 = (int)(__brev((unsigned)lane) >> 27);
#pragma unroll
  for (int t = 0; t < E; ++t) {
    int rt = 0;
#pragma unroll
    for (int b = 1, q = E >> 1; b < E; b <<= 1, q >>= 1)
      if (t & b) rt |= q;
    z[r5 * (E + 1) + rt] = v[t];
  }
  __syncwarp();
}

// Where frequency f of a transform of M = 32 E points sits after
// dif_fft_any<E>: natural order with a pad element every E (the register
// form), bit-reversed order (the shared-memory loop, E = 0).
template <int E>
__device__ __forceinline__ int fslot(int f, int logM) {
  if constexpr (E > 0) return f + f / E;
  else return (int)brev((unsigned)f, logM);
}
// Per-warp stride of the spectra in shared memory: room for the pad slots
template <int E>
__device__ __forceinline__ int fstride(int M) { return (E > 0) ? M + 32 : M; }

// The register form for M = 32 E (E > 0, chosen per launch so that each
// size gets its own register budget), the shared-memory loop otherwise.
template <int E, typename V>
__device__ __forceinline__ void dif_fft_any(V *z, int M, const V *tw, bool conj_tw, int lane) {
  __syncwarp();
  if constexpr (E > 0) dif_fft_reg<E>(z, tw, conj_tw, lane);
  else dif_fft(z, M, tw, conj_tw, lane);
}

// The flux form of the eta/zeta convection plus the GMAT_12 cross diffusion
// of a field (duct.F90:735-761; the TH version at 1210-1241 has visc =
// NU/PR) at one point from the field's neighbours and the face velocities.
// ORTH: GMAT_12 is zero, and the cross diffusion with its four corner values is
// left out.  The step's forward transforms: FP32 on 512 x 385 x 257 9.9 ->
// 8.7 ms, FP64 on 256 x 257 x 193 23.2 -> 18.1 ms.
template <typename T>
struct FluxG12 {
  T a, b, c, d, qv;
  __device__ FluxG12(const FftConst &fc, int k, int j, double visc)
      : a(from_f64<T>(fc.m.g12[fc.d.m3(k + 1, j, 2)])), b(from_f64<T>(fc.m.g12[fc.d.m3(k, j, 2)])),
        c(from_f64<T>(fc.m.g12[fc.d.m3(k, j + 1, 1)])), d(from_f64<T>(fc.m.g12[fc.d.m3(k, j, 1)])),
        qv(from_f64<T>(0.25 * visc)) {}
};
template <typename T>
__device__ __forceinline__ T flux_orth(T f, T fkp, T fkm, T fjp, T fjm, T u2, T u2p, T u3, T u3p) {
  const T h = (T)0.5;
  const T s1 = h * u2p * (f + fjp) - h * u2 * (f + fjm);
  const T s2 = h * u3p * (f + fkp) - h * u3 * (f + fkm);
  return -s1 - s2;
}
template <typename T>
__device__ __forceinline__ T flux_gen(const FluxG12<T> &g, T f, T fkp, T fkm, T fjp, T fjm, T fpp, T fpm, T fmp, T fmm,
                                      T u2, T u2p, T u3, T u3p) {
  const T h = (T)0.5;
  T s1 = h * u2p * (f + fjp) - h * u2 * (f + fjm);
  T s2 = h * u3p * (f + fkp) - h * u3 * (f + fkm);
  s1 = -s1 + g.qv * (g.a * (fpp + fjp - fjm - fpm) - g.b * (fmp + fjp - fjm - fmm));
  s2 = -s2 + g.qv * (g.c * (fpp + fkp - fmp - fkm) - g.d * (fkp + fpm - fkm - fmm));
  return s1 + s2;
}
// One or two consecutive values in the arithmetic type: two in one 8-byte load
// of an FP32 plane (a plane's lines start on even elements)
template <typename T> struct One {
  T x;
};
template <typename T> struct Two {
  T x, y;
};
template <typename T, typename P> __device__ __forceinline__ void ld_pts(One<T> &v, const P *p) { v.x = (T)(double)p[0]; }
template <typename T> __device__ __forceinline__ void ld_pts(Two<T> &v, const float *p) {
  const float2 w = *reinterpret_cast<const float2 *>(p);
  v.x = (T)(double)w.x, v.y = (T)(double)w.y;
}
template <typename T> __device__ __forceinline__ void ld_pts(Two<T> &v, const double *p) { v.x = (T)p[0], v.y = (T)p[1]; }
template <typename G, typename P> __device__ __forceinline__ G pts(const P *p) {
  G v;
  ld_pts(v, p);
  return v;
}
// The flux at the points from c on, its loads apart from its value so that
// several groups' loads can go out together; b is U2b, followed in memory by U3b
// (see the launch).
template <typename G> struct FluxIn {
  G f, kp, km, jp, jm, u2, u2p, u3, u3p, pp, pm, mp, mm;
};
template <typename G, bool ORTH, typename P>
__device__ __forceinline__ FluxIn<G> flux_load(const Dims &d, size_t c, const P *F, const P *U2b) {
  const size_t sK = d.LDX, sJ = (size_t)d.LDX * d.NZ2;
  const P *U3b = U2b + d.nphys();
  FluxIn<G> v;
  v.f = pts<G>(F + c), v.kp = pts<G>(F + c + sK), v.km = pts<G>(F + c - sK);
  v.jp = pts<G>(F + c + sJ), v.jm = pts<G>(F + c - sJ);
  v.u2 = pts<G>(U2b + c), v.u2p = pts<G>(U2b + c + sJ), v.u3 = pts<G>(U3b + c), v.u3p = pts<G>(U3b + c + sK);
  if constexpr (!ORTH) {
    v.pp = pts<G>(F + c + sK + sJ), v.pm = pts<G>(F + c + sK - sJ);
    v.mp = pts<G>(F + c - sK + sJ), v.mm = pts<G>(F + c - sK - sJ);
  }
  return v;
}
template <bool ORTH, typename T, typename G>
__device__ __forceinline__ G flux_value(const FluxG12<T> &g, const FluxIn<G> &v) {
  G r;
  if constexpr (ORTH)
    r.x = flux_orth(v.f.x, v.kp.x, v.km.x, v.jp.x, v.jm.x, v.u2.x, v.u2p.x, v.u3.x, v.u3p.x);
  else
    r.x = flux_gen(g, v.f.x, v.kp.x, v.km.x, v.jp.x, v.jm.x, v.pp.x, v.pm.x, v.mp.x, v.mm.x, v.u2.x, v.u2p.x, v.u3.x,
                   v.u3p.x);
  if constexpr (std::is_same_v<G, Two<T>>) {
    if constexpr (ORTH)
      r.y = flux_orth(v.f.y, v.kp.y, v.km.y, v.jp.y, v.jm.y, v.u2.y, v.u2p.y, v.u3.y, v.u3p.y);
    else
      r.y = flux_gen(g, v.f.y, v.kp.y, v.km.y, v.jp.y, v.jm.y, v.pp.y, v.pm.y, v.mp.y, v.mm.y, v.u2.y, v.u2p.y, v.u3.y,
                     v.u3p.y);
  }
  return r;
}
// The same along one x-line, point n to put(n, value), for the FP64 kernel.
// The choice is made for a whole line at once, so that either loop's loads
// stay together.
template <typename Put>
__device__ __forceinline__ void flux_line(Put put, const FftConst &fc, int k, int j, size_t base, int lane,
                                          const double *F, const double *U2b, double visc) {
  const Dims &d = fc.d;
  const int NX = d.NX;
  const size_t sK = d.LDX, sJ = (size_t)d.LDX * d.NZ2;
  const double *U3b = U2b + d.nphys();
  if (fc.orth) {
    for (int n = lane; n < NX; n += 32) {
      const size_t c = base + n;
      put(n, flux_orth(F[c], F[c + sK], F[c - sK], F[c + sJ], F[c - sJ], U2b[c], U2b[c + sJ], U3b[c], U3b[c + sK]));
    }
    return;
  }
  const FluxG12<double> g(fc, k, j, visc);
  for (int n = lane; n < NX; n += 32) {
    const size_t c = base + n;
    put(n, flux_gen(g, F[c], F[c + sK], F[c - sK], F[c + sJ], F[c - sJ], F[c + sK + sJ], F[c + sK - sJ],
                    F[c - sK + sJ], F[c - sK - sJ], U2b[c], U2b[c + sJ], U3b[c], U3b[c + sK]));
  }
}

// The FP32 register form asks for 8 blocks an SM (64 registers, spills of 8 to
// 48 bytes; 72 registers left 7): the step's forward transforms 10.6 -> 9.8 ms
// on 512 x 385 x 257.  A minimum of 0 leaves the other forms' allocation
// as the compiler chooses it.
template <typename T, int E, bool SHORT = false>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, (sizeof(T) == 4 && E > 0) ? 8 : 0)
    k_r2c(FftConst fc, R2cArgs args) {
  using V = typename Cx<T>::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *smem_c = reinterpret_cast<V *>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Dims &d = fc.d;
  const int nk = args.k1 - args.k0 + 1;
  // grid (ceil(nk / kWarpsPerBlock), nj): no index division (a 64-bit one
  // is a long integer sequence with FP64 steps)
  const int kw = (int)blockIdx.x * kWarpsPerBlock + warp;
  if (kw >= nk) return;
  const int k = args.k0 + kw;
  const int j = args.j0 + (int)blockIdx.y;
  const int M = fc.M;
  V *z = smem_c + (size_t)warp * fstride<E>(M);
  const size_t base = d.ip(0, k, j);
  constexpr bool kF = sizeof(T) == 4;
  const bool fin = kF && args.af != nullptr;  // FP32 copies of the inputs
  // Points go two at a time, and the loads of U pairs go out before any of them
  // is used: a load a turn leaves the memory waiting.  SHORT (NX <= 32): a point
  // a lane, as pairs would leave half the warp idle.
  using G = std::conditional_t<SHORT, One<T>, Two<T>>;
  constexpr int W = SHORT ? 1 : 2;
  const int items = SHORT ? 2 * M : M;
  auto batch = [&](auto U_, auto load, auto use) {
    constexpr int U = SHORT ? 1 : decltype(U_)::value, B = (E > 0 && E < U) ? E : U;
    for (int m0 = lane; m0 < items; m0 += 32 * B) {
      decltype(load(0)) v[B];
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (E > 0 || m0 + 32 * u < items) v[u] = load(m0 + 32 * u);
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (E > 0 || m0 + 32 * u < items) use(m0 + 32 * u, v[u]);
    }
  };
  constexpr std::integral_constant<int, 4> U4{};
  auto put = [&](V *y, int m, const G &v) {
    if constexpr (SHORT) reinterpret_cast<T *>(y)[m] = v.x;
    else y[m] = Cx<T>::make(v.x, v.y);
  };
  auto store = [&](int m, const G &v) { put(z, m, v); };
  auto flux = [&](V *y, auto *F, auto *b, double visc) {
    const FluxG12<T> g(fc, k, j, visc);
    auto line = [&](auto ORTH) {
      constexpr bool O = decltype(ORTH)::value;
      // a general pair is 26 values, an orthogonal one 18
      constexpr std::integral_constant<int, (kF && O) ? 2 : 1> UF{};
      batch(UF, [&](int m) { return flux_load<G, O>(d, base + W * m, F, b); },
            [&](int m, const FluxIn<G> &v) { put(y, m, flux_value<O>(g, v)); });
    };
    if (fc.orth) line(std::true_type{});
    else line(std::false_type{});
  };
  auto add = [&](V *y, auto *x, T es) {
    batch(U4, [&](int m) { return pts<G>(x + base + W * m); },
          [&](int m, const G &v) {
            if constexpr (SHORT) {
              T &o = reinterpret_cast<T *>(y)[m];
              o = o + es * v.x;
            } else {
              const V o = y[m];
              y[m] = Cx<T>::make(o.x + es * v.x, o.y + es * v.y);
            }
          });
  };
  if (args.pro == PRO_LOAD) {
    bool pairs = false;
    if constexpr (std::is_same_v<T, FF>) {
      // a float-float field: the pair as it is, no FP64 split
      pairs = args.alo != nullptr;
      if (pairs)
        batch(U4, [&](int m) {
          G v;
          if constexpr (SHORT) {
            v.x = FF(args.af[base + m], args.alo[base + m]);
          } else {
            const float2 h = *reinterpret_cast<const float2 *>(args.af + base + 2 * m);
            const float2 l = *reinterpret_cast<const float2 *>(args.alo + base + 2 * m);
            v.x = FF(h.x, l.x), v.y = FF(h.y, l.y);
          }
          return v;
        }, store);
    }
    // fin: an FP32 field (the increment of the state)
    if (!pairs) {
      if (fin) batch(U4, [&](int m) { return pts<G>(args.af + base + W * m); }, store);
      else batch(U4, [&](int m) { return pts<G>(args.a + base + W * m); }, store);
    }
  } else if (args.pro == PRO_PROD) {
    const T jac = from_f64<T>(fc.m.jac[d.m2(k, j)]);
    auto prod = [&](auto *a, auto *b) {
      struct In {
        G a, b;
      };
      batch(U4, [&](int m) { return In{pts<G>(a + base + W * m), pts<G>(b + base + W * m)}; },
            [&](int m, const In &v) {
              G r;
              r.x = jac * v.a.x * v.b.x;
              if constexpr (!SHORT) r.y = jac * v.a.y * v.b.y;
              put(z, m, r);
            });
    };
    if (fin) prod(args.af, args.bf);
    else prod(args.a, args.b);
  } else {
    if (fin) flux(z, args.af, args.bf, args.visc);
    else flux(z, args.a, args.b, args.visc);
  }
  if (args.pro != PRO_LOAD && (args.extra || args.extraf)) {
    // LES additions: jac * tau for a product, the precomputed terms for a flux
    const T es = (args.pro == PRO_PROD) ? from_f64<T>(fc.m.jac[d.m2(k, j)]) : (T)1.0;
    if (kF && args.extraf) add(z, args.extraf, es);
    else if (args.extra) add(z, args.extra, es);
  }
  // with fuse_flux the same line's flux term (PRO_FLUX of a2 against b2, and
  // its LES addition) goes through a second transform in the same warp
  const bool fuse = args.fuse_flux != 0;
  V *z2 = smem_c + (size_t)(kWarpsPerBlock + warp) * fstride<E>(M);
  if (fuse) {
    if (kF && args.a2f) flux(z2, args.a2f, args.b2f, args.visc2);
    else flux(z2, args.a2, args.b2, args.visc2);
    if (kF && args.extraf2) add(z2, args.extraf2, (T)1.0);
    else if (args.extra2) add(z2, args.extra2, (T)1.0);
  }
  __syncwarp();
  dif_fft_any<E>(z, M, tw_m<T>(fc), false, lane);
  if (fuse) dif_fft_any<E>(z2, M, tw_m<T>(fc), false, lane);
  // split: X[k] = E + W^k O, E = (Z_k + conj Z_{M-k})/2, O = -i (Z_k - conj Z_{M-k})/2
  cplx_t *dst = args.dst + d.ic(0, k, j);
  const T inv = from_f64<T>(fc.inv_nx);
  const T h = (T)0.5;
  const int NKX = d.NKX;
  const V *twn = tw_n<T>(fc);
  auto emit = [&](int kk, cplx_t o) {
    const int ik = fslot<E>(kk & (M - 1), fc.logM), im = fslot<E>((M - kk) & (M - 1), fc.logM);
    const V w = twn[kk];
    auto split = [&](const V *zz, T &tr, T &ti) {
      const V zk = zz[ik], zm = zz[im];
      const T er = h * (zk.x + zm.x), ei = h * (zk.y - zm.y);
      const T orr = h * (zk.y + zm.y), oi = -h * (zk.x - zm.x);
      tr = (er + (w.x * orr - w.y * oi)) * inv;
      ti = (ei + (w.x * oi + w.y * orr)) * inv;
    };
    T tr, ti;
    split(z, tr, ti);
    if (fuse) {
      // dst -= i kx X, then dst += X2: the two launches' FP64 updates in order
      T tr2, ti2;
      split(z2, tr2, ti2);
      if constexpr (kF) {
        const T kv = from_f64<T>(fc.kx[kk]);
        const cplx_t o1{o.re - f2d_bits((float)(T(0) * tr - kv * ti)), o.im - f2d_bits((float)(T(0) * ti + kv * tr))};
        dst[kk] = cplx_t{o1.re + f2d_bits((float)tr2), o1.im + f2d_bits((float)ti2)};
      } else {
        const double xr = (double)tr, xi = (double)ti, kv = fc.kx[kk];
        const cplx_t o1{o.re - (0.0 * xr - kv * xi), o.im - (0.0 * xi + kv * xr)};
        dst[kk] = cplx_t{o1.re + (double)tr2, o1.im + (double)ti2};
      }
      return;
    }
    if constexpr (kF) {
      // the FP32 result enters the FP64 field with one exact widening and
      // one FP64 add per component
      if (args.epi == EPI_STORE) {
        dst[kk] = cplx_t{f2d_bits((float)tr), f2d_bits((float)ti)};
      } else if (args.epi == EPI_ADD) {
        dst[kk] = cplx_t{o.re + f2d_bits((float)tr), o.im + f2d_bits((float)ti)};
      } else {
        const T kv = from_f64<T>(fc.kx[kk]);
        dst[kk] = cplx_t{o.re - f2d_bits((float)(T(0) * tr - kv * ti)), o.im - f2d_bits((float)(T(0) * ti + kv * tr))};
      }
      return;
    } else {
    const double xr = (double)tr, xi = (double)ti;
    if (args.epi == EPI_STORE) {
      dst[kk] = cplx_t{xr, xi};
    } else if (args.epi == EPI_ADD) {
      dst[kk] = cplx_t{o.re + xr, o.im + xi};
    } else {
      // CF = CF - CIKXP*CS with CIKXP = (0, kx)
      const double kv = fc.kx[kk];
      dst[kk] = cplx_t{o.re - (0.0 * xr - kv * xi), o.im - (0.0 * xi + kv * xr)};
    }
    }
  };
  constexpr int UE = SHORT ? 1 : 3;
  for (int k0 = lane; k0 <= NKX; k0 += 32 * UE) {
    cplx_t o[UE];
#pragma unroll
    for (int u = 0; u < UE; ++u)
      o[u] = (args.epi != EPI_STORE && k0 + 32 * u <= NKX) ? dst[k0 + 32 * u] : cplx_t{0.0, 0.0};
#pragma unroll
    for (int u = 0; u < UE; ++u)
      if (k0 + 32 * u <= NKX) emit(k0 + 32 * u, o[u]);
  }
  if (args.epi == EPI_STORE || args.zero_hi)
    for (int kk = NKX + 1 + lane; kk <= d.NX2P; kk += 32) dst[kk] = cplx_t{0.0, 0.0};
}

template <typename T, int E, bool SHORT = false>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_c2r(FftConst fc, C2rArgs args) {
  using V = typename Cx<T>::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *smem_c = reinterpret_cast<V *>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Dims &d = fc.d;
  const int nk = args.k1 - args.k0 + 1;
  // grid (ceil(nk / kWarpsPerBlock), nj): no index division (a 64-bit one
  // is a long integer sequence with FP64 steps)
  const int kw = (int)blockIdx.x * kWarpsPerBlock + warp;
  if (kw >= nk) return;
  const int k = args.k0 + kw;
  const int j = args.j0 + (int)blockIdx.y;
  const int M = fc.M, NKX = d.NKX;
  V *z = smem_c + (size_t)warp * fstride<E>(M);
  const cplx_t *src = args.src + d.ic(0, k, j);
  const cplx_t *src2 = args.src2 ? args.src2 + d.ic(0, k, j) : nullptr;
  // merge: Z'[k] = (X_k + conj X_{M-k}) + i (X_k - conj X_{M-k}) W^{-k}.
  // The spectrum is staged in z first, so that each mode's prologue (FP64
  // loads, the scale2 combination, the split into T) runs once; then each
  // lane merges the pair (k, M-k) in place (X_M = 0: k = 0 pairs with zero).
  // Loads go out four modes a lane at a time, before any of them is used: a
  // load a turn had 16 KB an SM on the way, and 3 TB/s is what that gives.
  constexpr int U = SHORT ? 1 : (E > 0 && E < 4) ? E : 4;
  for (int k0 = lane; k0 < M; k0 += 32 * U) {
    cplx_t v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = (k0 + 32 * u <= NKX) ? src[k0 + 32 * u] : cplx_t{0.0, 0.0};
    if (src2) {
      cplx_t w[U];
#pragma unroll
      for (int u = 0; u < U; ++u) w[u] = (k0 + 32 * u <= NKX) ? src2[k0 + 32 * u] : cplx_t{0.0, 0.0};
#pragma unroll
      for (int u = 0; u < U; ++u) {
        v[u].re = fma(args.scale2, w[u].re, v[u].re);
        v[u].im = fma(args.scale2, w[u].im, v[u].im);
      }
    }
    if (args.ik) {  // CIKXP * v
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const double kv = (k0 + 32 * u <= NKX) ? fc.kx[k0 + 32 * u] : 0.0, re = v[u].re;
        v[u].re = -(kv * v[u].im);
        v[u].im = kv * re;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int kk = k0 + 32 * u;
      if (kk >= M) break;
      if (kk == 0) v[u].im = 0.0;
      z[kk] = (kk <= NKX) ? Cx<T>::make(from_f64<T>(v[u].re), from_f64<T>(v[u].im)) : Cx<T>::make(T(0.0), T(0.0));
    }
  }
  __syncwarp();
  const V *twn = tw_n<T>(fc);
  auto merge = [&](V a, V b, V w) {
    const T sr = a.x + b.x, si = a.y - b.y;  // X_k + conj X_{M-k}
    const T dr = a.x - b.x, di = a.y + b.y;  // X_k - conj X_{M-k}
    const T tr = dr * w.x + di * w.y, ti = di * w.x - dr * w.y;  // (d)*conj(w)
    return Cx<T>::make(sr - ti, si + tr);   // + i*t
  };
  for (int kk = lane; kk <= (M >> 1); kk += 32) {
    const V a = z[kk];
    const V b = (kk == 0) ? Cx<T>::make(T(0.0), T(0.0)) : z[M - kk];
    z[kk] = merge(a, b, twn[kk]);
    if (kk != 0 && 2 * kk != M) z[M - kk] = merge(b, a, twn[M - kk]);
  }
  __syncwarp();
  dif_fft_any<E>(z, M, tw_m<T>(fc), true, lane);
  double *dst = args.dst ? args.dst + d.ip(0, k, j) : nullptr;
  float *dstf = args.dstf ? args.dstf + d.ip(0, k, j) : nullptr;
  if constexpr (std::is_same_v<T, FF>) {
    if (args.dstlo) {
      // float-float planes: the high part is also the field's FP32 copy
      float *dlo = args.dstlo + d.ip(0, k, j);
      for (int m = lane; m <= M; m += 32) {
        const V v = (m < M) ? z[fslot<E>(m, fc.logM)] : Cx<T>::make(T(0.0), T(0.0));
        *reinterpret_cast<float2 *>(dstf + 2 * m) = make_float2(v.x.hi, v.y.hi);
        *reinterpret_cast<float2 *>(dlo + 2 * m) = make_float2(v.x.lo, v.y.lo);
      }
      return;
    }
  }
  // two points at a time; the last pair is the padding x = NX, NX + 1
  for (int m = lane; m <= M; m += 32) {
    const V v = (m < M) ? z[fslot<E>(m, fc.logM)] : Cx<T>::make(T(0.0), T(0.0));
    if constexpr (sizeof(T) == 4) {
      if (dst) {
        dst[2 * m] = f2d_bits((float)v.x);
        dst[2 * m + 1] = f2d_bits((float)v.y);
      }
      if (dstf) *reinterpret_cast<float2 *>(dstf + 2 * m) = make_float2((float)v.x, (float)v.y);
    } else {
      if (dst) {
        dst[2 * m] = (double)v.x;
        dst[2 * m + 1] = (double)v.y;
      }
      if (dstf) *reinterpret_cast<float2 *>(dstf + 2 * m) = make_float2(d2f_bits((double)v.x), d2f_bits((double)v.y));
    }
  }
}

// ---------------------------------------------------------------------------
// The FP64 transforms.
//
// What bounds them: GB300's FP64 pipe, which takes a warp's instruction 64
// clocks a quarter SM whatever its active lanes (19 clocks an SM, measured).
// So the work is counted in warp instructions: every lane has a point in
// every one of them, and there are as few as the passes allow.
//   - Lines share a warp: a line of M = NX/2 complex points takes M/8 lanes
//     (M/16 at M = 512), 32 8/M lines a warp, where one line a warp left 16
//     lanes idle at NX = 64 and 28 at NX = 16.
//   - The complex transform goes in radix-8 and radix-4 passes in registers,
//     exchanged through shared memory (M = 256: three passes, 6,144 operations
//     a line against radix 2's 8,192).
//   - The split into (and the merge from) the real line's spectrum does modes k
//     and M - k together, whose sums and twiddle products differ in sign only:
//     ten or twelve operations for the two against sixteen for each; the scale
//     1/(2 NX) sits in the split's twiddles as an exponent.
// Measured: 98,945 lines of NX = 512 forward 2.09 -> 1.60 ms (the operations
// alone take 1.40), 4,225 lines of NX = 64 inverse 18.5 -> 12.3 us.
template <int M> struct Fft64 {
  static constexpr int PTS = (M == 512) ? 16 : 8;  // points a lane
  static constexpr int G = M / PTS;                // lanes a line
  static constexpr int LPW = 32 / G;               // lines a warp
  static constexpr int STRIDE = M + M / 8;         // a line in shared memory, padded
  // radices of the passes (0: no third pass)
  static constexpr int R1 = (M == 8 || M == 64 || M >= 128) ? 8 : 4;
  static constexpr int R2 = (M == 8) ? 0 : (M == 512 || M == 256 || M == 64 || M == 32) ? 8 : 4;
  static constexpr int R3 = (M == 512) ? 8 : (M == 256 || M == 128) ? 4 : 0;
};
// one pad element every 8, so that eight lanes a multiple of 8 elements apart
// read distinct banks
__device__ __forceinline__ int pad64(int e) { return e + (e >> 3); }

__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a times -i (INV: +i)
template <bool INV>
__device__ __forceinline__ double2 rot(double2 a) { return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x); }

template <bool INV>
__device__ __forceinline__ void fft4(double2 &a0, double2 &a1, double2 &a2, double2 &a3) {
  const double2 t0 = a0 + a2, t1 = a0 - a2, t2 = a1 + a3, t3 = rot<INV>(a1 - a3);
  a0 = t0 + t2;
  a1 = t1 + t3;
  a2 = t0 - t2;
  a3 = t1 - t3;
}
template <bool INV>
__device__ __forceinline__ void fft8(double2 *a) {
  constexpr double s = 0.70710678118654752440;
  double2 e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6], o0 = a[1], o1 = a[3], o2 = a[5], o3 = a[7];
  fft4<INV>(e0, e1, e2, e3);
  fft4<INV>(o0, o1, o2, o3);
  // W^1 and W^3 of order 8 are s (1 -+ i) and s (-1 -+ i): s goes into the sums
  const double2 p1 = o1 + rot<INV>(o1), r2 = rot<INV>(o2), p3 = rot<INV>(o3) - o3;
  a[0] = e0 + o0;
  a[4] = e0 - o0;
  a[1] = make_double2(fma(s, p1.x, e1.x), fma(s, p1.y, e1.y));
  a[5] = make_double2(fma(-s, p1.x, e1.x), fma(-s, p1.y, e1.y));
  a[2] = e2 + r2;
  a[6] = e2 - r2;
  a[3] = make_double2(fma(s, p3.x, e3.x), fma(s, p3.y, e3.y));
  a[7] = make_double2(fma(-s, p3.x, e3.x), fma(-s, p3.y, e3.y));
}

// One pass of radix R over blocks of B points of every line of the warp,
// z in place: output k1 of a butterfly takes the place of its input k1, times
// W_B^(n2 k1).  The last pass (B = R) puts its outputs in natural order, out(q,
// k1) the index of output k1 of block q.
template <int M, int R, int B, bool INV, typename Out>
__device__ __forceinline__ void pass64(double2 *z, const double2 *__restrict__ tw, int g, Out out) {
  using F = Fft64<M>;
  constexpr int m = B / R, N = F::PTS / R;  // butterflies a lane
  double2 a[N][R];
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const int b = g + u * F::G, q = b / m, n2 = b % m;
#pragma unroll
    for (int k = 0; k < R; ++k) a[u][k] = z[pad64(q * B + n2 + m * k)];
    if constexpr (R == 8) fft8<INV>(a[u]);
    else fft4<INV>(a[u][0], a[u][1], a[u][2], a[u][3]);
    if constexpr (m > 1) {
#pragma unroll
      for (int k = 1; k < R; ++k) {
        // W_M^t, t = n2 k M / B < M, from the half table
        const int t = n2 * k * (M / B);
        double2 w = tw[t & (M / 2 - 1)];
        if (t >= M / 2) w = make_double2(-w.x, -w.y);
        if (INV) w.y = -w.y;
        a[u][k] = cmul(a[u][k], w);
      }
    }
  }
  if constexpr (m == 1) __syncwarp();  // the outputs of one lane fall on the inputs of others
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const int b = g + u * F::G, q = b / m, n2 = b % m;
#pragma unroll
    for (int k = 0; k < R; ++k) z[pad64((m > 1) ? q * B + n2 + m * k : out(q, k))] = a[u][k];
  }
  __syncwarp();
}
// The warp's lines, each M complex points at z (this lane's line), natural
// order in and out.
template <int M, bool INV>
__device__ __forceinline__ void fft64(double2 *z, const double2 *tw, int g) {
  using F = Fft64<M>;
  auto none = [](int, int) { return 0; };
  __syncwarp();
  if constexpr (F::R2 == 0 && F::R3 == 0) {
    pass64<M, F::R1, M, INV>(z, tw, g, [](int, int k) { return k; });
  } else if constexpr (F::R3 == 0) {
    pass64<M, F::R1, M, INV>(z, tw, g, none);
    pass64<M, F::R2, F::R2, INV>(z, tw, g, [](int q, int k) { return q + F::R1 * k; });
  } else {
    pass64<M, F::R1, M, INV>(z, tw, g, none);
    pass64<M, F::R2, M / F::R1, INV>(z, tw, g, none);
    // block q = k1 R2 + k1'
    pass64<M, F::R3, F::R3, INV>(z, tw, g, [](int q, int k) {
      return q / F::R2 + F::R1 * (q % F::R2) + F::R1 * F::R2 * k;
    });
  }
}

// w 2^-e for a twiddle (zero stays zero), on the integer pipe
__device__ __forceinline__ double scale_tw(double w, int e) {
  const long long u = __double_as_longlong(w);
  return (u << 1) ? __longlong_as_double(u - ((long long)e << 52)) : w;
}

template <int M>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_r2c64(FftConst fc, R2cArgs args) {
  using F = Fft64<M>;
  constexpr int NX = 2 * M;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Dims &d = fc.d;
  const int nk = args.k1 - args.k0 + 1;
  const int kw = ((int)blockIdx.x * kWarpsPerBlock + warp) * F::LPW;  // the warp's first line
  if (kw >= nk) return;
  const int nl = min(F::LPW, nk - kw), k0 = args.k0 + kw;
  const int j = args.j0 + (int)blockIdx.y;
  double2 *zw = reinterpret_cast<double2 *>(smem_raw) + (size_t)warp * F::LPW * F::STRIDE;
  double2 *zw2 = zw + (size_t)kWarpsPerBlock * F::LPW * F::STRIDE;  // the fused flux's lines
  auto at = [&](double2 *w, int l, int n) -> double & {
    return reinterpret_cast<double *>(w + l * F::STRIDE + pad64(n >> 1))[n & 1];
  };
  if (args.pro == PRO_LOAD) {
    // flat over the warp's lines (short lines fill the lanes together)
    for (int t = lane; t < nl * NX; t += 32) at(zw, t / NX, t % NX) = args.a[d.ip(0, k0 + t / NX, j) + t % NX];
  } else {
    for (int l = 0; l < nl; ++l) {
      const int k = k0 + l;
      const size_t base = d.ip(0, k, j);
      const double jac = fc.m.jac[d.m2(k, j)];
      if (args.pro == PRO_PROD)
        for (int n = lane; n < NX; n += 32) at(zw, l, n) = jac * args.a[base + n] * args.b[base + n];
      else
        flux_line([&](int n, double v) { at(zw, l, n) = v; }, fc, k, j, base, lane, args.a, args.b, args.visc);
      if (args.extra) {
        // LES additions: jac * tau for a product, the precomputed terms for a flux
        const double es = (args.pro == PRO_PROD) ? jac : 1.0;
        for (int n = lane; n < NX; n += 32) at(zw, l, n) += es * args.extra[base + n];
      }
      if (args.fuse_flux) {
        flux_line([&](int n, double v) { at(zw2, l, n) = v; }, fc, k, j, base, lane, args.a2, args.b2, args.visc2);
        if (args.extra2)
          for (int n = lane; n < NX; n += 32) at(zw2, l, n) += args.extra2[base + n];
      }
    }
  }
  const bool fuse = args.fuse_flux != 0;
  fft64<M, false>(zw + (lane / F::G) * F::STRIDE, fc.tw_m, lane % F::G);
  if (fuse) fft64<M, false>(zw2 + (lane / F::G) * F::STRIDE, fc.tw_m, lane % F::G);
  // split: X_k = (s1 + u, d1 + v) / (2 NX), X_{M-k} = (s1 - u, v - d1) / (2 NX)
  // with s1 = Re(Z_k + Z_{M-k}), d1 = Im(Z_k - Z_{M-k}) and (u, v) the
  // product of W_NX^k with (Im(Z_k + Z_{M-k}), -Re(Z_k - Z_{M-k}))
  const int NKX = d.NKX;
  const double hi = 0.5 * fc.inv_nx;
  const int he = 1 + 31 - __clz(NX);
  auto split = [&](const double2 *z, int k, double2 w, double2 &x, double2 &y) {
    const double2 a = z[pad64(k & (M - 1))], b = z[pad64((M - k) & (M - 1))];
    const double s1 = a.x + b.x, d1 = a.y - b.y, s2 = a.y + b.y, d2 = a.x - b.x;
    const double u = w.x * s2 + w.y * d2, v = w.y * s2 - w.x * d2;
    x = make_double2(fma(hi, s1, u), fma(hi, d1, v));
    y = make_double2(fma(hi, s1, -u), fma(-hi, d1, v));
  };
  auto emit = [&](int l, int kk, double2 x, double2 x2) {
    cplx_t *dst = args.dst + d.ic(0, k0 + l, j) + kk;
    if (args.epi == EPI_STORE) {
      *dst = cplx_t{x.x, x.y};
      return;
    }
    const cplx_t o = *dst;
    if (args.epi == EPI_ADD) {
      *dst = cplx_t{o.re + x.x, o.im + x.y};
    } else {
      // CF = CF - CIKXP*CS with CIKXP = (0, kx), then the fused flux's X2
      const double kv = fc.kx[kk];
      cplx_t r{o.re + kv * x.y, o.im - kv * x.x};
      if (fuse) r = cplx_t{r.re + x2.x, r.im + x2.y};
      *dst = r;
    }
  };
  auto pair = [&](int l, int k) {
    const double2 *z = zw + l * F::STRIDE, *z2 = zw2 + l * F::STRIDE;
    const bool lo = k <= NKX, up = k > 0 && 2 * k < M && M - k <= NKX;
    if (!lo && !up) return;
    double2 w = fc.tw_n[k], x, y, x2 = make_double2(0.0, 0.0), y2 = x2;
    w = make_double2(scale_tw(w.x, he), scale_tw(w.y, he));
    split(z, k, w, x, y);
    if (fuse) split(z2, k, w, x2, y2);
    if (lo) emit(l, k, x, x2);
    if (up) emit(l, M - k, y, y2);
  };
  // k = 1..M/2 flat over the lines, k = 0 one lane a line
  for (int t = lane; t < nl * (M / 2); t += 32) pair(t / (M / 2), 1 + t % (M / 2));
  if (lane < nl) pair(lane, 0);
  if (args.epi == EPI_STORE || args.zero_hi)
    for (int l = 0; l < nl; ++l) {
      cplx_t *dst = args.dst + d.ic(0, k0 + l, j);
      for (int kk = NKX + 1 + lane; kk <= d.NX2P; kk += 32) dst[kk] = cplx_t{0.0, 0.0};
    }
}

template <int M>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_c2r64(FftConst fc, C2rArgs args) {
  using F = Fft64<M>;
  constexpr int NX = 2 * M;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Dims &d = fc.d;
  const int nk = args.k1 - args.k0 + 1;
  const int kw = ((int)blockIdx.x * kWarpsPerBlock + warp) * F::LPW;
  if (kw >= nk) return;
  const int nl = min(F::LPW, nk - kw), k0 = args.k0 + kw;
  const int j = args.j0 + (int)blockIdx.y;
  const int NKX = d.NKX;
  double2 *zw = reinterpret_cast<double2 *>(smem_raw) + (size_t)warp * F::LPW * F::STRIDE;
  auto X = [&](int l, int kk) {
    if (kk > NKX) return make_double2(0.0, 0.0);
    const size_t c = d.ic(0, k0 + l, j) + kk;
    cplx_t v = args.src[c];
    if (args.src2) {
      const cplx_t w = args.src2[c];
      v.re = v.re + args.scale2 * w.re;
      v.im = v.im + args.scale2 * w.im;
    }
    if (args.ik) {  // CIKXP * v
      const double kv = fc.kx[kk], re = v.re;
      v.re = -(kv * v.im);
      v.im = kv * re;
    }
    if (kk == 0) v.im = 0.0;
    return make_double2(v.re, v.im);
  };
  // merge: Z'_k = (sr - ti, si + tr), Z'_{M-k} = (sr + ti, tr - si) with s, d =
  // X_k +- conj X_{M-k} and t = d conj(W_NX^k); X_M = 0
  auto merge = [&](int l, int k) {
    double2 *z = zw + l * F::STRIDE;
    const double2 a = X(l, k), w = fc.tw_n[k];
    double sr = a.x, si = a.y, dr = a.x, di = a.y;
    if (k > 0 && M - k <= NKX) {
      const double2 b = X(l, M - k);
      sr = a.x + b.x;
      si = a.y - b.y;
      dr = a.x - b.x;
      di = a.y + b.y;
    }
    const double tr = dr * w.x + di * w.y, ti = di * w.x - dr * w.y;
    z[pad64(k)] = make_double2(sr - ti, si + tr);
    if (k > 0 && 2 * k < M) z[pad64(M - k)] = make_double2(sr + ti, tr - si);
  };
  for (int t = lane; t < nl * (M / 2); t += 32) merge(t / (M / 2), 1 + t % (M / 2));
  if (lane < nl) merge(lane, 0);
  fft64<M, true>(zw + (lane / F::G) * F::STRIDE, fc.tw_m, lane % F::G);
  for (int t = lane; t < nl * (NX / 2 + 1); t += 32) {
    // two points at a time; the last pair is the padding
    const int l = t / (NX / 2 + 1), e = t - l * (NX / 2 + 1);
    const double2 v = (e < M) ? zw[l * F::STRIDE + pad64(e)] : make_double2(0.0, 0.0);
    const size_t q = d.ip(0, k0 + l, j) + 2 * e;
    if (args.dst) {
      args.dst[q] = v.x;
      args.dst[q + 1] = v.y;
    }
    if (args.dstf) {
      args.dstf[q] = d2f_bits(v.x);
      args.dstf[q + 1] = d2f_bits(v.y);
    }
  }
}

// the FP64 launch of nk lines in each of nj rows; false: no such M
template <int M>
void run64(int nk, int nj, cudaStream_t s, const FftConst &fc, const R2cArgs *r, const C2rArgs *c) {
  using F = Fft64<M>;
  const dim3 grid((unsigned)((nk + kWarpsPerBlock * F::LPW - 1) / (kWarpsPerBlock * F::LPW)), (unsigned)nj);
  const size_t smem = sizeof(double2) * F::STRIDE * F::LPW * kWarpsPerBlock * ((r && r->fuse_flux) ? 2 : 1);
  if (r) k_r2c64<M><<<grid, 32 * kWarpsPerBlock, smem, s>>>(fc, *r);
  else k_c2r64<M><<<grid, 32 * kWarpsPerBlock, smem, s>>>(fc, *c);
}
bool launch64(int nk, int nj, cudaStream_t s, const FftConst &fc, const R2cArgs *r, const C2rArgs *c) {
  // Few lines leave the GPU idle, and what counts is one warp's chain of FP64
  // instructions: spread over a whole warp a line has fewer.  1,000 lines,
  // forward: NX = 16 7.9 us against 13.6, NX = 64 8.3 against 12.4, NX = 128
  // 10.3 against 14.4; 2,000 lines: equal at NX = 64 and 128; NX = 256 12.3
  // against 14.4 at 500 and 16.4 against 14.4 at 1,000; from NX = 512 on packed
  // lines are ahead with 260 lines as well (16.4 us against 20.5).
  const long lines = (long)nk * nj;
  if (fc.M <= 128 && lines < 2000 && lines * 2 * fc.M < 180000) return false;
  switch (fc.M) {
    case 8: run64<8>(nk, nj, s, fc, r, c); return true;
    case 16: run64<16>(nk, nj, s, fc, r, c); return true;
    case 32: run64<32>(nk, nj, s, fc, r, c); return true;
    case 64: run64<64>(nk, nj, s, fc, r, c); return true;
    case 128: run64<128>(nk, nj, s, fc, r, c); return true;
    case 256: run64<256>(nk, nj, s, fc, r, c); return true;
    case 512: run64<512>(nk, nj, s, fc, r, c); return true;
    default: return false;
  }
}

// Launch a transform with one line a warp (launch64 takes most FP64 ones).
// The register form of the FFT pays in the FP32 transforms (measured on 512 x 385 x 257: the inverse 0.34 -> 0.23 ms per
// launch; the forward ones, since each launch fuses a component's product
// and flux transforms, 13.9 -> 11.7 ms a step); in the float-float ones its
// extra registers cost more than the shared-memory passes it saves, so they
// keep the loop.
// What then bounds the FP32 ones is the loads on their way: with one a turn of
// each loop an SM waits on 16 KB at 3 TB/s.  So points are loaded two at a time
// and several pairs, or four modes, before any is used.  512 x 385 x 257, a
// step: forward 8.81 -> 7.84 ms, inverse 5.91 -> 4.95 (six modes at a time
// 5.55, at the cost of resident blocks); 128 x 129 x 97 0.63 -> 0.56 and 0.66 ->
// 0.60; 64 x 65 x 65 0.243 -> 0.233 and 0.401 -> 0.388; the float-float
// inverse of 256 x 193 x 129 2.18 -> 2.02.
// Lines of NX <= 32 keep a point and a mode a lane: pairs leave half a warp idle.
// Two steps of 32 x 257 x 193, forward 2.90 with pairs, 2.42 so; with LES 3.88
// and 3.18; 16 x 257 x 193 2.57 and 2.17, 3.41 and 2.79.
template <typename T>
void run_r2c(dim3 grid, size_t smem, cudaStream_t s, const FftConst &fc, const R2cArgs &a) {
  const unsigned nt = 32 * kWarpsPerBlock;
  if constexpr (std::is_same_v<T, float>) {
    switch (fc.M) {
      case 32: k_r2c<T, 1><<<grid, nt, smem, s>>>(fc, a); return;
      case 64: k_r2c<T, 2><<<grid, nt, smem, s>>>(fc, a); return;
      case 128: k_r2c<T, 4><<<grid, nt, smem, s>>>(fc, a); return;
      case 256: k_r2c<T, 8><<<grid, nt, smem, s>>>(fc, a); return;
      case 512: k_r2c<T, 16><<<grid, nt, smem, s>>>(fc, a); return;
      default: break;
    }
  }
  if (fc.M <= 16) k_r2c<T, 0, true><<<grid, nt, smem, s>>>(fc, a);
  else if constexpr (!std::is_same_v<T, float>) k_r2c<T, 0><<<grid, nt, smem, s>>>(fc, a);
}
template <typename T>
void run_c2r(dim3 grid, size_t smem, cudaStream_t s, const FftConst &fc, const C2rArgs &a) {
  const unsigned nt = 32 * kWarpsPerBlock;
  if constexpr (std::is_same_v<T, float>) {
    switch (fc.M) {
      case 32: k_c2r<T, 1><<<grid, nt, smem, s>>>(fc, a); return;
      case 64: k_c2r<T, 2><<<grid, nt, smem, s>>>(fc, a); return;
      case 128: k_c2r<T, 4><<<grid, nt, smem, s>>>(fc, a); return;
      case 256: k_c2r<T, 8><<<grid, nt, smem, s>>>(fc, a); return;
      case 512: k_c2r<T, 16><<<grid, nt, smem, s>>>(fc, a); return;
      default: break;
    }
  }
  if (fc.M <= 16) k_c2r<T, 0, true><<<grid, nt, smem, s>>>(fc, a);
  else if constexpr (!std::is_same_v<T, float>) k_c2r<T, 0><<<grid, nt, smem, s>>>(fc, a);
}
template <typename T>
void smem_attributes() {
  const int b = 96 * 1024;
  if constexpr (!std::is_same_v<T, float>) {
    EK_CUDA(cudaFuncSetAttribute(k_r2c<T, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_c2r<T, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  }
  if constexpr (std::is_same_v<T, double>) {
    EK_CUDA(cudaFuncSetAttribute(k_r2c64<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c64<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c64<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c64<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c64<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c64<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c64<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  }
  if constexpr (std::is_same_v<T, float>) {
    EK_CUDA(cudaFuncSetAttribute(k_c2r<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c<T, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c<T, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c<T, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_r2c<T, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_c2r<T, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_c2r<T, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_c2r<T, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    EK_CUDA(cudaFuncSetAttribute(k_c2r<T, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  }
}

FftConst make_const(Ctx &c) {
  FftConst f;
  f.d = c.d;
  f.M = c.d.NX / 2;
  int lg = 0;
  while ((1 << lg) < f.M) ++lg;
  f.logM = lg;
  f.tw_m = c.tw_m;
  f.tw_n = c.tw_n;
  f.tw_mf = c.tw_mf;
  f.tw_nf = c.tw_nf;
  f.tw_mff = c.tw_mff;
  f.tw_nff = c.tw_nff;
  f.kx = c.kx;
  f.inv_nx = 1.0 / c.d.NX;
  f.m = c.m;
  f.orth = c.orth ? 1 : 0;
  return f;
}

}  // namespace

// FP32 arithmetic for this transform?  fft_fp32 = 1: only the transforms
// marked low-precision (the nonlinear products and fluxes, whose results
// enter the step multiplied by the time step); 2: every transform.
bool fft_lowp(const Ctx &c, int lowp) { return c.p.fft_fp32 >= 2 || (c.p.fft_fp32 == 1 && lowp); }
// float-float for the other transforms under ff_arith
bool fft_ff(const Ctx &c, int lowp) { return c.p.ff_arith && !fft_lowp(c, lowp); }

void launch_r2c(Ctx &c, const R2cArgs &a) {
  const FftConst fc = make_const(c);
  const long nlines = (long)(a.k1 - a.k0 + 1) * (a.j1 - a.j0 + 1);
  if (nlines <= 0) return;
  const dim3 grid((unsigned)((a.k1 - a.k0 + 1 + kWarpsPerBlock - 1) / kWarpsPerBlock), (unsigned)(a.j1 - a.j0 + 1));
  if (a.fuse_flux && (a.pro != PRO_PROD || a.epi != EPI_SUB_IK))
    throw CudaError("r2c: a fused flux goes with a product and dst -= i kx X");
  // a fused launch holds both lines' spectra
  const size_t smem = sizeof(double2) * fc.M * kWarpsPerBlock * (a.fuse_flux ? 2 : 1);
  // algorithmic bytes: the input planes read (the flux's field, U2b and U3b;
  // a fused launch reads its product's second factor once, as the flux's
  // field) at the size of the copy the kernel reads, and the spectrum
  // (an FP32 kernel reading FP32 copies: 4 bytes an element; FP64 fields,
  // or float-float planes as hi and lo: 8)
  const bool lp = fft_lowp(c, a.lowp);
  const double elt = (lp && a.af) ? 4.0 : 8.0;
  const int nops = (a.pro == PRO_LOAD) ? 1 : (a.pro == PRO_PROD) ? (a.fuse_flux ? 4 : 2) : 3;
  const double epi = (a.epi == EPI_STORE) ? 16.0 * (c.d.NX2P + 1) : 32.0 * (c.d.NKX + 1);
  KScope ks(c, KC_R2C, nlines * (elt * c.d.NX * nops + epi));
  // FP32 spectra: 8 bytes an element, with the register form's pad slots
  const size_t smem_f = sizeof(float2) * (fc.M + 32) * kWarpsPerBlock * (a.fuse_flux ? 2 : 1);
  if (lp) run_r2c<float>(grid, smem_f, c.stream, fc, a);
  else if (fft_ff(c, a.lowp)) run_r2c<FF>(grid, smem, c.stream, fc, a);
  else if (!launch64(a.k1 - a.k0 + 1, a.j1 - a.j0 + 1, c.stream, fc, &a, nullptr))
    run_r2c<double>(grid, smem, c.stream, fc, a);
  after_launch(c);
}

void launch_c2r(Ctx &c, const C2rArgs &a) {
  const FftConst fc = make_const(c);
  const long nlines = (long)(a.k1 - a.k0 + 1) * (a.j1 - a.j0 + 1);
  if (nlines <= 0) return;
  const dim3 grid((unsigned)((a.k1 - a.k0 + 1 + kWarpsPerBlock - 1) / kWarpsPerBlock), (unsigned)(a.j1 - a.j0 + 1));
  const size_t smem = sizeof(double2) * fc.M * kWarpsPerBlock;
  // algorithmic bytes: the spectra read, the planes written (FP64, FP32 copy
  // and float-float low part as given)
  const double out = (a.dst ? 8.0 : 0.0) + (a.dstf ? 4.0 : 0.0) + (a.dstlo ? 4.0 : 0.0);
  KScope ks(c, KC_C2R, nlines * (16.0 * (c.d.NKX + 1) * (a.src2 ? 2 : 1) + out * (c.d.NX + 2)));
  const size_t smem_f = sizeof(float2) * (fc.M + 32) * kWarpsPerBlock;
  if (fft_lowp(c, a.lowp)) run_c2r<float>(grid, smem_f, c.stream, fc, a);
  else if (fft_ff(c, a.lowp)) run_c2r<FF>(grid, smem, c.stream, fc, a);
  else if (!launch64(a.k1 - a.k0 + 1, a.j1 - a.j0 + 1, c.stream, fc, nullptr, &a))
    run_c2r<double>(grid, smem, c.stream, fc, a);
  after_launch(c);
}

}  // namespace ek

namespace ek {
void fft_init_attributes() {
  static OncePerDevice once;
  once(current_device(), [] {
    smem_attributes<double>();
    smem_attributes<float>();
    smem_attributes<FF>();
  });
}
}  // namespace ek

// ---------------------------------------------------------------------------
// Context-free batched x-transforms: the FFT_X_TO_FOURIER_OP /
// FFT_X_TO_PHYSICAL_OP pair that the reference calls (e.g. duct.F90:700 and
// mpi_duct.F90:308) and whose source (fft.F90) is missing from its tree.
namespace ek {
namespace {

thread_local std::string t_last_error;

__global__ void k_twiddles(double2 *tw_m, double2 *tw_n, int nx) {
  const int M = nx / 2;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t <= M; t += gridDim.x * blockDim.x) {
    double s, c;
    if (t < M / 2) {
      sincospi(-2.0 * t / M, &s, &c);
      tw_m[t] = make_double2(c, s);
    }
    sincospi(-2.0 * t / nx, &s, &c);
    tw_n[t] = make_double2(c, s);
  }
}

bool fft_args_ok(int nx, int nkx, long nlines, const void *in, const void *out) {
  if (nx < 8 || nx > 1024 || (nx & (nx - 1))) {
    t_last_error = "nx must be a power of two in [8, 1024]";
    return false;
  }
  if (nkx < 0 || nkx >= nx / 2) {
    t_last_error = "nkx must be in [0, nx/2)";
    return false;
  }
  if (nlines < 0 || nlines > (1L << 30) || (nlines > 0 && (!in || !out))) {
    t_last_error = "bad line count or NULL buffer";
    return false;
  }
  return true;
}

// Twiddle tables of the context-free transforms: cudaMalloc'd once per
// (device, nx) and kept for the life of the process.  Their size in double2,
// shared with the fixed table of the allocation-free entry point below.
constexpr int twiddle_count(int nx) { return (nx / 2) / 2 + nx / 2 + 1; }
std::mutex g_tw_mu;
std::map<std::pair<int, int>, double2 *> g_tw_cache;
double2 *cached_twiddles(int nx, cudaStream_t s) {
  int dev = 0;
  EK_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_tw_mu);
  auto &cache = g_tw_cache;
  auto it = cache.find({dev, nx});
  if (it != cache.end()) return it->second;
  const int M = nx / 2;
  double2 *tw = nullptr;
  EK_CUDA(cudaMalloc(&tw, sizeof(double2) * twiddle_count(nx)));
  k_twiddles<<<4, 256, 0, s>>>(tw, tw + M / 2, nx);
  EK_CUDA(cudaPeekAtLastError());
  EK_CUDA(cudaStreamSynchronize(s));
  cache[{dev, nx}] = tw;
  return tw;
}

FftConst standalone_const(int nx, int nkx, long nlines, const double2 *tw) {
  FftConst f{};
  Dims &d = f.d;
  d.NX = nx;
  d.NKX = nkx;
  d.NX2P = nx / 2;
  d.LDX = nx + 2;
  d.LDC = nx / 2 + 1;
  d.NZ2 = (int)nlines;  // lines are indexed as (k, j = 0)
  d.NY2 = 1;
  f.M = nx / 2;
  int lg = 0;
  while ((1 << lg) < f.M) ++lg;
  f.logM = lg;
  f.tw_m = tw;
  f.tw_n = tw + f.M / 2;
  f.inv_nx = 1.0 / nx;
  return f;
}

int run_standalone(bool forward, int nx, int nkx, long nlines, const double *in, double *out, cudaStream_t s,
                   const double2 *tw) {
  if (nlines == 0) return EK_OK;
  const FftConst fc = standalone_const(nx, nkx, nlines, tw);
  const dim3 grid((unsigned)((nlines + kWarpsPerBlock - 1) / kWarpsPerBlock), 1u);
  const size_t smem = sizeof(double2) * fc.M * kWarpsPerBlock;
  if (forward) {
    R2cArgs a{};
    a.a = in;
    a.dst = reinterpret_cast<cplx_t *>(out);
    a.pro = PRO_LOAD;
    a.epi = EPI_STORE;
    a.k0 = 0; a.k1 = (int)nlines - 1; a.j0 = 0; a.j1 = 0;
    if (!launch64((int)nlines, 1, s, fc, &a, nullptr)) run_r2c<double>(grid, smem, s, fc, a);
  } else {
    C2rArgs a{};
    a.src = reinterpret_cast<const cplx_t *>(in);
    a.dst = out;
    a.k0 = 0; a.k1 = (int)nlines - 1; a.j0 = 0; a.j1 = 0;
    if (!launch64((int)nlines, 1, s, fc, nullptr, &a)) run_c2r<double>(grid, smem, s, fc, a);
  }
  EK_CUDA(cudaPeekAtLastError());
  return EK_OK;
}

int standalone(bool forward, int nx, int nkx, long nlines, const double *in, double *out, void *stream) {
  if (!fft_args_ok(nx, nkx, nlines, in, out)) return EK_ERR_ARG;
  try {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    fft_init_attributes();
    const double2 *tw = cached_twiddles(nx, s);
    return run_standalone(forward, nx, nkx, nlines, in, out, s, tw);
  } catch (const CudaError &e) {
    t_last_error = e.msg;
    return EK_ERR_CUDA;
  }
}

}  // namespace

const char *last_global_error() { return t_last_error.c_str(); }

}  // namespace ek

extern "C" int ekgpu_fft_table_count(void) {
  std::lock_guard<std::mutex> lk(ek::g_tw_mu);
  return (int)ek::g_tw_cache.size();
}

extern "C" int ekgpu_fft_x_to_fourier(int nx, int nkx, long nlines, const double *in_dev, double *out_dev,
                                      void *stream) {
  return ek::standalone(true, nx, nkx, nlines, in_dev, out_dev, stream);
}

extern "C" int ekgpu_fft_x_to_physical(int nx, int nkx, long nlines, const double *in_dev, double *out_dev,
                                       void *stream) {
  return ek::standalone(false, nx, nkx, nlines, in_dev, out_dev, stream);
}

// ---------------------------------------------------------------------------
// ekgpu_fft_x_to_fourier_noalloc: the forward transform above with its
// twiddle scratch in a fixed device array instead of cudaMalloc'd memory.
namespace ek {
namespace {

// Largest nx the array holds: (nx/4 + nx/2 + 1) twiddles = 769 for nx = 1024
// (12.3 KB, resident on every GPU that loads the library until exit).
constexpr int kNoAllocMaxNx = 1024;
constexpr int kNoAllocTw = kNoAllocMaxNx / 4 + kNoAllocMaxNx / 2 + 1;
static_assert(kNoAllocTw == twiddle_count(kNoAllocMaxNx), "the fixed table must hold the cached layout at nx = 1024");
static __device__ __align__(256) double2 g_noalloc_twiddles[kNoAllocTw];

// Device address of g_noalloc_twiddles, looked up once per device (the host
// symbol itself is only a stand-in and must never reach a kernel).
double2 *noalloc_scratch(int &err) {
  static std::mutex mu;
  static double2 *addr[128] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 128) {
    t_last_error = std::string("ekgpu_fft_x_to_fourier_noalloc: cudaGetDevice: ") + cudaGetErrorString(e);
    err = EK_ERR_CUDA;
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(mu);
  if (!addr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_twiddles);
    if (e != cudaSuccess || !p) {
      t_last_error = std::string("ekgpu_fft_x_to_fourier_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e);
      err = EK_ERR_CUDA;
      return nullptr;
    }
    addr[dev] = static_cast<double2 *>(p);
  }
  return addr[dev];
}

}  // namespace
}  // namespace ek

extern "C" int ekgpu_fft_x_to_fourier_noalloc(int nx, int nkx, long nlines, const double *in_dev, double *out_dev,
                                              void *stream) {
  using namespace ek;
  if (nx > kNoAllocMaxNx) {
    t_last_error = "ekgpu_fft_x_to_fourier_noalloc: nx exceeds the fixed scratch maximum of 1024";
    return EK_ERR_ARG;
  }
  if (!fft_args_ok(nx, nkx, nlines, in_dev, out_dev)) return EK_ERR_ARG;
  int err = EK_OK;
  double2 *tw = noalloc_scratch(err);
  if (!tw) return err;
  try {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    fft_init_attributes();
    // the whole table is rewritten on every call, before the transform reads it
    k_twiddles<<<4, 256, 0, s>>>(tw, tw + nx / 4, nx);
    EK_CUDA(cudaPeekAtLastError());
    return run_standalone(true, nx, nkx, nlines, in_dev, out_dev, s, tw);
  } catch (const CudaError &e) {
    t_last_error = e.msg;
    return EK_ERR_CUDA;
  }
}
