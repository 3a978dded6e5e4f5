// PME reciprocal-space kernels; see pme.h.
#include "pme.h"

#include <cuda.h>  // CUtensorMap (the encoder is fetched through the runtime)

#include <algorithm>
#include <atomic>
#include <cmath>
#include <functional>
#include <mutex>
#include <numeric>
#include <stdexcept>
#include <vector>

#include "common.h"
#include "device_util.cuh"

namespace apo {
namespace {

constexpr int kPlaneThreadsMax = 1024;
// dynamic shared memory a plane transform may use: the SM's 227 KB per
// block less the kernels' static digit-reversal table, and what is left of it
// beside the twiddles
constexpr size_t kPlaneSmemMax = 227 * 1024 - 1024;
constexpr size_t kPlaneSmemTw = kPlaneSmemMax - 512 * sizeof(float2);
// the tensor-map argument of launches that move their slabs with plain loads
const CUtensorMap kNoTensorMap{};
constexpr int kPencilThreads = 256;
// a pencil slab's complex columns x planes: at most 24 x 256 (set_tiles), and
// room to start it on 128 bytes
constexpr size_t kPencilSmemMax = 24 * 256 * sizeof(float2) + 128;

// ------------------------------------------------------------------------
// B-spline weights (Essmann et al. recursion, the reference's calc_one_theta,
// src/CudaPMERecip.cu:438-470)
// ------------------------------------------------------------------------
template <int ORDER>
__device__ __forceinline__ void bspline(float w, float (&th)[ORDER], float (&dth)[ORDER]) {
  th[ORDER - 1] = 0.f;
  th[1] = w;
  th[0] = 1.f - w;
#pragma unroll
  for (int k = 3; k <= ORDER - 1; ++k) {
    const float div = 1.f / (float)(k - 1);
    th[k - 1] = div * w * th[k - 2];
#pragma unroll
    for (int j = 1; j <= k - 2; ++j)
      th[k - j - 1] = div * ((w + j) * th[k - j - 2] + (k - j - w) * th[k - j - 1]);
    th[0] = div * (1.f - w) * th[0];
  }
  dth[0] = -th[0];
#pragma unroll
  for (int j = 1; j < ORDER; ++j) dth[j] = th[j - 1] - th[j];
  const float div = 1.f / (float)(ORDER - 1);
  th[ORDER - 1] = div * w * th[ORDER - 2];
#pragma unroll
  for (int j = 1; j <= ORDER - 2; ++j)
    th[ORDER - j - 1] =
        div * ((w + j) * th[ORDER - j - 2] + (ORDER - j - w) * th[ORDER - j - 1]);
  th[0] = div * (1.f - w) * th[0];
}

// grid anchoring of the reference (include/cuda_pme_spread.h:64-81):
// w = x/L + 2, fr = n (w - (floor(w+0.5) - 0.5)), points floor(fr)+0..p-1.
// Evaluated in FP64 from the exact global position (cluster origin + local
// offset): in FP32 the rounding of w near 2 (1.2e-7) times n shifts the
// B-spline fraction by up to n * 1.2e-7 grid units, which at a 216-point
// axis is the largest error of the reciprocal force.  The fraction itself
// is returned in FP32 for the spline recursion.
__device__ __forceinline__ void anchor(double x, double recip, int n, int &i0, float &w) {
  const double t = x * recip + 2.0;
  const double fr = (double)n * (t - (floor(t + 0.5) - 0.5));
  // non-finite or exploded coordinates must not index outside the grid
  if (!(fr >= 0.0 && fr < (double)n)) {
    i0 = fr >= (double)n ? n - 1 : 0;
    w = 0.f;
    return;
  }
  i0 = (int)fr;
  w = (float)(fr - (double)i0);
  if (i0 > n - 1) i0 = n - 1;
}

// global position of a sorted slot: the cluster origin (a multiple of
// 1/64 A, exact in FP32) plus the local offset, summed without rounding
__device__ __forceinline__ double3 global_pos(const float4 &p, const float4 *origin, int s) {
  if (!origin) return make_double3(p.x, p.y, p.z);
  const float4 o = origin[s >> 5];
  return make_double3((double)o.x + (double)p.x, (double)o.y + (double)p.y,
                      (double)o.z + (double)p.z);
}

// ------------------------------------------------------------------------
// small DFTs
// ------------------------------------------------------------------------
// (every product and sum below is rounded where it is written, so that all
// kernels that transform the same numbers get the same bits)
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)),
                     __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}

// cos / sin of 2*pi*k/R for the radices used (exact mathematical constants)
__device__ __forceinline__ constexpr float rcos(int R, int k) {
  return R == 3 ? (k == 0 ? 1.f : -0.5f)
       : R == 5 ? (k == 0 ? 1.f : (k == 1 || k == 4) ? 0.30901699437494745f : -0.8090169943749475f)
       : R == 6 ? (k == 0 ? 1.f : (k == 1 || k == 5) ? 0.5f : (k == 2 || k == 4) ? -0.5f : -1.f)
       : R == 7 ? (k == 0 ? 1.f : (k == 1 || k == 6) ? 0.6234898018587336f
                              : (k == 2 || k == 5) ? -0.22252093395631434f : -0.9009688679024191f)
       : R == 8 ? (k == 0 ? 1.f : (k == 1 || k == 7) ? 0.7071067811865476f
                              : (k == 2 || k == 6) ? 0.f : (k == 3 || k == 5) ? -0.7071067811865476f : -1.f)
       : 1.f;
}
__device__ __forceinline__ constexpr float rsin(int R, int k) {
  return R == 3 ? (k == 0 ? 0.f : k == 1 ? 0.8660254037844386f : -0.8660254037844386f)
       : R == 5 ? (k == 0 ? 0.f : k == 1 ? 0.9510565162951535f : k == 2 ? 0.5877852522924731f
                  : k == 3 ? -0.5877852522924731f : -0.9510565162951535f)
       : R == 6 ? (k == 0 || k == 3 ? 0.f : (k == 1 || k == 2) ? 0.8660254037844386f : -0.8660254037844386f)
       : R == 7 ? (k == 0 ? 0.f : k == 1 ? 0.7818314824680298f : k == 2 ? 0.9749279121818236f
                  : k == 3 ? 0.4338837391175582f : k == 4 ? -0.4338837391175582f
                  : k == 5 ? -0.9749279121818236f : -0.7818314824680298f)
       : R == 8 ? (k == 0 || k == 4 ? 0.f : (k == 1 || k == 3) ? 0.7071067811865476f
                  : k == 2 ? 1.f : (k == 5 || k == 7) ? -0.7071067811865476f : -1.f)
       : 0.f;
}

// y_k = sum_q x_q exp(+- 2 pi i q k / R), + when INV.  Each radix in its usual
// factored form (real arithmetic shared between y_k and y_{R-k}; 6 as 2 x 3
// and 8 as 2 x 4): 16 real additions for R = 4, 52 additions and 4
// multiplications for R = 8, where the R^2 products of the definition are 256
// multiply-adds.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y));
}
// a + i b when INV, else a - i b
template <bool INV>
__device__ __forceinline__ float2 cadd_i(float2 a, float2 b) {
  return INV ? make_float2(__fsub_rn(a.x, b.y), __fadd_rn(a.y, b.x))
             : make_float2(__fadd_rn(a.x, b.y), __fsub_rn(a.y, b.x));
}
// b + s a, and b + i s a
__device__ __forceinline__ float2 cfma(float s, float2 a, float2 b) {
  return make_float2(__fmaf_rn(s, a.x, b.x), __fmaf_rn(s, a.y, b.y));
}
__device__ __forceinline__ float2 cfma_i(float s, float2 a, float2 b) {
  return make_float2(__fmaf_rn(-s, a.y, b.x), __fmaf_rn(s, a.x, b.y));
}

template <bool INV>
__device__ __forceinline__ void dft2(float2 &a, float2 &b) {
  const float2 t = a;
  a = cadd(t, b);
  b = csub(t, b);
}
template <bool INV>
__device__ __forceinline__ void dft3(float2 &x0, float2 &x1, float2 &x2) {
  const float2 t = cadd(x1, x2), d = csub(x1, x2);
  const float2 m = cfma(-0.5f, t, x0);
  const float h = INV ? rsin(3, 1) : -rsin(3, 1);
  x0 = cadd(x0, t);
  x1 = cfma_i(h, d, m);
  x2 = cfma_i(-h, d, m);
}
template <bool INV>
__device__ __forceinline__ void dft4(float2 &x0, float2 &x1, float2 &x2, float2 &x3) {
  const float2 s02 = cadd(x0, x2), d02 = csub(x0, x2), s13 = cadd(x1, x3), d13 = csub(x1, x3);
  x0 = cadd(s02, s13);
  x2 = csub(s02, s13);
  x1 = cadd_i<INV>(d02, d13);
  x3 = cadd_i<!INV>(d02, d13);
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2 (&x)[R]) {
  if constexpr (R == 2) {
    dft2<INV>(x[0], x[1]);
  } else if constexpr (R == 3) {
    dft3<INV>(x[0], x[1], x[2]);
  } else if constexpr (R == 4) {
    dft4<INV>(x[0], x[1], x[2], x[3]);
  } else if constexpr (R == 6) {
    // index maps q = 3 q1 + 2 q2, k = 3 k1 + 4 k2 (mod 6): no twiddles between
    float2 a0 = x[0], b0 = x[3], a1 = x[2], b1 = x[5], a2 = x[4], b2 = x[1];
    dft2<INV>(a0, b0);
    dft2<INV>(a1, b1);
    dft2<INV>(a2, b2);
    dft3<INV>(a0, a1, a2);
    dft3<INV>(b0, b1, b2);
    x[0] = a0;
    x[4] = a1;
    x[2] = a2;
    x[3] = b0;
    x[1] = b1;
    x[5] = b2;
  } else if constexpr (R == 8) {
    dft4<INV>(x[0], x[2], x[4], x[6]);
    dft4<INV>(x[1], x[3], x[5], x[7]);
    // odd half times exp(+- 2 pi i k / 8)
    const float c = rcos(8, 1);
    const float2 o1 = cadd_i<INV>(x[3], x[3]), o3 = cadd_i<!INV>(x[7], x[7]);
    const float2 e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6], o0 = x[1], o2 = x[5];
    x[0] = cadd(e0, o0);
    x[4] = csub(e0, o0);
    x[1] = cfma(c, o1, e1);
    x[5] = cfma(-c, o1, e1);
    x[2] = cadd_i<INV>(e2, o2);
    x[6] = cadd_i<!INV>(e2, o2);
    x[3] = cfma(-c, o3, e3);
    x[7] = cfma(c, o3, e3);
  } else {  // 5 and 7: pairs q, R - q
    constexpr int H = R / 2;
    float2 t[H], d[H];
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      t[q - 1] = cadd(x[q], x[R - q]);
      d[q - 1] = csub(x[q], x[R - q]);
    }
    const float2 x0 = x[0];
    float2 y0 = x0;
#pragma unroll
    for (int q = 0; q < H; ++q) y0 = cadd(y0, t[q]);
    x[0] = y0;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      float2 m = x0, n = make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 1; q <= H; ++q) {
        m = cfma(rcos(R, (q * k) % R), t[q - 1], m);
        n = cfma(rsin(R, (q * k) % R), d[q - 1], n);
      }
      x[k] = cadd_i<INV>(m, n);
      x[R - k] = cadd_i<!INV>(m, n);
    }
  }
}

template <bool INV>
__device__ __forceinline__ float2 twiddle(const float2 *tw, int idx) {
  float2 w = tw[idx];
  if (INV) w.y = -w.y;
  return w;
}

// One stage on sub-blocks of length m of every line: decimation in frequency
// (butterfly, then twiddle) or in time (twiddle, then butterfly).  Lines start
// at buf + line * lstride; element e of a line is at e * estride.  The twiddle
// index j k n/m stays below n.  Consecutive threads take consecutive lines:
// their shared-memory accesses are lstride apart, free of bank conflicts for
// columns (lstride 1; with consecutive threads along a line the z pencils,
// estride 16, hit one bank with half a warp: 14.5 us a launch at 64^3 and 242
// us at 216^3 against 11.2 and 65), whatever the stage's radix.  Packed rows lie
// nx + 2 values apart, so theirs conflict gcd(nx + 2, 16)-fold: two-way where
// nx is a multiple of 4, four-way at nx = 90 or 210, eight-way at 54, 70 or 150,
// sixteen-way at 14, 30 or 126 (reciprocal space of 20 steps of a few atoms: 1.49
// ms on 128^3, 2.25 on 126^3; 3.28 and 3.26 with consecutive threads along a row).
template <int R, bool DIF, bool INV>
__device__ __forceinline__ void fft_stage(float2 *buf, int nlines, FastDiv by_lines, int lstride,
                                          int estride, int n, int m, FastDiv fmr, const float2 *tw) {
  const int mr = m / R, total = nlines * (n / R), nm = n / m;
  for (int b = threadIdx.x; b < total; b += blockDim.x) {
    const int rem = (int)fdiv((unsigned)b, by_lines), line = b - rem * nlines;
    const int blk = (int)fdiv((unsigned)rem, fmr), j = rem - blk * mr;
    float2 *p = buf + line * lstride + (blk * m + j) * estride;
    const int step = mr * estride;
    float2 x[R];
#pragma unroll
    for (int q = 0; q < R; ++q) x[q] = p[q * step];
    if (!DIF && j > 0) {
#pragma unroll
      for (int k = 1; k < R; ++k) x[k] = cmul(x[k], twiddle<INV>(tw, j * k * nm));
    }
    dft<R, INV>(x);
    if (DIF && j > 0) {
#pragma unroll
      for (int k = 1; k < R; ++k) x[k] = cmul(x[k], twiddle<INV>(tw, j * k * nm));
    }
#pragma unroll
    for (int k = 0; k < R; ++k) p[k * step] = x[k];
  }
}

template <bool DIF, bool INV>
__device__ __forceinline__ void stage(int R, float2 *buf, int nl, FastDiv by_nl, int ls, int es,
                                      int n, int m, FastDiv fmr, const float2 *tw) {
  switch (R) {
    case 2: fft_stage<2, DIF, INV>(buf, nl, by_nl, ls, es, n, m, fmr, tw); break;
    case 3: fft_stage<3, DIF, INV>(buf, nl, by_nl, ls, es, n, m, fmr, tw); break;
    case 4: fft_stage<4, DIF, INV>(buf, nl, by_nl, ls, es, n, m, fmr, tw); break;
    case 5: fft_stage<5, DIF, INV>(buf, nl, by_nl, ls, es, n, m, fmr, tw); break;
    case 6: fft_stage<6, DIF, INV>(buf, nl, by_nl, ls, es, n, m, fmr, tw); break;
    case 7: fft_stage<7, DIF, INV>(buf, nl, by_nl, ls, es, n, m, fmr, tw); break;
    case 8: fft_stage<8, DIF, INV>(buf, nl, by_nl, ls, es, n, m, fmr, tw); break;
    default: break;
  }
}

// natural order in, digit-reversed out
template <bool INV>
__device__ __forceinline__ void fft_dif(float2 *buf, int nl, FastDiv by_nl, int ls, int es, const FftAxis &a,
                        const float2 *tw) {
  int m = a.n;
  for (int s = 0; s < a.nrad; ++s) {
    stage<true, INV>(a.radix[s], buf, nl, by_nl, ls, es, a.n, m, a.dif_mr[s], tw);
    __syncthreads();
    m /= a.radix[s];
  }
}
// digit-reversed in, natural order out
template <bool INV>
__device__ __forceinline__ void fft_dit(float2 *buf, int nl, FastDiv by_nl, int ls, int es, const FftAxis &a,
                        const float2 *tw) {
  int m = 1;
  for (int s = a.nrad - 1; s >= 0; --s) {
    m *= a.radix[s];
    stage<false, INV>(a.radix[s], buf, nl, by_nl, ls, es, a.n, m, a.dit_mr[s], tw);
    __syncthreads();
  }
}

// digit-reversal table of an axis (positions of fft_dif's output, or their
// inverse) in shared memory, built by the whole block
__device__ __forceinline__ void fill_rev_table(short *tab, const FftAxis &a, bool inverse);

// natural index -> position in the output of fft_dif
__device__ __forceinline__ int dig_rev(int x, const FftAxis &a) {
  int p = 0, m = a.n;
  for (int s = 0; s < a.nrad; ++s) {
    const int R = a.radix[s];
    m /= R;
    p += (x % R) * m;
    x /= R;
  }
  return p;
}
// position in the output of fft_dif -> natural index
__device__ __forceinline__ int dig_unrev(int p, const FftAxis &a) {
  int k = 0, mult = 1, m = a.n;
  for (int s = 0; s < a.nrad; ++s) {
    const int R = a.radix[s];
    m /= R;
    const int d = p / m;
    p -= d * m;
    k += d * mult;
    mult *= R;
  }
  return k;
}

__device__ __forceinline__ void fill_rev_table(short *tab, const FftAxis &a, bool inverse) {
  for (int x = threadIdx.x; x < a.n; x += blockDim.x)
    tab[x] = (short)(inverse ? dig_unrev(x, a) : dig_rev(x, a));
}

// ------------------------------------------------------------------------
// tensor-memory-access (TMA) copies of pencil slabs: one thread issues a
// tiled bulk copy between global memory and shared memory; the load's
// completion is counted on an mbarrier (transaction bytes), waited for with
// a bounded number of polls
// ------------------------------------------------------------------------
constexpr int kTmaPollLimit = 1 << 22;

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// true once the phase `parity` has completed; false after kTmaPollLimit polls
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity) {
  for (int i = 0; i < kTmaPollLimit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z,
                                            unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, int x, int y, int z,
                                             const void *src) {
  asm volatile(
      "cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
          reinterpret_cast<unsigned long long>(map)),
      "r"(x), "r"(y), "r"(z), "r"(smem_u32(src))
      : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
// shared-memory writes of this thread become visible to the async proxy
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ------------------------------------------------------------------------
// the patch of grid points that a 32-slot cluster touches
// ------------------------------------------------------------------------
// The list's clusters are compact (an x-y column of about 7 A, 32 atoms high),
// so the p^3 points of their 32 atoms overlap: at 1 A and order 4 about
// 11^3 = 1,331 points instead of 2,048 additions, at order 6 13^3 = 2,197
// instead of 6,912, in rows of 11 to 13 neighbouring points instead of 4 to 6.
// From order 6 on spread sums a cluster's patch in shared memory and adds it
// to the grid row by row: a third of the grid additions, in rows that the L2
// takes in one go (order 6, 64^3: 25.6 -> 18.7 us a launch; 40 steps of 24,000
// atoms 7.53 -> 7.16 ms, of 107,000 18.96 -> 18.14, 40 piston steps 11.1 ->
// 10.0).  At order 4 the additions saved are fewer than the work of the patch
// costs (20 steps of 998,000 atoms 62.1 -> 64.4 ms with it), so it adds its
// points directly.  Gather reads the same patch row by row and takes its sums
// from shared memory.  A cluster whose atoms lie too far
// apart for the patch (coordinates that no list has sorted) takes the points
// one by one.
template <int ORDER>
struct PatchSize {  // points: 7.8 A columns at 0.85 A spacing with room to drift
  static constexpr int value = ORDER == 4 ? 4 : ORDER == 6 ? 4096 : 5120;
};
template <int ORDER>
struct Splines {
  static constexpr int kPitch = ORDER + 1;  // odd: 32 atoms' rows in 32 banks
  int i[3][32];                // first grid point, in the grid
  int l[3][32];                // the same, in the patch
  float q[32];
  float th[3][32][kPitch];
  int lo[3], ext[3];           // the patch: first grid point and points per axis
};

// splines of the 32 atoms of cluster blockIdx.x, one thread per (axis, atom)
// in the first three warps, and the patch they span; a barrier follows
template <int ORDER, bool DERIV>
__device__ __forceinline__ void cluster_splines(Splines<ORDER> &S,
                                                float (*dth)[32][Splines<ORDER>::kPitch],
                                                const float4 *__restrict__ xyzq,
                                                const float4 *__restrict__ origin, int nslot,
                                                int nx, int ny, int nz, double rLx, double rLy,
                                                double rLz) {
  if (threadIdx.x >= 96) return;
  const int dim = threadIdx.x >> 5, a = threadIdx.x & 31;
  const int s = blockIdx.x * 32 + a;
  const int n = dim == 0 ? nx : dim == 1 ? ny : nz;
  float q = 0.f, w = 0.f;
  int i0 = 0;
  if (s < nslot) {
    const float4 p = xyzq[s];
    const double3 g = global_pos(p, origin, s);
    q = p.w;
    anchor(dim == 0 ? g.x : dim == 1 ? g.y : g.z, dim == 0 ? rLx : dim == 1 ? rLy : rLz, n, i0, w);
  }
  float th[ORDER], dd[ORDER];
  bspline<ORDER>(w, th, dd);
  S.i[dim][a] = i0;
#pragma unroll
  for (int k = 0; k < ORDER; ++k) {
    S.th[dim][a][k] = th[k];
    if (DERIV) dth[dim][a][k] = dd[k];
  }
  if (dim == 0) S.q[a] = q;
  // the span of the charged atoms' first points, as distances (nearest image)
  // from the first such atom's
  const unsigned charged = __ballot_sync(0xffffffffu, q != 0.f);
  const int ref = __shfl_sync(0xffffffffu, i0, charged ? __ffs(charged) - 1 : 0);
  int d = i0 - ref;
  if (2 * d > n) d -= n;
  else if (2 * d < -n) d += n;
  const int lo = __reduce_min_sync(0xffffffffu, q != 0.f ? d : 0);
  const int hi = __reduce_max_sync(0xffffffffu, q != 0.f ? d : 0);
  S.l[dim][a] = d - lo;
  if (a == 0) {
    int first = ref + lo;
    if (first < 0) first += n;
    S.lo[dim] = first;
    S.ext[dim] = hi - lo + ORDER;
  }
}

// ------------------------------------------------------------------------
// spread
// ------------------------------------------------------------------------
template <int ORDER>
__global__ void __launch_bounds__(128) spread_kernel(const float4 *__restrict__ xyzq,
                                                     const int *__restrict__ counts,
                                                     const __grid_constant__ PmeDims d0,
                                                     int *__restrict__ qgrid,
                                                     const float4 *__restrict__ origin,
                                                     const PmeSysArgs *__restrict__ multi = nullptr,
                                                     const int *__restrict__ cl_sys = nullptr,
                                                     const double4 *__restrict__ dbox = nullptr) {
  constexpr int P3 = ORDER * ORDER * ORDER;
  constexpr int NI = (P3 + 31) / 32;  // points of an atom per lane
  __shared__ Splines<ORDER> S;
  __shared__ __align__(16) int patch[PatchSize<ORDER>::value];
  const int nslot = counts ? counts[0] : 0;
  if ((int)blockIdx.x * 32 >= nslot) return;
  const PmeDims *dp = &d0;
  if (multi) {  // one block = one 32-slot cluster of one system
    const PmeSysArgs &A = multi[cl_sys[blockIdx.x]];
    dp = &A.d;
    qgrid = A.qgrid;
  }
  const int nx = dp->nx, ny = dp->ny, nz = dp->nz;
  double rLx = dp->rLx, rLy = dp->rLy, rLz = dp->rLz;
  if (dbox) {
    rLx = 1.0 / dbox->x;
    rLy = 1.0 / dbox->y;
    rLz = 1.0 / dbox->z;
  }
  cluster_splines<ORDER, false>(S, nullptr, xyzq, origin, nslot, nx, ny, nz, rLx, rLy, rLz);
  __syncthreads();
  const int ex = S.ext[0], ey = S.ext[1], ez = S.ext[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // a patch wider than the grid would hold a point twice
  if (ORDER >= 6 && ex <= nx && ey <= ny && ez <= nz && ex * ey * ez <= PatchSize<ORDER>::value) {
    const int vol4 = (ex * ey * ez + 3) >> 2;
    for (int k = threadIdx.x; k < vol4; k += blockDim.x)
      reinterpret_cast<int4 *>(patch)[k] = make_int4(0, 0, 0, 0);
    // this lane's points of every atom: p^3 in order over the lanes
    int off[NI], xa[NI], yb[NI], zc[NI];
#pragma unroll
    for (int t = 0; t < NI; ++t) {
      const int pt = lane + 32 * t;
      xa[t] = pt % ORDER;
      yb[t] = (pt / ORDER) % ORDER;
      zc[t] = pt / (ORDER * ORDER);
      off[t] = (zc[t] * ey + yb[t]) * ex + xa[t];
    }
    __syncthreads();
#pragma unroll 2
    for (int a = warp; a < 32; a += 4) {
      const float q = S.q[a];
      if (q == 0.f) continue;  // warp-uniform
      int *base = patch + (S.l[2][a] * ey + S.l[1][a]) * ex + S.l[0][a];
#pragma unroll
      for (int t = 0; t < NI; ++t) {
        if (P3 % 32 && t == NI - 1 && zc[t] >= ORDER) continue;
        const float v = q * S.th[0][a][xa[t]] * S.th[1][a][yb[t]] * S.th[2][a][zc[t]];
        atomicAdd(base + off[t], __float2int_rn(v * kGridScale));
      }
    }
    __syncthreads();
    // row by row onto the grid, sixteen lanes a row
    const int xl = threadIdx.x & 15, rows = ey * ez;
    int z = 0, y = threadIdx.x >> 4;
    while (y >= ey) {
      y -= ey;
      ++z;
    }
    for (int r = threadIdx.x >> 4; r < rows; r += 8) {
      int gy = S.lo[1] + y, gz = S.lo[2] + z;
      if (gy >= ny) gy -= ny;
      if (gz >= nz) gz -= nz;
      int *row = qgrid + (size_t)nx * (gy + ny * gz);
      for (int x = xl; x < ex; x += 16) {
        const int v = patch[r * ex + x];
        int gx = S.lo[0] + x;
        if (gx >= nx) gx -= nx;
        if (v) atomicAdd(row + gx, v);
      }
      y += 8;
      while (y >= ey) {
        y -= ey;
        ++z;
      }
    }
    return;
  }
  for (int k = threadIdx.x; k < 32 * P3; k += blockDim.x) {
    const int a = k / P3, pt = k - a * P3;
    const float q = S.q[a];
    if (q == 0.f) continue;
    const int xa = pt % ORDER, yb = (pt / ORDER) % ORDER, zc = pt / (ORDER * ORDER);
    int x = S.i[0][a] + xa, y = S.i[1][a] + yb, z = S.i[2][a] + zc;
    if (x >= nx) x -= nx;
    if (y >= ny) y -= ny;
    if (z >= nz) z -= nz;
    const float v = q * S.th[0][a][xa] * S.th[1][a][yb] * S.th[2][a][zc];
    atomicAdd(&qgrid[x + nx * (y + ny * z)], __float2int_rn(v * kGridScale));
  }
}

// ------------------------------------------------------------------------
// plane transforms
// ------------------------------------------------------------------------
// The twiddles of a plane's two axes: copied to shared memory by the block
// (SMTW; the transforms read them at scattered places, each first touch a trip
// to the L2), or where the plane leaves no room for them, in global memory.
template <bool SMTW>
struct Twiddles {
  const float2 *x, *y;
  __device__ __forceinline__ Twiddles(const PmeDims &d, const float2 *twx, const float2 *twy,
                                      float2 *s_tw)
      : x(SMTW ? s_tw : twx), y(SMTW ? s_tw + 256 : twy) {
    if (SMTW) {
      for (int i = threadIdx.x; i < d.nx; i += blockDim.x) s_tw[i] = twx[i];
      for (int i = threadIdx.x; i < d.ny; i += blockDim.x) s_tw[256 + i] = twy[i];
    }
  }
};

// The grid dimensions are read through a pointer (to the kernel parameter or
// to the system's entry of the multi-system table), never copied: the FFT
// stages index their per-stage divisors at run time.
template <bool SMTW>
__global__ void __launch_bounds__(kPlaneThreadsMax) plane_fwd_kernel(const __grid_constant__ PmeDims d0, int *__restrict__ qgrid,
                                                                  float2 *__restrict__ cgrid,
                                                                  const float2 *__restrict__ twx,
                                                                  const float2 *__restrict__ twy,
                                                                  const PmeSysArgs *__restrict__ multi,
                                                                  const int *__restrict__ plane_sys) {
  extern __shared__ float2 buf[];
  int z = blockIdx.x;
  const PmeDims *dp = &d0;
  if (multi) {
    const PmeSysArgs &A = multi[plane_sys[blockIdx.x]];
    dp = &A.d;
    qgrid = A.qgrid;
    cgrid = A.cgrid;
    twx = A.tw;
    twy = A.tw + A.d.nx;
    z = blockIdx.x - A.plane0;
  }
  const PmeDims &d = *dp;
  __shared__ short s_rev[256];  // x -> position in the digit-reversed row
  __shared__ float2 s_tw[SMTW ? 512 : 1];
  const int nx = d.nx, ny = d.ny, nxc = d.nxc, nxcp = d.nxcp, rowp = nx + 2, h = nx / 2;
  // two neighbouring points of two rows a thread and turn (nx is even, so
  // pairs are 8-byte aligned), two turns in flight, the first while the
  // tables are made: a packed row takes both rows' points in one store
  int *plane = qgrid + (size_t)z * nx * ny;
  const int total = (ny / 2) * h;
  int2 v0[2], v1[2];
  const auto fetch = [&](int base) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = base + u * blockDim.x;
      if (i < total) {
        const int r = (int)fdiv((unsigned)i, d.by_hx), x = 2 * (i - r * h);
        v0[u] = *reinterpret_cast<int2 *>(plane + 2 * r * nx + x);
        v1[u] = *reinterpret_cast<int2 *>(plane + (2 * r + 1) * nx + x);
      }
    }
  };
  fetch(threadIdx.x);
  fill_rev_table(s_rev, d.ax, false);
  const Twiddles<SMTW> tw(d, twx, twy, s_tw);
  __syncthreads();
  for (int base = threadIdx.x; base < total; base += 2 * blockDim.x) {
    if (base != (int)threadIdx.x) fetch(base);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = base + u * blockDim.x;
      if (i < total) {
        const int r = (int)fdiv((unsigned)i, d.by_hx), x = 2 * (i - r * h);
        // ready for the next spread
        *reinterpret_cast<int2 *>(plane + 2 * r * nx + x) = make_int2(0, 0);
        *reinterpret_cast<int2 *>(plane + (2 * r + 1) * nx + x) = make_int2(0, 0);
        buf[r * rowp + s_rev[x]] =
            make_float2((float)v0[u].x * kInvGridScale, (float)v1[u].x * kInvGridScale);
        buf[r * rowp + s_rev[x + 1]] =
            make_float2((float)v0[u].y * kInvGridScale, (float)v1[u].y * kInvGridScale);
      }
    }
  }
  __syncthreads();
  fft_dit<false>(buf, ny / 2, d.by_rows, rowp, 1, d.ax, tw.x);
  // split the packed rows into the two half spectra, in place
  const int ngrp = (h + 1) / 2 + 1;
  for (int idx = threadIdx.x; idx < (ny / 2) * ngrp; idx += blockDim.x) {
    const int r = (int)fdiv((unsigned)idx, d.ax.by_ngrp), g = idx - r * ngrp;
    float2 *b = buf + r * rowp;
    if (g == ngrp - 1) {
      const float2 Z = b[h];
      b[h] = make_float2(Z.x, 0.f);
      b[nxc + h] = make_float2(Z.y, 0.f);
    } else {
      const int k1 = g, k2 = h - 1 - g;
      const float2 Z1 = b[k1], M1 = b[k1 ? nx - k1 : 0];
      const float2 Z2 = b[k2], M2 = b[nx - k2];
      const float2 A1 = make_float2(0.5f * (Z1.x + M1.x), 0.5f * (Z1.y - M1.y));
      const float2 B1 = make_float2(0.5f * (Z1.y + M1.y), -0.5f * (Z1.x - M1.x));
      const float2 A2 = make_float2(0.5f * (Z2.x + M2.x), 0.5f * (Z2.y - M2.y));
      const float2 B2 = make_float2(0.5f * (Z2.y + M2.y), -0.5f * (Z2.x - M2.x));
      b[k1] = A1;
      b[nxc + k1] = B1;
      if (k2 != k1) {
        b[k2] = A2;
        b[nxc + k2] = B2;
      }
    }
  }
  __syncthreads();
  // the in-place split leaves row y at y*nxc (rowp = 2 nxc: row 2r+1 starts
  // right after row 2r); in global memory rows have the even pitch nxcp
  fft_dif<false>(buf, nxc, d.ax.by_nxc, 1, nxc, d.ay, tw.y);
  float2 *out = cgrid + (size_t)z * ny * nxcp;
  for (int idx = threadIdx.x; idx < ny * nxcp; idx += blockDim.x) {
    const int y = (int)fdiv((unsigned)idx, d.ax.by_nxcp), kx = idx - y * nxcp;
    out[idx] = kx < nxc ? buf[y * nxc + kx] : make_float2(0.f, 0.f);
  }
}

template <bool SMTW>
__global__ void __launch_bounds__(kPlaneThreadsMax) plane_inv_kernel(const __grid_constant__ PmeDims d0,
                                                                  const float2 *__restrict__ cgrid,
                                                                  float *__restrict__ phi,
                                                                  const float2 *__restrict__ twx,
                                                                  const float2 *__restrict__ twy,
                                                                  const PmeSysArgs *__restrict__ multi,
                                                                  const int *__restrict__ plane_sys) {
  extern __shared__ float2 buf[];
  int z = blockIdx.x;
  const PmeDims *dp = &d0;
  if (multi) {
    const PmeSysArgs &A = multi[plane_sys[blockIdx.x]];
    dp = &A.d;
    cgrid = A.cgrid;
    phi = A.phi;
    twx = A.tw;
    twy = A.tw + A.d.nx;
    z = blockIdx.x - A.plane0;
  }
  const PmeDims &d = *dp;
  __shared__ short s_rev[256];  // x -> position in the digit-reversed row
  __shared__ float2 s_tw[SMTW ? 512 : 1];
  const int nx = d.nx, ny = d.ny, nxc = d.nxc, nxcp = d.nxcp, rowp = nx + 2, h = nx / 2;
  const float2 *in = cgrid + (size_t)z * ny * nxcp;
  fill_rev_table(s_rev, d.ax, false);
  const Twiddles<SMTW> tw(d, twx, twy, s_tw);
  // four loads in flight per thread before any store
  for (int base = threadIdx.x; base < ny * nxc; base += 4 * blockDim.x) {
    float2 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int idx = base + u * blockDim.x;
      if (idx < ny * nxc) {
        const int y = (int)fdiv((unsigned)idx, d.ax.by_nxc), kx = idx - y * nxc;
        v[u] = in[y * nxcp + kx];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int idx = base + u * blockDim.x;
      if (idx < ny * nxc) buf[idx] = v[u];
    }
  }
  __syncthreads();
  fft_dit<true>(buf, nxc, d.ax.by_nxc, 1, nxc, d.ay, tw.y);
  // pack pairs of half spectra into one complex row, in place
  const int ngrp = (h + 1) / 2 + 1;
  for (int idx = threadIdx.x; idx < (ny / 2) * ngrp; idx += blockDim.x) {
    const int r = (int)fdiv((unsigned)idx, d.ax.by_ngrp), g = idx - r * ngrp;
    float2 *b = buf + r * rowp;
    if (g == ngrp - 1) {
      const float2 A = b[h], B = b[nxc + h];
      b[h] = make_float2(A.x - B.y, A.y + B.x);
    } else {
      const int k1 = g, k2 = h - 1 - g;
      const float2 A1 = b[k1], B1 = b[nxc + k1], A2 = b[k2], B2 = b[nxc + k2];
      b[k1] = make_float2(A1.x - B1.y, A1.y + B1.x);
      if (k1 > 0) b[nx - k1] = make_float2(A1.x + B1.y, -A1.y + B1.x);
      if (k2 != k1) {
        b[k2] = make_float2(A2.x - B2.y, A2.y + B2.x);
        if (k2 > 0) b[nx - k2] = make_float2(A2.x + B2.y, -A2.y + B2.x);
      }
    }
  }
  __syncthreads();
  fft_dif<true>(buf, ny / 2, d.by_rows, rowp, 1, d.ax, tw.x);
  // natural order out: consecutive threads write consecutive pairs of points
  float *out = phi + (size_t)z * nx * ny;
  for (int i = threadIdx.x; i < (ny / 2) * h; i += blockDim.x) {
    const int r = (int)fdiv((unsigned)i, d.by_hx), x = 2 * (i - r * h);
    const float2 a = buf[r * rowp + s_rev[x]], b = buf[r * rowp + s_rev[x + 1]];
    *reinterpret_cast<float2 *>(out + 2 * r * nx + x) = make_float2(a.x, b.x);
    *reinterpret_cast<float2 *>(out + (2 * r + 1) * nx + x) = make_float2(a.y, b.y);
  }
}

// ------------------------------------------------------------------------
// z pencils: FFT, influence function, inverse FFT
// ------------------------------------------------------------------------
template <bool ENERGY, typename FT, bool VIRIAL = false, bool TMA = false>
__global__ void __launch_bounds__(kPencilThreads) pencil_kernel(const __grid_constant__ PmeDims d0, float2 *__restrict__ cgrid,
                                                                const float2 *__restrict__ twz,
                                                                const float *__restrict__ prefac,
                                                                const double *__restrict__ prefac_d,
                                                                long long *__restrict__ energy,
                                                                long long *__restrict__ virial,
                                                                const PmeSysArgs *__restrict__ multi,
                                                                const int *__restrict__ pencil_sys,
                                                                const __grid_constant__ CUtensorMap tmap,
                                                                unsigned *__restrict__ err,
                                                                const double4 *__restrict__ dbox = nullptr) {
  // TMA: the slab of ptx complex columns x nz arrives in (and leaves from)
  // buf as one tiled copy of the padded complex grid
  extern __shared__ float2 dyn[];
  float2 *const buf = dyn + ((128u - (smem_u32(dyn) & 127u)) & 127u) / sizeof(float2);
  __shared__ __align__(8) unsigned long long s_bar;
  __shared__ short s_unrev_z[256];
  __shared__ float2 s_tw[256];
  __shared__ double sh_e[kPencilThreads / 32];
  __shared__ double sh_v[6][kPencilThreads / 32];
  int blk = blockIdx.x;
  const PmeDims *dp = &d0;
  if (multi) {
    const PmeSysArgs &A = multi[pencil_sys[blockIdx.x]];
    dp = &A.d;
    cgrid = A.cgrid;
    twz = A.tw + A.d.nx + A.d.ny;
    prefac = A.prefac;
    prefac_d = A.prefac_d;
    energy = A.energy;
    virial = A.virial;
    blk = blockIdx.x - A.pencil0;
  }
  const PmeDims &d = *dp;
  const int nx = d.nx, ny = d.ny, nz = d.nz, nxc = d.nxc;
  float Lx = d.Lx, Ly = d.Ly, Lz = d.Lz;  // the box, or the device's copy of it
  if (dbox) {
    const double4 b = *dbox;
    Lx = (float)b.x;
    Ly = (float)b.y;
    Lz = (float)b.z;
  }
  const int TX = d.ptx, tiles_x = d.ptiles;
  const int py = blk / tiles_x, x0 = (blk - py * tiles_x) * TX;
  for (int i = threadIdx.x; i < nz; i += blockDim.x) s_tw[i] = twz[i];
  if (TMA) {
    if (threadIdx.x == 0) mbar_init(&s_bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
      mbar_expect_tx(&s_bar, (unsigned)(nz * TX * sizeof(float2)));
      tma_load_3d(buf, &tmap, 2 * x0, py, 0, &s_bar);
    }
    fill_rev_table(s_unrev_z, d.az, true);
    if (!mbar_wait(&s_bar, 0u)) {
      // the copy did not land: report it, give it a second bounded wait so
      // no write into this block's shared memory is left in flight, and leave
      // the slab untouched
      if (threadIdx.x == 0) atomicOr(err, (unsigned)kErrCopyTimeout);
      mbar_wait(&s_bar, 0u);
      return;
    }
  } else {
    fill_rev_table(s_unrev_z, d.az, true);
    for (int idx = threadIdx.x; idx < nz * TX; idx += blockDim.x) {
      const int zz = (int)fdiv((unsigned)idx, d.by_ptx), xt = idx - zz * TX, kx = x0 + xt;
      buf[idx] = kx < nxc ? cgrid[((size_t)zz * ny + py) * d.nxcp + kx] : make_float2(0.f, 0.f);
    }
  }
  __syncthreads();
  fft_dif<false>(buf, TX, d.by_ptx, 1, TX, d.az, s_tw);
  const int ky = dig_unrev(py, d.ay);
  const int nf1 = nx / 2 + (nx & 1), nf2 = ny / 2 + (ny & 1), nf3 = nz / 2 + (nz & 1);
  const FT m2 = (FT)(ky >= nf2 ? ky - ny : ky) / (FT)Ly;
  const FT pi = (FT)3.14159265358979323846;
  const FT fac = pi * pi / ((FT)d.kappa * (FT)d.kappa);
  const FT piv_inv = (FT)1 / ((FT)Lx * (FT)Ly * (FT)Lz * pi);
  const FT *pf = sizeof(FT) == 8 ? reinterpret_cast<const FT *>(prefac_d)
                                 : reinterpret_cast<const FT *>(prefac);
  const FT pyv = pf[nx + ky];
  double e = 0.0;
  double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int idx = threadIdx.x; idx < nz * TX; idx += blockDim.x) {
    const int pz = (int)fdiv((unsigned)idx, d.by_ptx), xt = idx - pz * TX, kx = x0 + xt;
    if (kx >= nxc) continue;
    const int kz = s_unrev_z[pz];
    FT eterm = 0;
    const FT m1 = (FT)(kx >= nf1 ? kx - nx : kx) / (FT)Lx;
    const FT m3 = (FT)(kz >= nf3 ? kz - nz : kz) / (FT)Lz;
    const FT msq = fma(m1, m1, fma(m2, m2, m3 * m3));
    if (kx != 0 || ky != 0 || kz != 0)
      eterm = exp(-fac * msq) * piv_inv * pf[kx] * pyv * pf[nx + ny + kz] / msq;
    const float2 q = buf[idx];
    if (ENERGY) {
      const FT mult = kx >= 1 ? (FT)2 : (FT)1;
      const FT t1 = mult * eterm * fma((FT)q.x, (FT)q.x, (FT)q.y * (FT)q.y);
      e += (double)t1;
      if (VIRIAL && eterm != (FT)0) {
        // reference scalar_sum (src/CudaPMERecip.cu:770-790): t1 (vterm m_a m_b - delta_ab)
        const FT vt = (FT)2 * (fac + (FT)1 / msq);
        v[0] += (double)(t1 * fma(vt * m1, m1, (FT)-1));
        v[1] += (double)(t1 * vt * m1 * m2);
        v[2] += (double)(t1 * vt * m1 * m3);
        v[3] += (double)(t1 * fma(vt * m2, m2, (FT)-1));
        v[4] += (double)(t1 * vt * m2 * m3);
        v[5] += (double)(t1 * fma(vt * m3, m3, (FT)-1));
      }
    }
    buf[idx] = make_float2((float)(q.x * eterm), (float)(q.y * eterm));
  }
  __syncthreads();
  fft_dit<true>(buf, TX, d.by_ptx, 1, TX, d.az, s_tw);
  if (TMA) {
    // columns past the grid's padded width are clipped by the copy
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) tma_store_3d(&tmap, 2 * x0, py, 0, buf);
  } else {
    for (int idx = threadIdx.x; idx < nz * TX; idx += blockDim.x) {
      const int zz = (int)fdiv((unsigned)idx, d.by_ptx), xt = idx - zz * TX, kx = x0 + xt;
      if (kx < nxc) cgrid[((size_t)zz * ny + py) * d.nxcp + kx] = buf[idx];
    }
  }
  if (ENERGY) {
    e = warp_sum(e);
    if ((threadIdx.x & 31) == 0) sh_e[threadIdx.x >> 5] = e;
    if (VIRIAL) {
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double t = warp_sum(v[k]);
        if ((threadIdx.x & 31) == 0) sh_v[k][threadIdx.x >> 5] = t;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < kPencilThreads / 32; ++w) t += sh_e[w];
      add_energy(energy + kEEwks, 0.5 * kCcelec * t);
    }
    if (VIRIAL && threadIdx.x < 6) {
      double t = 0.0;
      for (int w = 0; w < kPencilThreads / 32; ++w) t += sh_v[threadIdx.x][w];
      // xx xy xz yy yz zz -> row-major 3x3, W = -ccelec/2 * sum
      constexpr int kA[6] = {0, 1, 2, 4, 5, 8}, kB[6] = {0, 3, 6, 4, 7, 8};
      const long long iw = __double2ll_rn(-0.5 * kCcelec * t * kEnergyScale);
      add_fixed(virial + kA[threadIdx.x], iw);
      if (kB[threadIdx.x] != kA[threadIdx.x]) add_fixed(virial + kB[threadIdx.x], iw);
    }
  }
}

// ------------------------------------------------------------------------
// gather: 8 threads per atom, (y,z) pairs split across the 8, x loop inside.
// Order 4 reads its 4^3 points from the grid (gather4_kernel); orders 6
// and 8 from the cluster's patch in shared memory, with the splines of an
// atom worked out once instead of by each of its 8 threads (order 6, 64^3:
// 20.2 -> 16.6 us a launch; 40 steps of 24,000 atoms 7.16 -> 6.97 ms, of
// 107,000 18.1 -> 17.1).  At order 4 the patch holds more points than its
// atoms read (20 steps of 998,000 atoms 64.4 -> 65.6 ms with it).
// ------------------------------------------------------------------------
template <int ORDER>
__global__ void __launch_bounds__(256) gather_kernel(const float4 *__restrict__ xyzq,
                                                     const int *__restrict__ counts,
                                                     const __grid_constant__ PmeDims d0,
                                                     const float *__restrict__ phi,
                                                     long long *__restrict__ force, int stride,
                                                     const float4 *__restrict__ origin,
                                                     const PmeSysArgs *__restrict__ multi = nullptr,
                                                     const int *__restrict__ cl_sys = nullptr,
                                                     const double4 *__restrict__ dbox = nullptr) {
  __shared__ Splines<ORDER> S;
  __shared__ float dth[3][32][Splines<ORDER>::kPitch];
  __shared__ float patch[PatchSize<ORDER>::value];
  const int nslot = counts[0];
  if ((int)blockIdx.x * 32 >= nslot) return;
  const PmeDims *dp = &d0;
  if (multi) {  // one block = one 32-slot cluster of one system
    const PmeSysArgs &A = multi[cl_sys[blockIdx.x]];
    dp = &A.d;
    phi = A.phi;
  }
  const int nx = dp->nx, ny = dp->ny, nz = dp->nz;
  double rLx = dp->rLx, rLy = dp->rLy, rLz = dp->rLz;
  float Lx = dp->Lx, Ly = dp->Ly, Lz = dp->Lz;
  if (dbox) {
    const double4 b = *dbox;
    rLx = 1.0 / b.x;
    rLy = 1.0 / b.y;
    rLz = 1.0 / b.z;
    Lx = (float)b.x;
    Ly = (float)b.y;
    Lz = (float)b.z;
  }
  cluster_splines<ORDER, true>(S, dth, xyzq, origin, nslot, nx, ny, nz, rLx, rLy, rLz);
  __syncthreads();
  const int ex = S.ext[0], ey = S.ext[1], ez = S.ext[2];
  const bool in_patch = ex <= nx && ey <= ny && ez <= nz && ex * ey * ez <= PatchSize<ORDER>::value;
  if (in_patch) {  // row by row from the grid, sixteen lanes a row
    const int xl = threadIdx.x & 15, rows = ey * ez;
    int z = 0, y = threadIdx.x >> 4;
    while (y >= ey) {
      y -= ey;
      ++z;
    }
    for (int r = threadIdx.x >> 4; r < rows; r += 16) {
      int gy = S.lo[1] + y, gz = S.lo[2] + z;
      if (gy >= ny) gy -= ny;
      if (gz >= nz) gz -= nz;
      const float *row = phi + (size_t)nx * (gy + ny * gz);
      for (int x = xl; x < ex; x += 16) {
        int gx = S.lo[0] + x;
        if (gx >= nx) gx -= nx;
        patch[r * ex + x] = __ldg(row + gx);
      }
      y += 16;
      while (y >= ey) {
        y -= ey;
        ++z;
      }
    }
    __syncthreads();
  }
  const int a = threadIdx.x >> 3, sub = threadIdx.x & 7;
  const int s = blockIdx.x * 32 + a;
  const float q = S.q[a];
  float f1 = 0.f, f2 = 0.f, f3 = 0.f;
  if (q != 0.f) {
    float thx[ORDER], dx[ORDER];
#pragma unroll
    for (int t = 0; t < ORDER; ++t) {
      thx[t] = S.th[0][a][t];
      dx[t] = dth[0][a][t];
    }
    const int ix = S.i[0][a];
    const float *corner = patch + (S.l[2][a] * ey + S.l[1][a]) * ex + S.l[0][a];
#pragma unroll
    for (int k0 = 0; k0 < ORDER * ORDER; k0 += 8) {
      const int k = k0 + sub, b = k % ORDER, c = k / ORDER;
      if (ORDER * ORDER % 8 && k >= ORDER * ORDER) break;
      float sx = 0.f, sdx = 0.f;
      if (in_patch) {
        const float *row = corner + (c * ey + b) * ex;
#pragma unroll
        for (int t = 0; t < ORDER; ++t) {
          const float v = row[t];
          sx += thx[t] * v;
          sdx += dx[t] * v;
        }
      } else {
        int y = S.i[1][a] + b, z = S.i[2][a] + c;
        if (y >= ny) y -= ny;
        if (z >= nz) z -= nz;
        const float *row = phi + ((size_t)z * ny + y) * nx;
#pragma unroll
        for (int t = 0; t < ORDER; ++t) {
          int x = ix + t;
          if (x >= nx) x -= nx;
          const float v = __ldg(row + x);
          sx += thx[t] * v;
          sdx += dx[t] * v;
        }
      }
      const float tyb = S.th[1][a][b], tzc = S.th[2][a][c];
      f1 += sdx * tyb * tzc;
      f2 += sx * dth[1][a][b] * tzc;
      f3 += sx * tyb * dth[2][a][c];
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    f1 += __shfl_xor_sync(0xffffffffu, f1, o);
    f2 += __shfl_xor_sync(0xffffffffu, f2, o);
    f3 += __shfl_xor_sync(0xffffffffu, f3, o);
  }
  if (sub == 0 && q != 0.f) {
    const float qc = q * (float)kCcelec;
    add_fixed(force + s, to_fixed_force(qc * (float)nx / Lx * f1));
    add_fixed(force + stride + s, to_fixed_force(qc * (float)ny / Ly * f2));
    add_fixed(force + 2 * stride + s, to_fixed_force(qc * (float)nz / Lz * f3));
  }
}

// Order 4: the splines of the cluster's atoms worked out once, then a warp per
// atom with a lane per point of two layers (x fastest), so that a load takes
// eight rows of four neighbouring points; with a lane per row every load of
// the warp touched 32 lines and the kernel was bound by them (998,000 atoms
// on 216^3 170 -> 138 us a launch, 24 systems of 4,000 18.4 -> 18.0 ms a pass).
// Four atoms' loads are in flight together, and their twelve sums are taken
// with one halving exchange of sixteen values.
__global__ void __launch_bounds__(256) gather4_kernel(const float4 *__restrict__ xyzq,
                                                      const int *__restrict__ counts,
                                                      const __grid_constant__ PmeDims d0,
                                                      const float *__restrict__ phi,
                                                      long long *__restrict__ force, int stride,
                                                      const float4 *__restrict__ origin,
                                                      const PmeSysArgs *__restrict__ multi = nullptr,
                                                      const int *__restrict__ cl_sys = nullptr,
                                                      const double4 *__restrict__ dbox = nullptr) {
  __shared__ Splines<4> S;
  __shared__ float dth[3][32][Splines<4>::kPitch];
  const int nslot = counts[0];
  if ((int)blockIdx.x * 32 >= nslot) return;
  const PmeDims *dp = &d0;
  if (multi) {  // one block = one 32-slot cluster of one system
    const PmeSysArgs &A = multi[cl_sys[blockIdx.x]];
    dp = &A.d;
    phi = A.phi;
  }
  const int nx = dp->nx, ny = dp->ny, nz = dp->nz;
  double rLx = dp->rLx, rLy = dp->rLy, rLz = dp->rLz;
  float Lx = dp->Lx, Ly = dp->Ly, Lz = dp->Lz;
  if (dbox) {
    const double4 b = *dbox;
    rLx = 1.0 / b.x;
    rLy = 1.0 / b.y;
    rLz = 1.0 / b.z;
    Lx = (float)b.x;
    Ly = (float)b.y;
    Lz = (float)b.z;
  }
  cluster_splines<4, true>(S, dth, xyzq, origin, nslot, nx, ny, nz, rLx, rLy, rLz);
  __syncthreads();
  const int lane = threadIdx.x & 31, a0 = (threadIdx.x >> 5) * 4;
  const int xa = lane & 3, yb = (lane >> 2) & 3, zc = lane >> 4;
  float v[4][2];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int a = a0 + t;
    int x = S.i[0][a] + xa, y = S.i[1][a] + yb;
    if (x >= nx) x -= nx;
    if (y >= ny) y -= ny;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      int z = S.i[2][a] + zc + 2 * k;
      if (z >= nz) z -= nz;
      v[t][k] = __ldg(phi + ((size_t)z * ny + y) * nx + x);
    }
  }
  float f[16];  // 4 t + component
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int a = a0 + t;
    const float tx = S.th[0][a][xa], dx = dth[0][a][xa], ty = S.th[1][a][yb], dy = dth[1][a][yb];
    f[4 * t] = f[4 * t + 1] = f[4 * t + 2] = f[4 * t + 3] = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float tz = S.th[2][a][zc + 2 * k], dz = dth[2][a][zc + 2 * k];
      f[4 * t] += dx * v[t][k] * ty * tz;
      f[4 * t + 1] += tx * v[t][k] * dy * tz;
      f[4 * t + 2] += tx * v[t][k] * ty * dz;
    }
  }
  // lane L ends with the sum of value L / 2
  int o = 16;
#pragma unroll
  for (int half = 8; half >= 1; half >>= 1, o >>= 1) {
    const bool hi = lane & o;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = hi ? f[i] : f[i + half];
      const float keep = hi ? f[i + half] : f[i];
      f[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  f[0] += __shfl_xor_sync(0xffffffffu, f[0], 1);
  const int a = a0 + (lane >> 3), comp = (lane >> 1) & 3;
  const float q = S.q[a];
  if (!(lane & 1) && comp < 3 && q != 0.f) {
    const float n = (float)(comp == 0 ? nx : comp == 1 ? ny : nz);
    const float L = comp == 0 ? Lx : comp == 1 ? Ly : Lz;
    add_fixed(force + (size_t)comp * stride + blockIdx.x * 32 + a,
              to_fixed_force(q * (float)kCcelec * n / L * f[0]));
  }
}

// B-spline moduli as the reference's dftmod (src/CudaPMERecip.cu:2656-2678)
void bspline_moduli(int n, int order, std::vector<double> &out) {
  std::vector<double> th(order), arr(n + order + 2, 0.0);
  // weights at w = 0
  th[order - 1] = 0.0;
  th[1] = 0.0;
  th[0] = 1.0;
  for (int k = 3; k <= order - 1; ++k) {
    double div = 1.0 / (k - 1);
    th[k - 1] = 0.0;
    for (int j = 1; j <= k - 2; ++j) th[k - j - 1] = div * (j * th[k - j - 2] + (k - j) * th[k - j - 1]);
    th[0] = div * th[0];
  }
  {
    double div = 1.0 / (order - 1);
    th[order - 1] = 0.0;
    for (int j = 1; j <= order - 2; ++j)
      th[order - j - 1] = div * (j * th[order - j - 2] + (order - j) * th[order - j - 1]);
    th[0] = div * th[0];
  }
  for (int i = 2; i <= order + 1; ++i) arr[i - 1] = th[i - 2];
  out.assign(n, 0.0);
  for (int k = 0; k < n; ++k) {
    double s1 = 0, s2 = 0;
    for (int j = 0; j < n - 1; ++j) {
      double a = 2.0 * M_PI * k * j / n;
      s1 += arr[j] * std::cos(a);
      s2 += arr[j] * std::sin(a);
    }
    out[k] = s1 * s1 + s2 * s2;
  }
  for (int k = 0; k < n; ++k)
    if (out[k] < 1e-10) out[k] = 0.5 * (out[(k - 1 + n) % n] + out[(k + 1) % n]);
  for (int k = 0; k < n; ++k) out[k] = 1.0 / out[k];
}

template <typename T>
void dalloc(T *&p, size_t n) {
  if (p) cudaFree(p);
  p = nullptr;
  if (n) APO_CUDA(cudaMalloc(&p, n * sizeof(T)));
}

}  // namespace

// The tensor map of the pencil slabs: the padded complex grid viewed as
// floats [nz][ny][2 nxcp], a box of ptx complex columns x 1 row x nz planes.
// The encoder is the driver's, fetched through the runtime (no link to the
// driver library).
bool encode_pencil_map(CUtensorMap *map, float2 *cgrid, const PmeDims &d) {
  using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                              const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                              const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Encode fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<Encode>(p);
    else
      cudaGetLastError();
  }
  // at most 256 planes, rows and slabs of 16-byte multiples; a slab starts at
  // an even column, 16-byte aligned
  if (!fn || d.nz > 256 || (d.nxcp & 1) || (d.ptx & 1) || d.nxcp < d.ptx) return false;
  const cuuint64_t dims[3] = {2ull * d.nxcp, (cuuint64_t)d.ny, (cuuint64_t)d.nz};
  const cuuint64_t strides[2] = {2ull * d.nxcp * sizeof(float),
                                 2ull * d.nxcp * d.ny * sizeof(float)};
  const cuuint32_t box[3] = {2u * d.ptx, 1u, (cuuint32_t)d.nz};
  const cuuint32_t es[3] = {1u, 1u, 1u};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, cgrid, dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// shared memory of one plane transform: ny/2 packed rows of nx + 2 complex
static size_t plane_smem_bytes(int nx, int ny) {
  return (size_t)(ny / 2) * (nx + 2) * sizeof(float2);
}

// threads of a plane transform: one butterfly of about 8 points a thread and
// stage up to 1,024.  At 64^2 256 threads do every stage in one go (512 left
// half of them idle); a 216^2 plane has an SM to itself and needs the warps
// (20 steps of 998,000 atoms: 59.3 ms with 1,024 threads, 59.9 with 512, 61.2
// with 256).
static int plane_threads(int nx, int ny) {
  const int want = nx * ny / 16;
  return want <= 256 ? 256 : want <= 1024 ? 512 : 1024;
}
static size_t pencil_smem_bytes(const PmeDims &d) { return (size_t)d.nz * d.ptx * sizeof(float2) + 128; }

// The z pencils' slabs: about 16 complex columns, an even number (16-byte
// aligned slabs), chosen so that the last slab of a row is not left nearly
// empty (nxc = 33 is two slabs of 18, not 16 + 16 + 1)
static void set_tiles(PmeDims &d) {
  const int tiles = std::max(1, (d.nxc + 8) / 16);
  d.ptx = ((d.nxc + tiles - 1) / tiles + 1) & ~1;
  d.ptiles = (d.nxc + d.ptx - 1) / d.ptx;
  d.by_ptx = make_fastdiv((unsigned)d.ptx);
  d.by_rows = make_fastdiv((unsigned)(d.ny / 2));
  d.by_hx = make_fastdiv((unsigned)(d.nx / 2));
}

static void raise_smem_limits() {
  APO_CUDA(cudaFuncSetAttribute(plane_fwd_kernel<true>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, kPlaneSmemTw));
  APO_CUDA(cudaFuncSetAttribute(plane_fwd_kernel<false>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, kPlaneSmemMax));
  APO_CUDA(cudaFuncSetAttribute(plane_inv_kernel<true>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, kPlaneSmemTw));
  APO_CUDA(cudaFuncSetAttribute(plane_inv_kernel<false>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, kPlaneSmemMax));
  const auto raise = [](auto *k) {
    APO_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kPencilSmemMax));
  };
  raise(pencil_kernel<true, double, true, true>);
  raise(pencil_kernel<true, double, true, false>);
  raise(pencil_kernel<true, float, true, true>);
  raise(pencil_kernel<true, float, true, false>);
  raise(pencil_kernel<true, double, false, true>);
  raise(pencil_kernel<true, double, false, false>);
  raise(pencil_kernel<true, float, false, true>);
  raise(pencil_kernel<true, float, false, false>);
  raise(pencil_kernel<false, double, false, true>);
  raise(pencil_kernel<false, double, false, false>);
  raise(pencil_kernel<false, float, false, true>);
  raise(pencil_kernel<false, float, false, false>);
}

FastDiv make_fastdiv(unsigned d) {
  FastDiv f{0u, 0u};
  if (d <= 1) return f;
  unsigned l = 0;  // ceil(log2 d)
  while ((1u << l) < d) ++l;
  f.mul = (unsigned)(((1ull << (31 + l)) + d - 1) / d);
  f.shift = l - 1;
  return f;
}

void fill_axis_divisors(FftAxis &a) {
  int prod = 1;
  for (int s = 0; s < a.nrad; ++s) {
    prod *= a.radix[s];
    a.dif_mr[s] = make_fastdiv((unsigned)(a.n / prod));
  }
  int tail = 1;
  for (int s = a.nrad - 1; s >= 0; --s) {
    a.dit_mr[s] = make_fastdiv((unsigned)tail);
    tail *= a.radix[s];
  }
  a.by_nxc = make_fastdiv((unsigned)(a.n / 2 + 1));
  a.by_nxcp = make_fastdiv((unsigned)((a.n / 2 + 2) & ~1));
  a.by_ngrp = make_fastdiv((unsigned)((a.n / 2 + 1) / 2 + 1));
}

FftAxis Pme::plan_axis(int n) {
  // fewest stages, then smallest total radix
  std::vector<int> best;
  std::vector<int> cur;
  std::function<void(int)> rec = [&](int m) {
    if (m == 1) {
      if (best.empty() || cur.size() < best.size() ||
          (cur.size() == best.size() &&
           std::accumulate(cur.begin(), cur.end(), 0) < std::accumulate(best.begin(), best.end(), 0)))
        best = cur;
      return;
    }
    if (!best.empty() && cur.size() + 1 > best.size()) return;
    for (int R : {8, 7, 6, 5, 4, 3, 2}) {
      if (m % R == 0) {
        cur.push_back(R);
        rec(m / R);
        cur.pop_back();
      }
    }
  };
  rec(n);
  if (best.empty() || best.size() > 8)
    throw std::invalid_argument("PME grid size " + std::to_string(n) +
                                " must factor into 2, 3, 5 and 7");
  FftAxis a{};
  a.n = n;
  a.nrad = (int)best.size();
  for (size_t i = 0; i < best.size(); ++i) a.radix[i] = best[i];
  fill_axis_divisors(a);
  return a;
}

Pme::~Pme() { release(); }

void Pme::release() {
  if (qgrid) cudaFree(qgrid);
  if (cgrid) cudaFree(cgrid);
  if (phi) cudaFree(phi);
  if (m_tw) cudaFree(m_tw);
  if (m_prefac) cudaFree(m_prefac);
  if (m_prefac_d) cudaFree(m_prefac_d);
  qgrid = nullptr;
  cgrid = nullptr;
  phi = nullptr;
  m_tw = nullptr;
  m_prefac = nullptr;
  m_prefac_d = nullptr;
}

void Pme::setup(int nx, int ny, int nz, int order, double kappa, double Lx, double Ly,
                double Lz) {
  if (nx % 2 || ny % 2 || nz % 2)
    throw std::invalid_argument("PME grid dimensions must be even");
  if (nx > 256 || ny > 256 || nz > 256)
    throw std::invalid_argument("PME grid dimensions above 256 are not supported");
  if (order != 4 && order != 6 && order != 8)
    throw std::invalid_argument("PME spline order must be 4, 6 or 8");
  // a spline's p points wrap the grid at most once only when n >= p
  if (nx < order || ny < order || nz < order)
    throw std::invalid_argument("PME grid dimensions must be at least the spline order");
  const size_t plane_bytes = plane_smem_bytes(nx, ny);
  if (plane_bytes > kPlaneSmemMax)
    throw std::invalid_argument("PME plane does not fit in shared memory");
  release();
  m_d.nx = nx;
  m_d.ny = ny;
  m_d.nz = nz;
  m_d.nxc = nx / 2 + 1;
  m_d.nxcp = (m_d.nxc + 1) & ~1;
  m_d.order = order;
  m_d.Lx = (float)Lx;
  m_d.Ly = (float)Ly;
  m_d.Lz = (float)Lz;
  m_d.rLx = 1.0 / Lx;
  m_d.rLy = 1.0 / Ly;
  m_d.rLz = 1.0 / Lz;
  m_d.kappa = (float)kappa;
  m_d.ax = plan_axis(nx);
  m_d.ay = plan_axis(ny);
  m_d.az = plan_axis(nz);
  set_tiles(m_d);
  const size_t G = (size_t)nx * ny * nz;
  dalloc(qgrid, G);
  dalloc(cgrid, (size_t)nz * ny * m_d.nxcp);
  APO_CUDA(cudaMemset(cgrid, 0, (size_t)nz * ny * m_d.nxcp * sizeof(float2)));
  m_tma = encode_pencil_map(&m_tmap, cgrid, m_d);
  dalloc(phi, G);
  APO_CUDA(cudaMemset(qgrid, 0, G * sizeof(int)));
  std::vector<float2> tw;
  for (int n : {nx, ny, nz})
    for (int k = 0; k < n; ++k) {
      double a = 2.0 * M_PI * k / n;
      tw.push_back(make_float2((float)std::cos(a), (float)-std::sin(a)));
    }
  dalloc(m_tw, tw.size());
  APO_CUDA(cudaMemcpy(m_tw, tw.data(), tw.size() * sizeof(float2), cudaMemcpyHostToDevice));
  std::vector<double> pd, tmp;
  for (int n : {nx, ny, nz}) {
    bspline_moduli(n, order, tmp);
    pd.insert(pd.end(), tmp.begin(), tmp.end());
  }
  std::vector<float> pf(pd.begin(), pd.end());
  dalloc(m_prefac, pf.size());
  dalloc(m_prefac_d, pd.size());
  APO_CUDA(cudaMemcpy(m_prefac, pf.data(), pf.size() * sizeof(float), cudaMemcpyHostToDevice));
  APO_CUDA(cudaMemcpy(m_prefac_d, pd.data(), pd.size() * sizeof(double), cudaMemcpyHostToDevice));
  static bool attr = false;
  if (!attr) {
    raise_smem_limits();
    attr = true;
  }
}

void Pme::spread(const float4 *xyzq_s, const int *counts, cudaStream_t s,
                 const float4 *origin) {
  const int blocks = (max_slots + 31) / 32;
  switch (m_d.order) {
    case 4: spread_kernel<4><<<blocks, 128, 0, s>>>(xyzq_s, counts, m_d, qgrid, origin, nullptr, nullptr, m_dbox); break;
    case 6: spread_kernel<6><<<blocks, 128, 0, s>>>(xyzq_s, counts, m_d, qgrid, origin, nullptr, nullptr, m_dbox); break;
    case 8: spread_kernel<8><<<blocks, 128, 0, s>>>(xyzq_s, counts, m_d, qgrid, origin, nullptr, nullptr, m_dbox); break;
  }
  APO_LAUNCH_CHECK();
}

void Pme::forward(cudaStream_t s) {
  const size_t sm = plane_smem_bytes(m_d.nx, m_d.ny);
  (sm <= kPlaneSmemTw ? plane_fwd_kernel<true> : plane_fwd_kernel<false>)<<<m_d.nz, plane_threads(m_d.nx, m_d.ny), sm, s>>>(
      m_d, qgrid, cgrid, m_tw, m_tw + m_d.nx, nullptr, nullptr);
  APO_LAUNCH_CHECK();
}

void Pme::convolve(long long *energy, bool calc_energy, bool fp64, cudaStream_t s,
                   long long *virial) {
  const int grid = m_d.ptiles * m_d.ny;
  const size_t sm = pencil_smem_bytes(m_d);
  const float2 *twz = m_tw + m_d.nx + m_d.ny;
  const bool tma = tensor_copies() && m_err;
#define APO_PENCIL(E, FT, V)                                                                   \
  do {                                                                                         \
    if (tma)                                                                                   \
      pencil_kernel<E, FT, V, true><<<grid, kPencilThreads, sm, s>>>(                           \
          m_d, cgrid, twz, m_prefac, m_prefac_d, energy, virial, nullptr, nullptr, m_tmap, m_err, \
          m_dbox);                                                                             \
    else                                                                                       \
      pencil_kernel<E, FT, V, false><<<grid, kPencilThreads, sm, s>>>(                          \
          m_d, cgrid, twz, m_prefac, m_prefac_d, energy, virial, nullptr, nullptr, m_tmap, m_err, \
          m_dbox);                                                                             \
  } while (0)
  if (virial) {
    if (fp64) APO_PENCIL(true, double, true);
    else APO_PENCIL(true, float, true);
  } else if (fp64) {
    if (calc_energy) APO_PENCIL(true, double, false);
    else APO_PENCIL(false, double, false);
  } else {
    if (calc_energy) APO_PENCIL(true, float, false);
    else APO_PENCIL(false, float, false);
  }
#undef APO_PENCIL
  APO_LAUNCH_CHECK();
}

void Pme::backward(cudaStream_t s) {
  const size_t sm = plane_smem_bytes(m_d.nx, m_d.ny);
  (sm <= kPlaneSmemTw ? plane_inv_kernel<true> : plane_inv_kernel<false>)<<<m_d.nz, plane_threads(m_d.nx, m_d.ny), sm, s>>>(
      m_d, cgrid, phi, m_tw, m_tw + m_d.nx, nullptr, nullptr);
  APO_LAUNCH_CHECK();
}

void Pme::gather(const float4 *xyzq_s, const int *counts, long long *force, int stride,
                 cudaStream_t s, const float4 *origin) {
  const int blocks = (max_slots + 31) / 32;
  switch (m_d.order) {
    case 4: gather4_kernel<<<blocks, 256, 0, s>>>(xyzq_s, counts, m_d, phi, force, stride, origin, nullptr, nullptr, m_dbox); break;
    case 6: gather_kernel<6><<<blocks, 256, 0, s>>>(xyzq_s, counts, m_d, phi, force, stride, origin, nullptr, nullptr, m_dbox); break;
    case 8: gather_kernel<8><<<blocks, 256, 0, s>>>(xyzq_s, counts, m_d, phi, force, stride, origin, nullptr, nullptr, m_dbox); break;
  }
  APO_LAUNCH_CHECK();
}

void Pme::compute(const float4 *xyzq_s, const int *counts, long long *force, int stride,
                  long long *energy, bool calc_energy, bool fp64, cudaStream_t s,
                  long long *virial, const float4 *origin) {
  spread(xyzq_s, counts, s, origin);
  forward(s);
  convolve(energy, calc_energy, fp64, s, virial);
  backward(s);
  gather(xyzq_s, counts, force, stride, s, origin);
}

}  // namespace apo

// ---------------------------------------------------------------------------
// Many systems
// ---------------------------------------------------------------------------

namespace apo {

PmeMulti::~PmeMulti() { release(); }

void PmeMulti::release() {
  for (void *p : {(void *)m_args, (void *)m_plane_sys, (void *)m_pencil_sys, (void *)m_q,
                  (void *)m_c, (void *)m_phi, (void *)m_tw, (void *)m_pf, (void *)m_pfd})
    if (p) cudaFree(p);
  m_args = nullptr;
  m_plane_sys = m_pencil_sys = nullptr;
  m_q = nullptr;
  m_c = nullptr;
  m_phi = nullptr;
  m_tw = nullptr;
  m_pf = nullptr;
  m_pfd = nullptr;
}

void PmeMulti::setup(const std::vector<PmeSystemSpec> &systems, int order, long long *energy,
                     int energy_stride, int max_slots) {
  if (systems.empty()) throw std::invalid_argument("PmeMulti: no systems");
  if (order != 4 && order != 6 && order != 8)
    throw std::invalid_argument("PME spline order must be 4, 6 or 8");
  release();
  m_host.clear();
  m_order = order;
  m_max_slots = max_slots;
  size_t q = 0, c = 0, t = 0;
  std::vector<int> plane_sys, pencil_sys;
  std::vector<float2> tw;
  std::vector<double> pd;
  m_plane_smem = m_pencil_smem = 0;
  m_plane_threads = 0;
  for (size_t k = 0; k < systems.size(); ++k) {
    const PmeSystemSpec &y = systems[k];
    if (y.nx % 2 || y.ny % 2 || y.nz % 2 || y.nx <= 0 || y.ny <= 0 || y.nz <= 0)
      throw std::invalid_argument("PME grid dimensions must be even");
    if (y.nx > 256 || y.ny > 256 || y.nz > 256)
      throw std::invalid_argument("PME grid dimensions above 256 are not supported");
    if (y.nx < order || y.ny < order || y.nz < order)
      throw std::invalid_argument("PME grid dimensions must be at least the spline order");
    const size_t plane_bytes = plane_smem_bytes(y.nx, y.ny);
    if (plane_bytes > kPlaneSmemMax) throw std::invalid_argument("PME plane does not fit in shared memory");
    m_plane_smem = std::max(m_plane_smem, plane_bytes);
    PmeSysArgs A{};
    A.d.nx = y.nx;
    A.d.ny = y.ny;
    A.d.nz = y.nz;
    A.d.nxc = y.nx / 2 + 1;
    A.d.nxcp = (A.d.nxc + 1) & ~1;
    A.d.order = order;
    A.d.Lx = (float)y.Lx;
    A.d.Ly = (float)y.Ly;
    A.d.Lz = (float)y.Lz;
    A.d.rLx = 1.0 / y.Lx;
    A.d.rLy = 1.0 / y.Ly;
    A.d.rLz = 1.0 / y.Lz;
    A.d.kappa = (float)y.kappa;
    A.d.ax = Pme::plan_axis(y.nx);
    A.d.ay = Pme::plan_axis(y.ny);
    A.d.az = Pme::plan_axis(y.nz);
    set_tiles(A.d);
    m_pencil_smem = std::max(m_pencil_smem, pencil_smem_bytes(A.d));
    m_plane_threads = std::max(m_plane_threads, plane_threads(y.nx, y.ny));
    // offsets for now; turned into pointers once the buffers exist
    A.qgrid = reinterpret_cast<int *>(q);
    A.phi = reinterpret_cast<float *>(q);
    A.cgrid = reinterpret_cast<float2 *>(c);
    A.tw = reinterpret_cast<const float2 *>(t);
    A.prefac = reinterpret_cast<const float *>(t);
    A.prefac_d = reinterpret_cast<const double *>(t);
    A.energy = energy + k * (size_t)energy_stride;
    A.virial = A.energy + kNumEnergyTerms;
    A.plane0 = m_planes;
    A.pencil0 = m_pencils;
    const int tiles_x = A.d.ptiles;
    for (int z = 0; z < y.nz; ++z) plane_sys.push_back((int)k);
    for (int b = 0; b < tiles_x * y.ny; ++b) pencil_sys.push_back((int)k);
    m_planes += y.nz;
    m_pencils += tiles_x * y.ny;
    q += (size_t)y.nx * y.ny * y.nz;
    c += (size_t)y.nz * y.ny * A.d.nxcp;
    t += (size_t)y.nx + y.ny + y.nz;
    for (int n : {y.nx, y.ny, y.nz})
      for (int j = 0; j < n; ++j) {
        const double a = 2.0 * M_PI * j / n;
        tw.push_back(make_float2((float)std::cos(a), (float)-std::sin(a)));
      }
    std::vector<double> tmp;
    for (int n : {y.nx, y.ny, y.nz}) {
      bspline_moduli(n, order, tmp);
      pd.insert(pd.end(), tmp.begin(), tmp.end());
    }
    m_host.push_back(A);
  }
  APO_CUDA(cudaMalloc(&m_q, q * sizeof(int)));
  APO_CUDA(cudaMalloc(&m_phi, q * sizeof(float)));
  APO_CUDA(cudaMalloc(&m_c, c * sizeof(float2)));
  APO_CUDA(cudaMalloc(&m_tw, t * sizeof(float2)));
  APO_CUDA(cudaMalloc(&m_pf, t * sizeof(float)));
  APO_CUDA(cudaMalloc(&m_pfd, t * sizeof(double)));
  APO_CUDA(cudaMemset(m_q, 0, q * sizeof(int)));
  std::vector<float> pf(pd.begin(), pd.end());
  APO_CUDA(cudaMemcpy(m_tw, tw.data(), t * sizeof(float2), cudaMemcpyHostToDevice));
  APO_CUDA(cudaMemcpy(m_pf, pf.data(), t * sizeof(float), cudaMemcpyHostToDevice));
  APO_CUDA(cudaMemcpy(m_pfd, pd.data(), t * sizeof(double), cudaMemcpyHostToDevice));
  for (PmeSysArgs &A : m_host) {
    const size_t qo = reinterpret_cast<size_t>(A.qgrid), co = reinterpret_cast<size_t>(A.cgrid),
                 to = reinterpret_cast<size_t>(A.tw);
    A.qgrid = m_q + qo;
    A.phi = m_phi + qo;
    A.cgrid = m_c + co;
    A.tw = m_tw + to;
    A.prefac = m_pf + to;
    A.prefac_d = m_pfd + to;
  }
  APO_CUDA(cudaMalloc(&m_args, m_host.size() * sizeof(PmeSysArgs)));
  APO_CUDA(cudaMemcpy(m_args, m_host.data(), m_host.size() * sizeof(PmeSysArgs),
                      cudaMemcpyHostToDevice));
  APO_CUDA(cudaMalloc(&m_plane_sys, plane_sys.size() * sizeof(int)));
  APO_CUDA(cudaMemcpy(m_plane_sys, plane_sys.data(), plane_sys.size() * sizeof(int),
                      cudaMemcpyHostToDevice));
  APO_CUDA(cudaMalloc(&m_pencil_sys, pencil_sys.size() * sizeof(int)));
  APO_CUDA(cudaMemcpy(m_pencil_sys, pencil_sys.data(), pencil_sys.size() * sizeof(int),
                      cudaMemcpyHostToDevice));
  raise_smem_limits();
}

void PmeMulti::compute(const float4 *xyzq_s, const float4 *origin, const int *cl_sys,
                       const int *counts, long long *force, int stride, bool calc_energy,
                       bool calc_virial, bool fp64, cudaStream_t s) {
  const PmeDims &d0 = m_host[0].d;
  const int blocks = (m_max_slots + 31) / 32;
  switch (m_order) {
    case 4: spread_kernel<4><<<blocks, 128, 0, s>>>(xyzq_s, counts, d0, nullptr, origin, m_args, cl_sys); break;
    case 6: spread_kernel<6><<<blocks, 128, 0, s>>>(xyzq_s, counts, d0, nullptr, origin, m_args, cl_sys); break;
    case 8: spread_kernel<8><<<blocks, 128, 0, s>>>(xyzq_s, counts, d0, nullptr, origin, m_args, cl_sys); break;
  }
  APO_LAUNCH_CHECK();
  (m_plane_smem <= kPlaneSmemTw ? plane_fwd_kernel<true> : plane_fwd_kernel<false>)<<<m_planes, m_plane_threads, m_plane_smem, s>>>(d0, nullptr, nullptr, nullptr,
                                                                  nullptr, m_args, m_plane_sys);
  APO_LAUNCH_CHECK();
  if (calc_virial) {
    if (fp64)
      pencil_kernel<true, double, true><<<m_pencils, kPencilThreads, m_pencil_smem, s>>>(d0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, m_args, m_pencil_sys, kNoTensorMap, nullptr);
    else
      pencil_kernel<true, float, true><<<m_pencils, kPencilThreads, m_pencil_smem, s>>>(d0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, m_args, m_pencil_sys, kNoTensorMap, nullptr);
  } else if (calc_energy) {
    if (fp64)
      pencil_kernel<true, double><<<m_pencils, kPencilThreads, m_pencil_smem, s>>>(d0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, m_args, m_pencil_sys, kNoTensorMap, nullptr);
    else
      pencil_kernel<true, float><<<m_pencils, kPencilThreads, m_pencil_smem, s>>>(d0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, m_args, m_pencil_sys, kNoTensorMap, nullptr);
  } else {
    if (fp64)
      pencil_kernel<false, double><<<m_pencils, kPencilThreads, m_pencil_smem, s>>>(d0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, m_args, m_pencil_sys, kNoTensorMap, nullptr);
    else
      pencil_kernel<false, float><<<m_pencils, kPencilThreads, m_pencil_smem, s>>>(d0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, m_args, m_pencil_sys, kNoTensorMap, nullptr);
  }
  APO_LAUNCH_CHECK();
  (m_plane_smem <= kPlaneSmemTw ? plane_inv_kernel<true> : plane_inv_kernel<false>)<<<m_planes, m_plane_threads, m_plane_smem, s>>>(d0, nullptr, nullptr, nullptr,
                                                                  nullptr, m_args, m_plane_sys);
  APO_LAUNCH_CHECK();
  switch (m_order) {
    case 4: gather4_kernel<<<blocks, 256, 0, s>>>(xyzq_s, counts, d0, nullptr, force, stride, origin, m_args, cl_sys); break;
    case 6: gather_kernel<6><<<blocks, 256, 0, s>>>(xyzq_s, counts, d0, nullptr, force, stride, origin, m_args, cl_sys); break;
    case 8: gather_kernel<8><<<blocks, 256, 0, s>>>(xyzq_s, counts, d0, nullptr, force, stride, origin, m_args, cl_sys); break;
  }
  APO_LAUNCH_CHECK();
}

}  // namespace apo

// ---------------------------------------------------------------------------
// Reciprocal space from a static scratch area (no allocation of its own)
// ---------------------------------------------------------------------------
//
// The charge grid, complex grid, potential grid, twiddles, B-spline moduli,
// atom count and energy accumulator live in g_pme_static, a file-scope
// device array.  Its address is looked up once per device with
// cudaGetSymbolAddress (that first call also sets the plane kernels'
// shared-memory attribute, so it belongs before any stream capture).  What
// must be zero when a call's spread starts: the charge grid and the energy
// accumulator.  The array is zero at module load, every call clears both
// with cudaMemsetAsync before its first kernel, and plane_fwd leaves the
// charge grid zeroed again as it reads it.  The tables are recomputed on
// the device by every call, so nothing else carries over between calls;
// calls that overlap in time (two streams, two host threads) race on the
// area.

namespace apo {
namespace {

__device__ __align__(256) unsigned char g_pme_static[kPmeStaticScratchBytes];

constexpr int kStaticMaxDevices = 64;
std::mutex g_static_mu;
std::atomic<unsigned char *> g_static_base[kStaticMaxDevices];

inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

struct StaticLayout {
  size_t energy, counts, tw, prefac, prefac_d, qgrid, cgrid, phi, total;
};

StaticLayout static_layout(int nx, int ny, int nz) {
  StaticLayout l{};
  const size_t n3 = (size_t)nx + ny + nz;
  const size_t G = (size_t)nx * ny * nz;
  const size_t Gc = (size_t)nz * ny * ((nx / 2 + 2) & ~1);  // padded rows
  size_t o = 0;
  l.energy = o;   o += align256(kNumEnergyTerms * sizeof(long long));
  l.counts = o;   o += align256(4 * sizeof(int));
  l.tw = o;       o += align256(n3 * sizeof(float2));
  l.prefac = o;   o += align256(n3 * sizeof(float));
  l.prefac_d = o; o += align256(n3 * sizeof(double));
  l.qgrid = o;    o += align256(G * sizeof(int));
  l.cgrid = o;    o += align256(Gc * sizeof(float2));
  l.phi = o;      o += align256(G * sizeof(float));
  l.total = o;
  return l;
}

// The plan search of Pme::plan_axis (fewest stages, then the smallest sum
// of radices, radices tried from 8 down to 2) on fixed arrays.
struct FixedPlan {
  int cur[8], best[8], ncur = 0, nbest = -1, sbest = 0;
  void rec(int m) {
    if (m == 1) {
      int s = 0;
      for (int i = 0; i < ncur; ++i) s += cur[i];
      if (nbest < 0 || ncur < nbest || (ncur == nbest && s < sbest)) {
        for (int i = 0; i < ncur; ++i) best[i] = cur[i];
        nbest = ncur;
        sbest = s;
      }
      return;
    }
    if (ncur == 8 || (nbest >= 0 && ncur + 1 > nbest)) return;
    for (int R : {8, 7, 6, 5, 4, 3, 2}) {
      if (m % R == 0) {
        cur[ncur++] = R;
        rec(m / R);
        --ncur;
      }
    }
  }
};

bool fixed_plan_axis(int n, FftAxis &a) {
  FixedPlan p;
  p.rec(n);
  if (p.nbest < 0) return false;
  a = FftAxis{};
  a.n = n;
  a.nrad = p.nbest;
  for (int i = 0; i < p.nbest; ++i) a.radix[i] = p.best[i];
  fill_axis_divisors(a);
  return true;
}

// |b(k)|^2 of the order-p B-spline for grid size n, as bspline_moduli
__device__ double static_modulus(int n, int order, int k) {
  double th[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  th[0] = 1.0;
  for (int kk = 3; kk <= order; ++kk) {
    const double div = 1.0 / (kk - 1);
    th[kk - 1] = 0.0;
    for (int j = 1; j <= kk - 2; ++j) th[kk - j - 1] = div * (j * th[kk - j - 2] + (kk - j) * th[kk - j - 1]);
    th[0] = div * th[0];
  }
  // arr[i - 1] = th[i - 2] for i = 2..order+1: arr[j] = th[j - 1] for j = 1..order
  double s1 = 0.0, s2 = 0.0;
  for (int j = 1; j <= order && j < n - 1; ++j) {
    double sv, cv;
    sincospi(2.0 * (double)(((long long)k * j) % n) / n, &sv, &cv);
    s1 += th[j - 1] * cv;
    s2 += th[j - 1] * sv;
  }
  return s1 * s1 + s2 * s2;
}

__global__ void static_tables_kernel(PmeDims d, float2 *__restrict__ tw, float *__restrict__ prefac,
                                     double *__restrict__ prefac_d, int *__restrict__ counts,
                                     int natom) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) counts[0] = natom;
  int n, k;
  if (t < d.nx) { n = d.nx; k = t; }
  else if (t < d.nx + d.ny) { n = d.ny; k = t - d.nx; }
  else if (t < d.nx + d.ny + d.nz) { n = d.nz; k = t - d.nx - d.ny; }
  else return;
  double sv, cv;
  sincospi(2.0 * k / n, &sv, &cv);
  tw[t] = make_float2((float)cv, (float)-sv);
  double m = static_modulus(n, d.order, k);
  if (m < 1e-10)
    m = 0.5 * (static_modulus(n, d.order, (k - 1 + n) % n) + static_modulus(n, d.order, (k + 1) % n));
  prefac_d[t] = 1.0 / m;
  prefac[t] = (float)(1.0 / m);
}

__global__ void static_finish_kernel(const long long *__restrict__ acc, double *__restrict__ energy) {
  if (threadIdx.x == 0 && blockIdx.x == 0) energy[0] = (double)acc[kEEwks] / kEnergyScale;
}

unsigned char *static_base() {
  int dev = 0;
  APO_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kStaticMaxDevices)
    throw std::invalid_argument("pme_reciprocal_static: device ordinal out of range");
  unsigned char *b = g_static_base[dev].load(std::memory_order_acquire);
  if (b) return b;
  std::lock_guard<std::mutex> lock(g_static_mu);
  b = g_static_base[dev].load(std::memory_order_relaxed);
  if (!b) {
    void *p = nullptr;
    APO_CUDA(cudaGetSymbolAddress(&p, g_pme_static));
    raise_smem_limits();
    b = static_cast<unsigned char *>(p);
    g_static_base[dev].store(b, std::memory_order_release);
  }
  return b;
}

}  // namespace

size_t pme_static_scratch_bytes(int nx, int ny, int nz) { return static_layout(nx, ny, nz).total; }

void pme_reciprocal_static(const float4 *xyzq, int n, double Lx, double Ly, double Lz, int nx,
                           int ny, int nz, int order, double kappa, long long *grad, int stride,
                           double *energy, bool fp64, cudaStream_t s) {
  if (n < 0) throw std::invalid_argument("pme_reciprocal_static: negative atom count");
  if (n > 0 && (xyzq == nullptr || grad == nullptr))
    throw std::invalid_argument("pme_reciprocal_static: coordinate or gradient pointer is NULL");
  if (n > 0 && stride < n) throw std::invalid_argument("pme_reciprocal_static: stride < atom count");
  if (!(Lx > 0.0 && Ly > 0.0 && Lz > 0.0 && kappa > 0.0))
    throw std::invalid_argument("pme_reciprocal_static: box lengths and kappa must be positive");
  if (nx <= 0 || ny <= 0 || nz <= 0 || nx % 2 || ny % 2 || nz % 2 || nx > 256 || ny > 256 ||
      nz > 256)
    throw std::invalid_argument("pme_reciprocal_static: grid dimensions must be even, 2..256");
  if (order != 4 && order != 6 && order != 8)
    throw std::invalid_argument("pme_reciprocal_static: spline order must be 4, 6 or 8");
  if (nx < order || ny < order || nz < order)
    throw std::invalid_argument(
        "pme_reciprocal_static: grid dimensions must be at least the spline order");
  if (plane_smem_bytes(nx, ny) > kPlaneSmemMax)
    throw std::invalid_argument("pme_reciprocal_static: grid plane does not fit in shared memory");
  const StaticLayout l = static_layout(nx, ny, nz);
  if (l.total > kPmeStaticScratchBytes)
    throw std::invalid_argument(
        "pme_reciprocal_static: grid needs more scratch than the static area holds "
        "(8 MiB: about 5.5e5 grid points)");
  PmeDims d{};
  d.nx = nx;
  d.ny = ny;
  d.nz = nz;
  d.nxc = nx / 2 + 1;
  d.nxcp = (d.nxc + 1) & ~1;
  d.order = order;
  d.Lx = (float)Lx;
  d.Ly = (float)Ly;
  d.Lz = (float)Lz;
  d.rLx = 1.0 / Lx;
  d.rLy = 1.0 / Ly;
  d.rLz = 1.0 / Lz;
  d.kappa = (float)kappa;
  if (!fixed_plan_axis(nx, d.ax) || !fixed_plan_axis(ny, d.ay) || !fixed_plan_axis(nz, d.az))
    throw std::invalid_argument("pme_reciprocal_static: grid sizes must factor into 2, 3, 5 and 7");
  set_tiles(d);

  unsigned char *b = static_base();
  long long *acc = reinterpret_cast<long long *>(b + l.energy);
  int *counts = reinterpret_cast<int *>(b + l.counts);
  float2 *tw = reinterpret_cast<float2 *>(b + l.tw);
  float *prefac = reinterpret_cast<float *>(b + l.prefac);
  double *prefac_d = reinterpret_cast<double *>(b + l.prefac_d);
  int *qgrid = reinterpret_cast<int *>(b + l.qgrid);
  float2 *cgrid = reinterpret_cast<float2 *>(b + l.cgrid);
  float *phi = reinterpret_cast<float *>(b + l.phi);
  const size_t G = (size_t)nx * ny * nz;

  APO_CUDA(cudaMemsetAsync(acc, 0, kNumEnergyTerms * sizeof(long long), s));
  if (n == 0) {
    if (energy) APO_CUDA(cudaMemsetAsync(energy, 0, sizeof(double), s));
    return;
  }
  APO_CUDA(cudaMemsetAsync(qgrid, 0, G * sizeof(int), s));
  const int n3 = nx + ny + nz;
  static_tables_kernel<<<(n3 + 127) / 128, 128, 0, s>>>(d, tw, prefac, prefac_d, counts, n);
  APO_LAUNCH_CHECK();
  const int blocks = (n + 31) / 32;
  switch (order) {
    case 4: spread_kernel<4><<<blocks, 128, 0, s>>>(xyzq, counts, d, qgrid, nullptr); break;
    case 6: spread_kernel<6><<<blocks, 128, 0, s>>>(xyzq, counts, d, qgrid, nullptr); break;
    case 8: spread_kernel<8><<<blocks, 128, 0, s>>>(xyzq, counts, d, qgrid, nullptr); break;
  }
  APO_LAUNCH_CHECK();
  const size_t sm = plane_smem_bytes(nx, ny);
  (sm <= kPlaneSmemTw ? plane_fwd_kernel<true> : plane_fwd_kernel<false>)<<<nz, plane_threads(nx, ny), sm, s>>>(
      d, qgrid, cgrid, tw, tw + nx, nullptr, nullptr);
  APO_LAUNCH_CHECK();
  const int pgrid = d.ptiles * ny;
  const size_t psm = pencil_smem_bytes(d);
  const float2 *twz = tw + nx + ny;
  if (fp64)
    pencil_kernel<true, double><<<pgrid, kPencilThreads, psm, s>>>(d, cgrid, twz, prefac, prefac_d, acc, nullptr, nullptr, nullptr, kNoTensorMap, nullptr);
  else
    pencil_kernel<true, float><<<pgrid, kPencilThreads, psm, s>>>(d, cgrid, twz, prefac, prefac_d, acc, nullptr, nullptr, nullptr, kNoTensorMap, nullptr);
  APO_LAUNCH_CHECK();
  (sm <= kPlaneSmemTw ? plane_inv_kernel<true> : plane_inv_kernel<false>)<<<nz, plane_threads(nx, ny), sm, s>>>(
      d, cgrid, phi, tw, tw + nx, nullptr, nullptr);
  APO_LAUNCH_CHECK();
  switch (order) {
    case 4: gather4_kernel<<<blocks, 256, 0, s>>>(xyzq, counts, d, phi, grad, stride, nullptr); break;
    case 6: gather_kernel<6><<<blocks, 256, 0, s>>>(xyzq, counts, d, phi, grad, stride, nullptr); break;
    case 8: gather_kernel<8><<<blocks, 256, 0, s>>>(xyzq, counts, d, phi, grad, stride, nullptr); break;
  }
  APO_LAUNCH_CHECK();
  if (energy) {
    static_finish_kernel<<<1, 32, 0, s>>>(acc, energy);
    APO_LAUNCH_CHECK();
  }
}

}  // namespace apo
