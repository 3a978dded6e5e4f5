// Direct-space tile kernel; see nonbonded.h.
//
// One warp per work item (an i-cluster and a run of up to tiles_per_work of
// its j-tiles), persistent grid.  Lane l owns i-atom l for the whole work
// item: its force lives in registers.  The j-atoms of a tile that reach the
// i-cluster's live box are appended to a queue in shared memory that runs
// across the work item's tiles (a tile leaves 13 of its 32 on average, so
// batches of 8 within a tile would be a quarter fillers); 32 of them at a
// time are read back as warp-wide broadcasts, two by two for the packed
// arithmetic.  The j-forces are combined across the warp with a transpose
// reduction: 9 shuffles per component for every 8 j-atoms, after which lane L
// holds the full force of j-atom (L&3)*8 + (L>>2) and adds it to its slot, 32
// lanes at once.  Tiles with exclusions (and a cluster's tile with itself) do
// not go through the queue.  Bound by instruction issue (65 % of the slots busy at
// 107,000 atoms with 15 warps an SM, 57 % at 24,000 with 11) and, as much, by the
// latency of the pair chain and of the tiles' loads: with the queue, the
// tiles read 32 at a time and padding slots far away instead of tested, the
// kernel takes 81 us a launch on 24,000 atoms with four blocks an SM, 85 with the
// three it has there now (98.6 before, 40 steps 6.76 -> 6.41 ms), and 1.69 ms on
// 998,000 (2.15 before the pair function's and these changes, 20 steps 62.6 ->
// 58.9 ms).
#include "nonbonded.h"

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "device_util.cuh"
#include "nblist.h"
#include "nonbonded_pair.cuh"
#include "resident_grid.h"

namespace apo {

NbSetup make_nb_setup(double Lx, double Ly, double Lz, double kappa, double roff,
                      double ron) {
  NbSetup s;
  s.Lxd = Lx;
  s.Lyd = Ly;
  s.Lzd = Lz;
  s.Lx_lo = (float)(Lx - (double)(float)Lx);
  s.Ly_lo = (float)(Ly - (double)(float)Ly);
  s.Lz_lo = (float)(Lz - (double)(float)Lz);
  s.Lx = (float)Lx;
  s.Ly = (float)Ly;
  s.Lz = (float)Lz;
  s.roff2 = (float)(roff * roff);
  s.ron2 = (float)(ron * ron);
  s.kappa = (float)kappa;
  s.kappa2 = (float)(kappa * kappa);
  s.two_kappa_sqrtpi = (float)(2.0 * kappa / std::sqrt(M_PI));
  s.ewald_e2 = (float)(-kappa * kappa / std::log(2.0));
  // VDW_VFSW constants (src/CudaPMEDirectForce.cu:318-330)
  double roff3 = roff * roff * roff, ron3 = ron * ron * ron;
  double roff6 = roff3 * roff3, ron6 = ron3 * ron3;
  s.roffinv3 = (float)(1.0 / roff3);
  s.roffinv6 = (float)(1.0 / roff6);
  s.kp = (float)(0.365 * kappa);
  s.sw6 = s.sw12 = 0.f;
  if (ron < roff) {
    s.sw6 = (float)(1.0 / (roff3 - ron3));
    s.sw12 = (float)(1.0 / (roff6 - ron6));
    s.k6 = (float)(roff3 / (roff3 - ron3));
    s.k12 = (float)(roff6 / (roff6 - ron6));
    s.dv6 = (float)(-1.0 / (ron3 * roff3));
    s.dv12 = (float)(-1.0 / (ron6 * roff6));
  } else {
    s.k6 = 1.f;
    s.k12 = 1.f;
    s.dv6 = (float)(-1.0 / roff6);
    s.dv12 = (float)(-1.0 / (roff6 * roff6));
  }
  return s;
}

namespace {

using namespace nbdetail;

constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;

template <bool ENERGY, bool PER_PAIR, bool VIRIAL, bool MULTI>
__device__ __forceinline__ void nb_body(const NbArgs &a) {
  // the j-atoms that pass the box test, compacted: position and charge (for
  // the packed arithmetic as pairs of j-atoms: {x0 x1 y0 y1} and {z0 z1 q0
  // q1}), LJ type, and the list slot (queue) or tile lane (single tile).
  // Packed form: entries 0..63 are a queue carried across the tiles of a work
  // item, entries 64..95 a single tile with exclusions; PER_PAIR: 0..31.
  constexpr int kEnt = PER_PAIR ? 32 : 96;
  __shared__ float4 sh_xq[kWarps][kEnt];
  __shared__ __align__(16) int sh_tj[kWarps][kEnt];
  __shared__ int sh_js[kWarps][kEnt];
  extern __shared__ float2 sh_vdw[];
  int T = a.ntype;
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  // one system: the whole table once per block; several systems: one
  // ntype^2 slice per warp, reloaded when the warp's system changes
  const int tab_off = MULTI ? wib * kMaxMultiTypes * kMaxMultiTypes : 0;
  int cur_sys = -1;
  // the packed pair function takes the second coefficient negated
  const float vsign = PER_PAIR ? 1.f : -1.f;
  if (!MULTI) {
    for (int k = threadIdx.x; k < T * T; k += blockDim.x) {
      const float2 c = a.vdw[k];
      sh_vdw[k] = make_float2(c.x, vsign * c.y);
    }
    __syncthreads();
  }
  const unsigned lt_mask = (1u << lane) - 1u;
  const int nwork = a.counts[2];
  const int stride = a.stride;
  double e_elec = 0.0, e_vdw = 0.0;
  // one system: per-lane fixed-point sums of every work item's energies and
  // virial (integer sums: the total does not depend on which warp took
  // which item)
  long long ie_el = 0, ie_vdw = 0;
  long long ivir[6] = {0, 0, 0, 0, 0, 0};  // xx xy xz yy yz zz (VIRIAL)
  using Acc = typename std::conditional<PER_PAIR, long long, float>::type;

  int taken = 0;  // warp-uniform
  auto next = [&]() -> int {
    if (a.items_per_warp > 0 && taken >= a.items_per_warp) return nwork;
    ++taken;
    return next_work(a.sched, lane);
  };
  for (int w = next(); w < nwork; w = next()) {
    // work items are taken in a scattered order, w -> (w * 7919) mod nwork
    // (one to one unless nwork is a multiple of 7919): warps working at the
    // same time then add their j-forces to distant parts of the buffer
    // (chain23k: 116.7 -> 114.8 us a launch); the results do not depend on
    // the order
    const int wp = (nwork % 7919) ? (int)(((long long)w * 7919) % nwork) : w;
    const int4 wk = a.work[wp];
    const NbSetup st = a.setups[wk.w];
    if (MULTI && wk.w != cur_sys) {  // warp-uniform
      __syncwarp();
      T = st.ntype;
      for (int k = lane; k < T * T; k += 32) {
        const float2 c = a.vdw[st.vdw_off + k];
        sh_vdw[tab_off + k] = make_float2(c.x, vsign * c.y);
      }
      __syncwarp();
      cur_sys = wk.w;
    }
    const float4 oi = a.origin[wk.x];
    const int islot = wk.x * kTile + lane;
    const float4 xi = a.xyzq_s[islot];
    const bool ivalid = xi.x < 0.5f * kFarAway;
    const float qi = (PER_PAIR ? 1.f : -1.f) * xi.w * (float)kCcelec;
    // this lane's row of the LJ table
    const float2 *vrow = sh_vdw + tab_off + a.type_s[islot] * T;
    // box around the current positions of the i-cluster
    float lo_x = ivalid ? xi.x : INFINITY, lo_y = ivalid ? xi.y : INFINITY,
          lo_z = ivalid ? xi.z : INFINITY;
    float hi_x = ivalid ? xi.x : -INFINITY, hi_y = ivalid ? xi.y : -INFINITY,
          hi_z = ivalid ? xi.z : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo_x = fminf(lo_x, __shfl_xor_sync(0xffffffffu, lo_x, o));
      lo_y = fminf(lo_y, __shfl_xor_sync(0xffffffffu, lo_y, o));
      lo_z = fminf(lo_z, __shfl_xor_sync(0xffffffffu, lo_z, o));
      hi_x = fmaxf(hi_x, __shfl_xor_sync(0xffffffffu, hi_x, o));
      hi_y = fmaxf(hi_y, __shfl_xor_sync(0xffffffffu, hi_y, o));
      hi_z = fmaxf(hi_z, __shfl_xor_sync(0xffffffffu, hi_z, o));
    }
    Acc fix = 0, fiy = 0, fiz = 0;
    float vw[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // packed form: i-atom values in both halves, two partial sums per sum;
    // a padding slot sits kFarAway off, so none of its pairs is inside the
    // cutoff (its differences stay finite: their force factor is exactly 0)
    const F2 xi2x = f2(xi.x), xi2y = f2(xi.y), xi2z = f2(xi.z), qi2 = f2(qi);
    F2 fi2x = f2(0.f), fi2y = f2(0.f), fi2z = f2(0.f);
    F2 vw2[6] = {f2(0.f), f2(0.f), f2(0.f), f2(0.f), f2(0.f), f2(0.f)};

    // the pairs of this lane's i-atom with entries [e0, e0 + n) (e0 even, n
    // rounded up to whole batches of eight by fillers), and the j-forces
    // added to their slots
    auto consume = [&](auto with_excl, int e0, int n, unsigned excl, int slot0) {
      constexpr bool EXCL = decltype(with_excl)::value;
      float fjx = 0.f, fjy = 0.f, fjz = 0.f;  // force of entry (lane&3)*8 + (lane>>2)
      const int nbatch = (n + 7) >> 3;
      for (int b = 0; b < nbatch; ++b) {
        float fx[8], fy[8], fz[8];
#pragma unroll
        for (int pp = 0; pp < 4; ++pp) {
          const int r = e0 + b * 8 + 2 * pp;
          const float4 A = sh_xq[wib][r];      // x0 x1 y0 y1
          const float4 B = sh_xq[wib][r + 1];  // z0 z1 q0 q1
          const int2 tj = *reinterpret_cast<const int2 *>(&sh_tj[wib][r]);
          const F2 dx = xi2x - f2(A.x, A.y), dy = xi2y - f2(A.z, A.w), dz = xi2z - f2(B.x, B.y);
          const F2 r2 = fma2(dz, dz, fma2(dy, dy, dx * dx));
          bool in0 = f2lo(r2) < st.roff2, in1 = f2hi(r2) < st.roff2;
          if (EXCL) {
            in0 = in0 && !((excl >> sh_js[wib][r]) & 1u);
            in1 = in1 && !((excl >> sh_js[wib][r + 1]) & 1u);
          }
          const F2 f = pair_force2<ENERGY>(st, r2, in0, in1, qi2 * f2(B.z, B.w), vrow[tj.x],
                                           vrow[tj.y], e_elec, e_vdw);
          const F2 gx = f * dx, gy = f * dy, gz = f * dz;
          if (VIRIAL) {
            vw2[0] = fma2(gx, dx, vw2[0]);
            vw2[1] = fma2(gx, dy, vw2[1]);
            vw2[2] = fma2(gx, dz, vw2[2]);
            vw2[3] = fma2(gy, dy, vw2[3]);
            vw2[4] = fma2(gy, dz, vw2[4]);
            vw2[5] = fma2(gz, dz, vw2[5]);
          }
          fi2x = fi2x + gx;
          fi2y = fi2y + gy;
          fi2z = fi2z + gz;
          fx[2 * pp] = f2lo(gx);
          fx[2 * pp + 1] = f2hi(gx);
          fy[2 * pp] = f2lo(gy);
          fy[2 * pp + 1] = f2hi(gy);
          fz[2 * pp] = f2lo(gz);
          fz[2 * pp + 1] = f2hi(gz);
        }
        // the sums hold the gradient on i of each pair: the j-atom's is minus it
        const float rx = transpose_reduce8(fx, lane);
        const float ry = transpose_reduce8(fy, lane);
        const float rz = transpose_reduce8(fz, lane);
        if ((lane & 3) == b) {
          fjx = -rx;
          fjy = -ry;
          fjz = -rz;
        }
      }
      const int own = (lane & 3) * 8 + (lane >> 2);
      if (own < n) {
        const int js = slot0 + sh_js[wib][e0 + own];
        add_fixed(a.force + js, to_fixed_force(fjx));
        add_fixed(a.force + stride + js, to_fixed_force(fjy));
        add_fixed(a.force + 2 * stride + js, to_fixed_force(fjz));
      }
    };
    // entry e of the shared arrays: packed pairs
    auto put = [&](int e, float x, float y, float z, float q, int type, int js) {
      float *pa = reinterpret_cast<float *>(&sh_xq[wib][e & ~1]);
      const int h = e & 1;
      pa[h] = x;
      pa[2 + h] = y;
      pa[4 + h] = z;
      pa[6 + h] = q;
      sh_tj[wib][e] = type;
      sh_js[wib][e] = js;
    };
    // fillers up to a whole batch: out of everybody's reach, a padding
    // i-atom's among them
    auto pad = [&](int e0, int n, int ring) {
      const int nf = -n & 7;
      if (lane < nf) put((e0 + n + lane) & ring, 2.f * kFarAway, 2.f * kFarAway, 2.f * kFarAway, 0.f, 0, 0);
    };
    int head = 0, cnt = 0;  // the queue (uniform)
    // tiles are read 32 at a time, a tile a lane, with the shift of each one's
    // frame, and handed out by shuffles
    int2 my_tl = make_int2(0, 0);
    float my_sx = 0.f, my_sy = 0.f, my_sz = 0.f;

    for (int t = wk.y;;) {
      if constexpr (!PER_PAIR) {
        if (cnt >= 32 || (t >= wk.z && cnt > 0)) {
          const int n = min(cnt, 32);
          if (n < 32) {
            pad(head, n, 63);
            __syncwarp();
          }
          consume(std::false_type{}, head, n, 0u, 0);
          head ^= 32;
          cnt -= n;
          __syncwarp();
          continue;
        }
      }
      if (t >= wk.z) break;
      if (((t - wk.y) & 31) == 0) {  // the next 32 tiles, one a lane
        if (t + lane < wk.z) {
          my_tl = a.tiles[t + lane];
          const int code = tile_image(my_tl.y);
          // j cluster frame -> i cluster frame: origin difference (exact: both
          // origins are multiples of 1/64 A) plus the periodic image k L with
          // L as a two-float sum, so |offset| < rlist + 2 cluster edges
          // carries about one rounding
          const float4 oj = a.origin[my_tl.x];
          const int ic = code / 9, ib = (code - 9 * ic) / 3, ia = code - 9 * ic - 3 * ib;
          const float kx = (float)(ia - 1), ky = (float)(ib - 1), kz = (float)(ic - 1);
          my_sx = fmaf(kx, st.Lx, oj.x - oi.x) + kx * st.Lx_lo;
          my_sy = fmaf(ky, st.Ly, oj.y - oi.y) + ky * st.Ly_lo;
          my_sz = fmaf(kz, st.Lz, oj.z - oi.z) + kz * st.Lz_lo;
        }
      }
      const int src = (t - wk.y) & 31;
      ++t;
      const int2 tl = make_int2(__shfl_sync(0xffffffffu, my_tl.x, src),
                                __shfl_sync(0xffffffffu, my_tl.y, src));
      const int code = tile_image(tl.y);
      const int jslot = tl.x * kTile + lane;
      float4 xj = a.xyzq_s[jslot];
      xj.x += __shfl_sync(0xffffffffu, my_sx, src);
      xj.y += __shfl_sync(0xffffffffu, my_sy, src);
      xj.z += __shfl_sync(0xffffffffu, my_sz, src);
      // j-atoms that can reach the cutoff of some i-atom
      const float bx = fmaxf(0.f, fmaxf(lo_x - xj.x, xj.x - hi_x));
      const float by = fmaxf(0.f, fmaxf(lo_y - xj.y, xj.y - hi_y));
      const float bz = fmaxf(0.f, fmaxf(lo_z - xj.z, xj.z - hi_z));
      // (a padding slot lies kFarAway off)
      const bool jnear = bx * bx + by * by + bz * bz < st.roff2;
      const unsigned jmask = __ballot_sync(0xffffffffu, jnear);
      if (jmask == 0u) continue;
      const unsigned excl = tile_excl_word(a, tl, code, wk.x, lane);
      const int nj = __popc(jmask);
      const int rank = __popc(jmask & lt_mask);
      if constexpr (!PER_PAIR) {
        if (__any_sync(0xffffffffu, excl != 0u)) {
          // a tile with exclusions (or a cluster's tile with itself): on its own
          if (jnear) put(64 + rank, xj.x, xj.y, xj.z, xj.w, a.type_s[jslot], lane);
          pad(64, nj, 127);
          __syncwarp();
          consume(std::true_type{}, 64, nj, excl, tl.x * kTile);
          __syncwarp();
        } else {
          if (jnear) put((head + cnt + rank) & 63, xj.x, xj.y, xj.z, xj.w, a.type_s[jslot], jslot);
          cnt += nj;
          __syncwarp();
        }
        continue;
      }
      __syncwarp();
      if (jnear) {
        sh_xq[wib][rank] = xj;
        sh_tj[wib][rank] = a.type_s[jslot] | (lane << 16);
      }
      __syncwarp();

      Acc fjx = 0, fjy = 0, fjz = 0;  // force of compacted j (lane&3)*8 + (lane>>2)
      const int nbatch = (nj + 7) >> 3;
      for (int b = 0; b < nbatch; ++b) {
        Acc fx[8], fy[8], fz[8];
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          const int r = b * 8 + jj;
          fx[jj] = 0;
          fy[jj] = 0;
          fz[jj] = 0;
          if (r < nj) {  // uniform across the warp
            const float4 pj = sh_xq[wib][r];
            const int tj = sh_tj[wib][r];
            const float dx = xi.x - pj.x, dy = xi.y - pj.y, dz = xi.z - pj.z;
            const float r2raw = dx * dx + dy * dy + dz * dz;
            const bool in = ivalid && !((excl >> (tj >> 16)) & 1u) && r2raw < st.roff2;
            const float2 cc = vrow[tj & 0xffff];
            const float fij = pair_force<ENERGY>(st, r2raw, in, qi, pj.w, cc, e_elec, e_vdw);
            if (VIRIAL) {
              const float gx = fij * dx, gy = fij * dy, gz = fij * dz;
              vw[0] -= gx * dx;
              vw[1] -= gx * dy;
              vw[2] -= gx * dz;
              vw[3] -= gy * dy;
              vw[4] -= gy * dz;
              vw[5] -= gz * dz;
            }
            const long long gx = to_fixed_force(fij * dx);
            const long long gy = to_fixed_force(fij * dy);
            const long long gz = to_fixed_force(fij * dz);
            fix += gx;
            fiy += gy;
            fiz += gz;
            fx[jj] = -gx;
            fy[jj] = -gy;
            fz[jj] = -gz;
          }
        }
        const Acc rx = transpose_reduce8(fx, lane);
        const Acc ry = transpose_reduce8(fy, lane);
        const Acc rz = transpose_reduce8(fz, lane);
        if ((lane & 3) == b) {
          fjx = rx;
          fjy = ry;
          fjz = rz;
        }
      }
      const int rown = (lane & 3) * 8 + (lane >> 2);
      if (rown < nj) {
        const int jown = tl.x * kTile + (sh_tj[wib][rown] >> 16);
        add_fixed(a.force + jown, (long long)fjx);
        add_fixed(a.force + stride + jown, (long long)fjy);
        add_fixed(a.force + 2 * stride + jown, (long long)fjz);
      }
    }
    if (!PER_PAIR) {
      fix = f2lo(fi2x) + f2hi(fi2x);
      fiy = f2lo(fi2y) + f2hi(fi2y);
      fiz = f2lo(fi2z) + f2hi(fi2z);
      if (VIRIAL) {
#pragma unroll
        for (int k = 0; k < 6; ++k) vw[k] = -(f2lo(vw2[k]) + f2hi(vw2[k]));
      }
    }
    if (MULTI && ENERGY) {  // energies (and virial) belong to this work item's system
      long long *es = a.energy + (size_t)wk.w * a.energy_stride;
      warp_flush(e_elec, es + kEElec, lane);
      warp_flush(e_vdw, es + kEVdw, lane);
      e_elec = 0.0;
      e_vdw = 0.0;
      if (VIRIAL) {
        constexpr int kSlotM[6][2] = {{0, 0}, {1, 3}, {2, 6}, {4, 4}, {5, 7}, {8, 8}};
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          long long iw = __double2ll_rn((double)vw[k] * kEnergyScale);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) iw += __shfl_xor_sync(0xffffffffu, iw, o);
          if (lane == 0 && iw) {
            add_fixed(es + kNumEnergyTerms + kSlotM[k][0], iw);
            if (kSlotM[k][1] != kSlotM[k][0]) add_fixed(es + kNumEnergyTerms + kSlotM[k][1], iw);
          }
        }
      }
    }
    if (ENERGY && !MULTI) {
      ie_el += __double2ll_rn(e_elec * kEnergyScale);
      ie_vdw += __double2ll_rn(e_vdw * kEnergyScale);
      e_elec = 0.0;
      e_vdw = 0.0;
    }
    if (VIRIAL && !MULTI) {
#pragma unroll
      for (int k = 0; k < 6; ++k) ivir[k] += __double2ll_rn((double)vw[k] * kEnergyScale);
    }
    if (ivalid) {
      if (PER_PAIR) {
        add_fixed(a.force + islot, (long long)fix);
        add_fixed(a.force + stride + islot, (long long)fiy);
        add_fixed(a.force + 2 * stride + islot, (long long)fiz);
      } else {
        add_fixed(a.force + islot, to_fixed_force((float)fix));
        add_fixed(a.force + stride + islot, to_fixed_force((float)fiy));
        add_fixed(a.force + 2 * stride + islot, to_fixed_force((float)fiz));
      }
    }
  }
  retire_warp(a.sched, lane);
  if (ENERGY && !MULTI) {
    long long ie = ie_el, iv = ie_vdw;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ie += __shfl_xor_sync(0xffffffffu, ie, o);
      iv += __shfl_xor_sync(0xffffffffu, iv, o);
    }
    if (lane == 0) {
      add_fixed(a.energy + kEElec, ie);
      add_fixed(a.energy + kEVdw, iv);
    }
  }
  if (VIRIAL && !MULTI) {
    // xx xy xz yy yz zz -> row-major 3x3 (symmetric)
    constexpr int kSlot[6][2] = {{0, 0}, {1, 3}, {2, 6}, {4, 4}, {5, 7}, {8, 8}};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      long long iw = ivir[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) iw += __shfl_xor_sync(0xffffffffu, iw, o);
      if (lane == 0) {
        add_fixed(a.virial + kSlot[k][0], iw);
        if (kSlot[k][1] != kSlot[k][0]) add_fixed(a.virial + kSlot[k][1], iw);
      }
    }
  }
}

template <bool ENERGY, bool PER_PAIR, bool VIRIAL, bool MULTI>
__global__ void __launch_bounds__(kThreads) nb_kernel(NbArgs a) {
  nb_body<ENERGY, PER_PAIR, VIRIAL, MULTI>(a);
}
// with energies or the virial the packed form is held to 128 registers, four
// blocks an SM: it took 167 with both, three blocks (40 piston steps of 24,000 atoms 8.86
// -> 8.70 ms, an evaluation with virial 603 -> 577 us).  Without energies the
// compiler's own 122 (four blocks) stand.
template <bool ENERGY, bool PER_PAIR, bool VIRIAL, bool MULTI>
__global__ void __launch_bounds__(kThreads, 4) nb_energy_kernel(NbArgs a) {
  nb_body<ENERGY, PER_PAIR, VIRIAL, MULTI>(a);
}

// ---------------------------------------------------------------------------
// Grouped-queue variant.  The i-cluster is split into four 8-atom groups
// (the neighbour list orders each cluster as two z-halves of two x-halves,
// so a group is a compact 3.5 x 3.5 x 7 A block).  Every j-atom of a tile
// is tested against each group's live box and appended to that group's
// queue in shared memory (a 64-entry ring per group) with its position
// already in the i-cluster frame; the queues are consumed in batches of 8
// entries per group across tile boundaries.  Lane (g, l) computes the pairs
// of its i-atom with 8 entries of queue g, and the j-forces are combined
// over the group's 8 lanes (3 shuffle levels) before one atomic add per j.
// Fewer wasted pairs than testing all 32 i-atoms against a j that is only
// near part of the cluster, and no padding to 8 pairs per tile.
// ---------------------------------------------------------------------------

constexpr int kQ = 64;  // ring entries per group

__device__ __forceinline__ int sel4(int g, int a0, int a1, int a2, int a3) {
  return g == 0 ? a0 : g == 1 ? a1 : g == 2 ? a2 : a3;
}

// bits [start, start + n) of a 64-bit ring (n <= 64)
__device__ __forceinline__ unsigned long long ring_mask(int start, int n) {
  if (n <= 0) return 0ull;
  const unsigned long long m = n >= 64 ? ~0ull : ((1ull << n) - 1ull);
  const int s = start & 63;
  return s == 0 ? m : ((m << s) | (m >> (64 - s)));
}

template <bool ENERGY, bool PER_PAIR, bool VIRIAL, bool MULTI>
__global__ void __launch_bounds__(kThreads, 5) nbq_kernel(NbArgs a) {
  __shared__ float4 q_pos[kWarps][4][kQ];   // j position in the i frame, charge
  __shared__ int2 q_inf[kWarps][4][kQ];     // j slot, LJ type
  __shared__ float sh_box[kWarps][4][6];    // group boxes: lo xyz, hi xyz
  extern __shared__ float2 sh_vdw[];
  int T = a.ntype;
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int g = lane >> 3;
  const int tab_off = MULTI ? wib * kMaxMultiTypes * kMaxMultiTypes : 0;
  int cur_sys = -1;
  if (!MULTI) {
    for (int k = threadIdx.x; k < T * T; k += blockDim.x) sh_vdw[k] = a.vdw[k];
    __syncthreads();
  }
  const unsigned lt_mask = (1u << lane) - 1u;
  const int nwork = a.counts[2];
  const int stride = a.stride;
  double e_elec = 0.0, e_vdw = 0.0;
  double dv[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  // one system: per-lane fixed-point sums of every work item's energies and
  // virial (integer sums: the total does not depend on which warp took
  // which item)
  long long ie_el = 0, ie_vdw = 0;
  long long ivir[6] = {0, 0, 0, 0, 0, 0};
  using Acc = typename std::conditional<PER_PAIR, long long, float>::type;

  int taken = 0;  // warp-uniform
  auto next = [&]() -> int {
    if (a.items_per_warp > 0 && taken >= a.items_per_warp) return nwork;
    ++taken;
    return next_work(a.sched, lane);
  };
  for (int w = next(); w < nwork; w = next()) {
    const int4 wk = a.work[w];
    const NbSetup st = a.setups[wk.w];
    if (MULTI && wk.w != cur_sys) {  // warp-uniform
      __syncwarp();
      T = st.ntype;
      for (int k = lane; k < T * T; k += 32) sh_vdw[tab_off + k] = a.vdw[st.vdw_off + k];
      __syncwarp();
      cur_sys = wk.w;
    }
    const float4 oi = a.origin[wk.x];
    const int islot = wk.x * kTile + lane;
    const float4 xi = a.xyzq_s[islot];
    const bool ivalid = a.perm[islot] >= 0;
    const float qi = xi.w * (float)kCcelec;
    const int ti = a.type_s[islot] * T;
    // live box of this lane's group
    float lo_x = ivalid ? xi.x : INFINITY, lo_y = ivalid ? xi.y : INFINITY,
          lo_z = ivalid ? xi.z : INFINITY;
    float hi_x = ivalid ? xi.x : -INFINITY, hi_y = ivalid ? xi.y : -INFINITY,
          hi_z = ivalid ? xi.z : -INFINITY;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      lo_x = fminf(lo_x, __shfl_xor_sync(0xffffffffu, lo_x, o));
      lo_y = fminf(lo_y, __shfl_xor_sync(0xffffffffu, lo_y, o));
      lo_z = fminf(lo_z, __shfl_xor_sync(0xffffffffu, lo_z, o));
      hi_x = fmaxf(hi_x, __shfl_xor_sync(0xffffffffu, hi_x, o));
      hi_y = fmaxf(hi_y, __shfl_xor_sync(0xffffffffu, hi_y, o));
      hi_z = fmaxf(hi_z, __shfl_xor_sync(0xffffffffu, hi_z, o));
    }
    __syncwarp();
    if ((lane & 7) == 0) {
      sh_box[wib][g][0] = lo_x;
      sh_box[wib][g][1] = lo_y;
      sh_box[wib][g][2] = lo_z;
      sh_box[wib][g][3] = hi_x;
      sh_box[wib][g][4] = hi_y;
      sh_box[wib][g][5] = hi_z;
    }
    __syncwarp();
    Acc fix = 0, fiy = 0, fiz = 0;
    float vw[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    int h0 = 0, h1 = 0, h2 = 0, h3 = 0;   // ring heads (uniform)
    int t0 = 0, t1 = 0, t2 = 0, t3 = 0;   // ring tails (uniform)
    unsigned long long xmask = 0ull;      // excluded entries of my group, by ring position

    // consume up to 8 entries of every group
    auto batch = [&]() {
      const int head = sel4(g, h0, h1, h2, h3);
      const int cnt = min(8, sel4(g, t0, t1, t2, t3) - head);
      Acc fx[8], fy[8], fz[8];
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        const int pos = (head + jj) & (kQ - 1);
        // entries past this group's count are stale ring contents (possibly
        // not even finite): they are masked and their differences zeroed
        const float4 pj = q_pos[wib][g][pos];
        const int tj = q_inf[wib][g][pos].y;
        float dx = xi.x - pj.x, dy = xi.y - pj.y, dz = xi.z - pj.z;
        const float r2raw = dx * dx + dy * dy + dz * dz;
        const bool in = jj < cnt && ivalid && !((xmask >> pos) & 1ull) && r2raw < st.roff2;
        dx = in ? dx : 0.f;
        dy = in ? dy : 0.f;
        dz = in ? dz : 0.f;
        // stale entries: an in-range table index and a finite charge
        const float2 cc = sh_vdw[tab_off + ti + (in ? tj : 0)];
        const float fij = pair_force<ENERGY>(st, r2raw, in, qi, in ? pj.w : 0.f, cc, e_elec, e_vdw);
        if (VIRIAL) {
          const float gx = fij * dx, gy = fij * dy, gz = fij * dz;
          vw[0] -= gx * dx;
          vw[1] -= gx * dy;
          vw[2] -= gx * dz;
          vw[3] -= gy * dy;
          vw[4] -= gy * dz;
          vw[5] -= gz * dz;
        }
        if (PER_PAIR) {
          const long long gx = to_fixed_force(fij * dx);
          const long long gy = to_fixed_force(fij * dy);
          const long long gz = to_fixed_force(fij * dz);
          fix += gx;
          fiy += gy;
          fiz += gz;
          fx[jj] = -gx;
          fy[jj] = -gy;
          fz[jj] = -gz;
        } else {
          fix += fij * dx;
          fiy += fij * dy;
          fiz += fij * dz;
          fx[jj] = -fij * dx;
          fy[jj] = -fij * dy;
          fz[jj] = -fij * dz;
        }
      }
      const Acc rx = group_reduce8(fx, lane);
      const Acc ry = group_reduce8(fy, lane);
      const Acc rz = group_reduce8(fz, lane);
      const int own = lane & 7;
      if (own < cnt) {
        const int js = q_inf[wib][g][(head + own) & (kQ - 1)].x;
        if (PER_PAIR) {
          add_fixed(a.force + js, (long long)rx);
          add_fixed(a.force + stride + js, (long long)ry);
          add_fixed(a.force + 2 * stride + js, (long long)rz);
        } else {
          add_fixed(a.force + js, to_fixed_force((float)rx));
          add_fixed(a.force + stride + js, to_fixed_force((float)ry));
          add_fixed(a.force + 2 * stride + js, to_fixed_force((float)rz));
        }
      }
      xmask &= ~ring_mask(head, cnt > 0 ? cnt : 0);
      h0 += min(8, t0 - h0);
      h1 += min(8, t1 - h1);
      h2 += min(8, t2 - h2);
      h3 += min(8, t3 - h3);
      __syncwarp();
    };

    // one call site for the batch and one for the enqueue (code size: the
    // batch is an unrolled 8-pair loop): full batches while every group has
    // 8 waiting; before a tile, at most 32 waiting per group so that the tile
    // fits the rings; after the last tile, until the rings are empty
    int t = wk.y;
    for (;;) {
      const int fmin = min(min(t0 - h0, t1 - h1), min(t2 - h2, t3 - h3));
      const int fmax = max(max(t0 - h0, t1 - h1), max(t2 - h2, t3 - h3));
      if (fmin >= 8 || fmax > kQ - 32 || (t >= wk.z && fmax > 0)) {
        batch();
        continue;
      }
      if (t >= wk.z) break;
      const int2 tl = a.tiles[t];
      const int code = tile_image(tl.y);
      const float4 oj = a.origin[tl.x];
      const int ic = code / 9, ib = (code - 9 * ic) / 3, ia = code - 9 * ic - 3 * ib;
      const float kx = (float)(ia - 1), ky = (float)(ib - 1), kz = (float)(ic - 1);
      const float sx = fmaf(kx, st.Lx, oj.x - oi.x) + kx * st.Lx_lo;
      const float sy = fmaf(ky, st.Ly, oj.y - oi.y) + ky * st.Ly_lo;
      const float sz = fmaf(kz, st.Lz, oj.z - oi.z) + kz * st.Lz_lo;
      const int jslot = tl.x * kTile + lane;
      float4 xj = a.xyzq_s[jslot];
      xj.x += sx;
      xj.y += sy;
      xj.z += sz;
      const bool jvalid = a.perm[jslot] >= 0;
      const int tj = a.type_s[jslot];
      const unsigned excl = tile_excl_word(a, tl, code, wk.x, lane);
      const bool any_excl = __any_sync(0xffffffffu, ivalid && excl != 0u);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float *bb = sh_box[wib][h];
        const float bx = fmaxf(0.f, fmaxf(bb[0] - xj.x, xj.x - bb[3]));
        const float by = fmaxf(0.f, fmaxf(bb[1] - xj.y, xj.y - bb[4]));
        const float bz = fmaxf(0.f, fmaxf(bb[2] - xj.z, xj.z - bb[5]));
        const bool near = jvalid && bx * bx + by * by + bz * bz < st.roff2;
        const unsigned m = __ballot_sync(0xffffffffu, near);
        const int tail = h == 0 ? t0 : h == 1 ? t1 : h == 2 ? t2 : t3;
        if (near) {
          const int pos = (tail + __popc(m & lt_mask)) & (kQ - 1);
          q_pos[wib][h][pos] = xj;
          q_inf[wib][h][pos] = make_int2(jslot, tj);
        }
        if (any_excl && g == h && ivalid && excl != 0u) {
          unsigned mm = m & excl;   // excluded among the new entries, in order
          while (mm) {
            const int k = __ffs(mm) - 1;
            mm &= mm - 1u;
            xmask |= 1ull << ((tail + __popc(m & ((1u << k) - 1u))) & (kQ - 1));
          }
        }
        const int n = __popc(m);
        if (h == 0) t0 += n;
        else if (h == 1) t1 += n;
        else if (h == 2) t2 += n;
        else t3 += n;
      }
      __syncwarp();
      ++t;
    }

    if (VIRIAL) {
#pragma unroll
      for (int k = 0; k < 6; ++k) dv[k] += (double)vw[k];
    }
    if (MULTI && ENERGY) {
      long long *es = a.energy + (size_t)wk.w * a.energy_stride;
      warp_flush(e_elec, es + kEElec, lane);
      warp_flush(e_vdw, es + kEVdw, lane);
      e_elec = 0.0;
      e_vdw = 0.0;
      if (VIRIAL) {
        constexpr int kSlotM[6][2] = {{0, 0}, {1, 3}, {2, 6}, {4, 4}, {5, 7}, {8, 8}};
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          long long iw = __double2ll_rn(dv[k] * kEnergyScale);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) iw += __shfl_xor_sync(0xffffffffu, iw, o);
          if (lane == 0 && iw) {
            add_fixed(es + kNumEnergyTerms + kSlotM[k][0], iw);
            if (kSlotM[k][1] != kSlotM[k][0]) add_fixed(es + kNumEnergyTerms + kSlotM[k][1], iw);
          }
          dv[k] = 0.0;
        }
      }
    }
    if (ENERGY && !MULTI) {
      ie_el += __double2ll_rn(e_elec * kEnergyScale);
      ie_vdw += __double2ll_rn(e_vdw * kEnergyScale);
      e_elec = 0.0;
      e_vdw = 0.0;
      if (VIRIAL) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          ivir[k] += __double2ll_rn(dv[k] * kEnergyScale);
          dv[k] = 0.0;
        }
      }
    }
    if (ivalid) {
      if (PER_PAIR) {
        add_fixed(a.force + islot, (long long)fix);
        add_fixed(a.force + stride + islot, (long long)fiy);
        add_fixed(a.force + 2 * stride + islot, (long long)fiz);
      } else {
        add_fixed(a.force + islot, to_fixed_force((float)fix));
        add_fixed(a.force + stride + islot, to_fixed_force((float)fiy));
        add_fixed(a.force + 2 * stride + islot, to_fixed_force((float)fiz));
      }
    }
  }
  retire_warp(a.sched, lane);
  if (ENERGY && !MULTI) {
    long long ie = ie_el, iv = ie_vdw;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ie += __shfl_xor_sync(0xffffffffu, ie, o);
      iv += __shfl_xor_sync(0xffffffffu, iv, o);
    }
    if (lane == 0) {
      add_fixed(a.energy + kEElec, ie);
      add_fixed(a.energy + kEVdw, iv);
    }
  }
  if (VIRIAL && !MULTI) {
    constexpr int kSlot[6][2] = {{0, 0}, {1, 3}, {2, 6}, {4, 4}, {5, 7}, {8, 8}};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      long long iw = ivir[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) iw += __shfl_xor_sync(0xffffffffu, iw, o);
      if (lane == 0) {
        add_fixed(a.virial + kSlot[k][0], iw);
        if (kSlot[k][1] != kSlot[k][0]) add_fixed(a.virial + kSlot[k][1], iw);
      }
    }
  }
}

// persistent grid (resident blocks) or, with a bound on the items per warp,
// enough blocks for every work item the list can hold
int launch_grid(int resident, const NbArgs &a) {
  if (a.items_per_warp <= 0) return resident;
  const long long per_block = (long long)kWarps * a.items_per_warp;
  const long long need = ((long long)a.work_cap + per_block - 1) / per_block;
  return (int)std::max<long long>(resident, std::min<long long>(need, 1ll << 30));
}

template <bool E, bool P, bool V, bool M>
void launch_q(const NbArgs &a, cudaStream_t s) {
  static int grid = 0;
  size_t sm = M ? (size_t)kWarps * kMaxMultiTypes * kMaxMultiTypes * sizeof(float2)
                : (size_t)a.ntype * a.ntype * sizeof(float2);
  if (!grid) {
    int dev, nsm, per = 0;
    APO_CUDA(cudaGetDevice(&dev));
    APO_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    APO_CUDA(cudaFuncSetAttribute(nbq_kernel<E, P, V, M>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
    APO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, nbq_kernel<E, P, V, M>, kThreads,
                                                           64 * 1024 > sm ? sm : 64 * 1024));
    grid = nsm * (per > 0 ? per : 1);
  }
  nbq_kernel<E, P, V, M><<<launch_grid(grid, a), kThreads, sm, s>>>(a);
  APO_LAUNCH_CHECK();
}

template <bool M>
void dispatch_q(const NbArgs &a, bool energy, bool per_pair, bool virial, cudaStream_t s) {
  if (virial) {
    if (per_pair) launch_q<true, true, true, M>(a, s);
    else launch_q<true, false, true, M>(a, s);
  } else if (energy) {
    if (per_pair) launch_q<true, true, false, M>(a, s);
    else launch_q<true, false, false, M>(a, s);
  } else {
    if (per_pair) launch_q<false, true, false, M>(a, s);
    else launch_q<false, false, false, M>(a, s);
  }
}

// Lists of up to this many slots leave room on every SM: the persistent grid
// takes three blocks an SM where four fit, so that the blocks of the
// reciprocal-space kernels, which cannot fill the GPU on their own at these
// sizes, run beside it instead of after it (40 steps of 24,000 atoms 5.60 ->
// 5.05 ms, of 42,000 6.37 -> 5.95, 20 steps of 53,000 5.36 -> 5.12, of 80,000
// 7.47 -> 7.50, 40 of 107,000 15.35 -> 15.65; batches of 3 systems of 3,000
// atoms 1.35 -> 1.28 ms, of 12 3.18 -> 3.13, of 8 at order 6 3.47 -> 3.27).
// The precise form's kernel is longer and pays only at the smallest sizes (20
// Langevin steps at order 4 of 3,000 atoms 1.44 -> 1.30 ms, of 6,000 1.52 ->
// 1.43, of 9,000 1.69 -> 1.70, of 12,000 1.93 -> 1.99, of 24,000 2.98 -> 3.17;
// a batch of 12 systems of 3,000 4.18 -> 4.44).  Only for the forces
// alone: with energies (8.70 -> 9.08 ms) and with the virial (40 piston steps of
// 24,000 atoms 7.86 -> 8.11, of 53,000 9.28 -> 9.26) the kernel is so much
// longer than what runs beside it that it loses.
constexpr int kSharedSmSlots = 65536, kSharedSmSlotsPrecise = 10240;

template <bool E, bool P, bool V = false, bool M = false>
void launch_t(const NbArgs &a, cudaStream_t s) {
  void (*kernel)(NbArgs);
  if constexpr ((E || V) && !P) kernel = nb_energy_kernel<E, P, V, M>;
  else kernel = nb_kernel<E, P, V, M>;
  size_t sm = M ? (size_t)kWarps * kMaxMultiTypes * kMaxMultiTypes * sizeof(float2)
                : (size_t)a.ntype * a.ntype * sizeof(float2);
  const ResidentGrid &grid = resident_grid([&] {
    int dev, nsm, per = 0;
    APO_CUDA(cudaGetDevice(&dev));
    APO_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    APO_CUDA(cudaFuncSetAttribute(kernel,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
    APO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kThreads,
                                                           64 * 1024 > sm ? sm : 64 * 1024));
    ResidentGrid g;
    g.full = nsm * (per > 0 ? per : 1);
    g.shared = !E && !V && per > 3 ? nsm * 3 : g.full;
    return g;
  });
  const int resident = a.stride <= (P ? kSharedSmSlotsPrecise : kSharedSmSlots) ? grid.shared : grid.full;
  kernel<<<launch_grid(resident, a), kThreads, sm, s>>>(a);
  APO_LAUNCH_CHECK();
}

}  // namespace

void launch_nonbonded(const NbArgs &a, bool energy, bool per_pair, cudaStream_t s, bool virial) {
  if (!a.sched) throw std::invalid_argument("nonbonded: no schedule counters");
  if (a.ntype * a.ntype * sizeof(float2) > 64 * 1024)
    throw std::invalid_argument("nonbonded: too many LJ types for the shared table");
  if (virial && !a.virial) throw std::invalid_argument("nonbonded: virial requested without a buffer");
  if (a.variant == kNbGroupedQueues) return dispatch_q<false>(a, energy, per_pair, virial, s);
  if (a.variant == kNbOctetLists) return launch_nonbonded_octets(a, energy, per_pair, virial, false, s);
  if (virial) {
    if (per_pair) launch_t<true, true, true>(a, s);
    else if (energy) launch_t<true, false, true>(a, s);
    else launch_t<false, false, true>(a, s);
    return;
  }
  if (per_pair) {
    if (energy) launch_t<true, true>(a, s);
    else launch_t<false, true>(a, s);
  } else {
    if (energy) launch_t<true, false>(a, s);
    else launch_t<false, false>(a, s);
  }
}

void launch_nonbonded_multi(const NbArgs &a, bool energy, bool per_pair, cudaStream_t s,
                            bool virial) {
  if (!a.sched) throw std::invalid_argument("nonbonded: no schedule counters");
  if (a.energy_stride <= 0 && (energy || virial))
    throw std::invalid_argument("nonbonded: multi-system energies need an energy stride");
  if (a.variant == kNbGroupedQueues) return dispatch_q<true>(a, energy, per_pair, virial, s);
  if (a.variant == kNbOctetLists) return launch_nonbonded_octets(a, energy, per_pair, virial, true, s);
  if (virial) {
    if (per_pair) launch_t<true, true, true, true>(a, s);
    else launch_t<true, false, true, true>(a, s);
  } else if (energy) {
    if (per_pair) launch_t<true, true, false, true>(a, s);
    else launch_t<true, false, false, true>(a, s);
  } else {
    if (per_pair) launch_t<false, true, false, true>(a, s);
    else launch_t<false, false, false, true>(a, s);
  }
}

}  // namespace apo
