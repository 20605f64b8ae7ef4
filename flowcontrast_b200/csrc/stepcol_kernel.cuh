// FSLBM time step, FP64 column kernel for sm_100a (d1 = 2, the reference's order 2<->4 corrector).
//
// Planes marched one at a time, two FP64 rows of one column per thread:
//  - a 32 x 16 tile per CTA (32 x 8 for the smallest pipes), two tile rows per warp: a warp's 64-bit shared loads
//    read 32 consecutive doubles (two wavefronts, no bank conflict);
//  - p is staged with a one-cell halo and u,v,w with the corrector's 2*d1 halo, as two TMA boxes
//    per plane (no multicast) into a window of 7 planes (201 KB);
//  - no block-wide barrier in the march and no producer thread: per-slot "full" mbarriers count
//    TMA completion, planes leave the window in pairs and the last warp to release a pair
//    refills both slots (the bounded waits and failure path of step2_march);
//  - the predictor is step2_march's (x sums per row, carried times 216), the streamwise corrector
//    taps behind the output plane come from a register history of the thread's own column, the
//    taps ahead from the window, the output plane's centre from the predictor one plane earlier;
//  - grid = tiles x streamwise chunks in chunk-major order, odd chunks marching downwards, and a
//    cell's predictor adds its two neighbour planes' shares before its own plane's, so results do
//    not depend on the chunking.
// The shared-memory path (60 % of its wavefront slots) and the FP64 pipe (54 %) bound it. Two rows per
// thread share the predictor's rows: 54 shared loads per cell against 70 with one row and 512
// threads, 166 against 177 us a step at 512 x 128 x 128 in 25-step passes (164 over 2000 steps); the predictor's arithmetic per cell stays
// the same and 8 warps instead of 16 are enough (64 x 32 x 32: 6.8 us either way). Measured and not
// used: the plane two ahead carried into the predictor (51 loads, 1 % slower), the predictor
// instantiated apart for the seam planes (2 % slower).
// FP64 solves with other corrector orders, strides or masks per plane keep step_kernel.cuh.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>
#include "common.h"
#include "ptx.cuh"
#include "step_kernel.cuh"
#include "step2_kernel.cuh"

namespace fslbm {

template <int D1, int TY> struct ColTile {
  static constexpr int ES = int(sizeof(double));
  static constexpr int TX = 32;
  static constexpr int N = 2;                           // rows per thread
  static constexpr int THREADS = TX * TY / N;
  static constexpr int WARPS = THREADS / 32;
  static constexpr int R = 2 * D1;                      // farthest corrector tap
  static constexpr int HX = (R * ES + 15) / 16 * 16 / ES;   // x halo, TMA-aligned (16 bytes)
  static constexpr int HY = R;
  static constexpr int SW = TX + 2 * HX;                // row length of both boxes
  static constexpr int PH = TY + 2;                     // p rows (halo 1)
  static constexpr int UH = TY + 2 * HY;                // u,v,w rows
  static constexpr int PPLANE = (SW * PH * ES + 127) / 128 * 128 / ES;
  static constexpr int UPLANE = SW * UH;
  static constexpr int SLOT = PPLANE + 3 * UPLANE;
  static constexpr int S = 7;                           // window slots
  static constexpr int AHEAD = S - R - 1;
  static_assert(AHEAD >= 1, "window too small for the corrector reach");
  static constexpr uint32_t TX_BYTES = uint32_t((SW * PH + 3 * UPLANE) * ES);
  static constexpr size_t BAR_OFFSET = size_t(S) * SLOT * ES;
  static constexpr size_t SMEM_BYTES = BAR_OFFSET + S * sizeof(uint64_t) + S * sizeof(uint32_t);
  static_assert((PPLANE * ES) % 128 == 0 && (UPLANE * ES) % 16 == 0 && (SLOT * ES) % 128 == 0,
                "TMA destinations must stay aligned");
  static_assert((HX * ES) % 16 == 0, "TMA box x start must be 16-byte aligned");
  static_assert(SMEM_BYTES <= 227 * 1024, "window exceeds a CTA's shared memory");
};

// Marches one (tile, chunk) work item: the step of every cell of the tile's columns in the
// chunk's planes. Returns false when a bounded wait gave up (error flag set).
template <int D1, int TY>
__device__ __forceinline__ bool col_march(const CUtensorMap* tmap_p, const CUtensorMap* tmap_uvw,
                                          const Step2Geom& g, const StepConst<double>& k, int tile,
                                          int chunk, unsigned char* smem) {
  using Tl = ColTile<D1, TY>;
  static_assert(D1 == 2, "the march prologue below is written for d1 = 2 (R = 4)");
  constexpr int N = Tl::N, R = Tl::R, HX = Tl::HX, HY = Tl::HY, SW = Tl::SW, S = Tl::S;
  constexpr int PPL = Tl::PPLANE, UPL = Tl::UPLANE, SLOT = Tl::SLOT;

  auto slot_of = [](int m) { return int(unsigned(m) % unsigned(S)); };
  auto phase_of = [](int m) { return uint32_t((unsigned(m) / unsigned(S)) & 1u); };
  double* ring = reinterpret_cast<double*>(smem);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Tl::BAR_OFFSET);
  unsigned* released = reinterpret_cast<unsigned*>(full + S);

  const int tid = threadIdx.x, lane = tid & 31;
  const int tx = lane, ty = (tid >> 5) * N;            // N tile rows per warp

  // ---- work: one (tile, chunk); odd chunks march towards -z
  const int zb = int((long long)g.L * chunk / g.nchunks);
  const int ze = int((long long)g.L * (chunk + 1) / g.nchunks);
  const int dir = (chunk & 1) ? -1 : 1;
  const int nout = ze - zb, niter = nout + 2 * R;
  const int start = dir > 0 ? zb - R : ze - 1 + R;      // real plane of march index 0
  const int2 org = g.tiles[tile];
  const int x = org.x + tx, y0 = org.y + ty;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      released[s] = 0u;
    }
    mbar_init_fence();
  }

  auto issue = [&](int m) {            // load march plane m into its slot
    const int slot = slot_of(m);
    int zz = (start + dir * m) % g.L;
    if (zz < 0) zz += g.L;
    double* dst = ring + slot * SLOT;
    mbar_arrive_expect_tx(&full[slot], Tl::TX_BYTES);
    tma_load_4d(dst, tmap_p, &full[slot], org.x - HX, org.y - 1, zz, 0);
    tma_load_4d(dst + PPL, tmap_uvw, &full[slot], org.x - HX, org.y - HY, zz, 1);
  };
  if (tid == 0) {                      // the whole ring up front
    prefetch_tensormap(tmap_p);
    prefetch_tensormap(tmap_uvw);
    grid_dependency_wait();
    for (int m = 0; m < S && m < niter; ++m) issue(m);
  }
  // wall sums of the predictor (times 216, see the march) and fluid flag; nothing outside the box
  double ws0[N], wsx[N], wsy[N], fl[N];
  bool inside[N], some = false;
#pragma unroll
  for (int r = 0; r < N; ++r) {
    inside[r] = x < g.lxp && y0 + r < g.ly;
    ws0[r] = wsx[r] = wsy[r] = fl[r] = 0;
    if (inside[r]) {
      const ColCoef<double> c = reinterpret_cast<const ColCoef<double>*>(g.colcoef)[size_t(y0 + r) * g.lxp + x];
      ws0[r] = 216.0 * c.ws0; wsx[r] = 216.0 * c.wsx; wsy[r] = 216.0 * c.wsy; fl[r] = c.fluid;
    }
    some |= fl[r] != 0.0;
  }
  const bool warp_on = __any_sync(0xffffffffu, some);

  grid_dependency_wait();
  __syncthreads();
  // wait for march plane m, one verdict per warp; false after flagging a failure and letting this
  // CTA's loads land (bounded)
  auto arrive_wait = [&](int m) -> bool {
    if (mbar_wait_warp(&full[slot_of(m)], phase_of(m), kWaitLimitNs)) return true;
    if (lane == 0) {
      atomicOr(g.err, 1u);
      for (int q = m + 1; q < niter && q < m + 1 + S; ++q)
        mbar_wait_bounded(&full[slot_of(q)], phase_of(q), kWaitLimitNs / 8);
    }
    __syncwarp();
    return false;
  };
  // planes p - 1 and p (p = m - R odd) leave the window; see step2_march for the ordering
  auto release_produce = [&](int m) {
    __syncwarp();
    if (m >= R && ((m - R) & 1) && lane == 0) {
      const int slot = slot_of(m - R);
      const unsigned seen = atom_add_acq_rel_cta(&released[slot], 1u) + 1u;
      const int mn = m - R + S - 1;
      if (seen % unsigned(Tl::WARPS) == 0u && mn < niter) {
        fence_proxy_async_smem();
        issue(mn);
        if (mn + 1 < niter) issue(mn + 1);
      }
    }
  };

  if (!warp_on) {   // all-wall warps keep the pipeline protocol only
    for (int m = 0; m < niter; ++m) {
      if (!arrive_wait(m)) return false;
      release_produce(m);
    }
    return true;
  }

  const double gauge = g.gauge ? __ldcg(g.gauge) : 0.0;
  const size_t FS = size_t(g.lxp) * g.ly * g.L;
  double* outp = reinterpret_cast<double*>(g.out) + (size_t(start + dir * R) * g.ly + y0) * g.lxp + x;
  const long long ostep = (long long)dir * g.ly * g.lxp;     // output pointer step per plane
  const int po = (ty + 1) * SW + HX + tx;                     // p box
  const int uo = PPL + (ty + HY) * SW + HX + tx;              // u box (v, w at +UPL, +2 UPL)
  const double dir3 = 3.0 * double(dir);
  // folded update: u_new = K1 t1 + K2 t2 + K0 u + tb (u* + F)
  const double kam = __dmul_rn(__dmul_rn(k.tb, k.dtddy), k.m);
  const double kK0 = __fma_rn(kam, k.c0, k.cc), kK1 = __dmul_rn(kam, k.c1), kK2 = __dmul_rn(kam, k.c2);
  // the predictor's moments come times 216; the z-moment carries the march direction's sign
  const double ktb = __ddiv_rn(k.tb, 216.0), ktz = double(dir) * ktb;

  // own column of the four planes before the output plane: [field][plane parity][older, newer][row]
  double h[3][2][2][N];
  // per row: d2 / d1 = the shares that the two planes before the next predictor plane give to their
  // march-next planes (d2 to the output being completed), s1 = the self-plane moments of the newer
  double d2[N][3], d1[N][3], s1[N][3], comp[N][4];
#pragma unroll
  for (int r = 0; r < N; ++r)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      comp[r][j] = 0.0;
      if (j < 3) d2[r][j] = d1[r][j] = s1[r][j] = h[j][0][0][r] = h[j][0][1][r] = h[j][1][0][r] = h[j][1][1][r] = 0.0;
    }

  double cen[N][4], nxt[N][4];         // p, u, v, w of the output plane and of the one after it

  // predictor contribution of march plane ma (factorisation and scaling: step2_march)
  auto predictor = [&](int ma) {
    const double* ss = ring + slot_of(ma) * SLOT;
    const int sp = start + dir * ma;
    RowSide<double> above, here;         // rows r - 1 and r as their lower neighbours see them
    RowSums<double> mid;
#pragma unroll
    for (int j = -1; j <= N; ++j) {
      double p3[3], u3[3], v3[3], w3[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double* rq = ss + uo + j * SW + c - 1;
        p3[c] = ss[po + j * SW + c - 1];
        u3[c] = rq[0];
        v3[c] = rq[UPL];
        w3[c] = rq[2 * UPL];
      }
      if (j >= 0 && j < N) {
        cen[j][0] = nxt[j][0]; cen[j][1] = nxt[j][1]; cen[j][2] = nxt[j][2]; cen[j][3] = nxt[j][3];
        nxt[j][0] = p3[1]; nxt[j][1] = u3[1]; nxt[j][2] = v3[1]; nxt[j][3] = w3[1];
      }
      const RowSums<double> row = row_sums(p3, u3, v3, w3);
      if (j >= 1) {
        const int r = j - 1;
        const RowSide<double> below = row_side<1>(row);
        double A[3], X[3], Y[3];
        A[0] = fma2(4.0, mid.R0, add2(above.R0, below.R0));
        A[1] = fma2(4.0, mid.Rz, add2(above.Rz, below.Rz));
        A[2] = fma2(4.0, mid.Rw, add2(above.Rw, below.Rw));
        X[0] = fma2(4.0, mid.D0, add2(above.D0, below.D0));
        X[1] = fma2(4.0, mid.Dz, add2(above.Dz, below.Dz));
        X[2] = fma2(4.0, mid.Dw, add2(above.Dw, below.Dw));
        Y[0] = sub2(below.R0, above.R0);
        Y[1] = sub2(below.Rz, above.Rz);
        Y[2] = sub2(below.Rw, above.Rw);
        if (sp < 0 || sp >= g.L) {       // seam plane (CTA-uniform): the jump times the non-wall weight sums (x36)
          const double off = sp < 0 ? k.pin : -k.pin;
          A[0] = fma2(off, fma2(-1.0 / 6.0, ws0[r], 36.0), A[0]);
          X[0] = fma2(off, wsx[r] * (-1.0 / 6.0), X[0]);
          Y[0] = fma2(off, wsy[r] * (-1.0 / 6.0), Y[0]);
        }
        double s[3], d[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double(&m)[3] = i == 0 ? A : (i == 1 ? X : Y);
          const double e = fma2(m[2], 4.5, m[0]);
          s[i] = fma2(m[1], dir3, e);
          d[i] = fma2(-m[1], dir3, e);
        }
        // a cell adds its two neighbour planes' shares first, then its own plane's
#pragma unroll
        for (int i = 0; i < 3; ++i) comp[r][i] = fma2(s1[r][i], 4.0, add2(d2[r][i], s[i]));
        comp[r][3] = sub2(s[0], d2[r][0]);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          d2[r][i] = d1[r][i];
          d1[r][i] = d[i];
          s1[r][i] = i == 0 ? A[0] : (i == 1 ? X[0] : Y[0]);
        }
      }
      if (j >= 0) above = here;
      mid = row;
      here = row_side<-1>(row);
    }
  };

  // corrector and update of output march plane jo of parity PAR
  auto output = [&](int jo, auto par_c) {
    constexpr int PAR = decltype(par_c)::value;
    const double* so = ring + slot_of(jo) * SLOT;
    const double* sa1 = ring + slot_of(jo + D1) * SLOT + uo;   // march planes ahead
    const double* sa2 = ring + slot_of(jo + 2 * D1) * SLOT + uo;
    double pc[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
      pc[r] = cen[r][0];
      if (inside[r]) outp[r * g.lxp] = fma2(fma2(pc[r], ws0[r], comp[r][0]), 1.0 / 216.0, -gauge) * fl[r];   // walls get zero
    }
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const double* b = so + uo + f * UPL;
#pragma unroll
      for (int r = 0; r < N; ++r) {
        const double* q = b + r * SW;
        const double c = cen[r][1 + f];
        const double za1 = sa1[f * UPL + r * SW], za2 = sa2[f * UPL + r * SW];
        const double t1 = add2(add2(add2(q[-D1], q[D1]), add2(q[-D1 * SW], q[D1 * SW])), add2(h[f][PAR][1][r], za1));
        const double t2 = add2(add2(add2(q[-2 * D1], q[2 * D1]), add2(q[-2 * D1 * SW], q[2 * D1 * SW])),
                               add2(h[f][PAR][0][r], za2));
        const double mom = f == 2 ? comp[r][3] : fma2(pc[r], f == 0 ? wsx[r] : wsy[r], comp[r][1 + f]);
        // the small terms first: only the last operation rounds at the size of u
        double un = fma2(f == 2 ? ktz : ktb, mom, __dmul_rn(k.tb, f == 0 ? k.fx : (f == 1 ? k.fy : k.fz)));
        un = fma2(kK1, t1, fma2(kK2, t2, un));
        un = fma2(kK0, c, un);
        h[f][PAR][0][r] = h[f][PAR][1][r];
        h[f][PAR][1][r] = c;
        if (inside[r]) outp[(1 + f) * FS + r * g.lxp] = un * fl[r];
      }
    }
    outp += ostep;
  };

  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, 1>;
  // ---- prologue (R = 4): planes 0..3 enter the history when plane 4..7 arrive; planes 6..7 also
  // start the predictor sums of the first output
#pragma unroll 1
  for (int m = 0; m < 2 * R; ++m) {
    if (!arrive_wait(m)) return false;
    if (m >= 2 * R - 2) predictor(m - R + 1);
    if (m >= R) {
      const double* so = ring + slot_of(m - R) * SLOT + uo;
#pragma unroll
      for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int r = 0; r < N; ++r) {
          h[f][0][0][r] = h[f][0][1][r];
          h[f][0][1][r] = h[f][1][0][r];
          h[f][1][0][r] = h[f][1][1][r];
          h[f][1][1][r] = so[f * UPL + r * SW];
        }
    }
    release_produce(m);
  }
  // in march order the planes are now [0][0], [0][1], [1][0], [1][1]: swap the middle two
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const double t = h[f][0][1][r];
      h[f][0][1][r] = h[f][1][0][r];
      h[f][1][0][r] = t;
    }
  // ---- steady state, two planes per pass (the history's parity)
#pragma unroll 1
  for (int m = 2 * R; m < niter; m += 2) {
    if (!arrive_wait(m)) return false;
    predictor(m - R + 1);
    output(m - R, I0{});
    release_produce(m);
    if (m + 1 >= niter) break;
    if (!arrive_wait(m + 1)) return false;
    predictor(m - R + 2);
    output(m - R + 1, I1{});
    release_produce(m + 1);
  }
  return true;
}

// One pipe, one step: CTA b marches (tile b % ntiles, chunk b / ntiles).
template <int D1, int TY>
__global__ void __launch_bounds__(ColTile<D1, TY>::THREADS, 1)
    fslbm_col_kernel(const __grid_constant__ CUtensorMap tmap_p,
                     const __grid_constant__ CUtensorMap tmap_uvw, const Step2Geom g,
                     const StepConst<double> k) {
  extern __shared__ __align__(128) unsigned char smem[];
  col_march<D1, TY>(&tmap_p, &tmap_uvw, g, k, blockIdx.x % g.ntiles, blockIdx.x / g.ntiles, smem);
  if (threadIdx.x == 0 && blockIdx.x == 0 && g.step_counter) *g.step_counter += 1;
  grid_launch_dependents();
}

}  // namespace fslbm
