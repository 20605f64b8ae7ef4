// FSLBM time step, FP32 arithmetic, pairs of planes, for sm_100a (corrective stride 2, FP32 or FP16
// storage; corrector of 2 or 3 taps; one cross-section or one per plane).
//
// Same step as step_kernel.cuh (predictor factored by neighbour plane, coarse corrector,
// periodic +-pin seam, walls, gauge, body force), organised for throughput:
//  - a thread owns N rows of one column and marches along the pipe two planes at a time; the two
//    planes are the halves of packed FP32x2 operations (add2 / mul2 / fma2). Packing along the
//    march needs no register moves: the corrector's streamwise taps are an even number of planes
//    away, so its pairs are the window's pairs, and x and y neighbours of a pair are pairs too;
//  - the predictor's x sums of a row (RowSums) are formed once per row and serve the rows above
//    and below it within the thread;
//  - a 32 x TY tile per CTA; p is staged with a one-cell halo, u,v,w with the corrector's 2*d1
//    halo, by TMA into a window of SU pairs of planes (u,v,w) and SU - 2 pairs (p);
//  - the own columns of the last four pairs (centre and the four streamwise taps behind and at
//    the predictor's pair) live in tensor memory, written once by the predictor and read back
//    with tcgen05.ld: 24 N words per thread that would otherwise be registers (spills) or
//    shared-memory loads;
//  - results leave through a shared staging block per warp and one TMA store per plane, which
//    needs no per-store address or bounds arithmetic;
//  - no block-wide barrier in the march and no producer thread: per-pair "full" mbarriers count
//    TMA completion, each warp releases a pair after its last read of it, and the last warp to
//    release a pair refills its slot, so warps drift within the window and none waits for a
//    free slot;
//  - grid = tiles x streamwise chunks in chunk-major order, so concurrent CTAs work at nearby
//    planes and halos hit L2; odd chunks march downwards, so the planes two neighbouring
//    chunks share are read by both at the same time;
//  - warps whose cells are all wall keep the pipeline protocol but skip the arithmetic.
//
// What bounds it. FP32: with four rows per thread 8 warps of 209 registers issue on 48 % of the
// cycles (fixed-latency dependencies), the FMA pipes are busy 47 %, DRAM 29 %; FP16 storage:
// instruction issue, 67 % (conversions, rounding); small pipes: the march's K fill iterations. The
// form it replaces, two columns per thread with scalar FP32 and a register history, was bound by
// shared-memory wavefronts (17.3 M a launch, now 11.6 M) and instructions (59.9 M, now 41.0 M).
// Per step, that form against this one, one B200:
//   512 x 128 x 128   FP32 97.2 -> 83.9 us, FP16 storage 167 -> 125 us
//   300 x 120 x 120   FP32 61.7 -> 46.4 us
//   151 x 61 x 61     FP32 20.9 -> 13.0 us
// and against step_kernel.cuh, 10 steps: order 6 on 256 x 96 x 96 670 -> 367 us, a mask per plane on
// 192 x 96 x 96 488 -> 300 us.
// At 128 registers some forms spill (bytes stored a thread): 32 x 32 with masks per plane 36, FP16
// storage on 32 x 32 and 32 x 16 tiles 8, batched FP32 40, batched FP16 16 (32 x 32) and 24 (32 x 16).
#pragma once
#include <cstdint>
#include <type_traits>
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include "common.h"
#include "ptx.cuh"
#include "step_kernel.cuh"

namespace fslbm {

// TE is the storage type of the state (float, or __half for FP16 storage); arithmetic is FP32
// either way. Halo widths and paddings keep every TMA box start and destination on 16 bytes.
// K is the number of corrector taps per direction (2: the reference's order 2<->4 blend, 3: its
// order 4<->6 blend), SF the fields staged for a store at a time (4, or 2).
template <int TY, class TE = float, int K = 2, int ROWS = 2, int SF = 4> struct Step2Tile {
  static constexpr int D1 = 2;                          // corrective stride
  static constexpr int N = ROWS;                        // rows per thread
  static constexpr int STAGED = SF;                     // fields staged at a time
  static constexpr int ES = int(sizeof(TE));
  static constexpr int A16 = 16 / ES;                   // elements per 16 bytes
  static constexpr int TX = 32;
  static constexpr int WARPS = TY / N;                  // a warp owns 32 N cells (see the warp shapes)
  static constexpr int THREADS = 32 * WARPS;
  static constexpr int R = K * D1;                      // farthest corrector tap: K pairs of planes
  static constexpr int HX = (R + A16 - 1) / A16 * A16;  // x halo, TMA-aligned (16 bytes)
  static constexpr int HY = R;
  static constexpr int SW = TX + 2 * HX;                // row length of both boxes
  static constexpr int PH = TY + 2;                     // p rows (halo 1)
  static constexpr int UH = TY + 2 * HY;                // u,v,w rows
  static constexpr int PPL = (SW * PH * ES + 127) / 128 * 128 / ES;   // p plane, 128-byte aligned
  static constexpr int UPL = SW * UH;                                 // u, v or w plane
  static constexpr int VPL = (3 * UPL * ES + 127) / 128 * 128 / ES;   // u,v,w of one plane
  // Window, in pairs of planes. In use: the output pair and the K after it, of which the first is
  // the predictor's; one more is in flight. p is read by the predictor only.
  static constexpr int SU = K + 2, SP = 2;
  static constexpr uint32_t U_BYTES = uint32_t(3 * UPL * ES), P_BYTES = uint32_t(SW * PH * ES);
  static constexpr size_t P_OFFSET = size_t(SU) * 2 * VPL * ES;
  // staging of a warp's output pair: [plane][field][row][column] of the warp's cells
  static constexpr int STG = 2 * SF * N * 32;
  static constexpr size_t STG_OFFSET = P_OFFSET + size_t(SP) * 2 * PPL * ES;
  static constexpr size_t BAR_OFFSET = STG_OFFSET + size_t(WARPS) * STG * ES;   // a "full" mbarrier per slot
  static constexpr size_t REL_OFFSET = BAR_OFFSET + SU * sizeof(uint64_t);       // release counters, tensor memory base
  // FP16 storage: the tile's base of w (FP32) for columns org.x-1 .. org.x+TX and rows
  // org.y-1 .. org.y+TY
  static constexpr int BW = TX + 2, BH = TY + 2;
  static constexpr size_t BASE_OFFSET = (REL_OFFSET + (SU + 1) * sizeof(unsigned) + 15) / 16 * 16;
  static constexpr size_t BASE_BYTES = std::is_same<TE, __half>::value ? size_t(BW) * BH * sizeof(float) : 0;
  static constexpr size_t SMEM_BYTES = BASE_OFFSET + BASE_BYTES;
  // tensor memory: a ring of a warp's own columns of u, v, w of the predictor's pair and the K + 1
  // before it; warps w, w + 4, ... share the 32 lanes of subpartition w % 4
  static constexpr int TM_RING = K == 2 ? 4 : 8;
  static constexpr int TM_SLOT = 6 * N, TM_WARP = TM_RING * TM_SLOT;
  static constexpr int TM_NEED = TM_WARP * ((WARPS + 3) / 4);
  static constexpr int TM_COLS = TM_NEED <= 32 ? 32 : TM_NEED <= 64 ? 64 : TM_NEED <= 128 ? 128 : 256;
  // CTAs per SM (shared memory; 128 registers a thread at 16 warps per SM). FP32 32 x 16: 120 KB with
  // four fields staged, 112 KB with two, which leaves room for a second CTA.
  static constexpr int CTAS = K > 2 || TY == 32 ? 1 : TY == 16 ? (ES == 2 || SF == 2 ? 2 : 1) : 3;
  static_assert(TM_NEED <= TM_COLS && TM_COLS * CTAS <= 512, "tensor memory columns");
  static_assert((PPL * ES) % 128 == 0 && (VPL * ES) % 128 == 0 && (STG * ES) % 128 == 0,
                "TMA addresses must stay aligned");
  static_assert((HX * ES) % 16 == 0, "TMA box x start must be 16-byte aligned");
  static_assert(SMEM_BYTES <= 227 * 1024, "window exceeds a CTA's shared memory");
  static_assert(SF == 4 || SF == 2, "fields staged at a time");
  static_assert(TY % 8 == 0, "warp shapes within a 32-wide tile");
};

struct Step2Geom {
  int lxp, ly, L;
  int ntiles, nchunks;     // grid = ntiles * nchunks, chunk-major
  const int2* tiles;
  const uint8_t* mask;
  const void* colcoef;     // ColCoef<float>[lxp*ly]
  void* out;               // FP64 column kernel (the pair kernel stores through tensor maps)
  const double* gauge;
  unsigned* err;
  long long* step_counter;
  unsigned step_no;        // time step being computed (seed of the FP16 stochastic rounding)
  // FP16 storage: stored w is w - wb (per-column base, FP32); wgt is the base's share of a step
  // of the stored w. Null for other storage types.
  const float* wb;
  const float* wgt;
  bool early;              // tiles, colcoef and near are older than the previous kernel of the stream
  const uint32_t* near;    // masks per plane: packed wall sums per cell (pack_wall_sums), else null
};

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 f2(float2 a) { return a; }
__device__ __forceinline__ float lds1(const float* p) { return *p; }
__device__ __forceinline__ float lds1(const __half* p) { return __half2float(*p); }

// 32-bit integer hash (the "lowbias32" finaliser of C. Wellons' hash-prospector, public domain).
__device__ __forceinline__ uint32_t hash32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
  return x;
}

// FP32 -> FP16 with stochastic rounding: uniform noise below FP16's last kept bit is added to
// the magnitude, which is then truncated. The result is unbiased, so increments far below half
// an FP16 ulp (the body force and the slow relaxation of the step) survive in expectation
// instead of being rounded away. The kept bit is the 11th of the significand, 2^(e-10) for
// |x| in [2^e, 2^(e+1)), and fixed at 2^-24 below 2^-14 (FP16 subnormals, which the deviations
// of FP16 storage often reach): the noise is 13 random bits scaled to 2^(max(e,-14)-23), formed
// without a branch (measured +0.9 % on the FP16 step against branching on the subnormal range).
// In FP16's normal range the noise's lowest bit is x's FP32 resolution, so the sum is exact.
__device__ __forceinline__ __half sr_half(float x, uint32_t r) {
  const uint32_t ex = max(__float_as_uint(x) & 0x7f800000u, 0x38800000u);   // exponent of max(|x|, 2^-14)
  const float noise = float(r & 0x1fffu) * __uint_as_float(ex - (23u << 23));
  return __float2half_rz(x + copysignf(noise, x));
}

// Arithmetic on a pair of planes (.x the march-earlier plane, .y the later one): packed FP32x2
// instructions, each half rounded as the scalar operation.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }   // an operand modifier
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

template <class V> __device__ __forceinline__ V cst(float a);
template <> __device__ __forceinline__ float2 cst<float2>(float a) { return f2(a); }
template <> __device__ __forceinline__ double cst<double>(float a) { return double(a); }
__device__ __forceinline__ double add2(double a, double b) { return __dadd_rn(a, b); }   // FP64: one plane
__device__ __forceinline__ double neg2(double a) { return -a; }
__device__ __forceinline__ double sub2(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul2(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fma2(double a, double b, double c) { return __fma_rn(a, b, c); }

// x sums of one row at one column (V = float2: two planes; double: one plane, the FP64 kernel). With
// weights {4,1,1} over cx = 0, +1, -1 (R) or the difference +1 minus -1 (D), of the terms of the
// brackets as polynomials of cy:
//   0: q + 3 cx u + 4.5 cx^2 u^2        (P0 at cy = 0)
//   1: v (1 + 3 cx u)                   (P0 = 0 + 3 cy 1 + 4.5 cy^2 2)
//   2: v^2
//   z: w (1 + 3 cx u)                   (P1/3 = z + 3 cy m)
//   m: v w
//   w: w^2                              (P2/4.5)
template <class V> struct RowSums {
  V R0, D0, R1, D1, R2, D2, Rz, Dz, Rm, Dm, Rw, Dw;
};
template <class V> __device__ __forceinline__ V rsum(V l, V c, V r) { return fma2(cst<V>(4.0f), c, add2(l, r)); }

template <class V>
__device__ __forceinline__ RowSums<V> row_sums(const V (&p)[3], const V (&u)[3], const V (&v)[3], const V (&w)[3]) {
  V P[3], V1[3], V2[3], W[3], M[3], W2[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    V2[j] = mul2(v[j], v[j]);
    W2[j] = mul2(w[j], w[j]);
    M[j] = mul2(v[j], w[j]);
    const V s = add2(V2[j], W2[j]);
    if (j == 1) {
      P[j] = fma2(neg2(fma2(u[j], u[j], s)), cst<V>(1.5f), p[j]);
      V1[j] = v[j];
      W[j] = w[j];
    } else {
      const V cu = j == 2 ? u[j] : neg2(u[j]);               // cx u
      const V a = fma2(cu, cst<V>(3.0f), cst<V>(1.0f));
      // q + 3 cx u + 4.5 u^2 = p - 1.5 (v^2 + w^2) + cx u (3 cx u + 3)
      P[j] = fma2(cu, fma2(cu, cst<V>(3.0f), cst<V>(3.0f)), fma2(neg2(s), cst<V>(1.5f), p[j]));
      V1[j] = mul2(v[j], a);
      W[j] = mul2(w[j], a);
    }
  }
  RowSums<V> o;
  o.R0 = rsum(P[0], P[1], P[2]);   o.D0 = sub2(P[2], P[0]);
  o.R1 = rsum(V1[0], V1[1], V1[2]); o.D1 = sub2(V1[2], V1[0]);
  o.R2 = rsum(V2[0], V2[1], V2[2]); o.D2 = sub2(V2[2], V2[0]);
  o.Rz = rsum(W[0], W[1], W[2]);   o.Dz = sub2(W[2], W[0]);
  o.Rm = rsum(M[0], M[1], M[2]);   o.Dm = sub2(M[2], M[0]);
  o.Rw = rsum(W2[0], W2[1], W2[2]); o.Dw = sub2(W2[2], W2[0]);
  return o;
}

// A row's contribution to the output row one above (cy = -1) or below (cy = +1) it.
template <class V> struct RowSide {
  V R0, D0, Rz, Dz, Rw, Dw;
};
template <int CY, class V> __device__ __forceinline__ RowSide<V> row_side(const RowSums<V>& o) {
  auto cy = [](V a) { return CY > 0 ? a : neg2(a); };
  RowSide<V> s;
  s.R0 = fma2(cy(o.R1), cst<V>(3.0f), fma2(cst<V>(4.5f), o.R2, o.R0));
  s.D0 = fma2(cy(o.D1), cst<V>(3.0f), fma2(cst<V>(4.5f), o.D2, o.D0));
  s.Rz = fma2(cy(o.Rm), cst<V>(3.0f), o.Rz);
  s.Dz = fma2(cy(o.Dm), cst<V>(3.0f), o.Dz);
  s.Rw = o.Rw;
  s.Dw = o.Dw;
  return s;
}

// Tensor memory accesses of a warp: thread i reads and writes lane i of the warp's subpartition.
__device__ __forceinline__ void tm_store(uint32_t a, float2 v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void tm_load(float2 (&v)[2], uint32_t a) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y) : "r"(a) : "memory");
}
__device__ __forceinline__ void tm_wait_stores() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tm_load(float2 (&v)[4], uint32_t a) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[2].x), "=f"(v[2].y), "=f"(v[3].x),
                 "=f"(v[3].y)
               : "r"(a) : "memory");
}
// Completes the loads into v: their uses cannot move before the wait.
template <int M, int N> __device__ __forceinline__ void tm_wait_loads(float2 (&v)[M][N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < M; ++j)
#pragma unroll
    for (int r = 0; r < N; ++r) asm volatile("" : "+f"(v[j][r].x), "+f"(v[j][r].y));
}
// Allocation of a kernel's tensor memory by its first warp (whole warp); `slot` in shared memory
// receives the base address. Freed by the same warp before the kernel ends, on every path.
template <int COLS> __device__ __forceinline__ void tm_alloc(uint32_t* slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "n"(COLS)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int COLS> __device__ __forceinline__ void tm_free(uint32_t base) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(COLS) : "memory");
}

// Marches one (tile, chunk) work item of one pipe: the step of every cell of the tile's columns
// in the chunk's planes. `tmem` is the CTA's tensor memory, `reinit` re-arms the CTA's mbarriers
// when the CTA has marched an item before (persistent grids), `chained` waits for the stream's
// previous kernel before the state is read. Returns false when a bounded wait
// gave up (error flag set). The results are complete (visible to this thread) on return.
// The warp shape is a runtime argument: it only places each thread in the tile. 0: 32 columns x
// 2 rows; 1: 16 columns x 4 rows; 2: 8 columns x 8 rows (a thread's two rows are adjacent in all
// of them). The smaller shapes let warps over wall skip at a finer grain, which pays for small
// cross-sections. With the 160-byte FP32 row stride the shapes 0 and 1 read shared memory without
// bank conflicts (rows 2 apart are 16 banks apart), shape 2 two-way. The map changes no thread's
// arithmetic.
// tmap_out's box holds SF fields of the warp's cells.
template <int TY, class TE, int K = 2, bool MP = false, int ROWS = 2, int SF = 4>
__device__ __forceinline__ bool step2_march(const CUtensorMap* tmap_p, const CUtensorMap* tmap_uvw,
                                            const CUtensorMap* tmap_out, uint32_t tmem, const Step2Geom& g,
                                            const StepConst<float>& k, int tile, int chunk,
                                            unsigned char* smem, bool reinit, int shape, bool chained) {
  using Tl = Step2Tile<TY, TE, K, ROWS, SF>;
  constexpr int N = Tl::N, R = Tl::R, D1 = Tl::D1, HX = Tl::HX, HY = Tl::HY, SW = Tl::SW, SU = Tl::SU, SP = Tl::SP;
  constexpr int PPL = Tl::PPL, UPL = Tl::UPL, VPL = Tl::VPL;
  TE* uring = reinterpret_cast<TE*>(smem);
  TE* pring = reinterpret_cast<TE*>(smem + Tl::P_OFFSET);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Tl::BAR_OFFSET);
  unsigned* released = reinterpret_cast<unsigned*>(smem + Tl::REL_OFFSET);

  // position in the tile: the warp's cells start at (wx, wy), the thread's two rows at ty
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int wcols = 32 >> shape, wx = (warp & ((1 << shape) - 1)) * wcols, wy = (warp >> shape) * (N << shape);
  const int lrow = (lane >> (5 - shape)) * N, lcol = lane & (wcols - 1);
  const int tx = wx + lcol, ty = wy + lrow;

  // ---- work: one (tile, chunk); odd chunks march towards -z
  const int zb = int((long long)g.L * chunk / g.nchunks);
  const int nout = int((long long)g.L * (chunk + 1) / g.nchunks) - zb;
  const int dir = (chunk & 1) ? -1 : 1;
  const int nstage = (nout + 1) / 2 + 2 * K;            // pairs of planes: the outputs and K either side
  const int start = dir > 0 ? zb - R : zb + nout - 1 + R;   // real plane of march index 0
  const int2 org = g.tiles[tile];
  const int x = org.x + tx, y0 = org.y + ty;

  __syncthreads();   // a previous item (persistent grids) is fully consumed
  if (tid == 0) {
    for (int s = 0; s < SU; ++s) {
      if (reinit) mbar_inval(&full[s]);
      mbar_init(&full[s], 1);
      released[s] = 0u;
    }
    mbar_init_fence();
  }
  // stage j: u,v,w of the plane pair j (march planes 2j, 2j + 1) and p of the pair j - K + 1, which
  // the predictor reads in the iteration that waits for this stage
  auto plane_of = [&](int m) {
    int zz = start + dir * m;
    if (zz < 0 || zz >= g.L) zz %= g.L;
    return zz < 0 ? zz + g.L : zz;
  };
  auto issue = [&](int j) {
    uint64_t* bar = &full[unsigned(j) % unsigned(SU)];
    const bool with_p = j >= 2 * K - 2;
    mbar_arrive_expect_tx(bar, 2 * Tl::U_BYTES + (with_p ? 2 * Tl::P_BYTES : 0u));
    TE* du = uring + unsigned(j) % unsigned(SU) * (2 * VPL);
    tma_load_4d(du, tmap_uvw, bar, org.x - HX, org.y - HY, plane_of(2 * j), 1);
    tma_load_4d(du + VPL, tmap_uvw, bar, org.x - HX, org.y - HY, plane_of(2 * j + 1), 1);
    if (with_p) {
      const int m = 2 * (j - K + 1);
      TE* dp = pring + unsigned(j - K + 1) % unsigned(SP) * (2 * PPL);
      tma_load_4d(dp, tmap_p, bar, org.x - HX, org.y - 1, plane_of(m), 0);
      tma_load_4d(dp + PPL, tmap_p, bar, org.x - HX, org.y - 1, plane_of(m + 1), 0);
    }
  };
  if (tid == 0) {                      // the whole window up front, before the wall tables are read
    prefetch_tensormap(tmap_p);
    prefetch_tensormap(tmap_uvw);
    if (chained) grid_dependency_wait();
    for (int j = 0; j < SU && j < nstage; ++j) issue(j);
  }
  // Warps that compute (some fluid) and warps over fluid away from walls (no wall sums). With a
  // mask per plane (MP) g.near holds every cell's wall sums; one more plane holds kSolidCell for
  // the columns without any fluid.
  const size_t cplane = size_t(g.lxp) * g.ly;
  const long long col = (long long)y0 * g.lxp + x;
  auto coef = [&](int r) {             // extruded masks; outside the cross-section: nothing
    return x < g.lxp && y0 + r < g.ly ? reinterpret_cast<const ColCoef<float>*>(g.colcoef)[col + r * g.lxp]
                                      : ColCoef<float>{0.f, 0.f, 0.f, 0.f};
  };
  // The load is volatile and its address always valid, so nothing waits for it before its use a
  // predictor later; cells outside the cross-section are settled there.
  auto inside = [&](int r) { return x < g.lxp && y0 + r < g.ly; };
  auto walls = [&](int r, int z) -> uint32_t {
    uint32_t m;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(m) : "l"(g.near + (inside(r) ? z * cplane + col + r * g.lxp : 0)));
    return m;
  };
  bool some = false, every = true;
  if constexpr (MP) {
#pragma unroll
    for (int r = 0; r < N; ++r) some |= inside(r) && walls(r, g.L) != kSolidCell;   // over all planes
  } else {
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const ColCoef<float> c = coef(r);
      some |= c.fluid != 0.0f;
      every &= c.fluid != 0.0f && c.ws0 == 0.0f && c.wsx == 0.0f && c.wsy == 0.0f;
    }
  }
  const bool warp_on = __any_sync(0xffffffffu, some);
  const bool plain_column = __all_sync(0xffffffffu, every);

  // FP16 storage: the tile's base of w (zero outside the cross-section), read by the predictor
  if (chained) grid_dependency_wait();
  constexpr bool kBase = std::is_same<TE, __half>::value;
  float* wbs = reinterpret_cast<float*>(smem + Tl::BASE_OFFSET);
  if (kBase && g.wb)
    for (int i = tid; i < Tl::BW * Tl::BH; i += Tl::THREADS) {
      const int gx = org.x - 1 + i % Tl::BW, gy = org.y - 1 + i / Tl::BW;
      wbs[i] = (gx >= 0 && gy >= 0 && gx < g.lxp && gy < g.ly) ? g.wb[size_t(gy) * g.lxp + gx] : 0.0f;
    }
  __syncthreads();

  // Wait for stage j, one verdict per warp; false after flagging a failure (the whole warp
  // returns). Then any warp may have issued loads up to SU stages ahead: let them land (bounded).
  auto arrive_wait = [&](int j) -> bool {
    auto bar_of = [&](int q) { return &full[unsigned(q) % unsigned(SU)]; };
    auto parity = [](int q) { return (unsigned(q) / unsigned(SU)) & 1u; };
    if (mbar_wait_warp(bar_of(j), parity(j), kWaitLimitNs)) return true;
    if (lane == 0) {
      atomicOr(g.err, 1u);
      for (int q = j + 1; q < nstage && q <= j + SU; ++q) mbar_wait_bounded(bar_of(q), parity(q), kWaitLimitNs / 8);
    }
    __syncwarp();
    return false;
  };
  // Pair j leaves the window (u,v,w after it was the output pair, p of pair j + 1 after the
  // predictor read it, both in iteration j + 1). __syncwarp orders the warp's shared loads before
  // lane 0's acq_rel add to the slot's counter; the warp whose add completes the count has
  // acquired every warp's loads, orders them before its TMA writes with a proxy fence and refills
  // the slot with stage j + SU (and p of pair j + 3 into the slot of p of pair j + 1). A warp that
  // waits for stage s in iteration s - K + 1 needs every warp to have released pair s - SU, in
  // iteration s - SU + 1 = s - K - 1 at the latest, so no wait depends on itself. A slot's next
  // count starts only after its refill has landed, so the count is a multiple of WARPS exactly
  // when a pair is complete.
  auto release = [&](int j) {
    __syncwarp();
    if (lane == 0) {
      const unsigned seen = atom_add_acq_rel_cta(&released[unsigned(j) % unsigned(SU)], 1u) + 1u;
      if (seen % unsigned(Tl::WARPS) == 0u && j + SU < nstage) {
        fence_proxy_async_smem();
        issue(j + SU);
      }
    }
  };

#pragma unroll
  for (int j = 0; j < 2 * K - 2; ++j)
    if (!arrive_wait(j)) return false;
  if (!warp_on) {   // all-wall warps keep the pipeline protocol only
#pragma unroll 1
    for (int q = K - 1; q <= nstage - K; ++q) {
      if (!arrive_wait(q + K - 1)) return false;
      if (q == K - 1)
        for (int j = 0; j < K - 2; ++j) release(j);
      release(q - 1);
    }
    return true;
  }

  // the gauge may have been written by another CTA of the same (chained batched) launch: read
  // it from L2, not from a possibly stale L1 line
  const float gauge = g.gauge ? float(__ldcg(g.gauge)) : 0.0f;
  const int po = (ty + 1) * SW + HX + tx;               // p box
  const int uo = (ty + HY) * SW + HX + tx;              // u box (v, w at +UPL, +2 UPL)
  const float dir3 = 3.0f * float(dir);
  // folded update: u_new = K1 t1 + K2 t2 + K0 u + tb (u* + F), the corrector's taps t1 / t2 at
  // distance d1 / 2 d1, K0 = tb dtddy m c0 + (1 - tb), K1 = tb dtddy m c1, K2 = tb dtddy m c2
  const float kam = __fmul_rn(__fmul_rn(k.tb, k.dtddy), k.m);
  const float kK0 = __fmaf_rn(kam, k.c0, k.cc);
  float kKt[K];                                         // K1 .. KK
  kKt[0] = __fmul_rn(kam, k.c1);
  kKt[1] = __fmul_rn(kam, k.c2);
#pragma unroll
  for (int j = 2; j < K; ++j) kKt[j] = __fmul_rn(kam, k.ch[j - 2]);
  // the predictor's moments come times 216; the z-moment carries the march direction's sign
  const float ktb = __fdiv_rn(k.tb, 216.0f), ktz = __fmul_rn(float(dir), ktb);
  // FP16 storage: the rounding noise of a cell pair is keyed by its first cell, the field and the step
  const uint32_t seed = hash32(g.step_no * 0x9e3779b9u + 0x632be5abu);

  auto ldu = [&](const TE* q) { return make_float2(lds1(q), lds1(q + VPL)); };
  // ring of the own columns in tensor memory: pair j in slot j % TM_RING, field f of row r at
  // column f 2 N + 2 r
  const uint32_t tm = __shfl_sync(0xffffffffu, tmem + (uint32_t(warp & 3) << 21) + uint32_t((warp >> 2) * Tl::TM_WARP), 0);
  auto tm_slot = [&](int j) { return tm + (unsigned(j) & unsigned(Tl::TM_RING - 1)) * unsigned(Tl::TM_SLOT); };
#pragma unroll
  for (int j = 0; j < K - 1; ++j)        // pairs the predictor does not visit
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
      for (int r = 0; r < N; ++r)
        tm_store(tm_slot(j) + f * 2 * N + 2 * r, ldu(uring + j * 2 * VPL + uo + f * UPL + r * SW));
  // staging: the thread's place in the warp's block of wcols x (N << shape) cells
  TE* stg = reinterpret_cast<TE*>(smem + Tl::STG_OFFSET) + warp * Tl::STG;
  TE* sto = stg + lrow * wcols + lcol;
  // Predictor terms carried to the next iteration, per row: cp = the sums of the pair (its first
  // plane's are finished), sh = the self-plane moments of its second plane, dd = the shares that
  // its planes give their march-next planes, pc = p of the pair.
  float2 cp[N][4], dd[N][3], pc[N];
  float sh[N][3];
#pragma unroll
  for (int r = 0; r < N; ++r) {
    pc[r] = f2(0.f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      cp[r][j] = f2(0.f);
      if (j < 3) {
        dd[r][j] = f2(0.f);
        sh[r][j] = 0.f;
      }
    }
  }

#pragma unroll
  for (int j = 0; j < K - 2; ++j) release(j);
  // iteration q: predictor of pair q, which completes the sums of pair q - 1, and from q = K + 1 on
  // corrector and update of the output pair q - 1
  // Two iterations per pass rename the carried registers instead of moving them (FP32, two rows
  // per thread, one cross-section, tiles of 16 or 8 rows: -3 %); the other forms would spill (the
  // batched kernel's 32 x 32 tile: 14.55 against 13.21 ms per 32 steps of 64 pipes) or outgrow the
  // instruction cache (four rows: 4718 against 4415 us per 50 steps at 512 x 128 x 128).
  constexpr int kPass = !MP && !kBase && N == 2 && TY < 32 && SF == 4 ? 2 : 1;
#pragma unroll kPass
  for (int q = K - 1; q <= nstage - K; ++q) {
    if (!arrive_wait(q + K - 1)) {
      tm_wait_stores();
      if (lane == 0) bulk_wait_all();
      __syncwarp();
      return false;
    }
    const TE* sp0 = pring + unsigned(q) % unsigned(SP) * (2 * PPL) + po;
    const TE* su0 = uring + unsigned(q) % unsigned(SU) * (2 * VPL) + uo;          // predictor pair q
    const TE* sub = uring + unsigned(q - 1) % unsigned(SU) * (2 * VPL) + uo;      // output pair q - 1
    const TE* sua[K - 1];                                                         // pairs q + 1 ..
#pragma unroll
    for (int j = 0; j < K - 1; ++j) sua[j] = uring + unsigned(q + 1 + j) % unsigned(SU) * (2 * VPL) + uo;
    const int zp = start + dir * 2 * q;                                           // real plane of the pair's first
    // the output pair's wall sums (MP), loaded a predictor ahead of their use
    const bool second = 2 * (q - 1 - K) + 1 < nout;          // the chunk's plane count may be odd
    uint32_t code[N][2];
    if constexpr (MP) {
      const int z0 = q > K ? zp - 2 * dir : zb, z1 = q > K && second ? zp - dir : z0;
#pragma unroll
      for (int r = 0; r < N; ++r) {
        code[r][0] = walls(r, z0);
        code[r][1] = walls(r, z1);
      }
    }
    float nfirst[N][4];                  // finished sums of pair q's first plane
    float2 pcen[N];
    {
      RowSide<float2> above, here;       // rows r - 1 and r as their lower neighbours see them
      RowSums<float2> mid;
#pragma unroll
      for (int j = -1; j <= N; ++j) {
        float2 p3[3], u3[3], v3[3], w3[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const TE* qp = sp0 + j * SW + c - 1;
          const TE* qu = su0 + j * SW + c - 1;
          p3[c] = make_float2(lds1(qp), lds1(qp + PPL));
          u3[c] = ldu(qu);
          v3[c] = ldu(qu + UPL);
          w3[c] = ldu(qu + 2 * UPL);
        }
        if (j >= 0 && j < N) {
          pcen[j] = p3[1];
          const uint32_t ta = tm_slot(q) + 2 * j;
          tm_store(ta, u3[1]);
          tm_store(ta + 2 * N, v3[1]);
          tm_store(ta + 4 * N, w3[1]);
        }
        if (kBase && g.wb)               // w = stored deviation + the column's base
#pragma unroll
          for (int c = 0; c < 3; ++c) w3[c] = add2(w3[c], f2(wbs[(ty + 1 + j) * Tl::BW + tx + c]));
        const RowSums<float2> row = row_sums(p3, u3, v3, w3);
        if (j >= 1) {
          const int r = j - 1;
          const RowSide<float2> below = row_side<1>(row);
          // row-factored weights w(cx)w(cy) = {4,1,1}x{4,1,1}/36: A, X (cx moment), Y (cy moment)
          float2 A[3], X[3], Y[3];
          A[0] = fma2(f2(4.0f), mid.R0, add2(above.R0, below.R0));
          A[1] = fma2(f2(4.0f), mid.Rz, add2(above.Rz, below.Rz));
          A[2] = fma2(f2(4.0f), mid.Rw, add2(above.Rw, below.Rw));
          X[0] = fma2(f2(4.0f), mid.D0, add2(above.D0, below.D0));
          X[1] = fma2(f2(4.0f), mid.Dz, add2(above.Dz, below.Dz));
          X[2] = fma2(f2(4.0f), mid.Dw, add2(above.Dw, below.Dw));
          Y[0] = sub2(below.R0, above.R0);
          Y[1] = sub2(below.Rz, above.Rz);
          Y[2] = sub2(below.Rw, above.Rw);
          if (min(zp, zp + dir) < 0 || max(zp, zp + dir) >= g.L) {
            // seam planes (CTA-uniform): a wrapped plane adds the pressure jump to p on its
            // non-wall cells, i.e. the jump times their weight sums (raw units, x36)
            auto jump = [&](int z) { return z < 0 ? k.pin : (z >= g.L ? -k.pin : 0.0f); };
            const float2 off = make_float2(jump(zp), jump(zp + dir));
            float2 n0, nx, ny;
            if constexpr (MP) {
              float s0[2], sx[2], sy[2];
              for (int h = 0; h < 2; ++h) {
                const uint8_t* mz = g.mask + plane_of(2 * q + h) * cplane;
                s0[h] = sx[h] = sy[h] = 0.f;
                for (int cy = -1; cy <= 1; ++cy)
                  for (int cx = -1; cx <= 1; ++cx) {
                    const int gx = x + cx, gy = y0 + r + cy;
                    if (gx < 0 || gy < 0 || gx >= g.lxp || gy >= g.ly || mz[gy * g.lxp + gx] == kWall) continue;
                    const float w = (cx ? 1.f : 4.f) * (cy ? 1.f : 4.f);
                    s0[h] += w; sx[h] += cx * w; sy[h] += cy * w;
                  }
              }
              n0 = make_float2(s0[0], s0[1]); nx = make_float2(sx[0], sx[1]); ny = make_float2(sy[0], sy[1]);
            } else {
              const ColCoef<float> c = coef(r);
              n0 = f2(__fmaf_rn(-36.f, c.ws0, 36.f)); nx = f2(-36.f * c.wsx); ny = f2(-36.f * c.wsy);
            }
            A[0] = fma2(off, n0, A[0]);
            X[0] = fma2(off, nx, X[0]);
            Y[0] = fma2(off, ny, Y[0]);
          }
          // True sums are A0/36, dir A1/12, A2/8. A plane is the march-next neighbour of the plane
          // before it, itself, and the march-previous neighbour of the plane after: with
          // e = (A0 + A2)/6 and h = A1/6 the shares are e + h (next), (2/3) A0 (self) and e - h
          // (previous); for the z-moment h - e (previous), none (self) and e + h (next), times dir.
          // All are carried times 216 (the weights' common denominator): e = A0 + 4.5 A2,
          // h = 3 dir A1, self = 4 A0.
          float2 s[3], d[3];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const float2(&m)[3] = i == 0 ? A : (i == 1 ? X : Y);
            const float2 e = fma2(m[2], f2(4.5f), m[0]);
            s[i] = fma2(m[1], f2(dir3), e);
            d[i] = fma2(neg2(m[1]), f2(dir3), e);
          }
          // Each cell sums its two neighbour planes' shares first (a commutative add) and then
          // fuses its own plane's share, so its FP32 result depends neither on the march
          // direction nor on how the pipe is split into chunks and pairs. That makes batched and
          // served results equal to a solve stepped alone, bit for bit.
          const float2 self[3] = {A[0], X[0], Y[0]};
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            cp[r][i].y = __fmaf_rn(sh[r][i], 4.0f, __fadd_rn(dd[r][i].x, s[i].x));
            nfirst[r][i] = __fmaf_rn(self[i].x, 4.0f, __fadd_rn(dd[r][i].y, s[i].y));
          }
          cp[r][3].y = __fsub_rn(s[0].x, dd[r][0].x);
          nfirst[r][3] = __fsub_rn(s[0].y, dd[r][0].y);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            sh[r][i] = self[i].y;
            dd[r][i] = d[i];
          }
        }
        if (j >= 0) above = here;
        mid = row;
        here = row_side<-1>(row);
      }
    }
    if (q > K) {
      tm_wait_stores();
      const int zo = zp - 2 * dir;                           // real plane of the output pair's first
      // wall sums (times 216) and fluid flag of the rows: one value for both planes of an extruded mask
      using Sum = std::conditional_t<MP, float2, float>;
      auto both = [](float a, float b) {
        if constexpr (MP) return make_float2(a, b);
        else return a;
      };
      Sum ws0[N], wsx[N], wsy[N], wsz[N], fluid[N];
#pragma unroll
      for (int r = 0; r < N; ++r) {
        ws0[r] = wsx[r] = wsy[r] = wsz[r] = both(0.f, 0.f);
        fluid[r] = both(1.f, 1.f);
      }
      if constexpr (MP) {
        uint32_t any = 0;
#pragma unroll
        for (int r = 0; r < N; ++r) {
          if (!inside(r)) code[r][0] = code[r][1] = kSolidCell;
          any |= code[r][0] | code[r][1];
        }
        if (__any_sync(0xffffffffu, any != 0u)) {
#pragma unroll
          for (int r = 0; r < N; ++r) {
            auto sums = [&](uint32_t m, float& s0, float& sx, float& sy, float& sz, float& fl) {
              auto field = [&](int at) { return float(int(m << (25 - at)) >> 25); };
              s0 = float(m & 255u);
              sx = field(8);
              sy = field(15);
              sz = float(dir) * field(22);
              fl = m & kSolidCell ? 0.f : 1.f;
            };
            sums(code[r][0], ws0[r].x, wsx[r].x, wsy[r].x, wsz[r].x, fluid[r].x);
            sums(code[r][1], ws0[r].y, wsx[r].y, wsy[r].y, wsz[r].y, fluid[r].y);
          }
        }
      } else if (!plain_column) {
#pragma unroll
        for (int r = 0; r < N; ++r) {
          const ColCoef<float> c = coef(r);
          ws0[r] = 216.f * c.ws0; wsx[r] = 216.f * c.wsx; wsy[r] = 216.f * c.wsy;
          fluid[r] = c.fluid;
        }
      }
      float2 wg[N];
      if (kBase)
#pragma unroll
        for (int r = 0; r < N; ++r)
          wg[r] = f2(g.wgt && x < g.lxp && y0 + r < g.ly ? g.wgt[(y0 + r) * g.lxp + x] : 0.0f);
      if (lane == 0) bulk_wait_read();                       // the previous pair has left the staging
      __syncwarp();
      auto put = [&](int f, int r, float2 val) {
        val = mul2(val, f2(fluid[r]));                           // walls get zero
        TE* o = sto + f % SF * N * 32 + r * wcols;
        if constexpr (kBase) {
          // two cells share a hash word: the even column's lane forms the first plane's, the odd
          // column's the second plane's
          const bool odd = x & 1;
          const uint32_t cell = (uint32_t(zo + (odd ? dir : 0)) * uint32_t(g.ly) + uint32_t(y0 + r)) * uint32_t(g.lxp)
                                + (uint32_t(x) & ~1u);
          const uint32_t mine = hash32(((cell << 2) | uint32_t(f)) ^ seed);
          const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
          o[0] = sr_half(val.x, odd ? other >> 16 : mine);
          o[SF * N * 32] = sr_half(val.y, odd ? mine >> 16 : other);
        } else {
          o[0] = val.x;
          o[SF * N * 32] = val.y;
        }
      };
      auto flush = [&](int f0) {                                 // fields f0 .. f0 + SF - 1 leave the staging
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_4d(tmap_out, stg, org.x + wx, org.y + wy, zo, f0);
          if (second) tma_store_4d(tmap_out, stg + SF * N * 32, org.x + wx, org.y + wy, zo + dir, f0);
          bulk_commit();
        }
      };
#pragma unroll
      for (int r = 0; r < N; ++r)
        put(0, r, fma2(fma2(pc[r], f2(ws0[r]), cp[r][0]), f2(1.0f / 216.0f), f2(-gauge)));
      // own columns of pairs q, q - 1, ...: with kAhead the next field's arrive while a field is
      // computed (-1 % on the FP32 32 x 32 tile, -2 % with FP16 storage; in the FP32 batched
      // kernel the registers spill, +5 %)
      constexpr bool kAhead = N == 4 || kBase || (TY < 32 && SF == 4);
      float2 rings[kAhead ? 2 : 1][K + 2][N];
      auto load_ring = [&](int f) {
#pragma unroll
        for (int j = 0; j < K + 2; ++j) tm_load(rings[kAhead ? f & 1 : 0][j], tm_slot(q - j) + f * 2 * N);
      };
      if (kAhead) load_ring(0);
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        const TE* b = sub + f * UPL;
        float2 (&ring)[K + 2][N] = rings[kAhead ? f & 1 : 0];
        if (!kAhead) load_ring(f);
        float2 c[N + 2 * R];                                 // rows -R .. N + R - 1 of the own column
#pragma unroll
        for (int j = -R; j < N + R; ++j)
          if (j < 0 || j >= N) c[j + R] = ldu(b + j * SW);
        tm_wait_loads(ring);
        if (kAhead && f < 2) load_ring(f + 1);
#pragma unroll
        for (int r = 0; r < N; ++r) c[r + R] = ring[1][r];
#pragma unroll
        for (int r = 0; r < N; ++r) {
          const TE* t = b + r * SW;
          float2 taps[K];                                    // the six taps at distance 2 (j + 1)
#pragma unroll
          for (int j = 0; j < K; ++j) {
            const int o = D1 * (j + 1);
            const float2 ahead = j == 0 ? ring[0][r] : ldu(sua[j > 0 ? j - 1 : 0] + f * UPL + r * SW);
            taps[j] = add2(add2(add2(ldu(t - o), ldu(t + o)), add2(c[r + R - o], c[r + R + o])),
                           add2(ring[j + 2][r], ahead));
          }
          const float2 cm = cp[r][f == 2 ? 3 : 1 + f];
          const float2 mom = f == 2 && !MP ? cm : fma2(pc[r], f2(f == 0 ? wsx[r] : (f == 1 ? wsy[r] : wsz[r])), cm);
          // FP16 storage updates the stored deviation of w: the force's term becomes the column's
          // share of the step of the base (tb fz included), see launch_wgt
          const float2 tf = kBase && f == 2 && g.wgt ? wg[r] : f2(__fmul_rn(k.tb, f == 0 ? k.fx : (f == 1 ? k.fy : k.fz)));
          // the small terms first: only the last operation rounds at the size of u
          float2 un = fma2(f2(f == 2 ? ktz : ktb), mom, tf);
#pragma unroll
          for (int j = K - 1; j >= 0; --j) un = fma2(f2(kKt[j]), taps[j], un);
          un = fma2(f2(kK0), ring[1][r], un);
          if (SF == 2 && f == 1 && r == 0) {                     // p and u have left the staging
            if (lane == 0) bulk_wait_read();
            __syncwarp();
          }
          put(1 + f, r, un);
        }
        if (SF == 2 && f == 0) flush(0);
      }
      flush(4 - SF);
    }
#pragma unroll
    for (int r = 0; r < N; ++r) {
      pc[r] = pcen[r];
#pragma unroll
      for (int i = 0; i < 4; ++i) cp[r][i].x = nfirst[r][i];
    }
    release(q - 1);
  }
  if (lane == 0) bulk_wait_all();
  return true;
}

// One pipe, one step: CTA b marches (tile b % ntiles, chunk b / ntiles).
template <int TY, class TE, int K = 2, bool MP = false, int ROWS = 2>
__global__ void __launch_bounds__(Step2Tile<TY, TE, K, ROWS>::THREADS, Step2Tile<TY, TE, K, ROWS>::CTAS)
    fslbm_step2_kernel(const __grid_constant__ CUtensorMap tmap_p,
                       const __grid_constant__ CUtensorMap tmap_uvw,
                       const __grid_constant__ CUtensorMap tmap_out, const Step2Geom g,
                       const StepConst<float> k) {
  using Tl = Step2Tile<TY, TE, K, ROWS>;
  extern __shared__ __align__(128) unsigned char smem[];
  uint32_t* tm_base = reinterpret_cast<uint32_t*>(smem + Tl::REL_OFFSET) + Tl::SU;
  if (threadIdx.x < 32) tm_alloc<Tl::TM_COLS>(tm_base);
  if (!g.early) grid_dependency_wait();
  __syncthreads();
  const uint32_t tmem = *tm_base;
  step2_march<TY, TE, K, MP, ROWS>(&tmap_p, &tmap_uvw, &tmap_out, tmem, g, k, blockIdx.x % g.ntiles, blockIdx.x / g.ntiles,
                                   smem, false, 0, true);
  grid_launch_dependents();   // not earlier: waiting CTAs of the next step would share this one's SMs
  if (threadIdx.x == 0 && blockIdx.x == 0 && g.step_counter) *g.step_counter += 1;
  __syncthreads();
  if (threadIdx.x < 32) tm_free<Tl::TM_COLS>(tmem);
}

}  // namespace fslbm
