// tws_sweep.cu -- the temporally blocked step as a row sweep.
//
// Same arithmetic as the tiled kernels (flowUpdate.comp:34-62 then
// flowApply.comp:32-52, K steps per launch, bit-identical to the FP32
// transcription of the shaders), organised so that no halo is recomputed in y
// within a band:
//
// * A warp owns a strip of 128 columns, four per lane, and sweeps it down a
//   band of rows.  Row by row, time level s = 0..K-1 computes the outflow of
//   one row and the depth of the row above, which is the input row of level
//   s + 1 two rows further up; the last level writes its depth, flux and flow
//   map.  The y neighbours come from what the level keeps of its previous
//   rows, the x neighbours from the lane itself or its neighbour lanes (warp
//   shuffles).  Values of the outermost columns of the strip go stale one
//   more column per phase, so a strip yields 112 (K = 3, 4) or 120 (K = 2)
//   output columns; neighbouring strips overlap by the rest (their loads are
//   mostly L2 hits).  A band also loads 2K rows above and below it, whose
//   results are not written.
// * What bounds it: instruction issue, and on the largest grids HBM.  Four
//   cells a lane halve the shuffles, branches and address arithmetic per cell
//   against two, and the strip overlap falls from 23% to 14%.  What a level
//   keeps between rows is split so that three CTAs of four warps fit an SM
//   (168 registers a thread, 18 KB of shared memory a warp at K = 3): depths
//   and outflows that are read once, two rows later, wait in shared memory
//   (which also saves the moves that shift a register window); the slope
//   term of the last row pair, the x inflow and the outflow sum stay in
//   registers.  The loop over rows is not unrolled: two rows per trip double
//   the code and run 15-30% slower (instruction fetch).
// * Neighbouring cells share the slope term ka * (h - h_n) of their common
//   edge up to its sign, so each is computed once.
// * The columns of a lane are two packed f32x2 operands: each half is the
//   IEEE round-to-nearest result of its own operands.  A packed product that
//   feeds a packed sum is formed as a fused multiply-add of -0 (prod2), which
//   has the product's own bits and which the assembler cannot contract
//   further.
// * Loads: cp.async into shared memory, one row ahead of the row computed
//   (12 warps of 3 KB in flight cover the latency).  Cells off the grid are
//   zero-filled by the copy itself (the shaders' out-of-range image loads
//   read zero).  cp.async.wait_group and a warp barrier hand a row over.
// * The warps are persistent and take (strip, band) units from two per-grid
//   queues, border units and inner ones (sweep_next below).  A warp that finds
//   them empty takes over half of the rows that another has not begun
//   (range_pack below), so units under rain, at the border or on shores, which
//   take longer, do not hold the launch up.
//
// HBM traffic per launch: the state once in, once out (52 B per cell for FP32
// flux, 36 B for FP16), plus what L2 does not catch of the overlaps.
//
// Measured (CUDA events, Gcell-steps/s on moving water with a rain disk, K = 3;
// in brackets the two-columns-a-lane kernel with static bands that this
// replaced): 4096^2 268 (209), 8192^2 315 (250), 16384^2 339 (260), FP16 flux
// 320 (253).  16384^2 at 339 moves 5.9 TB/s of compulsory bytes, 0.86 of the
// copy rate; on smaller grids the halo rows of the bands (4096^2: 84 rows and
// 12) and the launch's end weigh more, and the scheduler issues in 57% of the
// cycles (three warps each: fixed-latency waits, shared memory, fetch).

#include <algorithm>

#include "tws_device.cuh"
#include "tws_internal.h"
#include "tws_pair.cuh"

namespace tws {
namespace {

constexpr int kSweepThreads = kSweepCtaThreads;
constexpr int kSweepWarps = kSweepThreads / 32;
constexpr int kSweepCols = 128;  // columns a warp loads: four per lane
// columns at either end of a strip that are not written: the 2K that go stale,
// in whole lanes
__host__ __device__ constexpr int kSweepHaloX(int k) { return (2 * k + 3) / 4 * 4; }

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// cp.async of `bytes` (<= size) from src; the rest of the `size` bytes is zero.
__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Shared memory of one warp, in bytes.
constexpr int kSweepRow = kSweepCols * 4;  // one float per column
constexpr int sweep_flux_row_bytes(bool f16) { return kSweepCols * (f16 ? 8 : 16); }
constexpr int kSweepSlotBytes = kSweepCols * 16;
// rows of the terrain ring: the row in flight, the current one and those the
// deeper levels still form h from (row r - 2(K - 1)): 2K, in a power of two
constexpr int sweep_b_rows(int k) { return k <= 2 ? 4 : 8; }
constexpr int kSweepDRows = 4;  // depth ring: the row in flight, rows r, r - 1 and r - 2
constexpr int sweep_warp_bytes(int k, bool f16) {
  return kSweepRow * (sweep_b_rows(k) + kSweepDRows + 2 * (k - 1)) + sweep_flux_row_bytes(f16) +
         (k - 1) * 2 * kSweepSlotBytes;
}

template <int K, bool F16>
struct SweepRing {
  static constexpr int PB = sweep_b_rows(K);
  static constexpr int B = 0;
  static constexpr int D = B + kSweepRow * PB;
  // depths of the two previous input rows of levels 1 .. K - 1
  static constexpr int DS = D + kSweepRow * kSweepDRows;
  static constexpr int F = DS + kSweepRow * 2 * (K - 1);
  // The new outflows of each level's two previous rows (all levels but the
  // last), one slot per row (the row computed in an iteration takes the slot
  // of the older one once it has been read): four channel planes.
  static constexpr int N = F + sweep_flux_row_bytes(F16);
  static constexpr int NSLOT = kSweepSlotBytes;
  static constexpr int WARP = sweep_warp_bytes(K, F16);
  static_assert(sweep_strip_columns(K) == kSweepCols - 2 * kSweepHaloX(K), "columns that count");
  static_assert(WARP == N + (K - 1) * 2 * NSLOT && PB >= 2 * K, "ring sizes");
};

// The rows of a warp's unit that nobody has claimed yet, one word per resident
// warp: [cur, end) of strip `strip`.  The owner claims kSweepClaim rows at a
// time from the front (one atomic add); a warp that finds the queue empty takes
// the back half of another's range (one compare-and-swap).  Equal words mean
// equal unclaimed rows, so a swap that succeeds is right whatever happened in
// between.  Nothing waits on anything.
constexpr int kSweepClaim = 8;     // rows of one claim
constexpr int kSweepStealTries = 6;
constexpr int kSweepMinSteal = 8; // unclaimed rows worth halving: a new unit computes
                                   // about six rows' worth of halo
__device__ __forceinline__ unsigned long long range_pack(int strip, int cur, int end) {
  return (unsigned long long)(unsigned)strip << 42 | (unsigned long long)(unsigned)end << 21 |
         (unsigned long long)(unsigned)cur;
}
__device__ __forceinline__ int range_cur(unsigned long long w) { return (int)(w & 0x1fffff); }
__device__ __forceinline__ int range_end(unsigned long long w) { return (int)(w >> 21 & 0x1fffff); }
__device__ __forceinline__ int range_strip(unsigned long long w) { return (int)(w >> 42); }

// A: StepArgs, or SweepArgs where the arguments come from a batch's table.
template <int K, bool F16, bool INTERIOR, class A>
__device__ __forceinline__ void sweep_unit(const A& a, const float* __restrict__ gb,
                                           const float* __restrict__ gd,
                                           const void* __restrict__ gf,
                                           float* __restrict__ d_out, void* __restrict__ f_out,
                                           float2* __restrict__ v_out, unsigned char* ring,
                                           int xs, int y0, int R, uint32_t mask,
                                           unsigned long long* word) {
  using RG = SweepRing<K, F16>;
  constexpr int HALO = 2 * K;
  const int lane = threadIdx.x & 31;
  const int W = a.W, H = a.H;
  const size_t pitch = (size_t)a.pitch;
  const pair_t kf2 = pk(a.kf, a.kf), ka2 = pk(a.ka, a.ka), cc2 = pk(a.c, a.c);
  const pair_t ncc2 = pk(-a.c, -a.c), nz2 = pk(a.neg_zero, a.neg_zero);
  const float2 fscale2 = make_float2(a.flux_scale, a.flux_scale);
  const float2 finv2 = make_float2(a.flux_inv_scale, a.flux_inv_scale);
  const bool closed = a.closed != 0;

  // this lane's columns gx .. gx + 3 (xs is a multiple of 4); `cols` of them
  // are on the grid, all on one side
  const int gx = xs + 4 * lane;
  const int cols = INTERIOR ? 4 : (gx < 0 ? 0 : min(4, max(0, W - gx)));
  const bool out_lane =
      lane >= kSweepHaloX(K) / 4 && lane < 32 - kSweepHaloX(K) / 4 && (INTERIOR || cols > 0);
  const int first_row = y0 - HALO;

  unsigned char* const lane16 = ring + 16 * lane;
  // ---- the copies of load step i: b and d of row first_row + i, the flux of
  // the row above it (which level 0 updates in the same iteration).  The
  // flux of the first two steps is never used.
  // Flux records go to shared memory in 16-byte chunks, lane l copying chunks
  // l, l + 32, ... of the row (whole sectors), chunk j at position j with its
  // low bits exchanged so that a lane's own chunks (4 in a row; FP16: 2) are
  // read back without bank conflicts.
  auto chunk = [](int j) { return F16 ? j ^ ((j >> 3) & 1) : j ^ ((j >> 3) & 3); };
  constexpr int CH = F16 ? 2 : 4;  // chunks of a lane
  // element index of row first_row + i (advanced with i), column xs or, at the
  // grid's edge, column 0
  long long g_in = (long long)first_row * (long long)pitch + (INTERIOR ? xs : 0);
  const int gx_in = max(0, gx), nb = 4 * cols;
  auto issue_row = [&](int i) {
    unsigned char* const sb = lane16 + RG::B + ((unsigned)i % RG::PB) * kSweepRow;
    unsigned char* const sd = lane16 + RG::D + ((unsigned)i % kSweepDRows) * kSweepRow;
    unsigned char* const sf = ring + RG::F;
    const unsigned char* const fb = reinterpret_cast<const unsigned char*>(gf);
    if constexpr (INTERIOR) {
      copy16(sb, gb + g_in + 4 * lane, 16);
      copy16(sd, gd + g_in + 4 * lane, 16);
      if (i >= 2) {
        const unsigned char* f = fb + (g_in - (long long)pitch) * (F16 ? 8 : 16) + 16 * lane;
#pragma unroll
        for (int k = 0; k < CH; ++k) copy16(sf + 16 * chunk(32 * k + lane), f + 512 * k, 16);
      }
    } else {
      // cells off the grid are cleared: a copy of n bytes zero-fills the rest
      // of its 16 (of no bytes: it reads nothing)
      const unsigned r = (unsigned)(first_row + i);  // rows above the grid wrap around
      const int n = r < (unsigned)H ? nb : 0;
      const long long g = n ? g_in + gx_in : 0;
      copy16(sb, gb + g, n);
      copy16(sd, gd + g, n);
      if (i >= 2) {
        const bool row_in = r - 1 < (unsigned)H;
#pragma unroll
        for (int k = 0; k < CH; ++k) {
          const int j = 32 * k + lane;
          const int c = xs + (F16 ? 2 * j : j);  // the chunk's first column
          const int m = row_in && c >= 0 ? min(F16 ? 2 : 1, max(0, W - c)) : 0;
          const long long h = m ? g_in - (long long)pitch + c : 0;
          copy16(sf + 16 * chunk(j), fb + h * (F16 ? 8 : 16), m * (F16 ? 8 : 16));
        }
      }
    }
    g_in += (long long)pitch;
  };
  auto read_b = [&](int i) -> Quad {  // terrain of load step i
    return load_quad(lane16 + RG::B + ((unsigned)i % RG::PB) * kSweepRow);
  };
  auto d_row = [&](int i) {  // depth of load step i
    return lane16 + RG::D + ((unsigned)i % kSweepDRows) * kSweepRow;
  };
  auto read_flux = [&]() -> Flux4 {
    const unsigned char* st = ring + RG::F;
    float4 c[4];
    if constexpr (F16) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint4 raw = *reinterpret_cast<const uint4*>(st + 16 * chunk(2 * lane + k));
        const float2 a0 = fmul2(__half22float2(*reinterpret_cast<const __half2*>(&raw.x)), finv2);
        const float2 a1 = fmul2(__half22float2(*reinterpret_cast<const __half2*>(&raw.y)), finv2);
        const float2 b0 = fmul2(__half22float2(*reinterpret_cast<const __half2*>(&raw.z)), finv2);
        const float2 b1 = fmul2(__half22float2(*reinterpret_cast<const __half2*>(&raw.w)), finv2);
        c[2 * k] = make_float4(a0.x, a0.y, a1.x, a1.y);
        c[2 * k + 1] = make_float4(b0.x, b0.y, b1.x, b1.y);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        c[k] = *reinterpret_cast<const float4*>(st + 16 * chunk(4 * lane + k));
    }
    return Flux4{pk4(c[0].x, c[1].x, c[2].x, c[3].x), pk4(c[0].y, c[1].y, c[2].y, c[3].y),
                 pk4(c[0].z, c[1].z, c[2].z, c[3].z), pk4(c[0].w, c[1].w, c[2].w, c[3].w)};
  };
  // The sources of row r on this lane's four cells, in source order (as
  // add_sources applies them): the unit's own one after another, not all that the
  // grid has (eight disks on 4096^2: 234 -> 255 Gcell-steps/s, 2896^2 172 -> 200).
  // A warp under a rain disk is the slowest of a
  // launch, so a DISK's four cells go side by side without a branch; the
  // brush, rare, is a rolled loop over the cells in `slot` (a call would take
  // registers from the whole kernel).
  auto sources4 = [&](Quad dq, unsigned char* slot, int r) -> Quad {
    if (!INTERIOR && (r < 0 || r >= H)) return dq;
#pragma unroll 1
    for (uint32_t left = mask; left; left &= left - 1) {
      const int k = __ffs((int)left) - 1;
      const DevSource& src = a.src[k];
      if (r < src.by0 || r > src.by1) continue;  // warp-uniform
      if (src.kind == TWS_SOURCE_DISK) {
        const long long dy = r - src.icy;
        const long long room = (long long)src.ir * src.ir - dy * dy;  // dx^2 allowed
        const uint32_t hy = rain_hash32((uint32_t)r);
        bool in[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const long long dx = gx + c - src.icx;
          in[c] = (INTERIOR || c < cols) && dx * dx <= room;
        }
        auto cell = [&](int c) { return rain_hash32((uint32_t)(gx + c) ^ hy); };
        dq.p[0] = rain2(dq.p[0], src.rate, cell(0), cell(1), in[0], in[1]);
        dq.p[1] = rain2(dq.p[1], src.rate, cell(2), cell(3), in[2], in[3]);
      } else {
        store_quad(slot, dq);
        float* const dv = reinterpret_cast<float*>(slot);
#pragma unroll 1
        for (int c = 0; c < cols; ++c) dv[c] = add_sources_inline(dv[c], gx + c, r, a, 1u << k);
        dq = load_quad(slot);
      }
    }
    return dq;
  };

  // ---- what level s carries from row to row in registers (every index is a
  // compile-time constant once the level loops are unrolled).  In iteration t
  // its outflow row is ys = first_row + t - 2s - 1, its depth row ys - 1.
  // Depths and the outflows of all levels but the last wait in shared memory
  // (a lane reads back only what it wrote).
  Quad Qm[K];           // ka * (h(ys - 1) - h(ys)): the +y slope term of row ys - 1,
                        // and minus the -y slope term of row ys
  Quad InX[K], Out[K];  // row ys - 1: inflow from the x neighbours, outflow sum
  // the last level: h of row ys; row ys - 1's x flow, +y and -y outflows, and
  // row ys - 2's +y outflow
  const Quad zero{{0, 0}};
  Quad h_c = zero, vx_m = zero, z_m = zero, w_m = zero, z_mm = zero;
#pragma unroll
  for (int s = 0; s < K; ++s) Qm[s] = InX[s] = Out[s] = zero;

  // Iterations, 4K more than the rows this warp has claimed so far: R of them
  // at first, and kSweepClaim more with every claim on the unit's range.
  int rows = R + 2 * HALO;
  bool more = word != nullptr;
  unsigned long long claim = 0;

  issue_row(0);
  copy_commit();

  auto row = [&](const int t) {
    const int r = first_row + t;
    // load step t has landed, for every lane
    copy_wait<0>();
    __syncwarp();
    const Flux4 f_row = read_flux();  // flux of row r - 1: level 0's outflow row
    Flux4 f_in = f_row;
    Quad d_in = load_quad(d_row(t));
    __syncwarp();  // the flux row has been read: the next one may take its place
    if (t + 1 < rows) issue_row(t + 1);
    copy_commit();
    // level 0's input row: the first step's sources, then h = d + b
    if (mask) {
      d_in = sources4(d_in, d_row(t), r);
      store_quad(d_row(t), d_in);
    }
    Quad h_in = add4(d_in, read_b(t));
    const int q = t & 1;

#pragma unroll
    for (int s = 0; s < K; ++s) {
      const int ys = r - 2 * s - 1;  // this level's outflow row
      // the y slope term of the row pair (ys, ys + 1)
      unsigned char* const ds = lane16 + RG::DS + ((s - 1) * 2 + q) * kSweepRow;
      unsigned char* const ds1 = lane16 + RG::DS + ((s - 1) * 2 + (q ^ 1)) * kSweepRow;
      const Quad dc = load_quad(s == 0 ? d_row(t - 1) : ds1);
      const Quad dm = load_quad(s == 0 ? d_row(t - 2) : ds);
      if (s > 0) {
        if (mask) d_in = sources4(d_in, ds, ys + 1);
        store_quad(ds, d_in);
        h_in = add4(d_in, read_b(t - 2 * s));
      }
      const Quad hc = s + 1 < K ? add4(dc, read_b(t - 2 * s - 1)) : h_c;
      if (s + 1 == K) h_c = h_in;
      // (the old value of what a level carries is used up before the new one is
      // formed, here and below, which saves moves)
      const Quad w_in = sub4(prod4(f_in.w, kf2, nz2), Qm[s]);
      Qm[s] = prod4(sub4(hc, h_in), ka2, nz2);
      // Rows above the band's first needed outflow row of this level (its
      // windows are filling): nothing below this level is needed either.
      if (t < 4 * s + 2) break;
      unsigned char* const slot = lane16 + RG::N + (s * 2 + q) * RG::NSLOT;

      // -- outflow of row ys, flowUpdate.comp:34-62.  Neighbouring cells share
      // the slope term of their common edge up to its sign (a - b and b - a
      // round alike, and so do the products).
      const float4 h4 = un4(hc);
      const float hr = __shfl_down_sync(0xffffffffu, h4.x, 1);
      const Quad qx = prod4(
          pk4(fsub(h4.x, h4.y), fsub(h4.y, h4.z), fsub(h4.z, h4.w), fsub(h4.w, hr)), ka2, nz2);
      const float4 q4 = un4(qx);
      const float ql = __shfl_up_sync(0xffffffffu, q4.w, 1);
      Flux4 nf;
      nf.x = max0q(add4(prod4(f_in.x, kf2, nz2), qx));
      const float4 fy = un4(prod4(f_in.y, kf2, nz2));
      nf.y = pk4(max0_fast(fsub(fy.x, ql)), max0_fast(fsub(fy.y, q4.x)),
                 max0_fast(fsub(fy.z, q4.y)), max0_fast(fsub(fy.w, q4.z)));
      nf.z = max0q(add4(prod4(f_in.z, kf2, nz2), Qm[s]));
      nf.w = max0q(w_in);
      if constexpr (!INTERIOR) {
        // Only what cells on the grid read of cells off it has to be zero:
        // the +x outflow of column -1, the -x outflow of column W, the +y
        // outflow of row -1 and the -y outflow of row H.  A closed wall has
        // no outflow across it either.
        if (ys < 0 || ys >= H) nf.z = nf.w = zero;
        if (closed && ys == H - 1) nf.z = zero;
        if (closed && ys == 0) nf.w = zero;
        const int wx = closed ? W - 1 : W;  // +x outflow is zero from here on
        const float4 ox = un4(nf.x), oy = un4(nf.y);
        nf.x = pk4(gx >= wx ? 0.0f : ox.x, gx + 1 >= wx ? 0.0f : ox.y,
                   gx + 2 >= wx ? 0.0f : ox.z, gx + 3 >= wx || gx < 0 ? 0.0f : ox.w);
        nf.y = pk4(gx >= W || (closed && gx == 0) ? 0.0f : oy.x, gx + 1 >= W ? 0.0f : oy.y,
                   gx + 2 >= W ? 0.0f : oy.z, gx + 3 >= W ? 0.0f : oy.w);
      }
      {
        const Quad sum = add4(add4(add4(nf.x, nf.y), nf.z), nf.w);
        const Quad sc = outflow_factors(sum, dc, cc2, ncc2, nz2);
        nf.x = prod4(nf.x, sc, nz2);
        nf.y = prod4(nf.y, sc, nz2);
        nf.z = prod4(nf.z, sc, nz2);
        nf.w = prod4(nf.w, sc, nz2);
      }
      if constexpr (F16) {
        auto quant = [&](Quad& v) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float2 o = quantize_f16x2(un(v.p[i]), fscale2, finv2);
            v.p[i] = pk(o.x, o.y);
          }
        };
        quant(nf.x);
        quant(nf.y);
        quant(nf.z);
        quant(nf.w);
      }

      // the outflows of row ys - 2 are level s + 1's input; row ys takes
      // their slot
      Quad Y0 = z_mm;
      if (s + 1 < K) {
        f_in.x = load_quad(slot);
        f_in.y = load_quad(slot + kSweepRow);
        f_in.z = load_quad(slot + 2 * kSweepRow);
        f_in.w = load_quad(slot + 3 * kSweepRow);
        Y0 = f_in.z;
        store_quad(slot, nf.x);
        store_quad(slot + kSweepRow, nf.y);
        store_quad(slot + 2 * kSweepRow, nf.z);
        store_quad(slot + 3 * kSweepRow, nf.w);
      }

      // -- depth of row ys - 1, flowApply.comp:32-41
      const Quad in = add4(add4(InX[s], nf.w), Y0);
      const Quad dn = max0q(add4(dm, prod4(sub4(in, Out[s]), cc2, nz2)));
      // this row's x inflow and outflow sum, for the depth of row ys
      const float4 nx = un4(nf.x), ny = un4(nf.y);
      const float X1r = __shfl_down_sync(0xffffffffu, ny.x, 1);
      const float X0l = __shfl_up_sync(0xffffffffu, nx.w, 1);
      InX[s] = pk4(fadd(ny.y, X0l), fadd(ny.z, nx.x), fadd(ny.w, nx.y), fadd(X1r, nx.z));
      Out[s] = add4(add4(add4(nf.x, nf.y), nf.z), nf.w);

      const int yd = ys - 1;
      if (s + 1 < K) {
        // level s + 1's input row yd; cells off the grid stay empty
        d_in = dn;
        if constexpr (!INTERIOR) {
          const int n = yd >= 0 && yd < H ? cols : 0;
          const float4 o = un4(dn);
          d_in =
              pk4(n > 0 ? o.x : 0.0f, n > 1 ? o.y : 0.0f, n > 2 ? o.z : 0.0f, n > 3 ? o.w : 0.0f);
        }
      } else {
        // the last level: the flux of row ys, the depth and the flow map
        // (flowApply.comp:45-46) of row yd go out
        const float4 nz = un4(nf.z), nw = un4(nf.w);
        if (t >= 4 * K - 1 && t < rows - 1 && out_lane && (INTERIOR || ys < H)) {
          const size_t g = (size_t)ys * pitch + (size_t)gx;
          const float4 c[4] = {make_float4(nx.x, ny.x, nz.x, nw.x),
                               make_float4(nx.y, ny.y, nz.y, nw.y),
                               make_float4(nx.z, ny.z, nz.z, nw.z),
                               make_float4(nx.w, ny.w, nz.w, nw.w)};
          if constexpr (F16) {
            uint2 h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const __half2 l = __float22half2_rn(fmul2(make_float2(c[k].x, c[k].y), fscale2));
              const __half2 u = __float22half2_rn(fmul2(make_float2(c[k].z, c[k].w), fscale2));
              h[k].x = *reinterpret_cast<const uint32_t*>(&l);
              h[k].y = *reinterpret_cast<const uint32_t*>(&u);
            }
            uint2* fo = reinterpret_cast<uint2*>(f_out) + g;
            if (INTERIOR || cols == 4) {
              store32(fo, __uint_as_float(h[0].x), __uint_as_float(h[0].y),
                      __uint_as_float(h[1].x), __uint_as_float(h[1].y), __uint_as_float(h[2].x),
                      __uint_as_float(h[2].y), __uint_as_float(h[3].x), __uint_as_float(h[3].y));
            } else {  // the grid's last columns
#pragma unroll
              for (int k = 0; k < 3; ++k)
                if (k < cols) fo[k] = h[k];
            }
          } else {
            float4* fo = reinterpret_cast<float4*>(f_out) + g;
            if (INTERIOR || cols == 4) {
              store32(fo, c[0].x, c[0].y, c[0].z, c[0].w, c[1].x, c[1].y, c[1].z, c[1].w);
              store32(fo + 2, c[2].x, c[2].y, c[2].z, c[2].w, c[3].x, c[3].y, c[3].z, c[3].w);
            } else {
#pragma unroll
              for (int k = 0; k < 3; ++k)
                if (k < cols) fo[k] = c[k];
            }
          }
        }
        if (t >= 4 * K && out_lane && (INTERIOR || yd < H)) {
          const size_t g = (size_t)yd * pitch + (size_t)gx;
          const float4 vx = un4(vx_m), vy = un4(sub4(sub4(nf.w, z_m), sub4(Y0, w_m)));
          const float4 d4 = un4(dn);
          if (INTERIOR || cols == 4) {
            *reinterpret_cast<float4*>(d_out + g) = d4;
            store32(v_out + g, vx.x, vy.x, vx.y, vy.y, vx.z, vy.z, vx.w, vy.w);
          } else {
            const float dk[3] = {d4.x, d4.y, d4.z};
            const float2 vk[3] = {make_float2(vx.x, vy.x), make_float2(vx.y, vy.y),
                                  make_float2(vx.z, vy.z)};
#pragma unroll
            for (int k = 0; k < 3; ++k)
              if (k < cols) {
                d_out[g + k] = dk[k];
                v_out[g + k] = vk[k];
              }
          }
        }
        vx_m = pk4(fsub(fsub(ny.y, nx.x), fsub(X0l, ny.x)),
                   fsub(fsub(ny.z, nx.y), fsub(nx.x, ny.y)),
                   fsub(fsub(ny.w, nx.z), fsub(nx.y, ny.z)),
                   fsub(fsub(X1r, nx.w), fsub(nx.z, ny.w)));
        z_mm = z_m;
        z_m = nf.z;
        w_m = nf.w;
      }
    }
  };
  auto extend = [&](const int t) {
    if (!more) return;
    if (t == rows - kSweepClaim) {  // asked for ahead of its use
      if (lane == 0) claim = atomicAdd(word, (unsigned long long)kSweepClaim);
    } else if (t == rows - 2) {
      const unsigned long long w = __shfl_sync(0xffffffffu, claim, 0);
      const int left = range_end(w) - range_cur(w);
      rows += max(0, min(kSweepClaim, left));
      more = left > kSweepClaim;
    }
  };
#pragma unroll 1
  for (int t = 0; t < rows; ++t) {
    row(t);
    extend(t);
  }
  copy_wait<0>();
  __syncwarp();  // every lane has read its last rows: the next unit may refill them
}

// Queue position i -> (strip, band): the units on the grid's border first
// (their cells take the slower edge path, and a launch ends with its slowest
// units), then the interior strip by strip, band by band.
__device__ __forceinline__ void sweep_unit_coords(int i, int S, int B, int& s, int& b) {
  if (S < 3 || B < 3) {
    s = i % S;
    b = i / S;
    return;
  }
  const int ne = 2 * S + 2 * (B - 2);
  if (i < S) {
    s = i;
    b = 0;
  } else if (i < 2 * S) {
    s = i - S;
    b = B - 1;
  } else if (i < 2 * S + (B - 2)) {
    s = 0;
    b = 1 + (i - 2 * S);
  } else if (i < ne) {
    s = S - 1;
    b = 1 + (i - 2 * S - (B - 2));
  } else {
    const int j = i - ne;
    s = 1 + j % (S - 2);
    b = 1 + j / (S - 2);
  }
}

// The bands of a launch: rows [0, tall_end) in bands of `tall` rows (the
// last one may be shorter), then rows [tall_end, H) in bands of `tail` rows.
// Short bands come last in the work queue, so that the launch ends on small
// units; tall bands recompute fewer halo rows per output row.
struct SweepBands {
  int tall, tall_end, tall_count, tail, count;
  int border_sms;  // SMs whose warps start on the units at the grid's border
};

// Band i of a partition with a tail: its first row and its height.
__device__ __forceinline__ void sweep_band(const SweepBands& sb, int H, int i, int& y0, int& R) {
  const bool tall = i < sb.tall_count;
  y0 = tall ? i * sb.tall : sb.tall_end + (i - sb.tall_count) * sb.tail;
  R = min(tall ? sb.tall : sb.tail, (tall ? sb.tall_end : H) - y0);
}

// The units at the grid's border come first in the order of sweep_unit_coords.
__host__ __device__ constexpr int sweep_border_units(int S, int B) {
  return S < 3 || B < 3 ? S * B : 2 * S + 2 * (B - 2);
}

// Two queues, the units at a grid's border and the inner ones.  The two are
// separate code, and warps of both on one SM stall each other on instruction
// fetch (a border unit then takes 1.6 times an inner one's time, against 1.1
// among its like), so the warps of `border_sms` SMs start on the border's units
// and all others on the inner ones; a queue that has run empty hands over to
// the other.  Words of `queue`: the border's next unit, warps done, the inner
// units' next.  4096^2 262 -> 268, 2896^2 213 -> 223, 2048^2 140 -> 154
// Gcell-steps/s against one queue, border first.
__device__ __forceinline__ int sweep_first_queue(int border_sms) {
  unsigned smid;
  asm("mov.u32 %0, %%smid;" : "=r"(smid));
  return (int)smid < border_sms ? 0 : 1;
}
__device__ __forceinline__ int sweep_next(int* queue, int border, int total, int& which,
                                          int& queues, int lane) {
  while (queues > 0) {
    int u = 0;
    if (lane == 0) u = atomicAdd(&queue[2 * which], 1);
    u = __shfl_sync(0xffffffffu, u, 0) + (which ? border : 0);
    if (u < (which ? total : border)) return u;
    which ^= 1;
    --queues;
  }
  return -1;
}

// The last warp to finish resets the queues for the next launch: every other
// warp has made its final claim by then, and the next launch reads them only
// after this grid has completed.
__device__ __forceinline__ void sweep_done(int* queue, int lane) {
  if (lane == 0) {
    __threadfence();
    if (atomicAdd(&queue[1], 1) == (int)(gridDim.x * kSweepWarps) - 1) {
      queue[0] = queue[1] = queue[2] = 0;
      __threadfence();
    }
  }
}

// Persistent warps (one wave): each takes units (strip, band) from the grid's
// queues until none is left, so warps that drew cheap units take more of them.
template <int K, bool F16>
__global__ void __launch_bounds__(kSweepThreads, (K <= 3 ? 3 : 2))
    sweep_kernel(const float* __restrict__ b, const float* __restrict__ d,
                 const void* __restrict__ f, const __grid_constant__ StepArgs a,
                 const SweepBands sb) {
  using RG = SweepRing<K, F16>;
  constexpr int VALID = kSweepCols - 2 * kSweepHaloX(K);
  extern __shared__ __align__(128) unsigned char sweep_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int strips = (a.W + VALID - 1) / VALID;
  const int bands = sb.count;
  const int total = strips * bands;
  // the previous launch on the stream has completed and its writes (the
  // state, and the queue it reset) are visible before any global access
  // (programmatic dependent launch)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  unsigned char* ring = sweep_smem + warp * RG::WARP;
  const int warps = gridDim.x * kSweepWarps, me = blockIdx.x * kSweepWarps + warp;
  unsigned long long* const word = a.ranges + me;
  uint32_t seed = (uint32_t)me;
  const int border = sweep_border_units(strips, bands);
  int which = sweep_first_queue(sb.border_sms), queues = 2;
  for (;;) {
    int si = 0, y0 = 0, y1 = 0;
    const int u = sweep_next(a.queue, border, total, which, queues, lane);
    const bool queued = u >= 0;
    if (queued) {
      int bi, R;
      sweep_unit_coords(u, strips, bands, si, bi);
      sweep_band(sb, a.H, bi, y0, R);
      y1 = y0 + R;
    }
    if (!queued) {
      // the queues are empty: the largest of 64 other warps' ranges, its back half
      bool got = false;
      for (int attempt = 0; attempt < kSweepStealTries && !got; ++attempt) {
        seed = seed * 1664525u + 1013904223u;  // (Numerical Recipes' generator)
        const unsigned v = (unsigned)(((unsigned long long)seed * (unsigned)warps) >> 32);
        unsigned long long w = 0;
        unsigned best = 0;
        unsigned victim = 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          unsigned j = v + lane + 32 * i;
          while (j >= (unsigned)warps) j -= (unsigned)warps;
          const unsigned long long x = *(volatile unsigned long long*)(a.ranges + j);
          const unsigned left = (unsigned)max(0, range_end(x) - range_cur(x));
          if (left > best) best = left, w = x, victim = j;
        }
        const unsigned top = __reduce_max_sync(0xffffffffu, best << 5 | (unsigned)lane);
        if ((int)(top >> 5) < kSweepMinSteal) continue;
        const int from = (int)(top & 31u);
        int mid = 0;
        if (lane == from) {
          const int cur = range_cur(w), end = range_end(w);
          mid = cur + (end - cur + 1) / 2;
          if (atomicCAS(a.ranges + victim, w, range_pack(range_strip(w), cur, mid)) != w) mid = 0;
        }
        mid = __shfl_sync(0xffffffffu, mid, from);
        if (mid == 0) continue;
        w = __shfl_sync(0xffffffffu, w, from);
        si = range_strip(w);
        y0 = mid;
        y1 = range_end(w);
        got = true;
      }
      if (!got) break;  // the whole warp
    }
    // the first rows are this warp's at once, the others can be taken over
    const int R = min(y1 - y0, kSweepClaim);
    const bool share = y1 - y0 > R;
    if (share && lane == 0) atomicExch(word, range_pack(si, y0 + R, y1));
    const int xs = si * VALID - kSweepHaloX(K);
    uint32_t mask = 0;
#pragma unroll
    for (int k = 0; k < TWS_MAX_SOURCES; ++k) {
      if (k < a.nsrc) {
        const DevSource& s = a.src[k];
        if (s.bx1 >= xs && s.bx0 < xs + kSweepCols && s.by1 >= y0 - 2 * K && s.by0 < y1 + 2 * K)
          mask |= 1u << k;
      }
    }
    const bool interior =
        xs >= 0 && xs + kSweepCols <= a.W && y0 - 2 * K >= 0 && y1 + 2 * K <= a.H;
    if (interior)
      sweep_unit<K, F16, true>(a, b, d, f, a.d_out, a.f_out, a.v_out, ring, xs, y0, R, mask,
                               share ? word : nullptr);
    else
      sweep_unit<K, F16, false>(a, b, d, f, a.d_out, a.f_out, a.v_out, ring, xs, y0, R, mask,
                                share ? word : nullptr);
  }
  sweep_done(a.queue, lane);
}

// What a sweep reads of its grid's step arguments, for a grid that a warp of a
// batch's launch drew: the values in registers, the sources in the batch's table.
struct SweepArgs {
  int W, H, pitch;
  float kf, ka, c;
  int closed, nsrc;
  float flux_scale, flux_inv_scale, neg_zero;
  const DevSource* src;
};

// The sweep over the units of many grids, from the same two queues; a taker of
// rows reads which grid they belong to from the unit that they were part of.
// Bound as the single grid's sweep, with more border: 20 FP32 grids of 128 to
// 2048 a side, 32 steps, 3440 -> 2660 us against the two-step tiles (a third of
// the units at borders), 16 of 2048^2, 48 steps, 17635 -> 11100.
template <int K, bool F16>
__global__ void __launch_bounds__(kSweepThreads, (K <= 3 ? 3 : 2))
    batch_sweep_kernel(const BatchGrid* __restrict__ grids, const BatchUnit* __restrict__ units,
                       int launch_idx, int* queue, unsigned long long* ranges) {
  using RG = SweepRing<K, F16>;
  extern __shared__ __align__(128) unsigned char sweep_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  asm volatile("griddepcontrol.wait;" ::: "memory");  // as in sweep_kernel
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  unsigned char* ring = sweep_smem + warp * RG::WARP;
  const int warps = gridDim.x * kSweepWarps, me = blockIdx.x * kSweepWarps + warp;
  unsigned long long* const word = ranges + me;
  uint32_t seed = (uint32_t)me;
  // the first entry: how many units there are, at the borders and in all
  const int4 head = __ldg(reinterpret_cast<const int4*>(units));
  const int4* const table = reinterpret_cast<const int4*>(units) + 1;
  int which = sweep_first_queue(head.z), queues = 2;
  for (;;) {
    int y0 = 0, y1 = 0;
    int u = sweep_next(queue, head.x, head.y, which, queues, lane);
    const bool queued = u >= 0;
    if (!queued) {
      // as in sweep_kernel (shared as a function, the search changed that kernel's
      // register allocation: 4096^2 262 -> 244 Gcell-steps/s)
      bool got = false;
      for (int attempt = 0; attempt < kSweepStealTries && !got; ++attempt) {
        seed = seed * 1664525u + 1013904223u;  // (Numerical Recipes' generator)
        const unsigned v = (unsigned)(((unsigned long long)seed * (unsigned)warps) >> 32);
        unsigned long long w = 0;
        unsigned best = 0;
        unsigned victim = 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          unsigned j = v + lane + 32 * i;
          while (j >= (unsigned)warps) j -= (unsigned)warps;
          const unsigned long long x = *(volatile unsigned long long*)(ranges + j);
          const unsigned left = (unsigned)max(0, range_end(x) - range_cur(x));
          if (left > best) best = left, w = x, victim = j;
        }
        const unsigned top = __reduce_max_sync(0xffffffffu, best << 5 | (unsigned)lane);
        if ((int)(top >> 5) < kSweepMinSteal) continue;
        const int from = (int)(top & 31u);
        int mid = 0;
        if (lane == from) {
          const int cur = range_cur(w), end = range_end(w);
          mid = cur + (end - cur + 1) / 2;
          if (atomicCAS(ranges + victim, w, range_pack(range_strip(w), cur, mid)) != w) mid = 0;
        }
        mid = __shfl_sync(0xffffffffu, mid, from);
        if (mid == 0) continue;
        w = __shfl_sync(0xffffffffu, w, from);
        u = range_strip(w);
        y0 = mid;
        y1 = range_end(w);
        got = true;
      }
      if (!got) break;  // the whole warp
    }
    const int4 un = __ldg(table + u);
    if (launch_idx >= batch_sweep_launches(un.w)) continue;
    const BatchGrid& G = grids[un.x];
    const int p = ((un.w >> 30) + launch_idx) & 1;
    const StepArgs& ga = G.a;
    const SweepArgs a{ga.W,      ga.H,    ga.pitch,      ga.kf,             ga.ka,       ga.c,
                      ga.closed, ga.nsrc, ga.flux_scale, ga.flux_inv_scale, ga.neg_zero, ga.src};
    if (queued) {
      y0 = un.z;
      y1 = min(y0 + batch_sweep_rows(un.w), a.H);
    }
    // the first rows are this warp's at once, the others can be taken over
    const int R = min(y1 - y0, kSweepClaim);
    const bool share = y1 - y0 > R;
    if (share && lane == 0) atomicExch(word, range_pack(u, y0 + R, y1));
    const int xs = un.y - kSweepHaloX(K);
    uint32_t mask = 0;
#pragma unroll
    for (int k = 0; k < TWS_MAX_SOURCES; ++k) {
      if (k < a.nsrc) {
        const DevSource& s = a.src[k];
        if (s.bx1 >= xs && s.bx0 < xs + kSweepCols && s.by1 >= y0 - 2 * K && s.by0 < y1 + 2 * K)
          mask |= 1u << k;
      }
    }
    const bool interior =
        xs >= 0 && xs + kSweepCols <= a.W && y0 - 2 * K >= 0 && y1 + 2 * K <= a.H;
    if (interior)
      sweep_unit<K, F16, true>(a, G.b, G.d[p], G.f[p], G.d[p ^ 1], G.f[p ^ 1], G.v, ring, xs, y0,
                               R, mask, share ? word : nullptr);
    else
      sweep_unit<K, F16, false>(a, G.b, G.d[p], G.f[p], G.d[p ^ 1], G.f[p ^ 1], G.v, ring, xs, y0,
                                R, mask, share ? word : nullptr);
  }
  sweep_done(queue, lane);
}

template <int K>
const void* sweep_fn(int flux_storage) {
  return flux_storage == TWS_FLUX_F16 ? reinterpret_cast<const void*>(&sweep_kernel<K, true>)
                                      : reinterpret_cast<const void*>(&sweep_kernel<K, false>);
}

const void* batch_sweep_fn(int flux_storage) {
  return flux_storage == TWS_FLUX_F16
             ? reinterpret_cast<const void*>(&batch_sweep_kernel<kBatchSweepK, true>)
             : reinterpret_cast<const void*>(&batch_sweep_kernel<kBatchSweepK, false>);
}

// SMs that start on `border` of `units` units: their share of the work, a border
// unit counted as kBorderCost inner ones.
constexpr double kBorderCost = 1.2;
}  // namespace
int sweep_border_sms(long long border, long long units, int sms) {
  const double w = kBorderCost * (double)border;
  return units > 0 ? (int)(w / (w + (double)(units - border)) * sms + 0.5) : 0;
}
namespace {

// One wave of persistent CTAs of a kernel.
cudaError_t sweep_ctas(const void* fn, size_t smem, long long* ctas, int* sm_count) {
  int per_sm = 0, sms = 0;
  const cudaError_t e = kernel_limits(fn, kSweepThreads, smem, &per_sm);
  if (e != cudaSuccess) return e;
  int dev = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    sms = 1;
  *sm_count = sms;
  *ctas = std::min<long long>((long long)per_sm * sms, kSweepMaxWarps / kSweepWarps);
  return cudaSuccess;
}

// A launch that may begin while the previous one on the stream ends.
cudaLaunchConfig_t sweep_config(long long blocks, size_t smem, cudaStream_t s,
                                cudaLaunchAttribute* attr) {
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(kSweepThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

}  // namespace

size_t sweep_smem_bytes(int k, int flux_storage) {
  return (size_t)kSweepWarps * sweep_warp_bytes(k, flux_storage == TWS_FLUX_F16);
}

cudaError_t launch_sweep_step(int k, int rows, int tail_rows, int flux_storage, const float* b,
                              const float* d, const void* f, const StepArgs& a, cudaStream_t s) {
  const void* fn = nullptr;
  switch (k) {
    case 2: fn = sweep_fn<2>(flux_storage); break;
    case 3: fn = sweep_fn<3>(flux_storage); break;
    case 4: fn = sweep_fn<4>(flux_storage); break;
    default: return cudaErrorInvalidValue;
  }
  if (rows < 1 || tail_rows < 0 || !a.queue || !a.ranges) return cudaErrorInvalidValue;
  const size_t smem = sweep_smem_bytes(k, flux_storage);
  long long ctas = 0;
  int sms = 0;
  const cudaError_t e0 = sweep_ctas(fn, smem, &ctas, &sms);
  if (e0 != cudaSuccess) return e0;
  const int valid = kSweepCols - 2 * kSweepHaloX(k);
  const long long strips = (a.W + valid - 1) / valid;
  // Band partition: uniform bands are made taller as long as every resident
  // warp has one; with a tail, about one short unit per resident warp ends the
  // queue (at most half of the rows).
  const long long warps = ctas * kSweepWarps;
  SweepBands sb{};
  sb.tall = rows;
  long long tail_bands = 0;
  if (tail_rows > 0) {
    tail_bands = std::min<long long>((warps + strips - 1) / strips, a.H / (2LL * tail_rows));
  } else if (strips <= warps) {
    const long long per_strip = warps / strips;
    sb.tall = (int)std::max<long long>(rows, (a.H + per_strip - 1) / per_strip);
  }
  sb.tail = tail_rows > 0 ? tail_rows : sb.tall;
  sb.tall_end = a.H - (int)(tail_bands * sb.tail);
  sb.tall_count = (sb.tall_end + sb.tall - 1) / sb.tall;
  sb.count = sb.tall_count + (int)tail_bands;
  const long long units = strips * sb.count;
  sb.border_sms = sweep_border_sms(sweep_border_units((int)strips, sb.count), units, sms);
  if (units > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  // four warps per unit where there are few units: the others take over rows
  const long long blocks = std::min(units, ctas);
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = sweep_config(blocks, smem, s, attr);
  using Fn = void (*)(const float*, const float*, const void*, StepArgs, SweepBands);
  const cudaError_t e =
      cudaLaunchKernelEx(&cfg, reinterpret_cast<Fn>(const_cast<void*>(fn)), b, d, f, a, sb);
  count_launch();
  return e;
}

int batch_sweep_columns() { return sweep_strip_columns(kBatchSweepK); }

cudaError_t batch_sweep_warps(int flux_storage, int* warps, int* sms) {
  long long ctas = 0;
  const cudaError_t e = sweep_ctas(batch_sweep_fn(flux_storage),
                                   sweep_smem_bytes(kBatchSweepK, flux_storage), &ctas, sms);
  *warps = (int)ctas * kSweepWarps;
  return e;
}

cudaError_t launch_batch_sweep(int flux_storage, const BatchGrid* grids, const BatchUnit* units,
                               int entries, int launch_idx, int* queue,
                               unsigned long long* ranges, cudaStream_t s) {
  const void* fn = batch_sweep_fn(flux_storage);
  const size_t smem = sweep_smem_bytes(kBatchSweepK, flux_storage);
  long long ctas = 0;
  int sms = 0;
  const cudaError_t e0 = sweep_ctas(fn, smem, &ctas, &sms);
  if (e0 != cudaSuccess) return e0;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = sweep_config(std::min<long long>(entries, ctas), smem, s, attr);
  using Fn = void (*)(const BatchGrid*, const BatchUnit*, int, int*, unsigned long long*);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, reinterpret_cast<Fn>(const_cast<void*>(fn)),
                                           grids, units, launch_idx, queue, ranges);
  count_launch();
  return e;
}

}  // namespace tws
