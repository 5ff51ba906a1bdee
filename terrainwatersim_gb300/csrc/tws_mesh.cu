// tws_mesh.cu -- grids of up to about a million cells advanced with their whole
// state on chip, spread over all SMs.
//
// One cooperative launch of at most one CTA per SM runs every step of a
// tws_step call.  A CTA owns a tile of the grid and computes a box of
// 64 x 16*RY cells around it: 16 warps stacked in y, RY rows each, two columns
// per lane.  A cell's four outflows and its depth stay in registers for the
// whole launch (RY = 9: the depth in shared memory), its terrain in shared
// memory, so a step touches no global memory:
//
//   outflow (flowUpdate.comp:34-62): x neighbours by warp shuffle, y
//     neighbours in the lane's own registers; the rows at a warp's upper and
//     lower edge come from the next warp through shared memory       barrier
//   depth (flowApply.comp:32-52), the same way                         barrier
//
// The box's outermost two cells go stale with every step, so the tile is the
// box less 2E cells a side and the CTAs exchange every E steps: each writes the
// cells of its tile's border into the inboxes of its (up to eight) neighbours,
// every value in one 8-byte word with the exchange's number, and reads its own
// inbox until every word carries that number.  No fence and no flag stands
// between a value and its reader (with the state buffers, a fence, a flag
// and a second read an exchange took 2.4 to 4.1 us).  Inboxes come in two
// halves used in turn: a word is overwritten two exchanges later, and its
// reader has then sent the exchange in between.  All CTAs are resident
// (cooperative launch), the waits are bounded like those of the tile kernels,
// and a wait that runs out sets the grid's error word.  A CTA takes a whole SM and
// may have to wait for one while another stream's kernels hold it, so the clocks of
// a wait count from when every CTA has begun.
//
// What bounds it: the latency of one step's dependent chain and two barriers on
// the smallest grids, instruction issue on the largest, and the exchange
// (a write to L2 and a read from it, about a microsecond) divided by E.  RY and E are
// chosen per grid from a measured cost model (mesh_shape).
//
// Measured (us per step of long calls, CUDA events, one rain disk; in brackets the
// two-step tiles): 64^2 1.3 (3.1), 256^2 1.6 (3.3), 512^2 2.4 (3.9), 1021 x 763
// 4.8 (6.2), 1024^2 6.2 (7.1).  Four columns per lane (boxes of 128 columns) issue
// less per cell but leave a quarter of the warps' parallelism: 256^2 2.5 against
// 1.4 without rain.
//
// The arithmetic is the tiled kernels', operation for operation.

#include <algorithm>

#include "tws_device.cuh"
#include "tws_internal.h"
#include "tws_pair.cuh"

namespace tws {
namespace {

constexpr int kMeshWarps = 16;
constexpr int kMeshThreads = 32 * kMeshWarps;
constexpr int kMeshCols = 64;
constexpr int kMeshRowBytes = kMeshCols * 4;
constexpr int kMeshBrushes = 2;  // brush sources a launch takes (one shared plane each)
constexpr size_t kMeshHeadBytes = 256;  // of the workspace: the count of CTAs that have begun
// An exchange waits for a neighbour's steps since the last one too, not for a load
// alone, so this much comes on top of the grid's wait limit (about 10 ms; the longest
// exchange of a sound launch takes microseconds).
constexpr long long kMeshExchangeCycles = 20000000;
// How long CTAs wait for others that have no SM yet (about half a minute).
constexpr long long kMeshBeginCycles = 60000000000;

struct MeshArgs {
  const float* b;
  float* d[2];  // the state as the launch finds it, and where the result goes
  void* f[2];
  int tiles_x, tiles_y;
  int hx, hy;    // halo columns and rows of the box
  int every;     // steps between exchanges
  int nsteps;
  int brushes;
  ulonglong2* inbox;  // two halves per CTA, `half` pairs of words each
  int half;
  unsigned epoch;     // number of the last exchange before this launch
  unsigned* begun;    // CTAs that have begun, of this launch and those before it
  unsigned all;       // what it says once all of this launch's have
  // clocks that a wait may take from when all have begun, and longer until then
  long long limit, begin_limit;
};

// Two words of an inbox: each a value and, in its high half, the number of the
// exchange that sent it.  A word is written and read as a whole.
__device__ __forceinline__ void words_store(ulonglong2* p, pair_t v, unsigned number) {
  const float2 f = un(v);
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p),
               "l"(pk(f.x, __uint_as_float(number))), "l"(pk(f.y, __uint_as_float(number)))
               : "memory");
}
__device__ __forceinline__ ulonglong2 words_load(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}

// Shared memory: terrain, depth (RY > 7), the rows that warps hand each other (two
// per warp and phase), the rain's cell hashes, the disks' cells, brush planes, then the stage of the
// cells an exchange brings.
__host__ __device__ constexpr int mesh_plane_bytes(int ry) { return kMeshWarps * ry * kMeshRowBytes; }
__host__ __device__ constexpr bool mesh_depth_shared(int ry) { return ry > 7; }
__host__ __device__ constexpr int mesh_smem_bytes(int ry, int brushes) {
  return mesh_plane_bytes(ry) * (2 + (mesh_depth_shared(ry) ? 1 : 0) + brushes) +
         2 * 2 * kMeshWarps * kMeshRowBytes + TWS_MAX_SOURCES * kMeshThreads * 4;
}
// Pairs of cells around a tile in its box (the box's columns are paired), and the
// inbox positions of a pair: channel * pairs + mesh_pair.
__host__ __device__ constexpr int mesh_pairs(int ry, int hx, int hy) {
  return 2 * hy * (kMeshCols / 2) + hx * (kMeshWarps * ry - 2 * hy);
}
// Position of the pair (row r, column pair c) among those of the box's outer frame,
// its halo (inner = 0), or of the frame inside that, the tile's border (inner = 1).
__device__ __forceinline__ int mesh_pair(int ry, int hx, int hy, int r, int c, int inner) {
  const int rows = kMeshWarps * ry, half = hx / 2, top = inner * hy, side = inner * half;
  if (r < top + hy) return (r - top) * (kMeshCols / 2) + c;
  if (r >= rows - top - hy) return (r - rows + top + 2 * hy) * (kMeshCols / 2) + c;
  return 2 * hy * (kMeshCols / 2) + (r - hy) * hx +
         (c < side + half ? c - side : c - kMeshCols / 2 + side + hx);
}
// One halo position: which of a CTA's border pairs a neighbour has there (-1: no such
// neighbour), and that neighbour's CTA; its sign bit says that no neighbour fills
// the CTA's own position.
struct MeshRoute {
  int src, dst;
};
constexpr int kMeshChannels = 5;  // depth and the four outflows

// After a wait that has run out once: until every CTA of the launch has begun (not
// inlined, nor a part of the waiting loop: with its state there, the steps' registers
// were allocated otherwise and 256^2 took 1655 us for 1000 steps, not 1620).  True
// if some CTA has not.
__device__ __noinline__ bool mesh_begin_runs_out(const unsigned* begun, unsigned all,
                                                 long long limit) {
  const long long t0 = clock64();
  while ((int)(*(const volatile unsigned*)begun - all) < 0)
    if (clock64() - t0 > limit) return true;
  return false;
}

template <int RY, bool F16>
__global__ void __launch_bounds__(kMeshThreads, 1)
    mesh_kernel(const __grid_constant__ StepArgs a, const __grid_constant__ MeshArgs m) {
  constexpr bool DSM = mesh_depth_shared(RY);
  constexpr int PLANE = mesh_plane_bytes(RY);
  extern __shared__ __align__(16) unsigned char mesh_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int W = a.W, H = a.H;
  const size_t pitch = (size_t)a.pitch;
  const int tx = blockIdx.x % m.tiles_x, ty = blockIdx.x / m.tiles_x;
  if (threadIdx.x == 0 && gridDim.x > 1) atomicAdd(m.begun, 1u);
  const int hx = m.hx, hy = m.hy;
  const int row0 = warp * RY;                                // box row of this warp's first row
  const int gx = tx * (kMeshCols - 2 * hx) - hx + 2 * lane;  // this lane's first column
  const int gy0 = ty * (kMeshWarps * RY - 2 * hy) - hy + row0;
  const int cols = gx < 0 ? 0 : min(2, max(0, W - gx));
  const bool closed = a.closed != 0;
  // A CTA whose box lies inside the grid skips the border's rules.  A box without
  // halo rows may end on the grid's first and last row, whose walls it then has; in
  // x every box has halo columns, and one that ends on a wall's column only has
  // it among the cells that go stale.
  const int by = gy0 - row0;
  const bool edge = gx - 2 * lane < 0 || gx - 2 * lane + kMeshCols > W || by <= 0 ||
                    by + kMeshWarps * RY >= H;
  // (the border's rules as bit masks of the lane's two cells: +x outflows, -x
  // outflows and depths that may be nonzero)
  auto cell_mask = [](bool lo, bool hi) {
    return (lo ? 0xffffffffull : 0ull) | (hi ? 0xffffffff00000000ull : 0ull);
  };
  const int wx = closed ? W - 1 : W;  // +x outflow is zero from here on
  const pair_t mask_x = cell_mask(gx < wx, gx >= 0 && gx + 1 < wx);
  const pair_t mask_y = cell_mask(gx < W && !(closed && gx == 0), gx + 1 < W);
  const pair_t mask_d = cell_mask(cols > 0, cols > 1);
  const bool edge_rows = gy0 <= 0 || gy0 + RY >= H;  // this warp's rows touch the border
  const bool col_own = 2 * lane >= hx && 2 * lane < kMeshCols - hx;
  const bool col_border = 2 * lane < 2 * hx || 2 * lane >= kMeshCols - 2 * hx;
  const pair_t kf2 = pk(a.kf, a.kf), ka2 = pk(a.ka, a.ka), cc2 = pk(a.c, a.c);
  const pair_t nz2 = pk(a.neg_zero, a.neg_zero);
  const float2 fscale2 = make_float2(a.flux_scale, a.flux_scale);
  const float2 finv2 = make_float2(a.flux_inv_scale, a.flux_inv_scale);

  // this lane's pair in row i of a plane, and the rows handed between warps
  unsigned char* const own = mesh_smem + (size_t)row0 * kMeshRowBytes + 8 * lane;
  unsigned char* const hand = mesh_smem + mesh_smem_bytes(RY, 0) -
                              TWS_MAX_SOURCES * kMeshThreads * 4 - PLANE -
                              2 * 2 * kMeshWarps * kMeshRowBytes + 8 * lane;
  auto at = [](unsigned char* p) -> pair_t& { return *reinterpret_cast<pair_t*>(p); };
  auto terrain = [&](int i) -> pair_t { return at(own + i * kMeshRowBytes); };
  // phase 0: h, phase 1: outflows; side 0: the warp's first row, 1: its last
  auto hand_row = [&](int phase, int w, int side) -> pair_t& {
    return at(hand + ((phase * kMeshWarps + w) * 2 + side) * kMeshRowBytes);
  };

  pair_t Fx[RY], Fy[RY], Fz[RY], Fw[RY];
  pair_t Dr[DSM ? 1 : RY];
  auto get_d = [&](int i) -> pair_t { return DSM ? at(own + PLANE + i * kMeshRowBytes) : Dr[DSM ? 0 : i]; };
  auto set_d = [&](int i, pair_t v) {
    if constexpr (DSM)
      at(own + PLANE + i * kMeshRowBytes) = v;
    else
      Dr[i] = v;
  };

  // State of the box's cells; cells off the grid keep the zero they are set to.
  // Predicated loads, all rows' in flight together: behind branches each row
  // waited for its own.
  auto load_state = [&](const float* d, const void* f) {
    constexpr int G = F16 ? 3 : RY;  // rows in flight (FP16 needs registers to convert from)
#pragma unroll
    for (int i0 = 0; i0 < RY; i0 += G) {
      uint4 raw[F16 ? G : 1];
#pragma unroll
      for (int i = i0; i < RY && i < i0 + G; ++i) {
        const int y = gy0 + i;
        const bool in = y >= 0 && y < H && cols > 0;
        const int p = in;
        const size_t g = in ? (size_t)y * pitch + (size_t)gx : 0;
        // (an even column's right neighbour lies in the row's padding at worst,
        // which is zero; what is loaded there is masked)
        pair_t dv = get_d(i);
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t"
                     "@q ld.global.b64 %0, [%1];\n\t}"
                     : "+l"(dv)
                     : "l"(d + g), "r"(p)
                     : "memory");
        set_d(i, dv & mask_d);
        if constexpr (F16) {
          raw[i - i0] = make_uint4(0u, 0u, 0u, 0u);
          asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t"
                       "@q ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                       : "+r"(raw[i - i0].x), "+r"(raw[i - i0].y), "+r"(raw[i - i0].z),
                         "+r"(raw[i - i0].w)
                       : "l"(reinterpret_cast<const uint2*>(f) + g), "r"(p)
                       : "memory");
        } else {
          float2 x = un(Fx[i]), yv = un(Fy[i]), z = un(Fz[i]), w = un(Fw[i]);
          asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %9, 0;\n\t"
                       "@q ld.global.f32 %0, [%8];\n\t"
                       "@q ld.global.f32 %1, [%8 + 4];\n\t"
                       "@q ld.global.f32 %2, [%8 + 8];\n\t"
                       "@q ld.global.f32 %3, [%8 + 12];\n\t"
                       "@q ld.global.f32 %4, [%8 + 16];\n\t"
                       "@q ld.global.f32 %5, [%8 + 20];\n\t"
                       "@q ld.global.f32 %6, [%8 + 24];\n\t"
                       "@q ld.global.f32 %7, [%8 + 28];\n\t}"
                       : "+f"(x.x), "+f"(yv.x), "+f"(z.x), "+f"(w.x), "+f"(x.y), "+f"(yv.y),
                         "+f"(z.y), "+f"(w.y)
                       : "l"(reinterpret_cast<const float4*>(f) + g), "r"(p)
                       : "memory");
          Fx[i] = pk(x.x, x.y) & mask_d;
          Fy[i] = pk(yv.x, yv.y) & mask_d;
          Fz[i] = pk(z.x, z.y) & mask_d;
          Fw[i] = pk(w.x, w.y) & mask_d;
        }
      }
      if constexpr (F16) {
#pragma unroll
        for (int i = i0; i < RY && i < i0 + G; ++i) {
          const int y = gy0 + i;
          const bool in = y >= 0 && y < H && cols > 0;
          const uint4 r = raw[i - i0];
          const float2 a0 = fmul2(__half22float2(*reinterpret_cast<const __half2*>(&r.x)), finv2);
          const float2 a1 = fmul2(__half22float2(*reinterpret_cast<const __half2*>(&r.y)), finv2);
          const float2 b0 = fmul2(__half22float2(*reinterpret_cast<const __half2*>(&r.z)), finv2);
          const float2 b1 = fmul2(__half22float2(*reinterpret_cast<const __half2*>(&r.w)), finv2);
          Fx[i] = in ? pk(a0.x, b0.x) : Fx[i];
          Fy[i] = in ? pk(a0.y, b0.y) : Fy[i];
          Fz[i] = in ? pk(a1.x, b1.x) : Fz[i];
          Fw[i] = in ? pk(a1.y, b1.y) : Fw[i];
        }
      }
    }
  };
  // depth and flux of row i to the state buffers
  auto store_state = [&](int i, float* d, void* f) {
    const size_t g = (size_t)(gy0 + i) * pitch + (size_t)gx;
    const float2 dv = un(get_d(i)), x = un(Fx[i]), y = un(Fy[i]), z = un(Fz[i]), w = un(Fw[i]);
    if (cols > 1)
      *reinterpret_cast<float2*>(d + g) = dv;
    else
      d[g] = dv.x;
    if constexpr (F16) {
      const __half2 p0 = __float22half2_rn(fmul2(make_float2(x.x, y.x), fscale2));
      const __half2 q0 = __float22half2_rn(fmul2(make_float2(z.x, w.x), fscale2));
      const __half2 p1 = __float22half2_rn(fmul2(make_float2(x.y, y.y), fscale2));
      const __half2 q1 = __float22half2_rn(fmul2(make_float2(z.y, w.y), fscale2));
      uint4 r;
      r.x = *reinterpret_cast<const uint32_t*>(&p0);
      r.y = *reinterpret_cast<const uint32_t*>(&q0);
      r.z = *reinterpret_cast<const uint32_t*>(&p1);
      r.w = *reinterpret_cast<const uint32_t*>(&q1);
      uint2* fo = reinterpret_cast<uint2*>(f) + g;
      if (cols > 1)
        *reinterpret_cast<uint4*>(fo) = r;
      else
        *fo = make_uint2(r.x, r.y);
    } else {
      float4* fo = reinterpret_cast<float4*>(f) + g;
      fo[0] = make_float4(x.x, y.x, z.x, w.x);
      if (cols > 1) fo[1] = make_float4(x.y, y.y, z.y, w.y);
    }
  };
  auto row_own = [&](int i) {  // row i of this warp is the tile's, and on the grid
    const int r = row0 + i, y = gy0 + i;
    return r >= hy && r < kMeshWarps * RY - hy && y >= 0 && y < H;
  };

  // ---- sources.  What does not depend on the depth is worked out once: for a
  // disk the cells of this lane that lie in it (two bits a row), for a brush its
  // increments (a plane), and the part of the rain's hash that the cell gives.
  uint32_t reach = 0;  // sources that reach the box
  uint32_t* const in_disk = reinterpret_cast<uint32_t*>(mesh_smem + mesh_smem_bytes(RY, 0)) -
                            TWS_MAX_SOURCES * kMeshThreads + threadIdx.x;
  unsigned char* const hash0 = own + mesh_smem_bytes(RY, 0) -
                               TWS_MAX_SOURCES * kMeshThreads * 4 - PLANE;
  unsigned char* const inc0 = own + mesh_smem_bytes(RY, 0);
  {
    int plane = 0;
    for (int k = 0; k < a.nsrc; ++k) {
      const DevSource& s = a.src[k];
      const int pl = plane;
      if (s.kind != TWS_SOURCE_DISK) ++plane;
      if (s.bx1 < gx - 2 * lane || s.bx0 >= gx - 2 * lane + kMeshCols || s.by1 < by ||
          s.by0 >= by + kMeshWarps * RY)
        continue;
      reach |= 1u << k;
      uint32_t bits = 0;
#pragma unroll 1
      for (int i = 0; i < RY; ++i) {
        float q[2] = {0.0f, 0.0f};
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int x = gx + c, y = gy0 + i;
          if (c >= cols || y < 0 || y >= H || x < s.bx0 || x > s.bx1 || y < s.by0 || y > s.by1)
            continue;
          if (s.kind == TWS_SOURCE_DISK) {
            const long long dx = x - s.icx, dy = y - s.icy;
            if (dx * dx + dy * dy <= (long long)s.ir * s.ir) bits |= 1u << (2 * i + c);
          } else {
            const float ax = fsub(s.cx, (float)x), ay = fsub(s.cy, (float)y);
            const float t = fdiv(fadd(fmul(ax, ax), fmul(ay, ay)), s.radius);
            q[c] = fmul(saturate01(fsub(1.0f, t)), s.rate);
          }
        }
        if (s.kind != TWS_SOURCE_DISK) {
          if (q[0] != 0.0f || q[1] != 0.0f) bits |= 3u << (2 * i);
          at(inc0 + pl * PLANE + i * kMeshRowBytes) = pk(q[0], q[1]);
        }
      }
      in_disk[k * kMeshThreads] = bits;
    }
    if (reach) {
#pragma unroll 1
      for (int i = 0; i < RY; ++i) {
        const uint32_t hy32 = rain_hash32((uint32_t)(gy0 + i));
        at(hash0 + i * kMeshRowBytes) = pk(__uint_as_float(rain_hash32((uint32_t)gx ^ hy32)),
                                           __uint_as_float(rain_hash32((uint32_t)(gx + 1) ^ hy32)));
      }
    }
  }
  // (a CTA under rain is the one that its neighbours wait for)
  auto sources = [&]() {
    int plane = 0;
#pragma unroll 1
    for (int k = 0; k < a.nsrc; ++k) {
      const bool disk = a.src[k].kind == TWS_SOURCE_DISK;
      const int pl = plane;
      if (!disk) ++plane;
      if (!((reach >> k) & 1u)) continue;
      const uint32_t bits = in_disk[k * kMeshThreads];
      if (!__any_sync(0xffffffffu, bits != 0u)) continue;
      const float rate = a.src[k].rate;
#pragma unroll
      for (int i = 0; i < RY; ++i) {
        if (!__any_sync(0xffffffffu, (bits >> (2 * i)) & 3u)) continue;
        if (disk) {
          const float2 ch = un(at(hash0 + i * kMeshRowBytes));
          set_d(i, rain2(get_d(i), rate, __float_as_uint(ch.x), __float_as_uint(ch.y),
                         (bits >> (2 * i)) & 1u, (bits >> (2 * i + 1)) & 1u));
        } else {
          const float2 inc = un(at(inc0 + pl * PLANE + i * kMeshRowBytes)), d = un(get_d(i));
          set_d(i, pk(inc.x != 0.0f ? fadd(d.x, inc.x) : d.x, inc.y != 0.0f ? fadd(d.y, inc.y) : d.y));
        }
      }
    }
  };

  // ---- the exchange's stages and routes
  const int pairs = mesh_pairs(RY, hx, hy);
  unsigned char* const stage = mesh_smem + mesh_smem_bytes(RY, m.brushes);
  unsigned char* const gather = stage + 8 * kMeshChannels * pairs;
  MeshRoute* const route = reinterpret_cast<MeshRoute*>(gather + 8 * kMeshChannels * pairs);
  for (int q = threadIdx.x; q < pairs; q += kMeshThreads) {
    // the halo position q as (row r, column pair c), and the direction (dx, dy)
    // from which a box takes it
    constexpr int C = kMeshCols / 2, ROWS = kMeshWarps * RY;
    int r, c;
    if (q < 2 * hy * C) {
      r = q / C;
      c = q - r * C;
      if (r >= hy) r += ROWS - 2 * hy;
    } else {
      const int t = q - 2 * hy * C;
      r = hy + t / hx;
      c = t % hx;
      if (c >= hx / 2) c += C - hx;
    }
    const int dx = c < hx / 2 ? -1 : (c >= C - hx / 2 ? 1 : 0);
    const int dy = r < hy ? -1 : (r >= ROWS - hy ? 1 : 0);
    auto exists = [&](int x, int y) { return x >= 0 && x < m.tiles_x && y >= 0 && y < m.tiles_y; };
    MeshRoute e{-1, 0};
    if (exists(tx - dx, ty - dy) && !a.drop_loads) {  // (the test hook sends nothing)
      e.src = mesh_pair(RY, hx, hy, r - dy * (ROWS - 2 * hy), c - dx * (C - hx), 1);
      e.dst = (ty - dy) * m.tiles_x + tx - dx;
    }
    if (!exists(tx + dx, ty + dy)) e.dst |= (int)0x80000000;
    route[q] = e;
  }

  // ---- the box's state
#pragma unroll
  for (int i = 0; i < RY; ++i) {
    const int y = gy0 + i;
    pair_t b = 0;
    if (y >= 0 && y < H && cols > 0) {
      const float2 v = __ldg(reinterpret_cast<const float2*>(m.b + (size_t)y * pitch + (size_t)gx));
      b = pk(v.x, cols > 1 ? v.y : 0.0f);
    }
    at(own + i * kMeshRowBytes) = b;
    set_d(i, 0);
    Fx[i] = Fy[i] = Fz[i] = Fw[i] = 0;
  }
  load_state(m.d[0], m.f[0]);

  unsigned epoch = m.epoch;
  for (int done = 0; done < m.nsteps;) {
    const int until = min(m.nsteps, done + m.every);
    for (; done < until; ++done) {
      const bool last = done + 1 == m.nsteps;
      if (reach) sources();
      // ---- outflows, flowUpdate.comp:34-62
      const pair_t h_first = add2(get_d(0), terrain(0));
      hand_row(0, warp, 0) = h_first;
      hand_row(0, warp, 1) = RY > 1 ? add2(get_d(RY - 1), terrain(RY - 1)) : h_first;
      __syncthreads();
      const pair_t h_up = warp > 0 ? hand_row(0, warp - 1, 1) : 0;
      const pair_t h_down = warp + 1 < kMeshWarps ? hand_row(0, warp + 1, 0) : 0;
      pair_t hc = h_first;
      pair_t qm = prod2(sub2(h_up, hc), ka2, nz2);
#pragma unroll
      for (int i = 0; i < RY; ++i) {
        const pair_t dc = get_d(i);
        const pair_t hp = i + 1 < RY ? add2(get_d(i + 1 < RY ? i + 1 : 0), terrain(i + 1)) : h_down;
        const pair_t qp = prod2(sub2(hc, hp), ka2, nz2);
        // neighbouring cells share the slope term of their common edge
        const float2 h2 = un(hc);
        const float hr = __shfl_down_sync(0xffffffffu, h2.x, 1);
        const pair_t qx = prod2(pk(fsub(h2.x, h2.y), fsub(h2.y, hr)), ka2, nz2);
        const float2 q2 = un(qx);
        const float ql = __shfl_up_sync(0xffffffffu, q2.y, 1);
        pair_t nx = max0p(add2(prod2(Fx[i], kf2, nz2), qx));
        const float2 fy = un(prod2(Fy[i], kf2, nz2));
        pair_t ny = pk(max0_fast(fsub(fy.x, ql)), max0_fast(fsub(fy.y, q2.x)));
        pair_t nz = max0p(add2(prod2(Fz[i], kf2, nz2), qp));
        pair_t nw = max0p(sub2(prod2(Fw[i], kf2, nz2), qm));
        if (edge) {
          // what cells on the grid read of cells off it is zero, and so is
          // the outflow across a closed wall
          nx &= mask_x;
          ny &= mask_y;
          if (edge_rows) {
            const int y = gy0 + i;
            if (y < 0 || y >= H) nz = nw = 0;
            if (closed && y == H - 1) nz = 0;
            if (closed && y == 0) nw = 0;
          }
        }
        // (outflow_factors2 with -t negated, not a second product: with that function
        // 200 steps on 1021 x 763 take 980 us, not 960)
        const pair_t sum = add2(add2(add2(nx, ny), nz), nw);
        const pair_t tq = prod2(sum, cc2, nz2);
        const float2 t = un(tq), d = un(dc);
        const bool over0 = t.x > d.x, over1 = t.y > d.y;
        float f0 = over0 ? d.x : 1.0f, f1 = over1 ? d.y : 1.0f;
        const bool div0 = over0 & (d.x != 0.0f), div1 = over1 & (d.y != 0.0f);
        if (div0 | div1) {
          const bool far = (fmaxf(t.x, t.y) > kDivMaxT) | (div0 & (d.x < kDivMinD)) |
                           (div1 & (d.y < kDivMinD));
          if (!far) {
            const float2 q = un(div2(dc, tq, pk(-t.x, -t.y)));
            f0 = div0 ? q.x : f0;
            f1 = div1 ? q.y : f1;
          } else {
            if (div0) f0 = fdiv(d.x, t.x);
            if (div1) f1 = fdiv(d.y, t.y);
          }
        }
        const pair_t sc = pk(f0, f1);
        nx = prod2(nx, sc, nz2);
        ny = prod2(ny, sc, nz2);
        nz = prod2(nz, sc, nz2);
        nw = prod2(nw, sc, nz2);
        if constexpr (F16) {
          auto quant = [&](pair_t v) {
            const float2 o = quantize_f16x2(un(v), fscale2, finv2);
            return pk(o.x, o.y);
          };
          nx = quant(nx);
          ny = quant(ny);
          nz = quant(nz);
          nw = quant(nw);
        }
        Fx[i] = nx;
        Fy[i] = ny;
        Fz[i] = nz;
        Fw[i] = nw;
        hc = hp;
        qm = qp;
      }
      // ---- depths and flow map, flowApply.comp:32-52
      hand_row(1, warp, 0) = Fw[0];
      hand_row(1, warp, 1) = Fz[RY - 1];
      __syncthreads();
      const pair_t z_up = warp > 0 ? hand_row(1, warp - 1, 1) : 0;
      const pair_t w_down = warp + 1 < kMeshWarps ? hand_row(1, warp + 1, 0) : 0;
#pragma unroll
      for (int i = 0; i < RY; ++i) {
        const pair_t Y0 = i > 0 ? Fz[i > 0 ? i - 1 : 0] : z_up;
        const pair_t Y1 = i + 1 < RY ? Fw[i + 1 < RY ? i + 1 : 0] : w_down;
        const float2 nx = un(Fx[i]), ny = un(Fy[i]);
        const float X1r = __shfl_down_sync(0xffffffffu, ny.x, 1);
        const float X0l = __shfl_up_sync(0xffffffffu, nx.y, 1);
        const pair_t in_x = pk(fadd(ny.y, X0l), fadd(X1r, nx.x));
        const pair_t sum = add2(add2(add2(Fx[i], Fy[i]), Fz[i]), Fw[i]);
        const pair_t in = add2(add2(in_x, Y1), Y0);
        pair_t dn = max0p(add2(get_d(i), prod2(sub2(in, sum), cc2, nz2)));
        if (edge) {  // cells off the grid stay empty
          dn &= mask_d;
          if (edge_rows && (gy0 + i < 0 || gy0 + i >= H)) dn = 0;
        }
        set_d(i, dn);
        if (last && col_own && cols > 0 && row_own(i)) {
          const float2 vx = make_float2(fsub(fsub(ny.y, nx.x), fsub(X0l, ny.x)),
                                        fsub(fsub(X1r, nx.y), fsub(nx.x, ny.y)));
          const float2 vy = un(sub2(sub2(Y1, Fz[i]), sub2(Y0, Fw[i])));
          float2* vo = a.v_out + (size_t)(gy0 + i) * pitch + (size_t)gx;
          if (cols > 1)
            *reinterpret_cast<float4*>(vo) = make_float4(vx.x, vy.x, vx.y, vy.y);
          else
            *vo = make_float2(vx.x, vy.x);
        }
      }
    }
    if (done == m.nsteps) break;

    // ---- exchange: the tile's border cells, gathered in shared memory, into the
    // neighbours' inboxes, all threads side by side
    ++epoch;
#pragma unroll
    for (int i = 0; i < RY; ++i) {
      const int r = row0 + i;
      const bool row_border = r < 2 * hy || r >= kMeshWarps * RY - 2 * hy;
      if (col_own && r >= hy && r < kMeshWarps * RY - hy && (row_border || col_border)) {
        unsigned char* const w = gather + 8 * mesh_pair(RY, hx, hy, r, lane, 1);
        at(w) = get_d(i);
        at(w + 8 * pairs) = Fx[i];
        at(w + 16 * pairs) = Fy[i];
        at(w + 24 * pairs) = Fz[i];
        at(w + 32 * pairs) = Fw[i];
      }
    }
    __syncthreads();
    ulonglong2* const part = m.inbox + ((epoch & 1u) ? m.half : 0);
    for (int q = threadIdx.x; q < pairs; q += kMeshThreads) {
      const MeshRoute e = route[q];
      if (e.src >= 0) {
        ulonglong2* const to = part + (size_t)(e.dst & 0x7fffffff) * 2 * m.half + q;
#pragma unroll
        for (int ch = 0; ch < kMeshChannels; ++ch)
          words_store(to + ch * pairs, at(gather + 8 * (ch * pairs + e.src)), epoch);
      }
    }
    // ---- and the own inbox into shared memory
    bool late = false;
    const ulonglong2* const own_part = part + (size_t)blockIdx.x * 2 * m.half;
    for (int q = threadIdx.x; q < pairs && !late; q += kMeshThreads) {
      if (route[q].dst < 0) continue;
      ulonglong2 w[kMeshChannels];
      for (int period = 0;; ++period) {  // the second one: from the last CTA's begin
        bool all = false;
        const long long t0 = clock64();
        do {
#pragma unroll
          for (int ch = 0; ch < kMeshChannels; ++ch) w[ch] = words_load(own_part + ch * pairs + q);
          all = true;
#pragma unroll
          for (int ch = 0; ch < kMeshChannels; ++ch)
            all &= (unsigned)(w[ch].x >> 32) == epoch && (unsigned)(w[ch].y >> 32) == epoch;
        } while (!all && clock64() - t0 <= m.limit);
        if (all) break;
        if (period > 0 || mesh_begin_runs_out(m.begun, m.all, m.begin_limit)) {
          late = true;
          break;
        }
      }
#pragma unroll
      for (int ch = 0; ch < kMeshChannels; ++ch)
        at(stage + 8 * (ch * pairs + q)) = pk(un(w[ch].x).x, un(w[ch].y).x);
    }
    if (__syncthreads_or(late)) {  // every thread leaves together
      if (threadIdx.x == 0) atomicExch(a.err, kDevErrWaitTimeout);
      return;
    }
#pragma unroll
    for (int i = 0; i < RY; ++i) {
      const int r = row0 + i, y = gy0 + i;
      if (!(col_own && r >= hy && r < kMeshWarps * RY - hy) && y >= 0 && y < H && cols > 0) {
        unsigned char* const w = stage + 8 * mesh_pair(RY, hx, hy, r, lane, 0);
        set_d(i, at(w));
        Fx[i] = at(w + 8 * pairs);
        Fy[i] = at(w + 16 * pairs);
        Fz[i] = at(w + 24 * pairs);
        Fw[i] = at(w + 32 * pairs);
      }
    }
    // (gather and stage are written again only after the next steps' barriers)
  }
#pragma unroll
  for (int i = 0; i < RY; ++i)
    if (col_own && cols > 0 && row_own(i)) store_state(i, m.d[1], m.f[1]);
}

using MeshFn = void (*)(const StepArgs, const MeshArgs);
constexpr int kMeshRows[] = {1, 2, 3, 4, 5, 7, 9};

MeshFn mesh_fn(int ry, int flux_storage) {
  const bool h = flux_storage == TWS_FLUX_F16;
  switch (ry) {
    case 1: return h ? mesh_kernel<1, true> : mesh_kernel<1, false>;
    case 2: return h ? mesh_kernel<2, true> : mesh_kernel<2, false>;
    case 3: return h ? mesh_kernel<3, true> : mesh_kernel<3, false>;
    case 4: return h ? mesh_kernel<4, true> : mesh_kernel<4, false>;
    case 5: return h ? mesh_kernel<5, true> : mesh_kernel<5, false>;
    case 7: return h ? mesh_kernel<7, true> : mesh_kernel<7, false>;
    case 9: return h ? mesh_kernel<9, true> : mesh_kernel<9, false>;
    default: return nullptr;
  }
}

// all shared memory of a launch
int mesh_launch_smem(const MeshShape& s) {
  return mesh_smem_bytes(s.ry, s.brushes) +
         (2 * kMeshChannels * 8 + (int)sizeof(MeshRoute)) * mesh_pairs(s.ry, s.hx, s.hy);
}

int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    return cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? v : 0;
  }();
  return n;
}

}  // namespace

bool mesh_shape(int W, int H, int brushes, MeshShape* out) {
  if (W < 1 || H < 1 || brushes > kMeshBrushes) return false;
  const int sms = std::min(sm_count(), kMeshMaxCtas);
  double best = 1e30;
  for (int ry : kMeshRows) {
    for (int e : {1, 2, 4, 6, 8}) {  // (odd ones: the exchange costs up to 1.2 us more)
      MeshShape s{};
      s.ry = ry;
      s.every = e;
      s.hx = 2 * e;
      s.hy = 2 * e;
      if (W <= kMeshCols - 4) s.hx = 2;  // one tile: only the empty columns around the grid
      if (H <= kMeshWarps * ry) s.hy = 0;
      const int ow = kMeshCols - 2 * s.hx, oh = kMeshWarps * ry - 2 * s.hy;
      // (a box's halo comes from the adjacent tiles alone)
      if (ow < 8 || oh < 1 || oh < s.hy || ow < s.hx) continue;
      s.brushes = brushes;
      if (mesh_launch_smem(s) > 227 * 1024) continue;
      s.tiles_x = (W + ow - 1) / ow;
      s.tiles_y = (H + oh - 1) / oh;
      if ((long long)s.tiles_x * s.tiles_y > sms) continue;
      const bool alone = s.tiles_x * s.tiles_y == 1;
      // microseconds per step, fitted to all shapes of 64^2 to 1024^2 grids (0.05
      // off on average): a step's own time, and an exchange's, which grows
      // with the cells it moves
      const double cost = 0.3 + 0.27 * ry + 0.01 * ry * ry +
                          (alone ? 0.0 : (1.3 + 0.28 * ry + 0.3 * std::max(0, e - 2)) / e);
      if (cost < best) {
        best = cost;
        *out = s;
      }
    }
  }
  return best < 1e30;
}

size_t mesh_inbox_bytes(const MeshShape& s) {
  return kMeshHeadBytes + sizeof(ulonglong2) * 2 * kMeshChannels * mesh_pairs(s.ry, s.hx, s.hy) * s.tiles_x *
         s.tiles_y;
}

cudaError_t launch_mesh(const MeshShape& s, int flux_storage, const float* b, float* const d[2],
                        void* const f[2], const StepArgs& a, int nsteps, void* inbox,
                        unsigned epoch, unsigned begun, cudaStream_t st) {
  MeshFn fn = mesh_fn(s.ry, flux_storage);
  if (!fn || nsteps < 1 || !inbox) return cudaErrorInvalidValue;
  const int smem = mesh_launch_smem(s);
  int per_sm = 0;  // (one: the cooperative launch checks it)
  const cudaError_t limit =
      kernel_limits(reinterpret_cast<const void*>(fn), kMeshThreads, (size_t)smem, &per_sm);
  if (limit != cudaSuccess) return limit;
  MeshArgs m{};
  m.b = b;
  for (int i = 0; i < 2; ++i) {
    m.d[i] = d[i];
    m.f[i] = f[i];
  }
  m.tiles_x = s.tiles_x;
  m.tiles_y = s.tiles_y;
  m.hx = s.hx;
  m.hy = s.hy;
  const bool alone = s.tiles_x * s.tiles_y == 1;
  m.every = alone ? nsteps : s.every;
  m.nsteps = nsteps;
  m.brushes = s.brushes;
  m.begun = static_cast<unsigned*>(inbox);
  m.all = begun + (unsigned)mesh_ctas(s);
  m.limit = std::min(a.wait_cycles, (long long)1 << 60) + kMeshExchangeCycles;
  m.begin_limit = kMeshBeginCycles;
  m.inbox = reinterpret_cast<ulonglong2*>(static_cast<char*>(inbox) + kMeshHeadBytes);
  m.half = kMeshChannels * mesh_pairs(s.ry, s.hx, s.hy);
  m.epoch = epoch;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(s.tiles_x * s.tiles_y));
  cfg.blockDim = dim3(kMeshThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = alone ? 0 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, a, m);
  if (e == cudaSuccess) count_launch();
  return e;
}

int mesh_exchanges(const MeshShape& s, int nsteps) {
  return s.tiles_x * s.tiles_y == 1 ? 0 : (nsteps + s.every - 1) / s.every - 1;
}

}  // namespace tws
