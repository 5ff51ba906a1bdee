// tws_internal.h -- shared declarations of the libtws implementation.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/tws.h"
#include "../../include/tws_testing.h"

namespace tws {

// ---------------------------------------------------------------------------
// Per-step source in the form the kernels read (bounding box precomputed).
struct DevSource {
  int kind;
  float cx, cy, radius, rate;
  int icx, icy, ir;    // DISK: integer centre and radius
  int bx0, by0, bx1, by1;  // inclusive bounding box of the cells it can touch
};

// Everything a step launch needs besides the tensor maps.
struct StepArgs {
  int W, H, pitch;
  float kf, ka, c;
  int closed;
  int nsrc;
  DevSource src[TWS_MAX_SOURCES];
  float* d_out;
  void* f_out;
  float2* v_out;
  float flux_scale;      // F16 storage: stored = f * flux_scale
  float flux_inv_scale;  // F16 storage: f = stored * flux_inv_scale
  float neg_zero;        // -0.0f, as data: a product formed as a * b + (-0) keeps its own
                         // rounding whatever the assembler does with a sum it feeds
  int* err;              // device error word (bounded-wait time-outs)
  long long wait_cycles; // bounded waits give up after this many SM clocks
  int drop_loads;        // test hook: tile loads arm their barrier but issue no copy
  int* queue;            // the sweep kernel's work queues: next border unit, warps done,
                         // next inner unit (zero between launches; the last warp of a
                         // launch resets them)
  unsigned long long* ranges;  // the sweep kernel's unclaimed rows, one word per resident
                         // warp (empty between launches)
};

// Kernel variants (temporal block depth K x tile).
struct StepVariant {
  int k;      // steps per launch
  int tx, ty; // interior tile
  int stages; // 1: one CTA per tile; 2: persistent CTAs, next tile prefetched
  int kind;   // kKindTile (TMA-staged tiles), kKindStream (register streaming, K = 1)
              // or kKindSweep (row sweep over column strips, K time levels in registers)
  int ry;     // kKindStream, kKindSweep: rows per warp strip
  int hx;     // x halo of the b/d boxes (2K rounded up to 4 floats)
  int bw, bh; // b/d box
  int fw, fh; // flux box
  int sw;     // F16 staging width in cells (whole pairs)
  int uni;    // unified layout: the flux box is the b/d box
  int ry_tail; // kKindSweep: rows of the short bands that end the work queue (0: none)
  size_t smem;
};

enum : int { kKindTile = 0, kKindStream = 1, kKindSweep = 2 };

// One member grid of a batch as the batched kernel reads it from device
// memory: its tensor maps, its step arguments and its buffers.  The maps are
// not in this table (which the host rewrites between chains) but in a block
// of the grid's own memory written once per kernel variant: tm[0] terrain,
// tm[1 + i] depth buffer i, tm[3 + i] flux buffer i.  A CTA makes the
// tensor-map proxy re-read them (an acquire fence, which costs a descriptor
// fetch per tile) only in the first chain after they were written: `fence`.
struct alignas(16) BatchGrid {
  const CUtensorMap* tm;
  int fence;
  int pad0_;
  StepArgs a;     // W, H, pitch, constants, sources, flux scale, error word
  const float* b;
  float* d[2];
  void* f[2];
  float2* v;
  // The kernel takes both from the unit records; here they make a changed
  // chain compare unequal with the table the device holds.
  int cur;        // buffer holding the state when the chain starts
  int launches;   // launches of this chain that advance this grid
};

// One work unit (tile) of a batched launch, as the batched kernel reads it:
// its grid (index into the BatchGrid table), tile origin, and meta =
// launches this chain gives the grid | (the grid's buffer parity at the chain
// start) << 30.  Entries past the chain's units have meta = 0.
// A unit of a batched sweep: x0 is its strip's first output column, and meta
// holds the unit's rows as well: launches | rows << 8 | parity << 30.  Its table
// begins with an entry of counts: units at the members' borders (they come
// first), all units, SMs that start on the border's.
struct BatchUnit {
  int grid, x0, y0, meta;
};
constexpr int kBatchSweepK = 3;  // steps per launch
constexpr int kBatchSweepMinRows = 16;
constexpr int kBatchSweepMaxLaunches = 255;
__host__ __device__ constexpr int batch_sweep_meta(int launches, int rows, int cur) {
  return launches | rows << 8 | cur << 30;
}
__host__ __device__ constexpr int batch_sweep_launches(int meta) { return meta & 0xff; }
__host__ __device__ constexpr int batch_sweep_rows(int meta) { return meta >> 8 & 0x3fffff; }

// Batched kernel variants (K steps per launch, tile) and their launcher.
// Launch `launch_idx` of a chain runs CTA u on units[u] (`blocks` CTAs, at
// least the chain's units) and advances a grid iff launch_idx < its launches.
int batch_variant_count();
int batch_variant_default();  // two steps per launch, unified 32x32 tiles
int batch_variant_sweep();    // the batched row sweep, three steps per launch
// A batch without a set variant takes the sweep from this many cells on, where its
// strips waste little more than the tiles (us for 48 steps with one disk a grid, sweep
// against tiles: 6 x 1024^2, below the line, 1749 (1818), 8 x 1024^2 2208 (2387), 32
// steps of 20 grids of 128 to 2048 a side 2830 (3437); FP16 24 x 1024^2 5896 (6179),
// 128 x 512^2 8757 (8752), 8 x 2048^2 6704 (7974)).  The line leaves room for sources:
// with two large disks a grid the tiles still lead on 8 x 1024^2 (sweep_is_faster).
constexpr long long kBatchSweepCells = 8LL << 20;
constexpr long long kBatchSweepF16Cells = 24LL << 20;
void batch_variant_info(int i, int* k, int* tx, int* ty, int* step_variant);
cudaError_t prepare_batch_variant(int variant, int flux_storage);  // outside any capture
cudaError_t launch_batch_step(int variant, int flux_storage, const BatchGrid* grids,
                              const BatchUnit* units, int launch_idx, int blocks, cudaStream_t s);
// tws_sweep.cu: the batched row sweep.  Its units are strips of
// batch_sweep_columns() columns in bands of rows; `queue` and `ranges` as in
// StepArgs, the batch's own.
int batch_sweep_columns();
cudaError_t batch_sweep_warps(int flux_storage, int* warps, int* sms);  // resident warps
cudaError_t launch_batch_sweep(int flux_storage, const BatchGrid* grids, const BatchUnit* units,
                               int entries, int launch_idx, int* queue,
                               unsigned long long* ranges, cudaStream_t s);
// SMs whose warps start on the units at the grids' borders
int sweep_border_sms(long long border, long long units, int sms);

// Device error codes written to StepArgs::err.
enum : int { kDevErrNone = 0, kDevErrWaitTimeout = 1 };

// Default limit of a bounded tile-load wait: about two seconds at 2 GHz, far
// beyond any real load, short enough that a lost load ends the kernel.
constexpr long long kDefaultWaitCycles = 4000000000LL;

// Host helpers implemented in tws_step.cu.
// Raises the kernel's shared memory limit on the current device to `smem` bytes, and
// the CTAs of `threads` threads that an SM then holds; both asked once per device.
cudaError_t kernel_limits(const void* fn, int threads, size_t smem, int* ctas_per_sm);
int step_variant_count();
const StepVariant& step_variant(int i);
constexpr long long kSmallStepTiles = 4096;  // of 32 x 32 cells
int step_variant_for(int k, int flux_storage, int W, int H);
// The automatic choice for grids of at least kLargeGridCells cells (FP16
// flux: kLargeF16Cells), or -1 (smaller ones).
constexpr long long kLargeGridCells = 7LL << 20;
constexpr long long kLargeF16Cells = 17LL << 20;
int step_variant_large_grid(int flux_storage, int W, int H);
// Tile variants read through the tensor maps, stream variants through the
// raw pointers (b, d, f of the current state).
cudaError_t launch_step(int variant, int flux_storage, const CUtensorMap* tm_b,
                        const CUtensorMap* tm_d, const CUtensorMap* tm_f, const float* b,
                        const float* d, const void* f, const StepArgs& a, cudaStream_t s);
// tws_sweep.cu: K = 2..4 steps per launch, bands of `rows` rows (the last bands
// `tail_rows` rows when it is above 0; with none, taller where every resident
// warp still gets a band)
cudaError_t launch_sweep_step(int k, int rows, int tail_rows, int flux_storage, const float* b,
                              const float* d, const void* f, const StepArgs& a, cudaStream_t s);
constexpr int kSweepCtaThreads = 128;  // four warps, each its own sweep
constexpr int kSweepMaxWarps = 4096;   // warps of a sweep launch (words of StepArgs::ranges)
constexpr int kSweepMaxUnits = 1 << 22;  // units of a batched sweep (a range word's strip field)
size_t sweep_smem_bytes(int k, int flux_storage);
// The column unit that the variant table names a sweep by: 64 columns less their
// halo.  A warp sweeps two such halves side by side (128 columns).
constexpr int sweep_column_unit(int k) { return 64 - 4 * k; }
constexpr int sweep_strip_columns(int k) { return 128 - 2 * ((2 * k + 3) / 4 * 4); }
// tws_stream.cu
cudaError_t launch_stream_step(int ry, int flux_storage, const float* b, const float* d,
                               const void* f, const StepArgs& a, cudaStream_t s);
cudaError_t encode_step_maps(int variant, int flux_storage, int W, int H, int pitch,
                             const float* b, const float* d, const void* f, CUtensorMap* tm_b,
                             CUtensorMap* tm_d, CUtensorMap* tm_f, std::string* why);

// tws_resident.cu: the whole grid in the shared memory of one cluster of up
// to kResidentMaxCluster CTAs, up to kResidentMaxSteps steps per launch.
constexpr int kResidentMaxCluster = 16;
constexpr int kResidentMaxSteps = 4096;
// cudaSuccess if a W x H grid fits a cluster of `ctas` CTAs (0: the automatic
// size, returned in *chosen) and the device can run that cluster
cudaError_t resident_supported(int W, int H, int flux_storage, int ctas, int* chosen);
cudaError_t launch_resident(int flux_storage, int ctas, const float* b, const float* d,
                            const void* f, const StepArgs& a, int nsteps, cudaStream_t s);

// tws_mesh.cu: grids of up to about a million cells with their state on chip
// across all SMs, all steps of a call in one cooperative launch.
struct MeshShape {
  int ry;                // rows per warp
  int every;             // steps between exchanges
  int hx, hy;            // halo of a CTA's box
  int tiles_x, tiles_y;  // CTAs
  int brushes;           // brush sources (a plane of shared memory each)
};
constexpr int kMeshMaxCtas = 256;
// Whether a W x H grid with that many brush sources fits, and how.
bool mesh_shape(int W, int H, int brushes, MeshShape* out);
// Exchanges of a launch.
int mesh_exchanges(const MeshShape& s, int nsteps);
// Bytes of the workspace (a count, and the CTAs' inboxes): zeroed once, then every
// exchange of every launch that uses it has a number of its own (never 0).
size_t mesh_inbox_bytes(const MeshShape& s);
inline int mesh_ctas(const MeshShape& s) { return s.tiles_x * s.tiles_y; }
// d[0], f[0]: the state; d[1], f[1]: where the result goes.  `epoch`: the number of
// the last exchange before, `begun`: the CTAs of all launches of several before.
cudaError_t launch_mesh(const MeshShape& s, int flux_storage, const float* b, float* const d[2],
                        void* const f[2], const StepArgs& a, int nsteps, void* inbox,
                        unsigned epoch, unsigned begun, cudaStream_t st);

// tws_aux.cu
cudaError_t launch_apply_source(float* d, int W, int H, int pitch, const DevSource& s,
                                cudaStream_t st);
cudaError_t launch_volume(const float* d, int W, int H, int pitch, double cell_area,
                          double* partials, int max_partials, double* out, cudaStream_t st);
int volume_partials_needed();
cudaError_t launch_generate_scene(uint64_t seed, int W, int H, int pitch, float height_scale,
                                  float fill, float* b, float* d, cudaStream_t st);
cudaError_t launch_reference_scene(uint32_t seed, int generation, int W, int H, int pitch,
                                   float height_scale, float* b, float* d, cudaStream_t st);
cudaError_t launch_flux_to_f32(const void* f, int flux_storage, float inv_scale, int W, int H,
                               int pitch, float* out_packed, cudaStream_t st);
cudaError_t launch_flux_from_f32(const float* in_packed, int flux_storage, float scale, int W,
                                 int H, int pitch, void* f, cudaStream_t st);
// Up to four row copies between packed arrays and the pitched state in one
// launch on the SMs (device-to-device copies on the copy engines are several
// times slower); a null source writes zeros.  Pitches and row lengths in
// floats; `vec` is filled by the launcher.
struct StageRows {
  const float* src[4];
  float* dst[4];
  int row_floats[4], src_pitch[4], dst_pitch[4], vec[4];
  int n;
  void add(const float* s, int sp, float* d, int dp, int floats) {
    src[n] = s;
    dst[n] = d;
    src_pitch[n] = sp;
    dst_pitch[n] = dp;
    row_floats[n] = floats;
    vec[n] = 1;
    ++n;
  }
};
cudaError_t launch_stage_rows(const StageRows& sr, int H, cudaStream_t st);

// tws_export.cu
cudaError_t launch_surface(const float* b, const float* d, const float2* v, int W, int H,
                           int pitch, const tws_surface_out& o, cudaStream_t s);
cudaError_t launch_export(const float* b, const float* d, const float2* v, int W, int H,
                          int pitch, float* terrain_rgba, uint16_t* flowmap, int mip_levels,
                          float* mips, cudaStream_t s);

DevSource make_dev_source(const tws_source& s);
// A launch that may be scheduled while the one before it on the stream finishes:
// the kernel waits for that one itself (griddepcontrol.wait) before it touches
// memory.
template <class... P, class... A>
cudaError_t launch_after_previous(void (*fn)(P...), dim3 grid, dim3 block, cudaStream_t s,
                                  A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, P(args)...);
}
void count_launch(uint64_t n = 1);

}  // namespace tws
