// Internal types and launchers of the 3D hybrid path (include/hybridmlem.h).
// Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace hybridmlem {

// The voxel grid and scanner constants in binary32 / int16 as the reference
// holds them: PixelGrid (src/2d/geometry/pixel_grid.h:22-37), VoxelGrid
// (src/3d/geometry/voxel_grid.h:19-24), GaussianKernel<float> members
// (src/2d/strip/gaussian_kernel.h:27-33).
struct GridF {
  int32_t nc, nr, np;
  float p;        // pixel size = plane thickness
  float z_left;
  float llc_x;    // lower_left_center
  float llc_y;
  float L;        // barrel length
  float ipz;      // 1 / sigma_z^2
  float ipdl;     // 1 / sigma_dl^2
  float norm_c;   // 1 / (2 pi^2) sqrt(ipz^2 ipdl)
  int32_t n_pixels;
};

// One kept frame event (FrameEvent, src/3d/hybrid/reconstruction.h:53-63),
// 32 bytes: the LOR, its pixel-info range, its plane range and the strip
// frame's (up, right, tan, sec).
struct __align__(16) Frame {
  int32_t lor;
  int32_t info_begin;
  int32_t info_end;
  int16_t plane_begin;
  int16_t plane_end;
  float up;
  float right;
  float tan;
  float sec;
};
static_assert(sizeof(Frame) == 32, "Frame is 32 bytes");

// Device view of the flattened geometry (GeometrySOA, geometry_soa.h:270-284).
struct GeometryDev {
  const float4* lor_md;     // per LOR: mid x, mid y, direction x, direction y
  const float* lor_len;     // per LOR: segment length
  const short2* pix;        // per info: pixel (x, y)
  const float* pos;         // per info: position along the LOR
  const float* w;           // per info: weight (normalised after the sensitivity)
  const int64_t* lbeg;      // per LOR
  const int64_t* lend;
  int64_t n_lors;
  int64_t n_infos;
};

// hybrid_setup.cu (compiled without FMA contraction: the frame arithmetic
// rounds as the reference's binary32 C++).
void launch_sensitivity(const GridF& g, const short2* pix, const float* w, int64_t n,
                        double* acc, float* sens, cudaStream_t st);
void launch_normalize(const GridF& g, const short2* pix, float* w, const float* sens,
                      int64_t n, cudaStream_t st);
void launch_frames(const GridF& g, const GeometryDev& geo, const int16_t* first,
                   const int16_t* second, const float* z_up, const float* z_dn,
                   const float* dl, int64_t n, Frame* frames, int32_t* keep,
                   cudaStream_t st);
void launch_compact(const Frame* frames, const int32_t* keep, const int64_t* offs, int64_t n,
                    Frame* out, int64_t* out_index, cudaStream_t st);
// Event-sized device memory: from a stream-ordered pool (plain allocations
// when pool is null).
struct EventMemory {
  cudaMemPool_t pool;
  cudaStream_t stream;
  cudaError_t alloc(void** p, size_t bytes) const {
    *p = nullptr;
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, stream) : cudaMalloc(p, bytes);
  }
  void free(void* p) const {
    if (!p) return;
    if (pool)
      cudaFreeAsync(p, stream);
    else
      cudaFree(p);
  }
};

// ---- the windowed iteration (hybrid_kernels.cu, "Windowed MLEM") ----
// Its shape: events are binned by LOR and by their first plane in slabs of
// tile_planes; a window holds `planes` planes, so it takes events of up to
// max_planes (planes 0: no windows).
struct WinPlan {
  int planes, max_planes, tile_planes, n_slabs;
};
// A windowed frame event, 32 bytes: the strip frame's constants and shape =
// pixel infos | planes << kWinRowBits | middle plane << 18.
constexpr int kWinRowBits = 11, kWinPlaneBits = 7, kWinPmBits = 14;
struct __align__(16) WinEvent {
  float up, tan, zc, cd;  // zc: z of the middle plane - right
  float na, nb;           // a'Sa = na up_p^2 + nb
  int32_t info_begin;
  uint32_t shape;
};
static_assert(sizeof(WinEvent) == 32, "WinEvent is 32 bytes");
// Up to kWinItemEvents events of one (LOR, slab) and the pixel infos they
// span; a task is 64 pixel infos of an item and the planes of its events that
// touch them (none: p0 == p1).
constexpr int kWinItemEvents = 512;
struct WinItem {
  int32_t e0, e1, lor, i0, i1;
};
struct WinTask {
  int32_t item, row0;
  int16_t p0, p1;
};
// Device arrays of the windowed events (allocated by order_frames in one
// block, `block`).
struct WinSet {
  WinPlan plan;
  int32_t n_events;   // windowed events: frames [0, n_events) of the order
  int32_t n_items, n_tasks;
  int64_t entries;    // window entries of all tasks
  char* block;
  WinEvent* events;
  WinItem* items;
  WinTask* tasks;
  double* D;          // zero between iterations
  float* inv;
  int32_t* list;      // events the windows leave to k_mlem
  int32_t* counters;  // next task of the two kernels, length of list
};
// The frame events in the iteration's order into `out`: (LOR, plane slab)
// order of the events the plan's windows take, then the others; without
// windows LOR order.  Fills ws (n_events 0: no windows; ws->block from mem).
// Synchronises mem's stream.
cudaError_t order_frames(const GridF& g, const GeometryDev& geo, const Frame* frames, int32_t n,
                         const WinPlan& plan, Frame* out, WinSet* ws, EventMemory mem);

// hybrid_kernels.cu
void launch_to_zfast(const GridF& g, const float* rho, float* rho_t, cudaStream_t st);
void launch_from_zfast(const GridF& g, const float* rho_t, float* rho, cudaStream_t st);
// One warp per event over frames[0 .. n_frames) and then the *n_list events
// win_frames[list[i]] (list, n_list may be null).  spill:
// mlem_spill_floats(n_blocks) floats of scratch for the per-warp weight slabs.
void launch_mlem(const GridF& g, const GeometryDev& geo, const float* sens, const Frame* frames,
                 int64_t n_frames, const Frame* win_frames, const int32_t* list,
                 const int32_t* n_list, const float* rho_t, float* acc_t, float* spill,
                 int n_blocks, cudaStream_t st);
// Windowed backprojection of ws's events into acc_t; counters are zeroed by
// the caller, and the events left in ws.list are launch_mlem's.
WinPlan plan_windows(const GridF& g, int max_planes);
void launch_win_events(const GridF& g, const GeometryDev& geo, const Frame* frames, int32_t n,
                       WinEvent* out, cudaStream_t st);
void launch_mlem_win(const GridF& g, const GeometryDev& geo, const float* sens,
                     const WinSet& ws, const float* rho_t, float* acc_t, int n_sm,
                     cudaStream_t st);
size_t mlem_spill_floats(int n_blocks);
int mlem_blocks_per_sm();
// out4: pixel infos, voxels, the largest event's pixel infos and planes
void launch_event_counts(const Frame* frames, int64_t n, unsigned long long* out4,
                         cudaStream_t st);
cudaError_t launch_atan2_probe(const float* a, const float* b, int64_t n, int which,
                               float* out, cudaStream_t st);

}  // namespace hybridmlem
