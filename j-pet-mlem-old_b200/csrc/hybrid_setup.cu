// Set-up kernels of the 3D hybrid path: the 2D sensitivity, the weight
// normalisation and the translation of responses to frame events.  This file
// is compiled with -fmad=false: every binary32 operation of the frame
// translation rounds where the reference's C++ says, so the pixel-info and
// plane ranges of each event equal the reference's bit for bit.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cuda/std/functional>

#include "hybrid_internal.h"

namespace hybridmlem {

namespace {

// calculate_sensitivity (src/3d/hybrid/reconstruction.h:226-237): the sum of
// the weights of every pixel info of each pixel.  Summed in binary64 (the
// reference sums sequentially in binary32; the two agree to the binary32
// rounding of the reference's own sum).
__global__ void k_sens_acc(int32_t nc, const short2* __restrict__ pix,
                           const float* __restrict__ w, int64_t n, double* acc) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const short2 p = pix[i];
    atomicAdd(acc + p.x + (int64_t)nc * p.y, (double)w[i]);
  }
}

__global__ void k_sens_round(const double* __restrict__ acc, float* sens, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    sens[i] = (float)acc[i];
}

// normalize_geometry_weights (reconstruction.h:239-261), one plane half.
__global__ void k_normalize(int32_t nc, const short2* __restrict__ pix, float* w,
                            const float* __restrict__ sens, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const short2 p = pix[i];
    w[i] = w[i] / sens[p.x + (int64_t)nc * p.y];
  }
}

// std::lower_bound / std::upper_bound over a sorted binary32 range.
__device__ int64_t lower_bound_f(const float* a, int64_t lo, int64_t hi, float v) {
  int64_t n = hi - lo;
  while (n > 0) {
    const int64_t half = n >> 1;
    if (a[lo + half] < v) {
      lo += half + 1;
      n -= half + 1;
    } else {
      n = half;
    }
  }
  return lo;
}

__device__ int64_t upper_bound_f(const float* a, int64_t lo, int64_t hi, float v) {
  int64_t n = hi - lo;
  while (n > 0) {
    const int64_t half = n >> 1;
    if (!(v < a[lo + half])) {
      lo += half + 1;
      n -= half + 1;
    } else {
      n = half;
    }
  }
  return lo;
}

// Reconstruction::plane (reconstruction.h:149): truncation to short.
__device__ __forceinline__ int16_t plane_of(const GridF& g, float z) {
  return (int16_t)(int)((z - g.z_left) / g.p);
}

// translate_to_frame + bb_intersects_grid_with_positive_weight
// (reconstruction.h:97-161), one response per thread.
__global__ void k_frames(const GridF g, const GeometryDev geo,
                         const int16_t* __restrict__ first, const int16_t* __restrict__ second,
                         const float* __restrict__ z_up, const float* __restrict__ z_dn,
                         const float* __restrict__ dl, int64_t n, Frame* frames,
                         int32_t* keep) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    keep[i] = 0;
    const int64_t a = first[i], b = second[i];
    // LOR::index on the pair as the reference reads it (lor.h:33-35)
    const int64_t li = a * (a + 1) / 2 + b;
    if (a < 0 || b < 0 || li >= geo.n_lors) continue;
    const float R = geo.lor_len[li] / 2;
    // Strip::Response::calculate_tan_y_z (src/2d/strip/response.h:22-37)
    const float zu = z_up[i], zd = z_dn[i], d = dl[i];
    const float tan = (zu - zd) / (2 * R);
    const float up = -0.5f * (d / sqrtf(1 + tan * tan));
    const float right = 0.5f * (zu + zd + (2 * up * tan));
    // GaussianKernel::ellipse_bb (src/2d/strip/gaussian_kernel.h:108-128)
    const float tan_sq = tan * tan;
    const float sec = sqrtf(1 + tan * tan);
    const float A = 4 * sec * sec * g.ipdl + 2 * tan_sq * g.ipz;
    const float B = -4 * tan * g.ipz;
    const float C = 2 * g.ipz;
    const float B_2 = (B / 2) * (B / 2);
    const float half_up = 3 / sqrtf(A - (B_2 / C));
    const float half_right = 3 / sqrtf(C - (B_2 / A));
    const int16_t pl = plane_of(g, right - half_right);
    const int16_t pr = plane_of(g, right + half_right);
    const int16_t pb = pl > 0 ? pl : (int16_t)0;
    const int16_t pe1 = (int16_t)(pr + 1);
    const int16_t pe = pe1 < (int16_t)g.np ? pe1 : (int16_t)g.np;
    const float y_up = up + half_up, y_dn = up - half_up;
    const float t_up = (y_up + R) / (2 * R);
    const float t_dn = (y_dn + R) / (2 * R);
    const int64_t lb = geo.lbeg[li], le = geo.lend[li];
    // upper_bound(t_up) + 1 and lower_bound(t_dn) (reconstruction.h:130-145);
    // the end may reach one info past the LOR's range, as in the reference,
    // and is clamped at the end of the arrays
    int64_t ie = upper_bound_f(geo.pos, lb, le, t_up) + 1;
    const int64_t ib = lower_bound_f(geo.pos, lb, le, t_dn);
    if (ie > geo.n_infos) ie = geo.n_infos;
    if (pe <= 0 || pb >= g.np) continue;
    bool ok = false;
    for (int64_t k = ib; k < ie && !ok; ++k) {
      const short2 p = geo.pix[k];
      ok = p.x >= 0 && p.x < g.nc && p.y >= 0 && p.y < g.nr && geo.w[k] > 0;
    }
    if (!ok) continue;
    Frame f;
    f.lor = (int32_t)li;
    f.info_begin = (int32_t)ib;
    f.info_end = (int32_t)ie;
    f.plane_begin = pb;
    f.plane_end = pe;
    f.up = up;
    f.right = right;
    f.tan = tan;
    f.sec = sec;
    frames[i] = f;
    keep[i] = 1;
  }
}

__global__ void k_compact(const Frame* __restrict__ frames, const int32_t* __restrict__ keep,
                          const int64_t* __restrict__ offs, int64_t n, Frame* out,
                          int64_t* out_index) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (!keep[i]) continue;
    out[offs[i]] = frames[i];
    out_index[offs[i]] = i;
  }
}

int grid_for(int64_t n) {
  const int64_t b = (n + 255) / 256;
  return (int)(b < 148 * 32 ? (b > 0 ? b : 1) : 148 * 32);
}

}  // namespace

void launch_sensitivity(const GridF& g, const short2* pix, const float* w, int64_t n,
                        double* acc, float* sens, cudaStream_t st) {
  cudaMemsetAsync(acc, 0, sizeof(double) * g.n_pixels, st);
  k_sens_acc<<<grid_for(n), 256, 0, st>>>(g.nc, pix, w, n, acc);
  k_sens_round<<<grid_for(g.n_pixels), 256, 0, st>>>(acc, sens, g.n_pixels);
}

void launch_normalize(const GridF& g, const short2* pix, float* w, const float* sens,
                      int64_t n, cudaStream_t st) {
  k_normalize<<<grid_for(n), 256, 0, st>>>(g.nc, pix, w, sens, n);
}

void launch_frames(const GridF& g, const GeometryDev& geo, const int16_t* first,
                   const int16_t* second, const float* z_up, const float* z_dn,
                   const float* dl, int64_t n, Frame* frames, int32_t* keep,
                   cudaStream_t st) {
  k_frames<<<grid_for(n), 256, 0, st>>>(g, geo, first, second, z_up, z_dn, dl, n, frames,
                                        keep);
}

void launch_compact(const Frame* frames, const int32_t* keep, const int64_t* offs, int64_t n,
                    Frame* out, int64_t* out_index, cudaStream_t st) {
  k_compact<<<grid_for(n), 256, 0, st>>>(frames, keep, offs, n, out, out_index);
}

namespace {

// Sort keys: (LOR, plane slab); the largest key for an event no window takes
// (counted): one without voxels or with more than a window holds, or whose
// infos are not its LOR's (and the one after them, where a frame may end), so
// that an item spans one LOR's infos however far apart its events' lie.
__global__ void k_order_keys(const Frame* __restrict__ frames, int32_t n, const GeometryDev geo,
                             const WinPlan w, uint64_t* keys, int32_t* index,
                             int32_t* n_general) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const Frame f = frames[i];
    uint64_t key = (uint64_t)f.lor;
    if (w.planes > 0) {
      const int rows = f.info_end - f.info_begin, planes = f.plane_end - f.plane_begin;
      if (rows > 0 && planes > 0 && rows < (1 << kWinRowBits) && planes <= w.max_planes &&
          f.info_begin >= geo.lbeg[f.lor] && f.info_end <= geo.lend[f.lor] + 1) {
        key = key * w.n_slabs + f.plane_begin / w.tile_planes;
      } else {
        key = (uint64_t)geo.n_lors * w.n_slabs;
        atomicAdd(n_general, 1);
      }
    }
    keys[i] = key;
    index[i] = i;
  }
}

__global__ void k_gather_frames(const Frame* __restrict__ frames, const int32_t* index,
                                int32_t n, Frame* out) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = frames[index[i]];
}

// flag[i] = 1 where a work item begins: at a new key and every
// kWinItemEvents events of it.
__global__ void k_item_flags(const uint64_t* __restrict__ keys, int32_t n, int32_t* flag) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    int32_t lo = 0, m = i;  // first event of the key, in [0, i]
    while (m > 0) {
      const int32_t half = m >> 1;
      if (keys[lo + half] < k) {
        lo += half + 1;
        m -= half + 1;
      } else {
        m = half;
      }
    }
    flag[i] = (i - lo) % kWinItemEvents == 0 ? 1 : 0;
  }
}

__global__ void k_item_begins(const int32_t* __restrict__ flag, const int64_t* __restrict__ offs,
                              int32_t n, int32_t n_items, int32_t* begin) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (flag[i]) begin[offs[i]] = i;
  if (blockIdx.x == 0 && threadIdx.x == 0) begin[n_items] = n;
}

// The items' pixel-info spans and numbers of tasks.  One warp per item.
__global__ void k_item_boxes(const Frame* __restrict__ frames, const int32_t* __restrict__ begin,
                             int32_t n_items, WinItem* items, int32_t* n_tasks) {
  const int lane = threadIdx.x & 31;
  const int32_t n_warps = gridDim.x * (blockDim.x >> 5);
  for (int32_t it = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < n_items;
       it += n_warps) {
    const int32_t e0 = begin[it], e1 = begin[it + 1];
    int i0 = 0x7FFFFFFF, i1 = 0;
    for (int32_t e = e0 + lane; e < e1; e += 32) {
      i0 = min(i0, frames[e].info_begin);
      i1 = max(i1, frames[e].info_end);
    }
    for (int o = 16; o > 0; o >>= 1) {
      i0 = min(i0, __shfl_xor_sync(0xffffffffu, i0, o));
      i1 = max(i1, __shfl_xor_sync(0xffffffffu, i1, o));
    }
    if (lane == 0) {
      items[it] = WinItem{e0, e1, frames[e0].lor, i0, i1};
      n_tasks[it] = (i1 - i0 + 63) / 64;
    }
  }
}

// The items' tasks, and the window entries they stage (planes by 32 and infos
// by 2, as the kernels take them).  One warp per item.
__global__ void k_item_tasks(const Frame* __restrict__ frames, const WinItem* __restrict__ items,
                             const int64_t* __restrict__ offs, int32_t n_items, WinTask* tasks,
                             unsigned long long* entries) {
  const int lane = threadIdx.x & 31;
  const int32_t n_warps = gridDim.x * (blockDim.x >> 5);
  unsigned long long sum = 0;
  for (int32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n_items;
       i += n_warps) {
    const WinItem it = items[i];
    WinTask* out = tasks + offs[i];
    for (int row0 = it.i0; row0 < it.i1; row0 += 64, ++out) {
      int p0 = 0x7FFF, p1 = 0;
      for (int32_t e = it.e0 + lane; e < it.e1; e += 32) {
        const Frame f = frames[e];
        if (f.info_begin < row0 + 64 && f.info_end > row0) {
          p0 = min(p0, (int)f.plane_begin);
          p1 = max(p1, (int)f.plane_end);
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        p0 = min(p0, __shfl_xor_sync(0xffffffffu, p0, o));
        p1 = max(p1, __shfl_xor_sync(0xffffffffu, p1, o));
      }
      if (p1 <= p0) p0 = p1 = 0;
      if (lane == 0) *out = WinTask{i, row0, (int16_t)p0, (int16_t)p1};
      sum += (unsigned long long)((min(64, it.i1 - row0) + 1) & ~1) * ((p1 - p0 + 31) & ~31);
    }
  }
  if (lane == 0 && sum) atomicAdd(entries, sum);
}

// Exclusive sums of 32-bit counts in 64 bits (DeviceScan adds in its initial
// value's type; ExclusiveSum's is the input's).
cudaError_t scan64(void* temp, size_t* temp_bytes, const int32_t* v, int64_t* out, int32_t n,
                   cudaStream_t st) {
  return cub::DeviceScan::ExclusiveScan(temp, *temp_bytes, v, out, cuda::std::plus<>{},
                                        int64_t{0}, n, st);
}

}  // namespace

cudaError_t order_frames(const GridF& g, const GeometryDev& geo, const Frame* frames, int32_t n,
                         const WinPlan& plan, Frame* out, WinSet* ws, EventMemory mem) {
  cudaStream_t st = mem.stream;
  *ws = WinSet{};
  ws->plan = plan;
  if (n <= 0) return cudaSuccess;
  const bool win = plan.planes > 0;
  const uint64_t n_keys = (uint64_t)geo.n_lors * (win ? (uint64_t)plan.n_slabs : 1) + 1;
  int end_bit = 1;
  while (end_bit < 64 && ((uint64_t)1 << end_bit) < n_keys) ++end_bit;
  // one scratch block: keys and indices, sorted keys and indices, offsets,
  // totals, CUB's own (sort and scan share it)
  const size_t nn = ((size_t)n + 64) & ~(size_t)63;
  size_t sort_bytes = 0, scan_bytes = 0;
  uint64_t* kn = nullptr;
  int32_t* in = nullptr;
  int64_t* on = nullptr;
  cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, kn, kn, in, in, n, 0,
                                                  end_bit, st);
  if (e == cudaSuccess)
    e = scan64(nullptr, &scan_bytes, in, on, n, st);
  if (e != cudaSuccess) return e;
  const size_t temp_bytes = std::max(sort_bytes, scan_bytes);
  void* block = nullptr;
  e = mem.alloc(&block, nn * (8 + 8 + 8 + 4 + 4) + 256 + temp_bytes);
  if (e != cudaSuccess) return e;
  uint64_t* keys = static_cast<uint64_t*>(block);
  uint64_t* keys_out = keys + nn;
  int64_t* offs = reinterpret_cast<int64_t*>(keys_out + nn);
  int32_t* index = reinterpret_cast<int32_t*>(offs + nn);
  int32_t* index_out = index + nn;
  unsigned long long* totals = reinterpret_cast<unsigned long long*>(index_out + nn);
  int32_t* d_general = reinterpret_cast<int32_t*>(totals + 1);
  void* temp = reinterpret_cast<char*>(totals) + 256;
  void* items_tmp = nullptr;
  auto done = [&](cudaError_t r) {
    mem.free(items_tmp);
    mem.free(block);
    if (r != cudaSuccess) {
      mem.free(ws->block);
      *ws = WinSet{};
    }
    const cudaError_t s = cudaStreamSynchronize(st);
    return r != cudaSuccess ? r : s;
  };
  // no memory for the windows: the ordered events go without
  auto no_windows = [&](cudaError_t r) {
    if (r != cudaErrorMemoryAllocation) return done(r);
    cudaGetLastError();
    return done(cudaSuccess);
  };
#define STEP(call)                              \
  do {                                          \
    e = (call);                                 \
    if (e != cudaSuccess) return done(e);       \
  } while (0)
  // total of an exclusive scan: its last offset plus the last value
  auto scan_total = [&](const int32_t* v, int32_t count, int64_t* total) {
    size_t tb = temp_bytes;
    cudaError_t r = scan64(temp, &tb, v, offs, count, st);
    int64_t last = 0;
    int32_t last_v = 0;
    if (r == cudaSuccess)
      r = cudaMemcpyAsync(&last, offs + (count - 1), 8, cudaMemcpyDeviceToHost, st);
    if (r == cudaSuccess)
      r = cudaMemcpyAsync(&last_v, v + (count - 1), 4, cudaMemcpyDeviceToHost, st);
    if (r == cudaSuccess) r = cudaStreamSynchronize(st);
    *total = last + last_v;
    return r;
  };
  STEP(cudaMemsetAsync(totals, 0, 16, st));
  k_order_keys<<<grid_for(n), 256, 0, st>>>(frames, n, geo, plan, keys, index, d_general);
  size_t tb = temp_bytes;
  STEP(cub::DeviceRadixSort::SortPairs(temp, tb, keys, keys_out, index, index_out, n, 0, end_bit,
                                       st));
  k_gather_frames<<<grid_for(n), 256, 0, st>>>(frames, index_out, n, out);
  STEP(cudaGetLastError());
  if (!win) return done(cudaSuccess);
  int32_t n_general = 0;
  STEP(cudaMemcpyAsync(&n_general, d_general, 4, cudaMemcpyDeviceToHost, st));
  STEP(cudaStreamSynchronize(st));
  const int32_t nf = n - n_general;
  if (nf <= 0) return done(cudaSuccess);
  int32_t* flag = index;  // the unsorted indices are done with
  k_item_flags<<<grid_for(nf), 256, 0, st>>>(keys_out, nf, flag);
  int64_t n_items = 0, n_tasks = 0;
  STEP(scan_total(flag, nf, &n_items));
  int32_t* begin = index_out;  // so are the sorted ones (n_items + 1 <= nn)
  k_item_begins<<<grid_for(nf), 256, 0, st>>>(flag, offs, nf, (int32_t)n_items, begin);
  e = mem.alloc(&items_tmp, (size_t)n_items * sizeof(WinItem));
  if (e != cudaSuccess) return no_windows(e);
  WinItem* items = static_cast<WinItem*>(items_tmp);
  k_item_boxes<<<grid_for(n_items * 32), 256, 0, st>>>(out, begin, (int32_t)n_items, items, flag);
  STEP(scan_total(flag, (int32_t)n_items, &n_tasks));
  // task numbers are ints (with room for the warps' last looks): no windows
  if (n_tasks > INT32_MAX - (1 << 20)) return done(cudaSuccess);
  // the set's own block
  auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t b_ev = up((size_t)nf * sizeof(WinEvent)), b_it = up((size_t)n_items * sizeof(WinItem)),
               b_ta = up((size_t)n_tasks * sizeof(WinTask)), b_D = up((size_t)nf * sizeof(double)),
               b_inv = up((size_t)nf * sizeof(float)), b_li = up((size_t)nf * sizeof(int32_t));
  void* own_p = nullptr;
  e = mem.alloc(&own_p, b_ev + b_it + b_ta + b_D + b_inv + b_li + 256);
  if (e != cudaSuccess) return no_windows(e);
  char* own = static_cast<char*>(own_p);
  ws->block = own;
  STEP(cudaMemcpyAsync(own + b_ev, items, (size_t)n_items * sizeof(WinItem),
                       cudaMemcpyDeviceToDevice, st));
  ws->events = reinterpret_cast<WinEvent*>(own);
  ws->items = reinterpret_cast<WinItem*>(own + b_ev);
  ws->tasks = reinterpret_cast<WinTask*>(own + b_ev + b_it);
  ws->D = reinterpret_cast<double*>(own + b_ev + b_it + b_ta);
  ws->inv = reinterpret_cast<float*>(own + b_ev + b_it + b_ta + b_D);
  ws->list = reinterpret_cast<int32_t*>(own + b_ev + b_it + b_ta + b_D + b_inv);
  ws->counters = reinterpret_cast<int32_t*>(own + b_ev + b_it + b_ta + b_D + b_inv + b_li);
  ws->n_events = nf;
  ws->n_items = (int32_t)n_items;
  ws->n_tasks = (int32_t)n_tasks;
  STEP(cudaMemsetAsync(ws->D, 0, b_D, st));
  k_item_tasks<<<grid_for(n_items * 32), 256, 0, st>>>(out, ws->items, offs, (int32_t)n_items,
                                                      ws->tasks, totals);
  launch_win_events(g, geo, out, nf, ws->events, st);
  STEP(cudaGetLastError());
  unsigned long long entries = 0;
  STEP(cudaMemcpyAsync(&entries, totals, 8, cudaMemcpyDeviceToHost, st));
  STEP(cudaStreamSynchronize(st));
  ws->entries = (int64_t)entries;
  return done(cudaSuccess);
#undef STEP
}

}  // namespace hybridmlem

// Exclusive scan of the keep flags (CUB), used by hybrid_capi.cu.
extern "C" cudaError_t hybridmlem_scan_keep(const int32_t* keep, int64_t* offs, int64_t n,
                                            void* temp, size_t* temp_bytes, cudaStream_t st) {
  return cub::DeviceScan::ExclusiveSum(temp, *temp_bytes, keep, offs, n, st);
}
