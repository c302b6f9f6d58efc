// Launch helpers of the single-lattice step kernels (kernels.cu, line.cu).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <utility>

namespace imx {

// Programmatic dependent launch of consecutive steps (launch_pdl): a step
// kernel may be scheduled while the previous one drains; pdl_wait holds it,
// before its first access to global memory, until the previous grid has
// completed and its writes are visible, and pdl_release lets the next one
// be scheduled.  Both are no-ops for a kernel launched without the attribute.
//
// A kernel releases the next step when it is done, not when it starts: blocks
// let in early sit waiting on the SMs that happen to have room, the rest of
// their grid is spread unevenly around them, and a small lattice's step lasts
// as long as its fullest SM.  us a step, released at the start | at the end:
// FP64 EXACT cavity 24^3 6.3 | 3.6, 32^3 6.5 | 4.2, FP32 cavity 48^3 6.5 |
// 4.5, FP64 reference cavity 48^3 13.4 | 11.0; above 56^3 the same.  Only a
// 2-byte staged grid that takes every slot of the device (FP16 96^3: 21.4 | 22.8)
// and the large lattices of step_box_kernel (FP64 vortex 30x180x170 93.9 | 94.7)
// release at the start.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch with programmatic stream serialisation: the kernel may start
// while the kernel before it on the stream finishes (see pdl_wait).
template <class... KArgs, class... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Tiles of a persistent kernel are handed out as its blocks come for them:
// with equal shares fixed beforehand the kernel lasts as long as its slowest
// SM, and SMs differ in the bandwidth they get.  counters[0] counts the
// tiles taken beyond the first ones, counters[1] the blocks that are done;
// the last block leaves both at zero for the next launch.  Every ticket's
// value has to be used before its block calls finish_tiles.  A block stops at
// the first stage without a tile, so its tickets have to grow in the order in
// which it works through its stages: one lane takes them, several at a time in
// one operation (the lanes of one atomic get their values in no stated order).
__device__ __forceinline__ int take_tiles(int* counters, int n) { return atomicAdd(counters, n); }
__device__ __forceinline__ int take_tile(int* counters) { return take_tiles(counters, 1); }
__device__ __forceinline__ void finish_tiles(int* counters) {  // one thread of the block, after all its tickets
  if (atomicAdd(counters + 1, 1) == static_cast<int>(gridDim.x) - 1) {
    counters[0] = 0;
    counters[1] = 0;
  }
}

// n / d of an index 0 <= n < 2^31 without a division: n m >> (31 + s) with
// s = ceil(log2 d), m = ceil(2^(31+s) / d): m d = 2^(31+s) + e, 0 <= e < d <=
// 2^s, and the excess n e / (d 2^(31+s)) is below 1 / d.
inline void item_magic(int d, uint32_t* m, int* s) {
  *s = 0;
  while ((int64_t(1) << *s) < d) ++*s;
  *m = static_cast<uint32_t>(((uint64_t(1) << (31 + *s)) + d - 1) / d);
}

__host__ __device__ __forceinline__ int item_quotient(int n, uint32_t m, int s) {
  return static_cast<int>((static_cast<uint64_t>(static_cast<uint32_t>(n)) * m) >> (31 + s));
}

constexpr int STEP_THREADS = 128;
constexpr int MAX_GRID_Y = 65535;

// Plane k of the step grid (blockIdx.y) is a line of items, rows of `width`
// items each, x fastest (an item is the cells one thread owns), and thread r
// of the line takes item r.  Blocks run across row ends, so a lattice of any
// extents fills its warps.
struct ItemMap {
  uint32_t m_width;
  int s_width;
  int width, plane;  // items of a row, of a plane
};

// Items of `cx` cells along x by `cy` along y, a value `elem` bytes.  Rows of
// a warp or more are rounded up to whole 32-byte sectors, so that no two
// warps share one where a warp starts in mid-row.
inline ItemMap item_map(int nx, int ny, int cx, int cy, int elem) {
  ItemMap im;
  im.width = (nx + cx - 1) / cx;
  const int sector = 32 / (cx * elem);
  if (im.width >= 32) im.width = (im.width + sector - 1) / sector * sector;
  im.plane = im.width * ((ny + cy - 1) / cy);
  item_magic(im.width, &im.m_width, &im.s_width);
  return im;
}
inline dim3 item_grid(const ItemMap& im, int nz) { return dim3((im.plane + STEP_THREADS - 1) / STEP_THREADS, nz, 1); }

// A positive number per device, found on first use there.  Safe to ask from
// several threads (two may find the same number at once).
class PerDevice {
 public:
  template <class Find>
  int get(int dev, Find&& find) {
    if (dev < 0 || dev >= MAX_DEVICES) return find();
    int n = n_[dev].load(std::memory_order_acquire);
    if (n <= 0) {
      n = find();
      n_[dev].store(n, std::memory_order_release);
    }
    return n;
  }

 private:
  static constexpr int MAX_DEVICES = 64;
  std::atomic<int> n_[MAX_DEVICES] = {};
};

// Blocks of a persistent kernel that the current device holds at once, kept
// in the kernel's `known`.  The first call on a device also raises the
// kernel's shared-memory limit there: the limit belongs to the device.
template <class K>
cudaError_t resident_blocks(PerDevice& known, K kernel, int threads, size_t smem, int* blocks) {
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  *blocks = known.get(dev, [&] {
    int sms = 0, per_sm = 0;
    err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (err == cudaSuccess) err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    return err == cudaSuccess ? per_sm * sms : 0;
  });
  if (err == cudaSuccess && *blocks <= 0) err = cudaErrorLaunchOutOfResources;
  return err;
}

}  // namespace imx
