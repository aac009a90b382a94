// Sharing one schedule row between the CTAs of a cluster: when, between how many, and the launch.
//
// The kernels keep one CTA on an SM, so a grid of few long rows leaves SMs idle for the whole launch
// (512 query rows of 32 heads against 16384 keys: 64 CTAs of 128 steps on 148 SMs).  Measured, one CTA
// a row -> shared: that forward 238 -> 137 us (two CTAs a row); dkv of causal 2 x 4096, 16 q heads
// on one kv head, d 64 (64 CTAs of 16 .. 512 steps) 733 -> 223 (four a tile).
#pragma once

#include <algorithm>
#include <functional>
#include <mutex>

#include "splash_common.cuh"

namespace sb {

constexpr int kMaxSplit = 8;  // portable cluster size
constexpr int kSplitMaxCtas = 1024;  // grids above this fill the chip several times over

// Steps (128-column tiles) of the rows, of the longest and of the average one, from the mask function; a table
// mask counts as full, whether it comes from the host or from the device: so both give the same bits.
// Not asked for calls whose rows come in an order of their own (q_sequence), nor for calls with segment ids,
// which cut rows at places that only the device knows.
struct RowWork {
  float longest, mean;  // 0: rows are left whole
  int64_t ctas;         // rows of the call (of all launches that make it up)
  int n_rows;           // those of one head; 0: a table, whose rows may have any length up to these; and e4m3 P, see fwd_split()
  int steps[kSplitMaxCtas];  // in any order

  void scale(int n) {
    longest *= (float)n;
    mean *= (float)n;
    for (int r = 0; r < n_rows; ++r) steps[r] *= n;
  }
};
struct ClusterCapacity {
  int clusters[kMaxSplit + 1];  // [n]: clusters of n CTAs that are resident at the same time; [1]: CTAs
};

// rows of `row_span` query rows (transposed = false) or key tiles (true) over `n_steps_full` tiles of the other side
inline RowWork estimate_row_work(const SplashMaskFn& fn, int n_rows, int row_span, int n_tiles,
                                 int64_t n_ctas, bool transposed = false) {
  RowWork w;
  w.longest = w.mean = 0.f;
  w.ctas = n_ctas;
  w.n_rows = 0;
  if (n_ctas > kSplitMaxCtas || n_rows > kSplitMaxCtas) return w;
  w.longest = w.mean = (float)n_tiles;
  if (fn.kind == SPLASH_MASK_TABLE) return w;
  w.n_rows = n_rows;
  int64_t sum = 0, most = 0;
  for (int r = 0; r < n_rows; ++r) {
    // the row sees columns lo .. hi of the other side
    const int64_t first = (int64_t)r * row_span, last = first + row_span - 1;
    int64_t lo = 0, hi = (int64_t)n_tiles * kTile - 1;
    const int64_t left = fn.kind == SPLASH_MASK_LOCAL && fn.has_left ? fn.left : -1;
    const int64_t right = fn.kind == SPLASH_MASK_CAUSAL ? 0 : (fn.has_right ? fn.right : -1);
    const bool has_right = fn.kind == SPLASH_MASK_CAUSAL || fn.has_right;
    const bool has_left = fn.kind == SPLASH_MASK_LOCAL && fn.has_left;
    if (fn.kind == SPLASH_MASK_CHUNKED) {  // query i sees keys (i / chunk) * chunk .. i
      if (!transposed) {
        lo = first / fn.chunk * fn.chunk;
        if (last < hi) hi = last;
      } else {
        lo = first;
        if ((last / fn.chunk + 1) * fn.chunk - 1 < hi) hi = (last / fn.chunk + 1) * fn.chunk - 1;
      }
    } else if (!transposed) {  // query i sees keys i + offset - left .. i + offset + right
      if (has_left && first + fn.offset - left > lo) lo = first + fn.offset - left;
      if (has_right && last + fn.offset + right < hi) hi = last + fn.offset + right;
    } else {            // key j is seen by queries j - offset - right .. j - offset + left
      if (has_right && first - fn.offset - right > lo) lo = first - fn.offset - right;
      if (has_left && last - fn.offset + left < hi) hi = last - fn.offset + left;
    }
    const int64_t n = hi < lo ? 0 : hi / kTile - lo / kTile + 1;
    w.steps[r] = (int)n;
    sum += n;
    if (n > most) most = n;
  }
  w.longest = (float)most;
  w.mean = n_rows > 0 ? (float)sum / n_rows : 0.f;
  return w;
}

// CTAs per row.  Time in steps: a CTA costs its steps and a fixed part (launch, prologue, epilogue; more for the addition
// across the cluster).  While everything is resident the longest row sets the time.  Beyond that the whole work over the slots does,
// or the longest row, or a slot's turns: of k room + 1 rows, longest first, some slot takes k + 1, each at least as long as the last
// of them and with a fixed part of its own.  (That is what grids a little above the resident ones pay: causal 3328, 2 / 1 heads, 26 rows, forward,
// 1 .. 8 CTAs a row: 50.9 33.5 27.4 25.2 *23.8 33.5 36.1 35.5 us, 22 clusters of six are resident.  Rows of one length go in whole
// waves by it.)  The constants are those of least time over 1240 calls of random sizes, forward and backward, causal and windows, every
// number of CTAs measured (148 SMs, 74 45 33 26 22 15 15 clusters of 2 .. 8), and were then held against 400 others: 1.006 of the best
// number's time in the mean.  Rows of different length as a tail of a tenth of the longest, and waves of equal ones, made that 1.014 forward, 1.020
// backward, up to 1.3 times the time of half a row for every grid's end (1.017, 1.038); this one 1.03 times at most.
// All numbers tried, us of the kernel, the rule's own marked *.  dkv, causal: 2 x 4096, 16 / 1 heads, d 64: 733 375 260 *223 254 249 315
// 278, d 128 837 438 307 *259 296 291 371 328; 1 x 4096, 8 / 2, fused: 310 173 128 *115 139 142 195 185; 2 x 2048, 16 / 4,
// d 64: 105 *74 96 100; window 1000, 1 x 8192, 8 / 1: 193 *110 153 128, 20 / 5, 320 tiles, whole backward: *286 319 364 400.
// Forward: 512 x 16384, 32 / 8: 238 *137 184 153, 80 / 8, 160 rows: 455 374 348 *348, 160 / 8: 700 *627 686 689;
// causal 4096, 8 / 2: 65 *55 75 88, d 64 61 *47 64; 4096, 16 / 2: *75 106.
//
// How long the rows of a table are only the device knows.  The whole work as if they were full, and half a row for the end,
// stands between full rows, which go in waves, and those of prefixes and triangles, which have none.  (Whole backward, d 128, us with 1 2 3 4
// CTAs a tile, the number by waves marked w: 4096, 20 / 5 heads, 160 tiles: prefix 343 *260
// 288 w301, lower triangle 341 *255 274 w292, full 644 *540 497 w479; 2 x 4096, 20 / 5, 320 tiles: *509 w497 554 588, *466 w484 534
// 566, *1037 w954 1047 1025; 8192, 20 / 5: *989 w916, *865 w869, *2005 w1795; 2 x 4096, 30 / 5, d 64: *476 w487, *431 w469, *970 w893.)
//
// Rows below 16 steps stay whole although the
// rule would share some (causal 2 x 1024, 8 heads, 64 CTAs of 2 .. 8 steps: 24.7 us, 20.9 with two CTAs a row),
// so that the bits of short rows do not depend on the batch and the heads beside them: in the forward those
// of fewer than 2048 keys, in dkv kv tiles of fewer than 16 (q tile, q head of the group) steps.
inline int split_for(RowWork& w, const ClusterCapacity& cap) {
  constexpr float kFewest = 16.f;
  const bool known = w.n_rows > 0;
  const float own = known ? 6.f : 3.f, merge = known ? 2.f : 1.f;
  if (w.longest < kFewest) return 1;
  bool sorted = false;
  auto time = [&](int n) {
    const float fixed = own + (n > 1 ? merge : 0.f);
    const float longest = w.longest / n + fixed, mean = w.mean / n + fixed;
    const int64_t room = cap.clusters[n];
    if (w.ctas <= room) return longest;
    const float all = (float)w.ctas * mean / room;
    if (!known) return all + 0.5f * longest;
    if (!sorted) std::sort(w.steps, w.steps + w.n_rows, std::greater<int>());
    sorted = true;
    float least = std::max(longest, all + 0.05f * w.longest / n);
    for (int64_t k = 1; k * room < w.ctas; ++k)
      least = std::max(least, (float)(k + 1) * ((float)w.steps[k * room * w.n_rows / w.ctas] / n + fixed));
    return least;
  };
  int best = 1;
  float least = (known ? 0.95f : 0.9f) * time(1);  // a split has to gain that much
  for (int n = 2; n <= kMaxSplit && n * 2 <= w.longest; ++n) {
    if (cap.clusters[n] <= 0) continue;
    const float t = time(n);
    if (t < least) {
      least = t;
      best = n;
    }
  }
  return best;
}

// The number for a call whose capacity the caller gives (clusters[n], n = 1 .. 8) or `device` knows.
template <typename Device>
inline int row_parts(RowWork& w, const int32_t* clusters, Device device) {
  if (!(w.longest > 0.f)) return 1;
  if (clusters == nullptr) {
    const ClusterCapacity* cap = device();
    return cap == nullptr ? SPLASH_ERR_CUDA : split_for(w, *cap);
  }
  ClusterCapacity cap;
  for (int n = 0; n <= kMaxSplit; ++n) cap.clusters[n] = clusters[n];
  if (cap.clusters[1] <= 0) return SPLASH_ERR_INVALID_ARGUMENT;
  return split_for(w, cap);
}

// What fits on the current device, asked once per kernel and device; also sets the kernel's shared-memory size.
inline const ClusterCapacity* cluster_capacity(const void* kernel, int variant, int threads, int smem) {
  static std::mutex mu;
  static ClusterCapacity table[64][16];
  static bool known[64][16] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || variant < 0 || variant >= 16) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  ClusterCapacity& c = table[dev][variant];
  if (!known[dev][variant]) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
    c.clusters[0] = 0;
    c.clusters[1] = sms;
    for (int n = 2; n <= kMaxSplit; ++n) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)n;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3((unsigned)(n * sms));
      cfg.blockDim = dim3((unsigned)threads);
      cfg.dynamicSmemBytes = (size_t)smem;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int count = 0;
      if (cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        count = 0;
      }
      c.clusters[n] = count;
    }
    known[dev][variant] = true;
  }
  return &c;
}

// Which steps of a row belong to which CTA of its cluster: those whose place along the walked axis (forward:
// the kv tile; dkv: the q tile plus the q head's number in its group) is the CTA's rank modulo the CTAs.
// Neighbours fall to different CTAs, so whole rows, windows and what is left of a diagonal all part evenly;
// and the part of a step depends on nothing but its place: tiles that are listed though they hold no live
// key (a partial block of several tiles, the other tile of a pair) leave every sum as it is without them.
// The entries of a row come in ascending order, mostly without a gap; that the entry n further on is the
// tile n further on shows it in one load.
template <bool kSplit>
struct PartWalk {
  const int4* entries;
  int beg, end, n;
  int first_tile, last_tile;

  __device__ __forceinline__ PartWalk(const int4* list, int from, int to, int parts) : entries(list), beg(from), end(to), n(parts) {
    first_tile = beg < end ? entries[beg].x : 0;
    last_tile = beg < end ? entries[end - 1].x : -1;
  }
  // tiles from the row's first one on to the first that is `residue` modulo n
  __device__ __forceinline__ int offset(int residue) const {
    const int d = (residue - first_tile) % n;
    return d < 0 ? d + n : d;
  }
  // the entry of tile `x`, or of the next one of the same part, looked for from `e` on (`end`: none)
  __device__ __forceinline__ int find(int e, int x) const {
    for (; e < end; ++e) {
      const int ahead = entries[e].x - x;
      if (ahead >= 0 && ahead % n == 0) return e;
    }
    return end;
  }
  // the first entry of the part that begins `offset` tiles behind the row's first
  __device__ __forceinline__ int first(int offset) const {
    const int x = first_tile + offset;
    if (x > last_tile) return end;
    return beg + offset < end && entries[beg + offset].x == x ? beg + offset : find(beg, x);
  }
  // the entry behind `e` in its part
  __device__ __forceinline__ int next(int e) const {
    const int x = entries[e].x + n;
    if (x > last_tile) return end;
    return e + n < end && entries[e + n].x == x ? e + n : find(e + 1, x);
  }
  // For loops that fetch an entry a step ahead of its use: where tile x = (tile of `e`) + n is if the row has no
  // gap before it (`end`: the row ends before x).  Where another tile is found there: find(e + 1, x).
  __device__ __forceinline__ int probe(int e, int x) const { return x > last_tile ? end : min(e + n, end - 1); }
};
template <>
struct PartWalk<false> {  // the whole row
  int beg;
  __device__ __forceinline__ PartWalk(const int4*, int from, int, int) : beg(from) {}
  __device__ __forceinline__ int offset(int) const { return 0; }
  __device__ __forceinline__ int first(int) const { return beg; }
  __device__ __forceinline__ int next(int e) const { return e + 1; }
};

template <typename... Params, typename... Args>
inline cudaError_t launch_clusters(void (*kernel)(Params...), unsigned rows, int n_split, int threads, int smem,
                                   cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(rows * (unsigned)n_split);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  if (n_split > 1) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)n_split;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (err != cudaSuccess) (void)cudaGetLastError();  // reported here: the next call's check is not to find it
  return err;
}

}  // namespace sb
