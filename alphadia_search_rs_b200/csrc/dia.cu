// DIAData construction on the device (DIADataBuilder::from_alpha_raw,
// src/dia_data_builder/mod.rs:11-139) and the DIAData getters.
//
// Layout in HBM, per quadrupole observation w (= delta_scan_idx):
//   slice_starts[slot(w)][b]  u32, b in [0, grid_len], CSR offsets by m/z bin
//   cycles[base(w) + i]       u16 cycle index of entry i
//   intens[base(w) + i]       f32 intensity of entry i
// Entries are ordered by (bin, cycle), ties in the order the reference visits
// peaks (spectrum index, then peak index), exactly like its stable sort_by_key.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <memory>

#include "common.cuh"

namespace ads {
namespace {

// The entries are put in order by a counting sort, a few observations at a time: the bins
// are counted in slice_starts itself, every peak keeping its number within its bin; the
// counts are scanned in place; every peak goes to its place as one 16-byte record; and a
// thread per bin puts its few records in (cycle, visit position) order and writes the
// entries.  Peaks of a group of observations, their counts and records fit the L2, so what
// crosses the memory bus is little more than the peaks once in and the entries once out,
// and the temporary memory is one group's (100 MB).  A radix sort of (window, bin, cycle)
// keys with peak indices for all moved 12 bytes a peak six times through 24 bytes a peak of
// temporaries: 324 M peaks in 25 ms of kernels and 100 ms of mapping and unmapping that
// memory; now 18 ms of kernels and none.  What bounds it: the counting's atomics in the L2
// (5 ms) and the records' scattered writes and reads there (10 ms).
constexpr int64_t kGroupItems = int64_t(1) << 22;
constexpr int kScanTile = 8192;       // bins of one scan block
constexpr int kScanThreads = 256;
constexpr int kBinRegs = 4;           // bins of up to this many entries are sorted in registers
constexpr int kBinThread = 24;        // up to this many by one thread in place
constexpr int kBinShared = 1024;      // up to this many by a block in shared memory
// Bins of many peaks undo that: a block sorts one, and peaks outside the grid all lie in its
// first and last bin.  A group with a bin of more than kBinShared peaks, or with more than
// 1 / kCrowdedShare of its peaks in bins of more than kBinThread, is told by its counts
// before any peak is placed, and sorted whole by a stable radix sort of (window, bin, cycle)
// keys afterwards, whose time does not depend on the bins.  60 M peaks, 10 % of them below the
// grid: 1166 -> 9.3 ms; 1 %: 88 -> 9.3; in 2000 bins: 20 -> 9.1; none crowded: 4.9.  The line:
// 12 M peaks of 16, 20 and 30 a bin in the mean 2.56, 3.12 and 3.95 ms counted, 2.32 sorted;
// a quarter of them in bins of 40, 200 and 700 2.13, 1.79 and 1.96, half 2.71, 2.15 and 2.38,
// against 2.26.
constexpr int kCrowdedShare = 8;

struct GroupCounts {
  unsigned int crowded;  // peaks in bins of more than kBinThread
  unsigned int widest;   // peaks of the widest of those bins
  unsigned int listed;   // of those bins, for order_large_bins_kernel
};
__host__ __device__ inline bool sorted_whole(const GroupCounts& c, int64_t items) {
  return c.widest > (unsigned)kBinShared || (int64_t)c.crowded * kCrowdedShare > items;
}

// A warp takes up to so many peaks of one spectrum: spectra of 150,000 peaks, a warp each,
// left most of the GPU idle (400 of them, 60 M peaks, 123 ms).
constexpr int kPiecePeaks = 2048;
constexpr int kPieceShift = 40;  // a piece: its spectrum, and above it its number in the spectrum

struct PeakPiece {
  int64_t s;      // spectrum
  int64_t first;  // its first peak, counted in the spectrum
  int64_t n;      // peaks
};
__device__ __forceinline__ PeakPiece peak_piece(int64_t id, const int64_t* pstart, const int64_t* pstop) {
  PeakPiece p;
  p.s = id & ((int64_t(1) << kPieceShift) - 1);
  p.first = (id >> kPieceShift) * kPiecePeaks;
  p.n = min(pstop[p.s] - pstart[p.s] - p.first, (int64_t)kPiecePeaks);
  return p;
}

// One observation of a group.
struct BuildWin {
  int64_t ss;       // element offset of its slice_starts
  int64_t base;     // its first entry
};

// A peak on its way to its bin: x intensity, y visit position in the observation, z cycle.
__device__ __forceinline__ uint64_t record_key(const uint4& r) { return (uint64_t)r.z << 32 | r.y; }

// The grid's first and last bin take every peak outside it: a warp's of them are numbered by
// one atomic (60 M peaks, 10 % of them below the grid: 14.9 -> 9.5 ms).  Whole warps call it.
__device__ __forceinline__ bool at_end(const GridView& g, uint32_t bin) { return bin == 0u || bin == g.n - 1u; }
__device__ __noinline__ uint32_t number_peak(uint32_t* count, const GridView& g, uint32_t bin, bool on, int lane) {
  const bool end = on && at_end(g, bin);
  const unsigned lo = __ballot_sync(0xffffffffu, end && bin == 0u), hi = __ballot_sync(0xffffffffu, end && bin != 0u);
  const unsigned own = bin == 0u ? lo : hi;
  const int first = __ffs(own) - 1;  // (of lanes at an end: the first of their bin)
  uint32_t number = 0;
  if (on && (!end || lane == first)) number = atomicAdd(count + bin, end ? (uint32_t)__popc(own) : 1u);
  const uint32_t base = __shfl_sync(0xffffffffu, number, end ? first : lane);
  return end ? base + (uint32_t)__popc(own & ((1u << lane) - 1u)) : number;
}

// One warp per piece of a spectrum (listed in window, then visit order): every peak's bin and
// its number within the bin (in order of arrival, which is any).
__global__ void __launch_bounds__(256) count_peaks_kernel(int64_t n_pieces, const int64_t* __restrict__ list,
                                                          const int64_t* __restrict__ item_off,
                                                          const int64_t* __restrict__ pstart,
                                                          const int64_t* __restrict__ pstop,
                                                          const int32_t* __restrict__ win, int win0,
                                                          const BuildWin* __restrict__ wins, int64_t item0,
                                                          const float* __restrict__ mz, GridView g,
                                                          uint2* __restrict__ bins,
                                                          uint32_t* __restrict__ starts) {
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n_pieces) return;
  const PeakPiece p = peak_piece(list[warp], pstart, pstop);
  const int64_t b = pstart[p.s] + p.first, n = p.n;
  uint2* to = bins + (item_off[p.s] + p.first - item0);
  uint32_t* count = starts + wins[win[p.s] - win0].ss + 1;
  // two peaks a lane at a time: their loads and atomics overlap
  for (int64_t k0 = 0; k0 < n; k0 += 64) {
    const int64_t k = k0 + lane;
    const bool on_a = k < n, on_b = k + 32 < n;
    const uint32_t bin_a = on_a ? grid_find_closest(g, __ldg(mz + b + k)) : 1u;
    const uint32_t bin_b = on_b ? grid_find_closest(g, __ldg(mz + b + k + 32)) : 1u;
    uint32_t number_a = 0, number_b = 0;
    if (__any_sync(0xffffffffu, at_end(g, bin_a) || at_end(g, bin_b))) {
      number_a = number_peak(count, g, bin_a, on_a, lane);
      number_b = number_peak(count, g, bin_b, on_b, lane);
    } else {
      if (on_a) number_a = atomicAdd(count + bin_a, 1u);
      if (on_b) number_b = atomicAdd(count + bin_b, 1u);
    }
    if (on_a) to[k] = make_uint2(bin_a, number_a);
    if (on_b) to[k + 32] = make_uint2(bin_b, number_b);
  }
}

// Inclusive scan of each observation's counts, in place: sums of tiles, their scan, the
// tiles.  counts[b + 1] becomes the end of bin b, which is what slice_starts holds there.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* sh, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) sh[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < kScanThreads / 32 ? sh[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < kScanThreads / 32) sh[lane] = wi - w;
    if (lane == 31) sh[32] = wi;
  }
  __syncthreads();
  const uint32_t r = sh[warp] + incl - v;
  *total = sh[32];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kScanThreads) tile_sums_kernel(int64_t grid_len, int tiles,
                                                                 const BuildWin* __restrict__ wins,
                                                                 const uint32_t* __restrict__ starts,
                                                                 uint32_t* __restrict__ sums,
                                                                 GroupCounts* __restrict__ counts) {
  __shared__ uint32_t sh[33];
  const int w = blockIdx.x / tiles, t = blockIdx.x - w * tiles;
  const uint32_t* c = starts + wins[w].ss + 1;
  uint32_t v = 0, total, crowded = 0, widest = 0;
  c += (int64_t)t * kScanTile;
  const int here = (int)min(grid_len - (int64_t)t * kScanTile, (int64_t)kScanTile);
#pragma unroll 8
  for (int i = threadIdx.x; i < here; i += kScanThreads) {
    const uint32_t n = c[i];
    v += n;
    if (n > (uint32_t)kBinThread) {
      crowded += n;
      widest = max(widest, n);
    }
  }
  __syncwarp();
  crowded = __reduce_add_sync(0xffffffffu, crowded);
  if (crowded) {
    widest = __reduce_max_sync(0xffffffffu, widest);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&counts->crowded, crowded);
      atomicMax(&counts->widest, widest);
    }
  }
  block_scan(v, sh, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(int tiles, uint32_t* __restrict__ sums) {
  __shared__ uint32_t sh[33];
  uint32_t* s = sums + (int64_t)blockIdx.x * tiles;
  uint32_t carry = 0;
  for (int t0 = 0; t0 < tiles; t0 += kScanThreads) {
    const int t = t0 + (int)threadIdx.x;
    uint32_t total;
    const uint32_t v = t < tiles ? s[t] : 0u;
    const uint32_t ex = block_scan(v, sh, &total);
    if (t < tiles) s[t] = carry + ex;
    carry += total;
  }
}

__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(int64_t grid_len, int tiles,
                                                                  const BuildWin* __restrict__ wins,
                                                                  const uint32_t* __restrict__ sums,
                                                                  uint32_t* __restrict__ starts) {
  __shared__ uint32_t sh[33];
  __shared__ uint32_t tile[kScanTile + kScanTile / 32];  // (padded: a thread's run is strided)
  const int w = blockIdx.x / tiles, t = blockIdx.x - w * tiles;
  uint32_t* c = starts + wins[w].ss + 1;
  const int64_t b0 = (int64_t)t * kScanTile;
  constexpr int kRun = kScanTile / kScanThreads;  // 32
  for (int i = threadIdx.x; i < kScanTile; i += kScanThreads)
    tile[i + i / 32] = b0 + i < grid_len ? c[b0 + i] : 0u;
  __syncthreads();
  uint32_t sum = 0, total;
  for (int i = 0; i < kRun; ++i) sum += tile[threadIdx.x * (kRun + 1) + i];
  uint32_t run = sums[blockIdx.x] + block_scan(sum, sh, &total);
  for (int i = 0; i < kRun; ++i) {
    const uint32_t v = tile[threadIdx.x * (kRun + 1) + i];
    run += v;
    tile[threadIdx.x * (kRun + 1) + i] = run;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kScanTile; i += kScanThreads)
    if (b0 + i < grid_len) c[b0 + i] = tile[i + i / 32];
}

// Every peak to its place, as a record.
__global__ void __launch_bounds__(256) place_peaks_kernel(
    int64_t n_pieces, const int64_t* __restrict__ list, const int64_t* __restrict__ item_off,
    const int64_t* __restrict__ pstart, const int64_t* __restrict__ pstop, const int32_t* __restrict__ win,
    const uint16_t* __restrict__ cyc, int win0, const BuildWin* __restrict__ wins, int64_t item0,
    const float* __restrict__ inten, const uint2* __restrict__ bins, const uint32_t* __restrict__ starts,
    uint4* __restrict__ recs, const GroupCounts* __restrict__ counts, int64_t items) {
  if (sorted_whole(*counts, items)) return;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n_pieces) return;
  const PeakPiece p = peak_piece(list[warp], pstart, pstop);
  const BuildWin w = wins[win[p.s] - win0];
  const int64_t b = pstart[p.s] + p.first, n = p.n, at = item_off[p.s] + p.first;
  const uint2* from = bins + (at - item0);
  const uint32_t* first = starts + w.ss;
  uint4* to = recs + (w.base - item0);
  const uint32_t c = cyc[p.s];
  const uint32_t vis0 = (uint32_t)(at - w.base);
#pragma unroll 4
  for (int64_t k = lane; k < n; k += 32) {
    const uint2 br = from[k];
    to[__ldg(first + br.x) + br.y] =
        make_uint4(__float_as_uint(__ldg(inten + b + k)), vis0 + (uint32_t)k, c, 0u);
  }
}

__device__ __forceinline__ void put_in_order(uint4& a, uint4& b) {
  if (record_key(a) > record_key(b)) {
    const uint4 t = a;
    a = b;
    b = t;
  }
}

// One thread per bin: its records in order, and its entries.  Larger bins are listed.
__global__ void __launch_bounds__(256) order_bins_kernel(int64_t grid_len, const BuildWin* __restrict__ wins,
                                                         int64_t item0, const uint32_t* __restrict__ starts,
                                                         uint4* recs, uint16_t* __restrict__ cyc,
                                                         float* __restrict__ inten, uint2* __restrict__ large,
                                                         GroupCounts* counts, int64_t items) {
  if (sorted_whole(*counts, items)) return;
  const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (b >= grid_len) return;
  const BuildWin bw = wins[blockIdx.y];
  const uint32_t e0 = starts[bw.ss + b], n = starts[bw.ss + b + 1] - e0;
  if (n == 0) return;
  if (n > kBinThread) {
    large[atomicAdd(&counts->listed, 1u)] = make_uint2(blockIdx.y, (unsigned)b);
    return;
  }
  uint4* r = recs + (bw.base - item0) + e0;
  uint16_t* c = cyc + bw.base + e0;
  float* y = inten + bw.base + e0;
  if (n <= kBinRegs) {
    uint4 v[kBinRegs];
#pragma unroll
    for (int i = 0; i < kBinRegs; ++i)
      v[i] = i < (int)n ? r[i] : make_uint4(0u, 0xffffffffu, 0xffffffffu, 0u);  // past every key
    put_in_order(v[0], v[1]);
    put_in_order(v[2], v[3]);
    put_in_order(v[0], v[2]);
    put_in_order(v[1], v[3]);
    put_in_order(v[1], v[2]);
#pragma unroll
    for (int i = 0; i < kBinRegs; ++i)
      if (i < (int)n) {
        c[i] = (uint16_t)v[i].z;
        y[i] = __uint_as_float(v[i].x);
      }
    return;
  }
  for (uint32_t a = 1; a < n; ++a) {
    const uint4 v = r[a];
    uint32_t j = a;
    for (; j > 0 && record_key(r[j - 1]) > record_key(v); --j) r[j] = r[j - 1];
    r[j] = v;
  }
  for (uint32_t a = 0; a < n; ++a) {
    const uint4 v = r[a];
    c[a] = (uint16_t)v.z;
    y[a] = __uint_as_float(v.x);
  }
}

// Bitonic sort of n records by a block, every exchange ascending (the first step of each
// merge mirrored), so that the missing records past n count as larger than all.
__device__ void block_sort(uint4* r, uint32_t n) {
  uint32_t p2 = 1;
  while (p2 < n) p2 <<= 1;
  for (uint32_t k = 2; k <= p2; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      const uint32_t flip = j == k >> 1 ? k - 1 : j;
      for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t o = i ^ flip;
        if (o > i && o < n) {
          uint4 a = r[i], b = r[o];
          if (record_key(a) > record_key(b)) {
            r[i] = b;
            r[o] = a;
          }
        }
      }
      __syncthreads();
    }
  }
}

// The bins that order_bins_kernel listed (none of a group that is sorted whole), a block each.
__global__ void __launch_bounds__(256) order_large_bins_kernel(const GroupCounts* __restrict__ counts,
                                                               const uint2* __restrict__ large,
                                                               const BuildWin* __restrict__ wins,
                                                               int64_t item0,
                                                               const uint32_t* __restrict__ starts,
                                                               const uint4* __restrict__ recs,
                                                               uint16_t* __restrict__ cyc,
                                                               float* __restrict__ inten) {
  __shared__ uint4 tile[kBinShared];
  const unsigned int m = counts->listed;
  for (unsigned int l = blockIdx.x; l < m; l += gridDim.x) {
    const uint2 id = large[l];
    const BuildWin bw = wins[id.x];
    const uint32_t e0 = starts[bw.ss + id.y], n = starts[bw.ss + id.y + 1] - e0;
    const uint4* r = recs + (bw.base - item0) + e0;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) tile[i] = r[i];
    __syncthreads();
    block_sort(tile, n);
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      cyc[bw.base + e0 + i] = (uint16_t)tile[i].z;
      inten[bw.base + e0 + i] = __uint_as_float(tile[i].x);
    }
    __syncthreads();
  }
}

// ---- groups that are sorted whole: every peak's key and intensity in visit order, a stable
// radix sort of the keys (window of the group, bin, cycle), the entries
constexpr int kKeyBinShift = 16;
constexpr int kKeyWinShift = 38;  // 22 bits of bin

__global__ void __launch_bounds__(256) key_peaks_kernel(
    int64_t n_pieces, const int64_t* __restrict__ list, const int64_t* __restrict__ item_off,
    const int64_t* __restrict__ pstart, const int64_t* __restrict__ pstop, const int32_t* __restrict__ win,
    const uint16_t* __restrict__ cyc, int win0, int64_t item0, const float* __restrict__ mz,
    const float* __restrict__ inten, GridView g, uint64_t* __restrict__ keys, float* __restrict__ vals) {
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n_pieces) return;
  const PeakPiece p = peak_piece(list[warp], pstart, pstop);
  const int64_t b = pstart[p.s] + p.first, to = item_off[p.s] + p.first - item0;
  const uint64_t rest = (uint64_t)(win[p.s] - win0) << kKeyWinShift | cyc[p.s];
  for (int64_t k = lane; k < p.n; k += 32) {
    keys[to + k] = rest | (uint64_t)grid_find_closest(g, __ldg(mz + b + k)) << kKeyBinShift;
    vals[to + k] = __ldg(inten + b + k);
  }
}

__global__ void __launch_bounds__(256) sorted_entries_kernel(int64_t n, const uint64_t* __restrict__ keys,
                                                             const float* __restrict__ vals,
                                                             uint16_t* __restrict__ cyc,
                                                             float* __restrict__ inten) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  cyc[i] = (uint16_t)keys[i];
  inten[i] = vals[i];
}

struct SpectrumTable {
  std::vector<int64_t> dsi, start, stop, cyc;
  std::vector<float> lo, hi, rt;
};

template <class T>
int fetch(const T* src, int64_t n, int loc, std::vector<T>& dst) {
  dst.resize((size_t)n);
  if (n == 0) return ADS_OK;
  if (!src) return fail(ADS_ERR_INVALID_ARGUMENT, "null array pointer");
  if (loc == ADS_MEM_DEVICE) {
    ADS_CUDA(cudaMemcpy(dst.data(), src, (size_t)n * sizeof(T), cudaMemcpyDeviceToHost));
  } else {
    std::memcpy(dst.data(), src, (size_t)n * sizeof(T));
  }
  return ADS_OK;
}

// Uploads the spectrum table (and host peak arrays), and builds cycles, intens and
// slice_starts.  `list`: the pieces of window w's spectra in visit order from first_piece[w].
int build_entries(AdsDia* d, const AdsRawArrays* raw, const std::vector<int32_t>& win_of_spec,
                  const std::vector<uint16_t>& cyc16, const std::vector<int64_t>& item_off,
                  int64_t n_items, const std::vector<int64_t>& list, const std::vector<int64_t>& first_piece,
                  int64_t n_slots, const GridView& g, cudaStream_t st) {
  const int64_t n_spec = raw->n_spectra;
  const int64_t stride = d->grid_len + 1;
  if (n_slots == 0 || n_items == 0) return ADS_OK;
  // device copies of the spectrum table and, if needed, the peak arrays
  DevBuf<int64_t> d_off, d_start, d_stop;
  DevBuf<int32_t> d_win;
  DevBuf<int64_t> d_list;
  DevBuf<uint16_t> d_cyc;
  DevBuf<float> d_mz, d_int;
  const float* mz = raw->peak_mz;
  const float* pint = raw->peak_intensity;
  const int64_t *pstart = raw->spectrum_peak_start_idx, *pstop = raw->spectrum_peak_stop_idx;
  ADS_TRY(d_off.alloc(n_spec));
  ADS_TRY(d_win.alloc(n_spec));
  ADS_TRY(d_cyc.alloc(n_spec));
  ADS_TRY(d_list.alloc(list.size()));
  ADS_CUDA(cudaMemcpyAsync(d_off.p, item_off.data(), n_spec * 8, cudaMemcpyHostToDevice, st));
  ADS_CUDA(cudaMemcpyAsync(d_win.p, win_of_spec.data(), n_spec * 4, cudaMemcpyHostToDevice, st));
  ADS_CUDA(cudaMemcpyAsync(d_cyc.p, cyc16.data(), n_spec * 2, cudaMemcpyHostToDevice, st));
  ADS_CUDA(cudaMemcpyAsync(d_list.p, list.data(), list.size() * 8, cudaMemcpyHostToDevice, st));
  if (raw->location != ADS_MEM_DEVICE) {
    ADS_TRY(d_start.alloc(n_spec));
    ADS_TRY(d_stop.alloc(n_spec));
    ADS_CUDA(cudaMemcpyAsync(d_start.p, pstart, n_spec * 8, cudaMemcpyHostToDevice, st));
    ADS_CUDA(cudaMemcpyAsync(d_stop.p, pstop, n_spec * 8, cudaMemcpyHostToDevice, st));
    ADS_TRY(d_mz.alloc(raw->n_peaks));
    ADS_TRY(d_int.alloc(raw->n_peaks));
    ADS_CUDA(cudaMemcpyAsync(d_mz.p, raw->peak_mz, raw->n_peaks * 4, cudaMemcpyHostToDevice, st));
    ADS_CUDA(cudaMemcpyAsync(d_int.p, raw->peak_intensity, raw->n_peaks * 4, cudaMemcpyHostToDevice, st));
    pstart = d_start.p;
    pstop = d_stop.p;
    mz = d_mz.p;
    pint = d_int.p;
  }
  ADS_TRY(d->cycles.alloc(n_items + kEntrySlack));  // (16-byte copies may reach past the last entry)
  ADS_TRY(d->intens.alloc(n_items + kEntrySlack));
  ADS_TRY(d->slice_starts.alloc((size_t)(n_slots * stride)));
  ADS_CUDA(cudaMemsetAsync(d->slice_starts.p, 0, d->slice_starts.bytes(), st));

  // the observations that hold peaks, in groups of up to kGroupItems peaks (or one)
  struct Group {
    int64_t w0, w1, items, pieces;
    int slots;
  };
  std::vector<Group> groups;
  std::vector<BuildWin> wins((size_t)d->n_obs, BuildWin{0, 0});
  int64_t most_items = 0;
  int most_slots = 0;
  for (int64_t w = 0; w < d->n_obs; ++w) {
    wins[w] = BuildWin{d->win[w].ss_off, d->win[w].base};
    if (d->num_peaks[w] == 0) continue;
    if (groups.empty() || groups.back().items + d->num_peaks[w] > kGroupItems || groups.back().w1 != w ||
        groups.back().slots == 1024)  // (slots are a grid dimension)
      groups.push_back(Group{w, w, 0, 0, 0});
    Group& gr = groups.back();
    gr.w1 = w + 1;
    gr.items += d->num_peaks[w];
    gr.pieces += first_piece[w + 1] - first_piece[w];
    ++gr.slots;
    most_items = std::max(most_items, gr.items);
    most_slots = std::max(most_slots, gr.slots);
  }
  const int tiles = (int)((d->grid_len + kScanTile - 1) / kScanTile);
  DevBuf<BuildWin> d_wins;
  DevBuf<uint32_t> sums;
  DevBuf<uint2> bins, large;
  DevBuf<uint4> recs;
  DevBuf<GroupCounts> counts;
  ADS_TRY(d_wins.alloc(wins.size()));
  // (a group that is sorted whole has its keys in `bins` and the rest of the sort's buffers
  // in `recs`, in four multiples of 64 peaks)
  const size_t most_up = ((size_t)most_items + 63) / 64 * 64;
  ADS_TRY(bins.alloc(most_up));
  ADS_TRY(recs.alloc(most_up));
  ADS_TRY(sums.alloc((size_t)most_slots * tiles));
  ADS_TRY(large.alloc((size_t)(most_items / (kBinThread + 1) + 1)));
  ADS_TRY(counts.alloc(groups.size()));
  ADS_CUDA(cudaMemcpyAsync(d_wins.p, wins.data(), wins.size() * sizeof(BuildWin), cudaMemcpyHostToDevice, st));
  ADS_CUDA(cudaMemsetAsync(counts.p, 0, counts.bytes(), st));
  for (size_t k = 0; k < groups.size(); ++k) {
    const Group& gr = groups[k];
    const int64_t item0 = d->win[gr.w0].base;
    const BuildWin* gw = d_wins.p + gr.w0;
    const int64_t* gl = d_list.p + first_piece[gr.w0];
    const int sg = (int)((gr.pieces + 7) / 8);
    count_peaks_kernel<<<sg, 256, 0, st>>>(gr.pieces, gl, d_off.p, pstart, pstop, d_win.p, (int)gr.w0, gw, item0,
                                           mz, g, bins.p, d->slice_starts.p);
    ADS_LAUNCH_CHECK();
    tile_sums_kernel<<<gr.slots * tiles, kScanThreads, 0, st>>>(d->grid_len, tiles, gw, d->slice_starts.p, sums.p,
                                                                counts.p + k);
    ADS_LAUNCH_CHECK();
    scan_sums_kernel<<<gr.slots, kScanThreads, 0, st>>>(tiles, sums.p);
    ADS_LAUNCH_CHECK();
    scan_tiles_kernel<<<gr.slots * tiles, kScanThreads, 0, st>>>(d->grid_len, tiles, gw, sums.p, d->slice_starts.p);
    ADS_LAUNCH_CHECK();
    place_peaks_kernel<<<sg, 256, 0, st>>>(gr.pieces, gl, d_off.p, pstart, pstop, d_win.p, d_cyc.p, (int)gr.w0, gw,
                                           item0, pint, bins.p, d->slice_starts.p, recs.p, counts.p + k, gr.items);
    ADS_LAUNCH_CHECK();
    order_bins_kernel<<<dim3((unsigned)((d->grid_len + 255) / 256), (unsigned)gr.slots), 256, 0, st>>>(
        d->grid_len, gw, item0, d->slice_starts.p, recs.p, d->cycles.p, d->intens.p, large.p, counts.p + k,
        gr.items);
    ADS_LAUNCH_CHECK();
    order_large_bins_kernel<<<148 * 4, 256, 0, st>>>(counts.p + k, large.p, gw, item0, d->slice_starts.p,
                                                     recs.p, d->cycles.p, d->intens.p);
    ADS_LAUNCH_CHECK();
  }
  // the groups whose bins are too full for that
  std::vector<GroupCounts> told(groups.size());
  ADS_CUDA(cudaMemcpyAsync(told.data(), counts.p, counts.bytes(), cudaMemcpyDeviceToHost, st));
  ADS_CUDA(cudaStreamSynchronize(st));
  DevBuf<unsigned char> tmp;
  for (size_t k = 0; k < groups.size(); ++k) {
    const Group& gr = groups[k];
    if (!sorted_whole(told[k], gr.items)) continue;
    const int64_t item0 = d->win[gr.w0].base;
    uint64_t* keys_b = reinterpret_cast<uint64_t*>(recs.p);
    float* vals_a = reinterpret_cast<float*>(keys_b + most_up);
    cub::DoubleBuffer<uint64_t> keys(reinterpret_cast<uint64_t*>(bins.p), keys_b);
    cub::DoubleBuffer<float> vals(vals_a, vals_a + most_up);
    int end_bit = kKeyWinShift;
    while ((gr.slots - 1) >> (end_bit - kKeyWinShift)) ++end_bit;
    size_t need = 0;
    ADS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, need, keys, vals, gr.items, 0, end_bit, st));
    ADS_TRY(tmp.reserve(need + 16));
    key_peaks_kernel<<<(int)((gr.pieces + 7) / 8), 256, 0, st>>>(
        gr.pieces, d_list.p + first_piece[gr.w0], d_off.p, pstart, pstop, d_win.p, d_cyc.p, (int)gr.w0, item0, mz,
        pint, g, keys.Current(), vals.Current());
    ADS_LAUNCH_CHECK();
    ADS_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, need, keys, vals, gr.items, 0, end_bit, st));
    sorted_entries_kernel<<<(unsigned)((gr.items + 255) / 256), 256, 0, st>>>(
        gr.items, keys.Current(), vals.Current(), d->cycles.p + item0, d->intens.p + item0);
    ADS_LAUNCH_CHECK();
  }
  ADS_CUDA(cudaStreamSynchronize(st));
  return ADS_OK;
}

// The run's WinIndex on the device.  Left out (windows are then scanned) where its lists
// would exceed kWinIndexMax entries: hundreds of windows all over one another (a run of 300
// windows that meet at their limits has 1500).
constexpr size_t kWinIndexMax = size_t(1) << 16;

int build_win_index(AdsDia* d) {
  std::vector<float> v;
  std::vector<int> open;
  for (int64_t w = 0; w < d->n_obs; ++w) {
    const WinInfo& wi = d->win[w];
    if (wi.ss_off < 0 || !(wi.lo <= wi.hi)) continue;  // holds no peaks, or no m/z
    v.push_back(wi.lo);
    v.push_back(wi.hi);
    open.push_back((int)w);
  }
  std::sort(v.begin(), v.end());
  v.erase(std::unique(v.begin(), v.end()), v.end());
  const int m = (int)v.size();
  auto at = [&](float x) { return (int)(std::lower_bound(v.begin(), v.end(), x) - v.begin()); };
  // windows hold the classes from their lower limit's to their upper limit's
  std::vector<int> off(2 * (size_t)m + 2, 0);
  size_t total = 0;
  for (int w : open) total += 2 * (size_t)(at(d->win[w].hi) - at(d->win[w].lo)) + 1;
  if (total > kWinIndexMax) return ADS_OK;
  for (int w : open)
    for (int k = 2 * at(d->win[w].lo) + 1; k <= 2 * at(d->win[w].hi) + 1; ++k) ++off[k + 1];
  for (size_t k = 1; k < off.size(); ++k) off[k] += off[k - 1];
  std::vector<int> cur(off.begin(), off.end() - 1), list(total);
  for (int w : open)  // ascending, so every class's list is in window order
    for (int k = 2 * at(d->win[w].lo) + 1; k <= 2 * at(d->win[w].hi) + 1; ++k) list[cur[k]++] = w;
  std::vector<int> host(3 * (size_t)m + 2 + total);
  if (m) std::memcpy(host.data(), v.data(), (size_t)m * 4);
  std::copy(off.begin(), off.end(), host.begin() + m);
  std::copy(list.begin(), list.end(), host.begin() + 3 * (size_t)m + 2);
  ADS_TRY(d->win_index_dev.alloc(host.size()));
  ADS_CUDA(cudaMemcpy(d->win_index_dev.p, host.data(), host.size() * 4, cudaMemcpyHostToDevice));
  d->win_index_m = m;
  d->win_index_ok = true;
  return ADS_OK;
}

int dia_create(const AdsRawArrays* raw, int device, AdsDia** out) {
  if (!raw || !out) return fail(ADS_ERR_INVALID_ARGUMENT, "null argument");
  *out = nullptr;
  if (raw->location != ADS_MEM_HOST && raw->location != ADS_MEM_DEVICE)
    return fail(ADS_ERR_INVALID_ARGUMENT, "location must be ADS_MEM_HOST or ADS_MEM_DEVICE");
  const int64_t n_spec = raw->n_spectra, n_peaks = raw->n_peaks;
  if (n_spec <= 0)
    return fail(ADS_ERR_INVALID_ARGUMENT, "DIAData needs at least one spectrum");
  if (n_peaks < 0) return fail(ADS_ERR_INVALID_ARGUMENT, "n_peaks < 0");
  if (n_peaks > 0 && (!raw->peak_mz || !raw->peak_intensity))
    return fail(ADS_ERR_INVALID_ARGUMENT, "null peak array");
  int n_dev = 0;
  if (cudaGetDeviceCount(&n_dev) != cudaSuccess || n_dev == 0) {
    cudaGetLastError();
    return fail(ADS_ERR_CUDA, "no CUDA device available");
  }
  if (device < 0 || device >= n_dev) return fail(ADS_ERR_INVALID_ARGUMENT, "bad device index");
  DeviceGuard dg(device);

  SpectrumTable t;
  const int L = raw->location;
  ADS_TRY(fetch(raw->spectrum_delta_scan_idx, n_spec, L, t.dsi));
  ADS_TRY(fetch(raw->spectrum_peak_start_idx, n_spec, L, t.start));
  ADS_TRY(fetch(raw->spectrum_peak_stop_idx, n_spec, L, t.stop));
  ADS_TRY(fetch(raw->spectrum_cycle_idx, n_spec, L, t.cyc));
  ADS_TRY(fetch(raw->isolation_lower_mz, n_spec, L, t.lo));
  ADS_TRY(fetch(raw->isolation_upper_mz, n_spec, L, t.hi));
  ADS_TRY(fetch(raw->spectrum_rt, n_spec, L, t.rt));

  // validation the reference leaves to panics or silent truncation
  int64_t max_dsi = t.dsi[0];
  for (int64_t s = 0; s < n_spec; ++s) {
    if (t.start[s] < 0 || t.stop[s] < t.start[s] || t.stop[s] > n_peaks)
      return fail(ADS_ERR_INVALID_ARGUMENT,
                  "spectrum " + std::to_string(s) + ": peak range outside [0, n_peaks] or start > stop");
    if (t.cyc[s] < 0 || t.cyc[s] > 65535)
      return fail(ADS_ERR_INVALID_ARGUMENT,
                  "spectrum " + std::to_string(s) + ": cycle index outside [0, 65535]");
    max_dsi = std::max(max_dsi, t.dsi[s]);
  }
  if (max_dsi > (int64_t(1) << 20))
    return fail(ADS_ERR_INVALID_ARGUMENT, "delta_scan_idx above 2^20");
  const int64_t n_obs = max_dsi >= 0 ? max_dsi + 1 : 0;

  auto d = new AdsDia();
  std::unique_ptr<AdsDia> guard(d);
  d->device = device;
  d->n_obs = n_obs;
  d->grid_len = (int64_t)host_grid().size();
  d->win.assign((size_t)n_obs, WinInfo{0.0f, 0.0f, 0, -1});
  d->num_cycles.assign((size_t)n_obs, 0);
  d->num_peaks.assign((size_t)n_obs, 0);
  d->rt_values = t.rt;

  // RT index from MS1 scans (src/rt_index/mod.rs:53-75)
  for (int64_t s = 0; s < n_spec; ++s)
    if (t.dsi[s] == 0) d->rt.push_back(t.rt[s]);
  const int64_t n_rt = (int64_t)d->rt.size();
  d->delta_t = n_rt > 1 ? (d->rt[n_rt - 1] - d->rt[0]) / (float)(n_rt - 1) : 1.0f;

  // per observation: isolation window of the first spectrum, unique cycles,
  // peak counts (src/dia_data_builder/mod.rs:57-91)
  std::vector<char> seen_first((size_t)n_obs, 0);
  std::vector<int32_t> win_of_spec((size_t)n_spec, -1);
  std::vector<uint16_t> cyc16((size_t)n_spec);
  std::vector<int64_t> first_piece((size_t)n_obs + 1, 0);
  std::vector<int64_t> last_cycle((size_t)n_obs, -1);
  std::vector<char> unsorted((size_t)n_obs, 0);  // cycles that step back: counted below
  for (int64_t s = 0; s < n_spec; ++s) {
    cyc16[s] = (uint16_t)t.cyc[s];
    const int64_t w = t.dsi[s];
    if (w < 0) continue;
    win_of_spec[s] = (int32_t)w;
    if (!seen_first[w]) {
      seen_first[w] = 1;
      d->win[w].lo = t.lo[s];
      d->win[w].hi = t.hi[s];
    }
    d->num_peaks[w] += t.stop[s] - t.start[s];
    first_piece[w + 1] += (t.stop[s] - t.start[s] + kPiecePeaks - 1) / kPiecePeaks;
    if (t.cyc[s] > last_cycle[w]) {
      ++d->num_cycles[w];
      last_cycle[w] = t.cyc[s];
    } else if (t.cyc[s] < last_cycle[w]) {
      unsorted[w] = 1;
    }
  }
  // the pieces of the spectra by window, in visit order
  for (int64_t w = 0; w < n_obs; ++w) first_piece[w + 1] += first_piece[w];
  std::vector<int64_t> pieces((size_t)first_piece[n_obs]);
  {
    std::vector<int64_t> cursor(first_piece.begin(), first_piece.end() - 1);
    for (int64_t s = 0; s < n_spec; ++s)
      for (int64_t i = 0; win_of_spec[s] >= 0 && i * kPiecePeaks < t.stop[s] - t.start[s]; ++i)
        pieces[cursor[win_of_spec[s]]++] = s | i << kPieceShift;
  }
  if (std::find(unsorted.begin(), unsorted.end(), 1) != unsorted.end()) {
    std::vector<std::vector<int64_t>> c((size_t)n_obs);
    for (int64_t s = 0; s < n_spec; ++s)
      if (t.dsi[s] >= 0 && unsorted[t.dsi[s]]) c[t.dsi[s]].push_back(t.cyc[s]);
    for (int64_t w = 0; w < n_obs; ++w) {
      if (!unsorted[w]) continue;
      std::sort(c[w].begin(), c[w].end());
      d->num_cycles[w] = std::unique(c[w].begin(), c[w].end()) - c[w].begin();
    }
  }

  // entry bases and slice_starts slots (observations without peaks get none)
  int64_t n_slots = 0, n_items = 0;
  for (int64_t w = 0; w < n_obs; ++w) {
    if (d->num_peaks[w] > 0xFFFFFFFFll)
      return fail(ADS_ERR_INVALID_ARGUMENT, "more than 2^32-1 peaks in one observation");
    d->win[w].base = n_items;
    n_items += d->num_peaks[w];
    if (d->num_peaks[w] > 0) {
      d->win[w].ss_off = n_slots * (d->grid_len + 1);
      ++n_slots;
    }
  }
  std::vector<int64_t> item_off((size_t)n_spec, 0);
  {
    std::vector<int64_t> cursor((size_t)std::max<int64_t>(n_obs, 1), 0);
    for (int64_t w = 0; w < n_obs; ++w) cursor[w] = d->win[w].base;
    for (int64_t s = 0; s < n_spec; ++s) {
      const int64_t w = t.dsi[s];
      if (w < 0) continue;
      item_off[s] = cursor[w];
      cursor[w] += t.stop[s] - t.start[s];
    }
  }
  d->n_entries = n_items;

  // maximum depth of overlapping (non-empty) isolation windows, closed intervals
  {
    std::vector<std::pair<float, int>> ev;
    for (int64_t w = 0; w < n_obs; ++w)
      if (d->num_peaks[w] > 0 && d->win[w].lo <= d->win[w].hi) {
        ev.emplace_back(d->win[w].lo, -1);  // opens sort first at equal m/z
        ev.emplace_back(d->win[w].hi, +1);
      }
    std::sort(ev.begin(), ev.end());
    int depth = 0, best = 0;
    for (auto& e : ev) {
      depth += (e.second < 0) ? 1 : -1;
      best = std::max(best, depth);
    }
    d->max_overlap = best;
  }

  if (raw->cycle) {
    int64_t nc = 1;
    for (int i = 0; i < 4; ++i) {
      if (raw->cycle_shape[i] < 0) return fail(ADS_ERR_INVALID_ARGUMENT, "negative cycle shape");
      nc *= raw->cycle_shape[i];
      d->cycle_shape[i] = raw->cycle_shape[i];
    }
    d->cycle.assign(raw->cycle, raw->cycle + nc);
  }

  GridView g;
  ADS_TRY(device_grid(device, &g));
  cudaStream_t st;
  ADS_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  const int rc = build_entries(d, raw, win_of_spec, cyc16, item_off, n_items, pieces, first_piece, n_slots, g, st);
  cudaStreamDestroy(st);
  if (rc != ADS_OK) return rc;

  ADS_TRY(d->win_dev.alloc(std::max<int64_t>(n_obs, 1)));
  if (n_obs)
    ADS_CUDA(cudaMemcpy(d->win_dev.p, d->win.data(), n_obs * sizeof(WinInfo), cudaMemcpyHostToDevice));
  ADS_TRY(build_win_index(d));
  ADS_TRY(d->rt_dev.alloc(std::max<int64_t>(n_rt, 1)));
  if (n_rt) ADS_CUDA(cudaMemcpy(d->rt_dev.p, d->rt.data(), n_rt * 4, cudaMemcpyHostToDevice));
  // copies from pageable memory may return before their DMA ends; searches read these
  // tables from non-blocking streams
  ADS_CUDA(cudaDeviceSynchronize());
  *out = guard.release();
  return ADS_OK;
}

}  // namespace
}  // namespace ads

using namespace ads;

extern "C" {

const char* ads_version(void) { return "alphadia-search-b200 0.1.0"; }

int ads_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int ads_dia_create(const AdsRawArrays* raw, int device, AdsDia** out) {
  return guarded([&] { return dia_create(raw, device, out); });
}

int ads_dia_destroy(AdsDia* dia) {
  return guarded([&] {
    if (dia) {
      DeviceGuard dg(dia->device);
      delete dia;
    }
    return ADS_OK;
  });
}

int64_t ads_dia_num_observations(const AdsDia* dia) { return dia ? dia->n_obs : 0; }

int64_t ads_dia_memory_footprint_bytes(const AdsDia* dia) {
  if (!dia) return 0;
  // src/dia_data/mod.rs:90-105 + src/quadrupole_observation/mod.rs:110-128 with
  // 64-bit Rust layouts: Vec = 24 bytes, usize = 8, [f32; 2] = 8.
  int64_t total = (int64_t)dia->rt.size() * 4 + 24;
  for (int64_t w = 0; w < dia->n_obs; ++w)
    total += 8 + 8 + 3 * 24 + (dia->grid_len + 1) * 4 + dia->num_peaks[w] * (2 + 4);
  return total;
}

int64_t ads_dia_device_bytes(const AdsDia* dia) {
  if (!dia) return 0;
  return (int64_t)(dia->slice_starts.bytes() + dia->cycles.bytes() + dia->intens.bytes() +
                   dia->intens_bf16.bytes() + dia->win_dev.bytes() + dia->win_index_dev.bytes() +
                   dia->rt_dev.bytes());
}

int ads_dia_rt_values(const AdsDia* dia, float* out, int64_t cap, int64_t* n) {
  return guarded([&] {
    if (!dia) return fail(ADS_ERR_INVALID_ARGUMENT, "null handle");
    const int64_t m = (int64_t)dia->rt_values.size();
    if (n) *n = m;
    if (out) std::memcpy(out, dia->rt_values.data(), (size_t)std::min(m, cap) * 4);
    return ADS_OK;
  });
}

int ads_dia_cycle(const AdsDia* dia, float* out, int64_t cap, int64_t shape[4]) {
  return guarded([&] {
    if (!dia) return fail(ADS_ERR_INVALID_ARGUMENT, "null handle");
    if (shape)
      for (int i = 0; i < 4; ++i) shape[i] = dia->cycle_shape[i];
    if (out)
      std::memcpy(out, dia->cycle.data(),
                  (size_t)std::min<int64_t>((int64_t)dia->cycle.size(), cap) * 4);
    return ADS_OK;
  });
}

int ads_dia_rt_index(const AdsDia* dia, float* out, int64_t cap, int64_t* n, float* delta_t) {
  return guarded([&] {
    if (!dia) return fail(ADS_ERR_INVALID_ARGUMENT, "null handle");
    const int64_t m = (int64_t)dia->rt.size();
    if (n) *n = m;
    if (delta_t) *delta_t = dia->delta_t;
    if (out) std::memcpy(out, dia->rt.data(), (size_t)std::min(m, cap) * 4);
    return ADS_OK;
  });
}

int ads_dia_observation_info(const AdsDia* dia, int64_t obs, float* lo, float* hi,
                             int64_t* num_cycles, int64_t* num_peaks) {
  return guarded([&] {
    if (!dia || obs < 0 || obs >= dia->n_obs)
      return fail(ADS_ERR_INVALID_ARGUMENT, "bad observation index");
    if (lo) *lo = dia->win[obs].lo;
    if (hi) *hi = dia->win[obs].hi;
    if (num_cycles) *num_cycles = dia->num_cycles[obs];
    if (num_peaks) *num_peaks = dia->num_peaks[obs];
    return ADS_OK;
  });
}

int ads_dia_copy_observation(const AdsDia* dia, int64_t obs, uint32_t* ss, uint16_t* cyc,
                             float* inten) {
  return guarded([&] {
    if (!dia || obs < 0 || obs >= dia->n_obs)
      return fail(ADS_ERR_INVALID_ARGUMENT, "bad observation index");
    DeviceGuard dg(dia->device);
    const auto& w = dia->win[obs];
    const int64_t n = dia->num_peaks[obs];
    if (ss) {
      if (w.ss_off < 0)
        std::memset(ss, 0, (size_t)(dia->grid_len + 1) * 4);
      else
        ADS_CUDA(cudaMemcpy(ss, dia->slice_starts.p + w.ss_off, (dia->grid_len + 1) * 4,
                            cudaMemcpyDeviceToHost));
    }
    if (cyc && n)
      ADS_CUDA(cudaMemcpy(cyc, dia->cycles.p + w.base, n * 2, cudaMemcpyDeviceToHost));
    if (inten && n) {
      if (dia->bf16_only) {  // the stored bfloat16 values, widened
        std::vector<uint16_t> b((size_t)n);
        ADS_CUDA(cudaMemcpy(b.data(), dia->intens_bf16.p + w.base, n * 2, cudaMemcpyDeviceToHost));
        for (int64_t i = 0; i < n; ++i) {
          const uint32_t bits = (uint32_t)b[(size_t)i] << 16;
          std::memcpy(inten + i, &bits, 4);
        }
      } else {
        ADS_CUDA(cudaMemcpy(inten, dia->intens.p + w.base, n * 4, cudaMemcpyDeviceToHost));
      }
    }
    return ADS_OK;
  });
}

int64_t ads_mz_grid_len(void) { return (int64_t)host_grid().size(); }

int ads_mz_grid(float* out, int64_t cap) {
  return guarded([&] {
    const auto& g = host_grid();
    if (!out) return fail(ADS_ERR_INVALID_ARGUMENT, "null output");
    std::memcpy(out, g.data(), (size_t)std::min<int64_t>((int64_t)g.size(), cap) * 4);
    return ADS_OK;
  });
}

}  // extern "C"
