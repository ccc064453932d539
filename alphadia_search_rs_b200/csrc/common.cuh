// Internal declarations shared by the engine's translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "ads_gpu.h"

namespace ads {

// ------------------------------------------------------------------ errors
void set_error(const std::string& msg);
void clear_error();
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what, const char* file, int line);

#define ADS_TRY(expr)                   \
  do {                                  \
    int _rc = (expr);                   \
    if (_rc != ADS_OK) return _rc;      \
  } while (0)

#define ADS_CUDA(expr)                                                  \
  do {                                                                  \
    cudaError_t _e = (expr);                                            \
    if (_e != cudaSuccess) return ::ads::cuda_fail(_e, #expr, __FILE__, __LINE__); \
  } while (0)

#define ADS_LAUNCH_CHECK() ADS_CUDA(cudaGetLastError())

// Runs `body` and converts C++ exceptions to status codes so nothing crosses
// the C boundary.
template <class F>
int guarded(F&& body) {
  try {
    clear_error();
    return body();
  } catch (const std::bad_alloc&) {
    return fail(ADS_ERR_OUT_OF_MEMORY, "host allocation failed");
  } catch (const std::exception& e) {
    return fail(ADS_ERR_INTERNAL, e.what());
  } catch (...) {
    return fail(ADS_ERR_INTERNAL, "unknown exception");
  }
}

// Device-current guard: restores the previous device on scope exit.
struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (dev != prev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

// ------------------------------------------------------------ device memory
// Every device buffer of the engine comes from one memory pool per device that
// keeps up to kPoolKeepBytes of freed memory for reuse, so that building a
// library or a candidate collection per call does not map and unmap device pages
// each time.  pool_alloc and pool_free are ordered on a private stream of the pool, and
// pool_free first waits for the device to go idle (the guarantee cudaFree gives), so no
// kernel still in flight can see its memory handed out again; the forms below leave the
// waits out where the caller knows the order.
constexpr uint64_t kPoolKeepBytes = uint64_t(4) << 30;
int pool_alloc(int device, size_t bytes, void** out);
void pool_free(int device, void* p);
// Frees p once the work enqueued on `st` so far is done (no host synchronisation): for
// memory that only `st` uses.
void pool_free_async(int device, void* p, cudaStream_t st);

// Memory for `st` only, from where it stands: no host synchronisation.
int pool_alloc_async(int device, size_t bytes, cudaStream_t st, void** out);
// Frees p, which no work in flight uses: no host synchronisation.
void pool_free_idle(int device, void* p);

// Owning device buffer (move-only) on the current device's pool.
template <class T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  int dev = -1;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n), dev(o.dev) {
    o.p = nullptr;
    o.n = 0;
  }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      n = o.n;
      dev = o.dev;
      o.p = nullptr;
      o.n = 0;
    }
    return *this;
  }
  ~DevBuf() { release(); }
  void release() {
    if (p) pool_free(dev, p);
    p = nullptr;
    n = 0;
  }
  // release() for a buffer that only `st` has used: ordered after its work on `st`.
  void release_async(cudaStream_t st) {
    if (p) pool_free_async(dev, p, st);
    p = nullptr;
    n = 0;
  }
  // release() for a buffer that no work in flight uses.
  void release_idle() {
    if (p) pool_free_idle(dev, p);
    p = nullptr;
    n = 0;
  }
  // alloc() for a buffer that `st` uses first (any other stream after an event of `st`).
  int alloc_on(size_t count, cudaStream_t st) {
    release();
    if (count == 0) return ADS_OK;
    int d = 0;
    ADS_CUDA(cudaGetDevice(&d));
    void* q = nullptr;
    ADS_TRY(pool_alloc_async(d, count * sizeof(T), st, &q));
    p = static_cast<T*>(q);
    n = count;
    dev = d;
    return ADS_OK;
  }
  // Allocates exactly `count` elements on the current device (frees the previous
  // buffer).
  int alloc(size_t count) {
    release();
    if (count == 0) return ADS_OK;
    int d = 0;
    ADS_CUDA(cudaGetDevice(&d));
    void* q = nullptr;
    ADS_TRY(pool_alloc(d, count * sizeof(T), &q));
    p = static_cast<T*>(q);
    n = count;
    dev = d;
    return ADS_OK;
  }
  // Grows to at least `count` elements, keeping nothing.
  int reserve(size_t count) { return count <= n ? ADS_OK : alloc(count); }
  size_t bytes() const { return n * sizeof(T); }
};

// A call's temporary memory on one stream: allocated and freed in its order (an allocation
// with a host synchronisation and a release after a device-wide one took 10 to 15 us each,
// more than the kernels of a small call between them).
template <class T>
struct TmpBuf : DevBuf<T> {
  cudaStream_t st;
  explicit TmpBuf(cudaStream_t s) : st(s) {}
  ~TmpBuf() { this->release_async(st); }
  int alloc(size_t count) {
    this->release_async(st);
    return this->alloc_on(count, st);
  }
};

// ---------------------------------------------------------------- m/z grid
// The global 1-ppm grid (src/mz_index/mod.rs:4-25).  Each of its steps, cur * 1e-6 rounded
// to cur's last place, is a whole number of such places (8 to 17), and the number changes
// only 39 times between 150 and 2000 m/z: the float bit patterns of the 2.6 M points are 40
// arithmetic sequences.  A bound is found from its sequence by one division, without
// reading the grid (a bracket by a table of the bit patterns and a search of the grid inside
// it were 5 dependent loads from 12 MB).
struct GridRun {
  uint32_t bits;   // bit pattern of the first point
  uint32_t next;   // of the next run's first point
  uint32_t magic;  // floor(2^32 / step) + 1: x * magic >> 32 = x / step for x * step < 2^32
  uint32_t at;     // index of the first point; the step in the top 8 bits
};
constexpr int kRunShift = 16;  // bit patterns per entry of run_of (runs are longer, but three)

struct GridView {
  const float* grid = nullptr;
  const GridRun* runs = nullptr;
  const uint8_t* run_of = nullptr;  // run of the first bit pattern of each 2^kRunShift
  uint32_t n = 0;       // grid length
  uint32_t bits0 = 0;   // bit pattern of grid[0]
  float first = 0.0f;
  float last = 0.0f;
};

const std::vector<float>& host_grid();
int device_grid(int device, GridView* out);

// Gaussian kernel of PeakGroupSelection::new (src/kernel/mod.rs:13-56).
std::vector<float> gaussian_kernel(float fwhm_rt, float sigma_scale_rt, int64_t kernel_width,
                                   float rt_resolution);

__device__ __forceinline__ uint32_t f2bits(float x) { return __float_as_uint(x); }

// The last grid point at or below x (g.first <= x <= g.last): its index, its bit pattern, the
// step to the next point and how far above it x is (in bit patterns).
struct GridPoint {
  uint32_t at, bits, step, above;
};
__device__ __forceinline__ GridPoint grid_point(const GridView& g, float x) {
  const uint32_t bx = f2bits(x);
  uint32_t k = __ldg(g.run_of + ((bx - g.bits0) >> kRunShift));
  uint4 r = __ldg(reinterpret_cast<const uint4*>(g.runs) + k);
  while (bx >= r.y) r = __ldg(reinterpret_cast<const uint4*>(g.runs) + ++k);
  const uint32_t d = bx - r.x, step = r.w >> 24, q = __umulhi(d, r.z);
  return GridPoint{(r.w & 0xFFFFFFu) + q, r.x + q * step, step, d - q * step};
}

// First i with grid[i] >= x (lower_bound), exact for every float x, NaN -> 0.
__device__ __forceinline__ uint32_t grid_lower_bound(const GridView& g, float x) {
  if (!(x > g.first)) return 0;
  if (x > g.last) return g.n;
  const GridPoint p = grid_point(g, x);
  return p.at + (p.above ? 1u : 0u);
}

// First i with grid[i] > x (upper_bound), exact, NaN -> 0.
__device__ __forceinline__ uint32_t grid_upper_bound(const GridView& g, float x) {
  if (!(x >= g.first)) return 0;
  if (!(x < g.last)) return g.n;
  return grid_point(g, x).at + 1u;
}

// MZIndex::find_closest_index (src/mz_index/mod.rs:55-90): nearest grid point,
// ties to the lower index, clamped to the ends.
__device__ __forceinline__ uint32_t grid_find_closest(const GridView& g, float mz) {
  if (!(mz > g.first)) return 0;
  if (!(mz < g.last)) return g.n - 1;
  const GridPoint p = grid_point(g, mz);
  if (p.above == 0) return p.at;
  const float ld = fabsf(__fsub_rn(__uint_as_float(p.bits + p.step), mz));
  const float rd = fabsf(__fsub_rn(__uint_as_float(p.bits), mz));
  return ld < rd ? p.at + 1u : p.at;
}

// Fragment m/z ordering key: NaN sorts after every number (ties by library
// position), so the output positions always form a permutation.
__device__ __forceinline__ float mz_key(float m) { return m != m ? INFINITY : m; }

// ln(x) of a float rounded to the nearest float: evaluated in double and rounded
// once.  (The reference calls glibc logf, which is not correctly rounded for
// about 1e-3 of its inputs: there the two differ by one ulp.)
__device__ __forceinline__ float ln_rn(float x) { return __double2float_rn(log((double)x)); }

// The same, kept out of line for rarely taken paths (keeps hot loops small).
static __device__ __noinline__ float ln_rn_slow(float x) {
  return __double2float_rn(log((double)x));
}

// Table for ln_fast: for j in [0, 256), c_j = 1 + j/256, {1/c_j, ln(c_j)} in double.
constexpr int kLnTableBits = 8;
constexpr int kLnTableSize = 1 << kLnTableBits;
int device_ln_table(int device, const double2** out);
std::vector<double2> host_ln_table();  // the values device_ln_table uploads

// The same value as ln_rn(x) for every float x, computed faster: x = 2^e * m,
// m = c_j * (1 + r) with 0 <= r < 2^-8, ln(1 + r) by its Taylor series to r^5,
// all in double; e*ln2 + ln(c_j) and r*p(r) are non-negative for x > 1, so the
// result y carries a relative error below 2^-42.  Rounding y to float is then correct unless the 29
// bits of y's significand below float precision lie within 2^14 units of the
// halfway pattern (about one input in 2^14); there ln_rn decides.  Checked against
// ln_rn for every float in (1, inf).  `tab` is the table of device_ln_table
// (usually staged in shared memory).
//
// The coefficients come as an argument: kernels pass them in their parameters, which the
// double-precision instructions read in place (as literals each took two moves per use,
// 50 of the search kernel's 1160 instructions per fragment row).
//
// ln_table: *y = ln(x) unless it returns true, when ln_rn must decide (x < 1, infinite or
// NaN, or a result too near a rounding boundary).  x = 1 gives exactly 0.
struct LnCoef {
  double ln2 = 0.6931471805599453094172321, c2 = -1.0 / 2.0, c3 = 1.0 / 3.0, c4 = -1.0 / 4.0,
         c5 = 1.0 / 5.0, one = 1.0;
};

__device__ __forceinline__ bool ln_table(float x, const double2* tab, const LnCoef& k, float* y) {
  const uint32_t b = __float_as_uint(x);
  const int e = (int)(b >> 23) - 127;
  const uint32_t j = (b >> (23 - kLnTableBits)) & (kLnTableSize - 1);
  const double m = (double)__uint_as_float((b & 0x007FFFFFu) | 0x3F800000u);
  const double2 t = tab[j];
  const double r = fma(m, t.x, -1.0);
  // 1 - r/2 + r^2/3 - r^3/4 + r^4/5 as (1 - r/2) + r^2 * ((1/3 - r/4) + r^2/5): three
  // dependent steps after r instead of four; e*ln2 + ln(c_j) forms alongside
  const double r2 = r * r;
  const double c0 = fma(r, k.c2, k.one);
  const double c1 = fma(r, k.c4, k.c3);
  const double p = fma(r2, fma(r2, k.c5, c1), c0);
  const double v = fma(p, r, fma((double)e, k.ln2, t.y));
  *y = __double2float_rn(v);
  const uint32_t low = (uint32_t)__double2loint(v) & 0x1FFFFFFFu;
  return b - 0x3F800000u >= 0x40000000u || low - (0x10000000u - 0x4000u) < 0x8000u;
}

__device__ __forceinline__ float ln_fast(float x, const double2* tab, const LnCoef& k,
                                         bool* slow = nullptr) {
  float y;
  if (ln_table(x, tab, k, &y)) {
    if (slow) *slow = x > 1.0f && x < INFINITY;
    return ln_rn_slow(x);
  }
  return y;
}

// ------------------------------------------------------------- structures
struct WinInfo {
  float lo, hi;      // isolation window, inclusive at both ends
  int64_t base;      // first entry of this observation in the entry arrays
  int64_t ss_off;    // element offset of its slice_starts, -1 if it holds no peaks
};

// The non-empty windows that hold an m/z, by lookup: the m distinct window limits v
// (ascending) cut the axis into 2m + 1 classes, the limits themselves (2i + 1) and what lies
// below (2i) or above them (2m); class k's windows are list[off[k]] .. list[off[k + 1] - 1],
// in window order.
struct WinIndex {
  const float* v = nullptr;
  const int* off = nullptr;
  const int* list = nullptr;
  int m = 0;
};

__device__ __forceinline__ void find_windows(const WinIndex& w, float x, int* off, int* len) {
  *off = *len = 0;
  if (!(x == x)) return;  // NaN lies in no window
  int lo = 0, hi = w.m;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(w.v + mid) < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  const int k = lo < w.m && __ldg(w.v + lo) == x ? 2 * lo + 1 : 2 * lo;
  *off = __ldg(w.off + k);
  *len = __ldg(w.off + k + 1) - *off;
}

}  // namespace ads

// Elements a run's entry arrays are allocated past their last entry: the search copies
// them 16 bytes at a time from 16-byte boundaries (15 bytes at 2 bytes an entry).
namespace ads {
constexpr int kEntrySlack = 8;
}

// A number that no other run of the process has or had (an address may come again).
namespace ads {
uint64_t new_id();
}

struct AdsDia {
  const uint64_t id = ads::new_id();
  int device = 0;
  int64_t n_obs = 0;
  int64_t grid_len = 0;
  std::vector<ads::WinInfo> win;
  std::vector<int64_t> num_cycles, num_peaks;
  ads::DevBuf<ads::WinInfo> win_dev;
  ads::DevBuf<uint32_t> slice_starts;  // [slots x (grid_len + 1)]
  ads::DevBuf<uint16_t> cycles;
  ads::DevBuf<float> intens;
  ads::DevBuf<uint16_t> intens_bf16;   // built on first BF16 search
  bool bf16_only = false;              // f32 intensities released (ads_dia_keep_bf16_only)
  int64_t n_entries = 0;
  int max_overlap = 0;                 // max number of non-empty windows covering one m/z
  ads::DevBuf<int> win_index_dev;      // WinIndex: v, off, list
  int win_index_m = 0;
  bool win_index_ok = false;           // false: too many overlaps to list (windows are scanned)
  ads::WinIndex win_index() const {
    const int* p = win_index_dev.p;
    return ads::WinIndex{reinterpret_cast<const float*>(p), p + win_index_m, p + 3 * win_index_m + 2,
                         win_index_m};
  }
  std::vector<float> rt;               // MS1 retention times (RT index)
  float delta_t = 1.0f;
  ads::DevBuf<float> rt_dev;
  std::vector<float> rt_values;        // every spectrum's RT (DIAData.rt_values)
  std::vector<float> cycle;
  int64_t cycle_shape[4] = {0, 0, 0, 0};
  std::mutex mu;
};

struct AdsLib {
  int device = 0;
  int64_t n_prec = 0, n_frag = 0;
  int64_t max_frag = 0;  // max fragments of one precursor
  int64_t min_frag = 0;  // min fragments of one precursor
  ads::DevBuf<char> arena;  // every array below lives in this one allocation
  uint64_t* pidx_p = nullptr;  // precursor arrays, sorted by precursor_idx
  float* pmz_p = nullptr;
  float* prt_p = nullptr;
  float* ptol_p = nullptr;     // optional per-precursor RT half-window
  uint32_t* prow_p = nullptr;  // input row of each sorted precursor
  uint64_t* fstart_p = nullptr;
  uint64_t* fstop_p = nullptr;
  uint8_t* naa_p = nullptr;    // precursor_naa (scoring), sorted like the other precursor arrays
  float* fmz_p = nullptr;      // fragment arrays, input order
  float* fmzl_p = nullptr;     // fragment_mz_library (scoring's IDF)
  float* fint_p = nullptr;
  uint8_t* fnum_p = nullptr;
  uint8_t* ftype_p = nullptr;
  bool has_tol = false;
  float max_tol = 0.0f;
  // recorded after the library's device-side preparation (the precursor sort); every
  // stream that reads the arrays waits on it (lib_ready_on)
  cudaEvent_t ready = nullptr;
  // InverseDocumentFrequency (src/idf/mod.rs:13-33): fragments of the library per
  // m/z grid bin, built on the first scoring call
  std::mutex mu;
  ads::DevBuf<uint32_t> idf_counts;
  float idf_total = -1.0f;  // fragments the histogram counts (< 0: this library's own)
  AdsLib() = default;
  AdsLib(const AdsLib&) = delete;
  AdsLib& operator=(const AdsLib&) = delete;
  ~AdsLib() {
    if (ready) cudaEventDestroy(ready);
  }
};

namespace ads {
// Orders `st` after the library's preparation (from_arrays returns once its uploads
// have landed; the sort behind them may still be queued).
inline int lib_ready_on(const AdsLib* l, cudaStream_t st) {
  if (l->ready) ADS_CUDA(cudaStreamWaitEvent(st, l->ready, 0));
  return ADS_OK;
}
}  // namespace ads

// Candidate columns on the device (CandidateCollection, src/candidate/entry.rs:41-179).
struct AdsCandidates {
  int device = 0;
  cudaEvent_t done = nullptr;
  int64_t cap = -1;
  ads::DevBuf<char> arena;  // all columns and counters in one allocation
  uint64_t* pidx_p = nullptr;
  uint64_t* rank_p = nullptr;
  uint64_t* center_p = nullptr;
  uint64_t* start_p = nullptr;
  uint64_t* stop_p = nullptr;
  float* score_p = nullptr;
  int64_t* count_p = nullptr;
  int* err_p = nullptr;
  int64_t count = 0;
  bool pending = false;
  // `done` was recorded behind everything that a search has enqueued on the buffers, in
  // part or whole (false while one is being enqueued)
  bool covered = false;
  ~AdsCandidates() {
    if (done) {
      // what searches have enqueued on the buffers has ended, and every reader waits for its
      // own copies or kernels before it returns: nothing uses them any more (else the arena
      // goes by the release that waits for the device)
      const bool ended = covered && cudaEventSynchronize(done) == cudaSuccess;
      cudaEventDestroy(done);
      if (ended) arena.release_idle();
    }
  }
};

