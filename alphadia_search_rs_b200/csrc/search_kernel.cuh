// The fused per-precursor search kernel: XIC gather -> Gaussian convolution ->
// ln(x + 1) * w -> ordered score sum -> 5-point local maxima -> top-K.
// Included by search.cu inside namespace ads::{anonymous}; uses its helpers
// (kFull, rust_bsearch_u16, lower_bound_u16).
//
// One warp per precursor; warps pull precursors from an atomic counter and never
// wait on each other after the block has staged its tables.  The warp walks the
// precursor's kept fragments in order and, for each one,
//   1. gathers the fragment's XIC row into its shared-memory row: the CSR
//      entries of every (fragment, window) pair are read up to 128 at a time and
//      added to the row in CSR order (the reference's `dense_xic[c] += intensity`);
//   2. convolves the row: lane l owns S consecutive output cycles per pass of
//      32*S cycles and holds the S + 2h inputs they need in registers;
//   3. adds ln(conv + 1) * w_f to its own columns' scores.  Fragments are taken
//      in order, which is the reference's row-major accumulation
//      (src/score/scalar.rs:16-22).
// Then 5-point local maxima over the scores and a warp top-K.  All f32
// arithmetic is explicitly rounded and in the reference's order, so results
// equal the reference's except for its logf (see ln_rn).

struct SearchArgs {
  int64_t n_prec;
  const int* list;                // nullable: the precursors to search, else 0..n_prec-1
  const unsigned int* list_len;   // device length of `list`
  const int* nf;
  const int* cs;
  const int* ce;
  const int* nwin;
  const int* wins;
  int maxw;
  const float* fw;
  const uint32_t* blo;
  const uint32_t* bhi;
  int kf;
  const WinInfo* win;
  const uint32_t* ss;
  const uint16_t* cyc;
  const float* inten;
  const uint16_t* inten_bf16;  // bfloat16 copy of `inten` (BF16-storage searches)
  const double2* ln_tab;
  float kw[kMaxHalf + 1];  // kernel taps w[0..h]; w[h] is the centre (h <= kMaxHalf)
  const float* kw_dev;     // the taps in device memory when h > kMaxHalf, else null
  unsigned long long kw2[kMaxHalf + 1];  // the same taps, each twice (packed f32x2 operands)
  unsigned long long zero2;   // +0.0f twice
  unsigned long long nzero2;  // -0.0f twice
  LnCoef ln;
  int h;
  int k_out;   // candidates kept per precursor
  int c_max;   // largest cycle range of the precursors this launch searches
  int ncell;   // cycles a warp's row holds: passes * 32 * S >= c_max
  int gather_mode;
  int scan_thresh;
  float* grow;  // per-warp working sets of a long-window launch (GROW), else null
  unsigned long long* work;
  int* err;
  int* cand_n;
  float* cand_score;
  int* cand_center;
  unsigned long long* stats;  // nullable
};

// The scanning gather copies up to kStageEntries CSR entries of a (fragment, window)
// range into the warp's staging area in shared memory, asynchronously and 16 bytes per
// lane: intensities first, then cycles, each from the 16-byte boundary at or below the
// range's first entry.
constexpr int kStageEntries = 128;
constexpr int kStageCycOff = kStageEntries * 4 + 16;                   // bytes
constexpr int kStageWords = (kStageCycOff + kStageEntries * 2 + 16) / 4;
// Bin ranges of more entries than this are binary-searched per bin instead of scanned.
constexpr int kScanThreshFp32 = 256, kScanThreshBf16 = 384;
constexpr int kBitOff = 32;         // bitmap bit of cycle c is c + kBitOff (room for -h)
constexpr int kSmemMaxCycles = 2048;  // longest RT window (cycles) a warp's shared-memory plan
                                      // holds; longer windows run with GROW
constexpr int kTouchCap = 256;      // accepted cells a row records for clearing; beyond it the
                                    // row is zeroed whole

__host__ __device__ inline int maxima_cap(int ncell) { return ncell / 4 + 8; }

// Shared-memory address of stored index i (cycle + off) in a score array whose
// lanes own S consecutive cycles: one pad word after every S cells, so that the 32
// lanes of a warp, reading at the same offset within their segments, hit 32
// different banks.
template <int S>
__device__ __forceinline__ int xaddr(int i) {
  return i + i / S;
}

// The XIC row is read as 8-byte pairs of cells (u, u + 1), u even within a lane's
// segment, so its segments of S cells (S even) sit at an even stride of
// row_stride(S) words whose half is odd: the 16 lanes of each half-warp then hit 16
// different bank pairs.
__host__ __device__ constexpr int row_stride(int S) {
  return ((S + 2) / 2) % 2 == 1 ? S + 2 : S + 4;
}

template <int S>
__device__ __forceinline__ int raddr(int i) {
  return i + (i / S) * (row_stride(S) - S);
}

// Floor division, for offsets known at compile time.
__host__ __device__ constexpr int floordiv(int a, int b) {
  return a >= 0 ? a / b : -((-a + b - 1) / b);
}

// Per-warp shared-memory plan, in 4-byte words.  The block's ln table (double2 x
// 256 = 1024 words), kernel taps (h + 1 words, at least 32) and the warps' staging
// areas come first.  `ncell` (passes * 32 * S) sizes the bitmap, which every lane reads;
// the row and the scores, of which only lanes with an output below c_max touch theirs,
// are sized by c_max (a 801-cycle class of S = 16 would else hold 1024 cycles).
struct WarpPlan {
  int row, bm, cells, score, lst, mval, midx, total;
  int off;        // stored index of cycle c is c + off (off >= h, a multiple of S)
  int row_words;  // words of the row, a multiple of 4
  int lead;       // bitmap words below bm[0]: a window reaching h cycles before cycle 0
                  // reads them (always zero)
  int bw;         // bitmap words from bm[0]
  int mx;         // maxima capacity
};
__host__ __device__ inline int block_header_words(int h) {
  return kLnTableSize * 4 + ((h + 1 + 31) / 32) * 32;
}

__host__ __device__ inline WarpPlan warp_plan(int S, int h, int ncell, int c_max) {
  WarpPlan w;
  const int cc = (c_max + S - 1) / S * S;
  w.off = (h + S - 1) / S * S;
  const int span = cc + h + w.off + S;  // stored indices [0, span) cover every read
  w.row_words = (span + (span / S + 1) * (row_stride(S) - S) + 3) & ~3;
  int o = 0;
  w.row = o;
  o += w.row_words;
  w.lead = h > kBitOff ? (h - kBitOff + 31) / 32 : 0;
  w.bw = (ncell + h + kBitOff + 31) / 32 + 2;
  w.bm = o + w.lead;
  o += w.lead + w.bw;
  w.cells = o;  // cells accepted by the current row (16 bits each)
  o += kTouchCap / 2;
  w.score = o + 4;  // 4 words of margin below: the maxima scan reads 2 cycles early, and
                    // idle lanes of the score terms work on the lowest
  o += cc + cc / S + 12;
  o = (o + 1) & ~1;
  // one pass of convolved values as (value, score address) pairs, and a warp of idle ones;
  // before it, while the row is gathered, the accepted entries' intensities (kTouchCap words)
  w.lst = o;
  o += 2 * 32 * (S + 1);
  w.mx = maxima_cap(ncell);
  if (2 * w.mx <= 2 * 32 * S) {
    // the maxima are collected after the precursor's last row is scored, when the
    // output list is free
    w.mval = w.lst;
    w.midx = w.lst + w.mx;
  } else {
    w.mval = o;
    o += w.mx;
    w.midx = o;
    o += w.mx;
  }
  w.total = (o + 3) & ~3;
  return w;
}

__host__ __device__ inline size_t search_smem_bytes(int nw, int S, int h, int ncell, int c_max,
                                                    bool grow = false) {
  return (size_t)(block_header_words(h) +
                  nw * (kStageWords + (grow ? 0 : warp_plan(S, h, ncell, c_max).total))) * 4;
}

// Launch bounds of an instance.  The FP32 shared-memory instances for half widths 10
// and 11 (kernel sizes 20-22) at 128 threads and 5 blocks per SM: up to 102 registers,
// 20 warps (on 3000 x 300 data with 301-cycle windows 9 % faster than 256 x 2, without
// spills worth noting).  Everything else at 256 x 2 (128 registers): the BF16 instances
// (the 20-warp shape was 1.5 % slower on the uneven workload), half width 16 (spilled
// up to 256 bytes and ran 13 % slower at kernel size 31), the generic half width and the
// global-memory (long-window) instances.
template <int H, bool FAST, bool GROW>
struct LaunchShape {
  static constexpr bool narrow = !FAST && !GROW && (H == 10 || H == 11);
  static constexpr int threads = narrow ? 128 : 256;
  static constexpr int blocks = narrow ? 5 : 2;
};
__host__ __device__ constexpr int launch_threads(int h, bool fast, bool grow) {
  return (!fast && !grow && (h == 10 || h == 11)) ? 128 : 256;
}

// Per-warp work counters of the statistics pass (ON); 32 bits suffice for one warp's
// share of a launch.  In the searching instances (ON = false) they hold nothing and
// compile to no instruction.
template <bool ON>
struct Count;
template <>
struct Count<true> {
  unsigned int v = 0;
  __device__ Count& operator+=(unsigned int x) {
    v += x;
    return *this;
  }
  __device__ unsigned int get() const { return v; }
};
template <>
struct Count<false> {
  __device__ Count& operator+=(unsigned int) { return *this; }
  __device__ unsigned int get() const { return 0u; }
};
template <bool ON>
struct Counters {
  Count<ON> read, acc, off, pairs, bins1, frag;
};

// A value that is the same in all lanes, as the result of a warp reduction, which the
// compiler knows to be uniform: branches and loops on it need no reconvergence code, and
// the collectives inside them no divergence check (24 of 1160 instructions per fragment
// row, and as many again for the barriers around them).
__device__ __forceinline__ int uniform(int x) {
  return (int)__reduce_max_sync(kFull, (unsigned)x);
}
// Lane q's value (x >= 0), uniform as above.
__device__ __forceinline__ unsigned from_lane(unsigned x, int q, int lane) {
  return __reduce_max_sync(kFull, lane == q ? x : 0u);
}

// One fragment row being gathered.  Accepted entries are appended, in CSR order, to a list
// (cell, intensity) and added to the row 32 at a time, so that the adds run with full
// warps however few entries of a chunk lie in the RT window (7 of 32 on average on
// 3000 x 300 data); the list is also what the next row clears.
struct RowList {
  float* row;
  uint32_t* bm;
  uint16_t* cells;  // entry i at i % kTouchCap
  float* vals;      // likewise
  int n;            // entries appended (warp-uniform)
  int done;         // of them added to the row
};

// The rare case of add_entries: lanes that hit the same cycle are grouped and summed
// by their lowest lane in lane order (kept out of line: it is seldom taken).
static __device__ __noinline__ void add_grouped(bool act, int cell, int addr, int first, int lane,
                                                float* row, const float* vals) {
  const int key = act ? cell : (-1 - lane);
  const unsigned grp = __match_any_sync(kFull, key);
  if (act && lane == __ffs(grp) - 1) {
    float acc = row[addr];
    unsigned g = grp;
#pragma unroll 1
    while (g) {
      const int l = __ffs(g) - 1;
      acc = __fadd_rn(acc, vals[(first + l) % kTouchCap]);
      g &= g - 1;
    }
    row[addr] = acc;
  }
}

// Adds the next m (1 to 32) listed entries to the XIC row in list order (the reference's
// `dense_xic[c] += intensity`, src/quadrupole_observation/mod.rs:96-105).  Setting a
// cell's bit tells whether it was touched before, by an earlier entry or by another lane:
// if none was, every cell holds 0 and takes its intensity.  If one lane's was (a third of
// the rows), that lane adds after the others have stored: to what an earlier entry left, or
// to another lane's intensity, where 0 + a + b and 0 + b + a round alike.  Else the lanes
// are grouped by cell and summed by their lowest lane one rounded add at a time.
template <int S>
__device__ __forceinline__ void add_entries(RowList& r, int m, int off, int lane) {
  __syncwarp();
  const int i = (r.done + lane) % kTouchCap;
  const bool act = lane < m;
  const int cell = r.cells[i];
  const float v = r.vals[i];
  const int addr = raddr<S>(cell + off);
  const uint32_t bit = 1u << (cell & 31);
  bool again = false;
  if (act) again = (atomicOr(r.bm + ((cell + kBitOff) >> 5), bit) & bit) != 0u;
  const unsigned later = __ballot_sync(kFull, again);
  if ((later & (later - 1u)) == 0u) {
    if (act && !again) r.row[addr] = v;
    __syncwarp();
    if (again) r.row[addr] = __fadd_rn(r.row[addr], v);
  } else {
    add_grouped(act, cell, addr, r.done, lane, r.row, r.vals);
  }
  r.done += m;
}

// Appends the lanes' entries marked `in`, in lane order.
template <int S>
__device__ __forceinline__ void append_entries(RowList& r, bool in, int cell, float v, int off,
                                               int lane) {
  const unsigned act = __ballot_sync(kFull, in);
  if (in) {
    const int at = (r.n + __popc(act & lanemask_lt())) % kTouchCap;
    r.cells[at] = (uint16_t)cell;
    r.vals[at] = v;
  }
  r.n += __popc(act);
  if (r.n - r.done >= 32) add_entries<S>(r, 32, off, lane);
}

// The same for two consecutive entries per lane.
template <int S>
__device__ __forceinline__ void append_pairs(RowList& r, bool in0, bool in1, int cell0, int cell1,
                                             float v0, float v1, int off, int lane) {
  const unsigned act0 = __ballot_sync(kFull, in0), act1 = __ballot_sync(kFull, in1);
  const int at = r.n + __popc(act0 & lanemask_lt()) + __popc(act1 & lanemask_lt());
  if (in0) {
    r.cells[at % kTouchCap] = (uint16_t)cell0;
    r.vals[at % kTouchCap] = v0;
  }
  if (in1) {
    const int to = (at + (in0 ? 1 : 0)) % kTouchCap;
    r.cells[to] = (uint16_t)cell1;
    r.vals[to] = v1;
  }
  r.n += __popc(act0) + __popc(act1);
#pragma unroll 1
  while (r.n - r.done >= 32) add_entries<S>(r, 32, off, lane);
}

// Is `pos` the first entry of one of the bins (b0, b1)?  (slice_starts[b] == pos)
// Kept out of line: only entries at the window's first cycle ask.
static __device__ __noinline__ bool bin_starts_at(const uint32_t* ssw, uint32_t b0, uint32_t b1,
                                                  uint32_t pos) {
  uint32_t lo = b0 + 1, hi = b1;
#pragma unroll 1
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(ssw + mid) < pos)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo < b1 && __ldg(ssw + lo) == pos;
}

// Entries of one run, addressed by absolute CSR position (64 bits: a run may hold more
// than 2^32 entries).
template <bool FAST>
__device__ __forceinline__ float ld_intensity(const SearchArgs& a, int64_t q) {
  if (FAST) return __uint_as_float((uint32_t)__ldg(a.inten_bf16 + q) << 16);
  return __ldg(a.inten + q);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Starts copying entries [q0, q0 + m) (m <= kStageEntries) into the staging area: lane k
// takes 16-byte pieces k, k + 32 of the intensities' pieces followed by the cycles'.  A
// range of up to about 76 FP32 (120 BF16) entries is one instruction of the warp; through
// registers, 64 (96) entries took 4 to 6 loads and as many live registers across the
// stencil.
template <bool FAST>
__device__ __forceinline__ void stage_entries(const SearchArgs& a, int64_t q0, int m, uint32_t stage,
                                              int lane) {
  constexpr int PI = FAST ? 8 : 4;  // intensities in 16 bytes
  const char* in = FAST ? reinterpret_cast<const char*>(a.inten_bf16) + (q0 & ~(int64_t)7) * 2
                        : reinterpret_cast<const char*>(a.inten) + (q0 & ~(int64_t)3) * 4;
  const char* cy = reinterpret_cast<const char*>(a.cyc) + (q0 & ~(int64_t)7) * 2;
  const int ni = ((int)(q0 & (PI - 1)) + m + PI - 1) / PI;
  const int nc = ((int)(q0 & 7) + m + 7) / 8;
  // (piece k of the cycles, counted from the intensities' first)
  const char* cy0 = cy - ni * 16;
  const uint32_t cyc_stage = stage + kStageCycOff - ni * 16;
#pragma unroll 1
  for (int k0 = 0; k0 < ni + nc; k0 += 32) {
    const int k = k0 + lane;
    if (k < ni + nc) cp_async16((k < ni ? stage : cyc_stage) + k * 16, (k < ni ? in : cy0) + k * 16);
  }
}

__device__ __forceinline__ void stage_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}

__device__ __forceinline__ bool scans(const SearchArgs& a, uint32_t n) {
  return a.gather_mode == 1 || (a.gather_mode == 0 && n <= (uint32_t)a.scan_thresh);
}

// The CSR ranges of a precursor's (fragment, window) pairs, fetched 32 at a time
// (lane q holds pair pb + q), and the pair whose first entries are staged.
struct PairCursor {
  int pb = -64;
  uint32_t rs = 0, n = 0, b0 = 0, b1 = 0;
  int wsel = 0;
  int64_t wbase = 0;
  int pre_pi = -1;
};

// The pair in lane q of the cursor.
struct Pair {
  int64_t q;   // absolute position of its first entry
  uint32_t n;  // entries
};
__device__ __forceinline__ Pair pair_of(const PairCursor& pc, int q, int lane) {
  return Pair{__shfl_sync(kFull, pc.wbase + pc.rs, q), from_lane(pc.n, q, lane)};
}

// An entry at the window's first cycle counts only if it is the last of its bin there
// (where Rust's binary_search lands, src/quadrupole_observation/mod.rs:91-94): is the
// next entry, entry `tn` of the pair's n, in another bin or at another cycle?  Out of
// line: about one range in fifty holds such an entry.
static __device__ __noinline__ bool last_at_start(const SearchArgs& a, int wsel, uint32_t b0,
                                                  uint32_t b1, uint32_t rs, int64_t q, uint32_t tn,
                                                  uint32_t n, int cs) {
  if (tn >= n || bin_starts_at(a.ss + a.win[wsel].ss_off, b0, b1, rs + tn)) return true;
  return (int)__ldg(a.cyc + q + tn) != cs;
}

// The rare strategy of gather_pair, out of line: per bin, binary-search the first kept
// entry and the first entry at or past stop, then read only the kept entries.
struct SearchedPair {
  int n, done;           // of the row list
  unsigned read, offs;   // entries and offsets read
};
template <int S, bool FAST>
static __device__ __noinline__ SearchedPair gather_searched(const SearchArgs& a, uint32_t b0,
                                                            uint32_t b1, int wsel, int64_t wbase,
                                                            int cs, int C, int lane, RowList r,
                                                            int off) {
  SearchedPair out{0, 0, 0, 0};
  const uint32_t* ssw = a.ss + a.win[wsel].ss_off;
  const uint16_t* cy = a.cyc + wbase;
#pragma unroll 1
  for (uint32_t bb = b0; bb < b1; bb += 32) {
    const uint32_t b = bb + lane;
    const bool vb = b < b1;
    int64_t pos = 0, cnt = 0;
    if (vb) {
      const int64_t s0 = __ldg(ssw + b), s1 = __ldg(ssw + b + 1);
      pos = s0 + rust_bsearch_u16(cy + s0, s1 - s0, cs);
      const int64_t end = pos + lower_bound_u16(cy + pos, s1 - pos, cs + C);
      cnt = end - pos;
    }
    out.offs += 2u * (unsigned int)__popc(__ballot_sync(kFull, vb));
    int64_t incl = cnt;
#pragma unroll 1
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += t;
    }
    const int64_t total = __shfl_sync(kFull, incl, 31);
    const int64_t excl = incl - cnt;
    out.read += (unsigned int)total;
#pragma unroll 1
    for (int64_t t0 = 0; t0 < total; t0 += 32) {
      const int64_t t = t0 + lane;
      int l = 0;
#pragma unroll 1
      for (int st = 16; st >= 1; st >>= 1) {
        const int c = l + st;
        const int64_t ec = __shfl_sync(kFull, excl, c);
        if (ec <= t) l = c;
      }
      const int64_t opos = __shfl_sync(kFull, pos, l);
      const int64_t oex = __shfl_sync(kFull, excl, l);
      const bool vt = t < total;
      const int64_t q = opos + (t - oex);
      const int c = vt ? (int)__ldg(cy + q) : 0;
      const float v = vt ? ld_intensity<FAST>(a, wbase + q) : 0.0f;
      append_entries<S>(r, vt, c - cs, v, off, lane);
    }
  }
  out.n = r.n;
  out.done = r.done;
  return out;
}

// fill_xic_slice for the (fragment, window) pair in lane `pq` of the cursor: its entries
// inside the RT window are listed, in CSR order.  Two exact strategies: scan, which reads
// every entry of the range and keeps start < cycle < stop plus, per bin, the last entry
// at cycle == start; or, for long ranges, gather_searched.  `staged`: the range's first
// kStageEntries entries are already on their way.
template <int S, bool FAST, bool STATS>
__device__ __forceinline__ void gather_pair(const SearchArgs& a, const PairCursor& pc, int pq,
                                            Pair pr, bool staged, int cs, int C, int lane,
                                            uint32_t stage, const unsigned char* stage_p,
                                            RowList& r, int off, Counters<STATS>& k) {
  if (scans(a, pr.n)) {
    k.read += pr.n;
#pragma unroll 1
    for (uint32_t q0 = 0; q0 < pr.n; q0 += kStageEntries) {
      const int m = (int)min(pr.n - q0, (uint32_t)kStageEntries);
      const int64_t q = pr.q + q0;
      if (!staged) {
        __syncwarp();  // the area's previous entries have been read
        stage_entries<FAST>(a, q, m, stage, lane);
      }
      staged = false;
      stage_wait();
      // two consecutive entries per lane, from the even position at or below the first
      const int odd = (int)(q & 1);
      const uint32_t* sc = reinterpret_cast<const uint32_t*>(stage_p + kStageCycOff) + ((q & 7) >> 1);
      const float2* sf = reinterpret_cast<const float2*>(stage_p) + ((q & 3) >> 1);
      const uint32_t* sh = reinterpret_cast<const uint32_t*>(stage_p) + ((q & 7) >> 1);
#pragma unroll 1
      for (int i0 = 0; i0 < m + odd; i0 += 64) {
        const int t = i0 + 2 * lane - odd;
        const int i = min((i0 >> 1) + lane, kStageEntries / 2);  // the area's last pair
        const uint32_t cc = sc[i];
        float2 v;
        if (FAST) {
          const uint32_t b = sh[i];
          v = make_float2(__uint_as_float(b << 16), __uint_as_float(b & 0xffff0000u));
        } else {
          v = sf[i];
        }
        const int cell0 = (int)(cc & 0xffffu) - cs, cell1 = (int)(cc >> 16) - cs;
        bool in0 = (unsigned)t < (unsigned)m && (unsigned)cell0 < (unsigned)C;
        bool in1 = t + 1 < m && (unsigned)cell1 < (unsigned)C;
        if (__any_sync(kFull, (in0 && cell0 == 0) || (in1 && cell1 == 0))) {
          const uint32_t rs = __shfl_sync(kFull, pc.rs, pq);
          const uint32_t b0 = __shfl_sync(kFull, pc.b0, pq), b1 = __shfl_sync(kFull, pc.b1, pq);
          const int wsel = __shfl_sync(kFull, pc.wsel, pq);
#pragma unroll 1
          for (int e = 0; e < 2; ++e) {
            const bool ask = e == 0 ? in0 && cell0 == 0 : in1 && cell1 == 0;
            if (ask) {
              const bool keep = last_at_start(a, wsel, b0, b1, rs, pr.q, q0 + (uint32_t)(t + e) + 1,
                                              pr.n, cs);
              if (e == 0)
                in0 = keep;
              else
                in1 = keep;
            }
          }
        }
        append_pairs<S>(r, in0, in1, cell0, cell1, v.x, v.y, off, lane);
      }
    }
  } else {
    const SearchedPair sp = gather_searched<S, FAST>(
        a, __shfl_sync(kFull, pc.b0, pq), __shfl_sync(kFull, pc.b1, pq),
        __shfl_sync(kFull, pc.wsel, pq), __shfl_sync(kFull, pc.wbase, pq), cs, C, lane, r, off);
    r.n = uniform(sp.n);
    r.done = uniform(sp.done);
    k.read += sp.read;
    k.off += sp.offs;
  }
}

// Any bit set in bm[lo, lo + n)?  (n >= 1; lo may be negative: the shift and mask
// below are floor division and remainder on two's-complement ints, and the words
// below bm[0] that such a range reaches are reserved and zero)
__device__ __forceinline__ bool bits_any(const uint32_t* bm, int lo, int n) {
  const int last = lo + n - 1;
  const int w0 = lo >> 5, w1 = last >> 5;
  uint32_t acc = 0;
#pragma unroll 1
  for (int w = w0; w <= w1; ++w) {
    uint32_t v = bm[w];
    if (w == w0) v &= 0xffffffffu << (lo & 31);
    if (w == w1) v &= 0xffffffffu >> (31 - (last & 31));
    acc |= v;
  }
  return acc != 0u;
}

// Packed f32x2 arithmetic (sm_100a): one instruction performs two independent f32
// operations, each rounded to nearest exactly like __fadd_rn / __fmul_rn /
// __fmaf_rn, so a packed result is bit-identical to the two scalar ones.
//
// ptxas contracts a packed multiply followed by a packed add into one fused
// multiply-add even with explicit .rn rounding and --fmad=false (measured on
// sm_100a: about half of 12-term chains differed).  The exact path therefore forms
// each rounded product as fma(a, b, -0), with the -0 a kernel argument that ptxas
// cannot see: fma(a, b, -0) = round(a * b) bit for bit, and an fma followed by an
// add is not contractible.  The +0 of the reference's `0 + x * w` is a kernel
// argument for the same reason.
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pk2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}

__device__ __forceinline__ void unpk2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// One output of convolution_scalar (src/convolution/scalar.rs:30-50) read from the
// row in shared memory: x[j]*w[h] first, then (x[j-d] + x[j+d]) * w[h-d] for
// d = h..1.  Any half width; used off the main path.  FAST (BF16 storage) fuses
// each multiply-add.
template <int S, bool FAST>
__device__ __forceinline__ float conv_at(const float* row, int off, const float* kw_s, int h,
                                         int j) {
  float s = __fadd_rn(0.0f, __fmul_rn(row[raddr<S>(j + off)], kw_s[h]));
#pragma unroll 1
  for (int t = 0; t < h; ++t) {
    const float lr = __fadd_rn(row[raddr<S>(j - h + t + off)], row[raddr<S>(j + h - t + off)]);
    s = FAST ? __fmaf_rn(lr, kw_s[t], s) : __fadd_rn(s, __fmul_rn(lr, kw_s[t]));
  }
  return s;
}

// ln(1 + c) for the BF16-storage path: the hardware log2 (absolute error about
// 2^-21) where ln(1 + c) >= ln(17/16), and the series c - c^2/2 + ... + c^7/7
// (relative error below 2^-26) for |c| < 1/16, so that small terms keep their
// relative accuracy.
__device__ __forceinline__ float ln1p_fast(float c) {
  float p = __fmaf_rn(c, -1.0f / 7.0f, 1.0f / 6.0f);
  p = __fmaf_rn(c, p, -1.0f / 5.0f);
  p = __fmaf_rn(c, p, 1.0f / 4.0f);
  p = __fmaf_rn(c, p, -1.0f / 3.0f);
  p = __fmaf_rn(c, p, 1.0f / 2.0f);
  p = __fmaf_rn(c, -p, 1.0f);  // 1 - c/2 + c^2/3 - ...
  const float series = __fmul_rn(c, p);
  return fabsf(c) < 0.0625f ? series : __logf(__fadd_rn(c, 1.0f));
}

// s + ln(c + 1) * w (src/score/scalar.rs:16-22): one rounded operation at a time with the
// exact ln; FAST (BF16 storage) takes the hardware log2 and a fused multiply-add.  Called
// by whole warps: the slow path of the exact ln is behind one vote.
template <bool FAST>
__device__ __forceinline__ float score_term(float s, float c, float w, const double2* lnt,
                                            const LnCoef& k) {
  if (FAST) return __fmaf_rn(ln1p_fast(c), w, s);
  const float x = __fadd_rn(c, 1.0f);
  float y;
  const bool slow = ln_table(x, lnt, k, &y);
  if (__any_sync(kFull, slow)) y = slow ? ln_rn_slow(x) : y;
  return __fadd_rn(s, __fmul_rn(y, w));
}

// Where the list of a pass's outputs, (value, score index) pairs, is appended to: a
// shared-memory address, or (GROW) a pointer.
template <bool GROW>
struct OutEnd;
template <>
struct OutEnd<false> {
  uint32_t to;
  __device__ OutEnd(float2* at) : to((uint32_t)__cvta_generic_to_shared(at)) {}
  // Appends (v, at) where bit m of mk is set: test, store, advance, all predicated (a
  // branch around each store cost three times as much).
  __device__ __forceinline__ void put(uint32_t mk, int m, float v, int at) {
    asm volatile(
        "{\n .reg .pred q;\n .reg .b32 t;\n and.b32 t, %1, %2;\n setp.ne.u32 q, t, 0;\n"
        " @q st.shared.v2.b32 [%0], {%3, %4};\n @q add.u32 %0, %0, 8;\n}"
        : "+r"(to)
        : "r"(mk), "r"(1u << m), "r"(__float_as_uint(v)), "r"(at)
        : "memory");
  }
};
template <>
struct OutEnd<true> {
  float2* to;
  __device__ OutEnd(float2* at) : to(at) {}
  __device__ __forceinline__ void put(uint32_t mk, int m, float v, int at) {
    if ((mk >> m) & 1u) *to++ = make_float2(v, __int_as_float(at));
  }
};

// Spreads every set bit of x over the LEN bits at and below it: bit m of the result is set
// where any of bits m .. m + LEN - 1 is.
template <int LEN, class U>
__device__ __forceinline__ U spread_down(U x) {
  int reach = 1;
#pragma unroll
  for (int g = 0; g < 5; ++g)
    if (2 * reach <= LEN) {
      x |= x >> reach;
      reach *= 2;
    }
  if (reach < LEN) x |= x >> (LEN - reach);
  return x;
}

template <bool FAST>
__device__ __forceinline__ void score_add(float* score, int addr, float c, float w,
                                          const double2* lnt, const LnCoef& k) {
  if (FAST)
    score[addr] = __fmaf_rn(ln1p_fast(c), w, score[addr]);
  else
    score[addr] = __fadd_rn(score[addr], __fmul_rn(ln_fast(__fadd_rn(c, 1.0f), lnt, k), w));
}

// An unsigned key ordered like the value (-0 as +0), at least 1; NaN has key 0.
__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t b = __float_as_uint(__fadd_rn(v, 0.0f));
  const uint32_t k = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  return v != v ? 0u : k;
}

// Moves the cursor to pairs [pi, pi + 32).
__device__ __forceinline__ void load_pairs(const SearchArgs& a, int64_t p, int pi, int nwin,
                                           int npairs, int lane, PairCursor& pc) {
  pc.pb = pi;
  const int pj = pi + lane;
  pc.rs = pc.n = 0;
  pc.b0 = pc.b1 = 0;
  pc.wsel = 0;
  pc.wbase = 0;
  if (pj < npairs) {
    const int fj = nwin == 1 ? pj : pj / nwin, wj = pj - fj * nwin;
    const int64_t fo = p * a.kf + fj;
    pc.b0 = a.blo[fo];
    pc.b1 = a.bhi[fo];
    pc.wsel = a.wins[p * a.maxw + wj];
    if (pc.b1 > pc.b0) {
      const WinInfo w = a.win[pc.wsel];
      pc.wbase = w.base;
      pc.rs = __ldg(a.ss + w.ss_off + pc.b0);
      pc.n = __ldg(a.ss + w.ss_off + pc.b1) - pc.rs;
    }
  }
}

// Starts staging pair pi's first entries (after the area's last ones have been read).
template <bool FAST>
__device__ __forceinline__ void stage_pair(const SearchArgs& a, int64_t p, int pi, int nwin,
                                           int npairs, int lane, PairCursor& pc, uint32_t stage) {
  pc.pre_pi = -1;
  if (pi >= npairs) return;
  if (pi >= pc.pb + 32) load_pairs(a, p, pi, nwin, npairs, lane, pc);
  const Pair pr = pair_of(pc, pi - pc.pb, lane);
  if (pr.n > 0 && scans(a, pr.n)) {
    __syncwarp();
    stage_entries<FAST>(a, pr.q, (int)min(pr.n, (uint32_t)kStageEntries), stage, lane);
    pc.pre_pi = pi;
  }
}

// Gathers fragment f's XIC row: its (fragment, window) pairs in window order (the
// reference's DenseXICObservation::new, src/dense_xic_observation/mod.rs:30-64).
template <int S, bool FAST, bool STATS>
__device__ __forceinline__ void gather_row(const SearchArgs& a, int64_t p, int f, int nwin,
                                           int npairs, int cs, int C, int lane, PairCursor& pc,
                                           uint32_t stage, const unsigned char* stage_p, RowList& r,
                                           int off, Counters<STATS>& k) {
#pragma unroll 1
  for (int wi = 0; wi < nwin; ++wi) {
    const int pi = f * nwin + wi;
    if (pi >= pc.pb + 32) load_pairs(a, p, pi, nwin, npairs, lane, pc);
    const int q = pi - pc.pb;
    const Pair pr = pair_of(pc, q, lane);
    if (STATS) {
      const uint32_t b0 = __shfl_sync(kFull, pc.b0, q), b1 = __shfl_sync(kFull, pc.b1, q);
      if (b1 > b0) {
        k.off += 2u;
        k.pairs += 1u;
        k.bins1 += b1 - b0 + 1;
      }
    }
    if (pr.n == 0) continue;
    gather_pair<S, FAST, STATS>(a, pc, q, pr, pi == pc.pre_pi, cs, C, lane, stage,
                                stage_p, r, off, k);
  }
  if (r.done < r.n) add_entries<S>(r, r.n - r.done, off, lane);
}

// The last gathered row's cells (and bitmap words) back to zero.
template <int S>
__device__ __forceinline__ void clear_row(RowList& r, const WarpPlan& P, int lane) {
  if (r.n > kTouchCap) {
    float4* r4 = reinterpret_cast<float4*>(r.row);
#pragma unroll 1
    for (int i = lane; i < P.row_words / 4; i += 32) r4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int i = lane; i < P.bw; i += 32) r.bm[i] = 0u;
  } else {
#pragma unroll 1
    for (int i = lane; i < r.n; i += 32) {
      const int c = r.cells[i];
      r.row[raddr<S>(c + P.off)] = 0.0f;
      r.bm[(c + kBitOff) >> 5] = 0u;
    }
  }
  r.n = r.done = 0;
  __syncwarp();
}

// A row whose weight is not finite, out of line: ln(conv + 1) * w is NaN even where conv
// is zero, so every column takes its term, as in the reference.
template <int S, bool FAST>
static __device__ __noinline__ void score_every_column(const SearchArgs& a, const float* row, int off,
                                                       const float* kw_s, int h, int C, float wf,
                                                       float* score, const double2* lnt, int lane) {
#pragma unroll 1
  for (int j = lane; j < C; j += 32) {
    const float c = (j >= h && j < C - h) ? conv_at<S, FAST>(row, off, kw_s, h, j) : 0.0f;
    score_add<FAST>(score, xaddr<S>(j), c, wf, lnt, a.ln);
  }
}

// Strict 5-point local maxima of a precursor's scores (src/peak_group_selection/mod.rs:33-43),
// collected in cycle order, and the top K of them by (value descending, cycle
// ascending), the reference's stable sort (src/peak_group_selection/mod.rs:45-61),
// written to the candidate slots.  `score` holds cycle j at xaddr<S>(j), with two
// readable words below cycle 0 and S + 2 cycles past C.
template <int S>
__device__ __forceinline__ void pick_top_k(const SearchArgs& a, int64_t p, int cs, int C,
                                           const float* score, float* mval, int* midx, int mx,
                                           int lane) {
  const int passes = (C + 32 * S - 1) / (32 * S);
  // lane l's maxima of a pass go after those of lanes < l
  int nmax = 0;
#pragma unroll 1
  for (int ps = 0; ps < passes; ++ps) {
    const int seg = ps * 32 + lane;
    const float* sb = score + seg * (S + 1);
    uint32_t mk = 0;
    if (seg * S < C - 2 && seg * S + S > 2) {
      float v[S + 4];
#pragma unroll
      for (int t = 0; t < S + 4; ++t) v[t] = sb[(t - 2) + floordiv(t - 2, S)];
#pragma unroll
      for (int m = 0; m < S; ++m) {
        const int i = seg * S + m;
        const bool is = i >= 2 && i < C - 2 && v[m] < v[m + 1] && v[m + 1] < v[m + 2] &&
                        v[m + 2] > v[m + 3] && v[m + 3] > v[m + 4];
        mk |= (uint32_t)is << m;
      }
    }
    const int cnt = __popc(mk);
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += t;
    }
    int pos = nmax + incl - cnt;
#pragma unroll 1
    while (mk) {
      const int m = __ffs(mk) - 1;
      if (pos < mx) {
        mval[pos] = sb[m];
        midx[pos] = seg * S + m;
      }
      ++pos;
      mk &= mk - 1;
    }
    nmax += __shfl_sync(kFull, incl, 31);
  }
  __syncwarp();
  if (nmax > mx) {  // cannot happen: maxima are at least 4 cycles apart
    if (lane == 0) atomicOr(a.err, 4);
    nmax = mx;
  }
  const int kk = min(a.k_out, nmax);
  // one selection per candidate: every lane holds the best of its maxima (lane,
  // lane + 32, ...), two reductions find the best value and its first cycle, and the lane
  // that held it looks for its next.  Sorting 32 at a time took ten times the instructions
  // for the usual 3 or 5 candidates.
  uint32_t key = 0;
  int at = -1;
  bool look = true;
#pragma unroll 1
  for (int r = 0; r < kk; ++r) {
    if (look) {
      key = 0;
#pragma unroll 1
      for (int q = lane; q < nmax; q += 32) {
        const uint32_t x = order_key(mval[q]);
        if (x > key) {
          key = x;
          at = q;
        }
      }
    }
    const uint32_t top = __reduce_max_sync(kFull, key);
    // maxima are listed in cycle order, so the first in the list is the first cycle
    const unsigned pos = __reduce_min_sync(kFull, key == top ? (unsigned)at : 0xffffffffu);
    look = (unsigned)at == pos && key == top;
    if (look) {
      a.cand_score[p * a.k_out + r] = mval[pos];
      a.cand_center[p * a.k_out + r] = cs + midx[pos];
      mval[pos] = __int_as_float(0x7fc00000);  // taken: key 0
    }
  }
  __syncwarp();
  if (lane == 0) a.cand_n[p] = kk;
}

// Per-warp work counters to the statistics pass's totals.
template <bool STATS>
__device__ __forceinline__ void flush_counters(const SearchArgs& a, const Counters<STATS>& k,
                                               int lane) {
  if (STATS && a.stats && lane == 0) {
    atomicAdd(a.stats + 0, (unsigned long long)k.pairs.get());
    atomicAdd(a.stats + 1, (unsigned long long)k.bins1.get());
    atomicAdd(a.stats + 2, (unsigned long long)k.frag.get());
    atomicAdd(a.stats + 3, (unsigned long long)k.read.get());
    atomicAdd(a.stats + 4, (unsigned long long)k.acc.get());
    atomicAdd(a.stats + 5, (unsigned long long)k.off.get());
  }
}

// GROW: the warp's working set (row, tags, bitmap, scores, lists, maxima) lives in
// a global buffer of P.total words per warp (`a.grow`) instead of shared memory, for
// RT windows longer than kSmemMaxCycles; the code and every operation are the same.
// STATS: the statistics pass's work counters (compiled in only for it).
template <int H, int S, bool FAST, bool GROW, bool STATS>
__global__ void __launch_bounds__(LaunchShape<H, FAST, GROW>::threads, LaunchShape<H, FAST, GROW>::blocks)
    search_kernel(const __grid_constant__ SearchArgs a) {
  extern __shared__ __align__(16) float smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = H > 0 ? H : a.h;
  const WarpPlan P = warp_plan(S, h, a.ncell, a.c_max);
  double2* lnt = reinterpret_cast<double2*>(smem_raw);
  float* kw_s = smem_raw + kLnTableSize * 4;
  const int nw = blockDim.x >> 5;
  float* areas = smem_raw + block_header_words(h);
  const unsigned char* stage_p = reinterpret_cast<const unsigned char*>(areas + warp * kStageWords);
  const uint32_t stage = (uint32_t)__cvta_generic_to_shared(stage_p);
  float* wb = GROW ? a.grow + ((size_t)blockIdx.x * nw + warp) * (size_t)P.total
                   : areas + nw * kStageWords + warp * P.total;
  float* row = wb + P.row;
  uint32_t* bm = reinterpret_cast<uint32_t*>(wb + P.bm);
  float* score = wb + P.score;
  float* mval = wb + P.mval;
  int* midx = reinterpret_cast<int*>(wb + P.midx);
  float2* lst = reinterpret_cast<float2*>(wb + P.lst);
  // r.n: also the cells the previous row left to clear
  RowList r{row, bm, reinterpret_cast<uint16_t*>(wb + P.cells), wb + P.lst, 0, 0};
  {
    float4* r4 = reinterpret_cast<float4*>(row);
#pragma unroll 1
    for (int i = lane; i < P.row_words / 4; i += 32) r4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int i = lane - P.lead; i < P.bw; i += 32) bm[i] = 0u;
  }

#pragma unroll 1
  for (int i = threadIdx.x; i < kLnTableSize; i += blockDim.x) lnt[i] = a.ln_tab[i];
#pragma unroll 1
  for (int i = threadIdx.x; i <= a.h; i += blockDim.x) kw_s[i] = a.kw_dev ? a.kw_dev[i] : a.kw[i];
  __syncthreads();
  Counters<STATS> k;

  const unsigned n_work = a.list ? (unsigned)uniform((int)*a.list_len) : (unsigned)a.n_prec;
#pragma unroll 1
  for (;;) {
    unsigned pw = 0;
    if (lane == 0) pw = (unsigned)min(atomicAdd(a.work, 1ull), 0xffffffffull);
    pw = __reduce_max_sync(kFull, pw);
    if (pw >= n_work) break;
    const int64_t p = a.list ? (int64_t)uniform(a.list[pw]) : (int64_t)pw;
    const int F = uniform(a.nf[p]);
    const int cs = uniform(a.cs[p]);
    const int C = uniform(a.ce[p]) - cs;
    if (F == 0 || C <= 0) {
      if (lane == 0) a.cand_n[p] = 0;
      continue;
    }
    if (C > a.c_max) {
      if (lane == 0) {
        a.cand_n[p] = 0;
        atomicOr(a.err, 2);
      }
      continue;
    }
    const int nwin = uniform(a.nwin[p]);
    const int npairs = F * nwin;
    const int passes = (C + 32 * S - 1) / (32 * S);
    k.frag += F;
    // fragment weights, lane f holding fragment f's (fetched once per precursor)
    const float wf_lane = lane < F ? __ldg(a.fw + p * a.kf + lane) : 0.0f;
    PairCursor pc;
    // f = -1: only starts the first row's entries on their way
#pragma unroll 1
    for (int f = -1; f < F; ++f) {
      if (f >= 0) {
        // ---- 1. gather: the fragment's pairs in window order
        clear_row<S>(r, P, lane);
        gather_row<S, FAST, STATS>(a, p, f, nwin, npairs, cs, C, lane, pc, stage, stage_p, r, P.off, k);
        k.acc += (unsigned int)r.n;
      }
      // the next fragment's first pair arrives while this row is convolved
      stage_pair<FAST>(a, p, (f + 1) * nwin, nwin, npairs, lane, pc, stage);
      if (f < 0) {
#pragma unroll 1
        for (int i = lane; i <= C + C / S; i += 32) score[i] = 0.0f;  // cycles [0, C) with pads
        continue;
      }
      __syncwarp();
      float wf = __shfl_sync(kFull, wf_lane, f & 31);
      if (f >= 32) wf = __ldg(a.fw + p * a.kf + f);
      if (!isfinite(wf)) {
        score_every_column<S, FAST>(a, row, P.off, kw_s, h, C, wf, score, lnt, lane);
        __syncwarp();
        continue;
      }
      if (r.n == 0) continue;  // no entry accepted: every term is +0
      // ---- 2./3. convolution of this lane's cycles, then the score terms of the
      // outputs of the valid range [h, C - h) that a touched cycle reaches.  Every other
      // output is zero and adds ln(1) * w = +0, which leaves a score as it is, so only
      // those are listed (warp-compacted, in lane order) and take a logarithm.
#pragma unroll 1
      for (int ps = 0; ps < passes; ++ps) {
        const int j0 = ps * 32 * S + lane * S;
        uint32_t mk = 0;  // outputs j0 + m to list
        bool act;
        if (H > 0) {
          // bits j0 - H .. j0 + S - 1 + H of the touched cycles, each spread over the
          // 2H + 1 outputs it reaches
          const int lo = j0 - H + kBitOff;
          const uint32_t* bw = bm + (lo >> 5);
          uint32_t x;
          if (S + 2 * H <= 32) {
            x = spread_down<2 * H + 1>(__funnelshift_r(bw[0], bw[1], lo));
          } else {
            const uint32_t x0 = bw[0], x1 = bw[1], x2 = bw[2];
            x = (uint32_t)spread_down<2 * H + 1>(
                ((unsigned long long)__funnelshift_r(x1, x2, lo) << 32) | __funnelshift_r(x0, x1, lo));
          }
          const int m0 = max(H - j0, 0), m1 = max(min(C - H - j0, S), 0);
          mk = x & ((1u << m1) - 1u) & (0xffffffffu << m0);
          act = mk != 0u;
        } else {
          act = j0 + S > h && j0 < C - h && bits_any(bm, j0 - h + kBitOff, S + 2 * h);
        }
        if (!__any_sync(kFull, act)) continue;
        float cv[S];
        if (H > 0) {
          // cells u in [UB, UE) of this lane's segment as 8-byte pairs (u even; a lane
          // without outputs computes the first segment's); every output is formed in the
          // reference's order: 0 + x[j]*w[h], then + (x[j-d] + x[j+d]) * w[h-d] for
          // d = h..1, two outputs (m, m + 1) per packed instruction.  For odd d the pair
          // sums straddle the register pairs and are formed by two scalar adds.
          constexpr int UB = -((H + 1) & ~1);
          constexpr int UE = (S + H + 1) & ~1;
          constexpr int NX = UE - UB;
          const float* rb = row + ((act ? ps * 32 + lane : 0) + P.off / S) * row_stride(S);
          float xv[NX];
#pragma unroll
          for (int q = 0; q < NX; q += 2) {
            const int u = UB + q;
            const float2 v =
                *reinterpret_cast<const float2*>(rb + u + floordiv(u, S) * (row_stride(S) - S));
            xv[q] = v.x;
            xv[q + 1] = v.y;
          }
          f32x2 acc[S / 2];
#pragma unroll
          for (int m = 0; m < S; m += 2)
            acc[m / 2] = add2(a.zero2, fma2(pk2(xv[m - UB], xv[m + 1 - UB]), a.kw2[H], a.nzero2));
#pragma unroll
          for (int t = 0; t < H; ++t) {
            const int d = H - t;
#pragma unroll
            for (int m = 0; m < S; m += 2) {
              f32x2 lr;
              if (d % 2 == 0)
                lr = add2(pk2(xv[m - d - UB], xv[m - d + 1 - UB]),
                          pk2(xv[m + d - UB], xv[m + d + 1 - UB]));
              else
                lr = pk2(__fadd_rn(xv[m - d - UB], xv[m + d - UB]),
                         __fadd_rn(xv[m + 1 - d - UB], xv[m + 1 + d - UB]));
              acc[m / 2] = FAST ? fma2(lr, a.kw2[t], acc[m / 2])
                                : add2(acc[m / 2], fma2(lr, a.kw2[t], a.nzero2));
            }
          }
#pragma unroll
          for (int m = 0; m < S; m += 2) unpk2(acc[m / 2], cv[m], cv[m + 1]);
        } else if (act) {
#pragma unroll
          for (int m = 0; m < S; ++m) {
            const int j = j0 + m;
            cv[m] = (j >= h && j < C - h) ? conv_at<S, FAST>(row, P.off, kw_s, h, j) : 0.0f;
          }
          const int m0 = max(h - j0, 0), m1 = min(C - h - j0, S);
#pragma unroll
          for (int m = 0; m < S; ++m)
            mk |= (uint32_t)(m >= m0 && m < m1 && cv[m] != 0.0f) << m;
        }
        const int cnt = __popc(mk);
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += t;
        }
        const int total = (int)__reduce_add_sync(kFull, (unsigned)cnt);
        const int sbase = (ps * 32 + lane) * (S + 1);  // score index of cycle j0
        OutEnd<GROW> end(lst + (incl - cnt));
#pragma unroll
        for (int m = 0; m < S; ++m) end.put(mk, m, cv[m], sbase + m);
        // idle entries up to a whole warp, which work on a word below the scores
        lst[total + lane] = make_float2(0.0f, __int_as_float(-4));
        __syncwarp();
#pragma unroll 1
        for (int i0 = 0; i0 < total; i0 += 32) {
          const float2 e = lst[i0 + lane];
          float* sp = score + __float_as_int(e.y);
          *sp = score_term<FAST>(*sp, e.x, wf, lnt, a.ln);
        }
        __syncwarp();
      }
      __syncwarp();
    }
    __syncwarp();

    pick_top_k<S>(a, p, cs, C, score, mval, midx, P.mx, lane);
  }
  flush_counters<STATS>(a, k, lane);
}
