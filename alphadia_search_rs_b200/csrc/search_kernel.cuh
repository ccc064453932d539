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
//   2. convolves the segments of 4 output cycles that a touched cycle reaches, one per
//      lane, the 4 + 2h inputs in registers;
//   3. adds ln(conv + 1) * w_f to the scores of the non-zero outputs.  Fragments are taken
//      in order, which is the reference's row-major accumulation
//      (src/score/scalar.rs:16-22).
// Then 5-point local maxima over the scores and a warp top-K.  All f32
// arithmetic is explicitly rounded and in the reference's order, so results
// equal the reference's except for its logf (see ln_rn).
//
// What bounds it: instruction issue (73 % of the cycles with 20 warps per SM, 1070
// instructions per fragment row of 4-24 fragments and windows of up to 801 cycles; memory
// 9 % busy).  Hence entries staged by asynchronous 16-byte copies and listed before they are
// added, work only on the segments that a cell reaches, rolled loops, rare cases out of line.
// A lane owning 4 to 16 consecutive cycles of every row, with the gather in registers, issued
// on 56 %: 200,000 uneven precursors FP32 6.08 -> 3.60 ms, 500,000 BF16 12.29 -> 7.70, 66,667
// with 12 fragments and 301 cycles 1.53 -> 1.00.

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
  uint32_t scan_thresh;  // longest range that is scanned
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
constexpr int kSeg = 4;               // output cycles of one segment
constexpr int kSmemMaxCycles = 2048;  // longest RT window (cycles) a warp's shared-memory plan
                                      // holds; longer windows run with GROW
constexpr int kTouchCap = 256;        // accepted cells a row records for clearing; beyond it the
                                      // row is zeroed whole
// Listed outputs: up to 31 left over, 4 per lane of one round, a warp of idle ones.
constexpr int kOutCap = 31 + 32 * kSeg + 32;
// Listed outputs that a lane takes the logarithm of at a time: the logarithm is a chain of
// dependent double operations, and 20 warps per SM do not hide it (1, 2, 3, 4 at a time:
// 200,000 uneven precursors FP32 3.77, 3.65, 3.60, 3.78 ms; 500,000 BF16 7.79, 7.71, 7.70,
// 7.82; windows of 4000 cycles 0.987, 0.903, 0.872, 0.909).
constexpr int kTerms = 3;

__host__ __device__ inline int maxima_cap(int c_max) { return c_max / 4 + 8; }

// Per-warp shared-memory plan, in 4-byte words.  The block's ln table (double2 x
// 256 = 1024 words), kernel taps (h + 1 words, at least 32) and the warps' staging
// areas come first.
struct WarpPlan {
  int row, bm, cells, segbits, segs, score, lst, mval, midx, total;
  int off;        // the row holds cycle c at c + off (off >= h, a multiple of kSeg)
  int row_words;  // words of the row, a multiple of 4
  int bw;         // words of the touched-cycle bitmap
  int sw;         // words of the segment bitmap
  int mx;         // maxima capacity
};
__host__ __device__ inline int block_header_words(int h) {
  return kLnTableSize * 4 + ((h + 1 + 31) / 32) * 32;
}

__host__ __device__ inline WarpPlan warp_plan(int h, int c_max) {
  WarpPlan w;
  const int cc = (c_max + kSeg - 1) / kSeg * kSeg;
  w.off = (h + kSeg - 1) / kSeg * kSeg;
  w.row_words = cc + 2 * w.off + kSeg;
  int o = 0;
  w.row = o;
  o += w.row_words;
  w.score = o + 4;  // 4 words of margin on both sides: the maxima scan reads them, and idle
                    // lanes of the score terms work on the lowest
  o += cc + 8;
  w.bm = o;  // a bit per touched cycle
  w.bw = (cc + 31) / 32;
  o += w.bw;
  w.segbits = o;  // a bit per segment that a touched cycle reaches
  w.sw = (cc / kSeg + 31) / 32 + 1;
  o += w.sw;
  w.segs = o;  // those segments, listed (16 bits each)
  o += (cc / kSeg + 1) / 2;
  w.cells = o;  // cells accepted by the current row (16 bits each)
  o += kTouchCap / 2;
  o = (o + 1) & ~1;
  // non-zero outputs as (value, score index) pairs; before them, while the row is gathered,
  // the accepted entries' intensities (kTouchCap words); after the last row, the maxima
  w.lst = o;
  w.mx = maxima_cap(cc);
  w.mval = o;
  w.midx = o + w.mx;
  int lw = 2 * kOutCap;
  if (lw < kTouchCap) lw = kTouchCap;
  if (lw < 2 * w.mx) lw = 2 * w.mx;
  o += lw;
  w.total = (o + 3) & ~3;
  return w;
}

__host__ __device__ inline size_t search_smem_bytes(int nw, int h, int c_max, bool grow = false) {
  return (size_t)(block_header_words(h) +
                  nw * (kStageWords + (grow ? 0 : warp_plan(h, c_max).total))) * 4;
}

// Launch bounds of an instance: shared-memory instances at 128 threads and 5 blocks per SM
// (up to 102 registers, 20 warps), the global-memory (long-window) ones at 256 x 2.  With
// 6 to 8 blocks (80 to 64 registers) up to 164 bytes of spills meet the little L1 that the
// warps' shared memory leaves: 200,000 uneven precursors FP32 4.04 ms -> 4.39 to 5.22 ms;
// at 256 x 2 500,000 uneven BF16 took 9.38 ms against 8.26 ms.
template <bool GROW>
struct LaunchShape {
  static constexpr int threads = GROW ? 256 : 128;
  static constexpr int blocks = GROW ? 2 : 5;
};

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
  float* row;         // cycle 0's cell
  uint32_t* bm;       // touched cycles
  uint32_t* segbits;  // segments they reach
  uint16_t* cells;  // entry i at i % kTouchCap
  float* vals;      // likewise
  int n;            // entries appended (warp-uniform)
  int done;         // of them added to the row
};

// The rare case of add_entries: lanes that hit the same cycle are grouped and summed
// by their lowest lane in lane order (kept out of line: it is seldom taken).
static __device__ __noinline__ void add_grouped(bool act, int cell, int first, int lane,
                                                float* row, const float* vals) {
  const int key = act ? cell : (-1 - lane);
  const unsigned grp = __match_any_sync(kFull, key);
  if (act && lane == __ffs(grp) - 1) {
    float acc = row[cell];
    unsigned g = grp;
#pragma unroll 1
    while (g) {
      const int l = __ffs(g) - 1;
      acc = __fadd_rn(acc, vals[(first + l) % kTouchCap]);
      g &= g - 1;
    }
    row[cell] = acc;
  }
}

// Adds the next m (1 to 32) listed entries to the XIC row in list order (the reference's
// `dense_xic[c] += intensity`, src/quadrupole_observation/mod.rs:96-105).  Setting a
// cell's bit tells whether it was touched before, by an earlier entry or by another lane:
// if none was, every cell holds 0 and takes its intensity.  If one lane's was (a third of
// the rows), that lane adds after the others have stored: to what an earlier entry left, or
// to another lane's intensity, where 0 + a + b and 0 + b + a round alike.  Else the lanes
// are grouped by cell and summed by their lowest lane one rounded add at a time.
template <int H>
__device__ __forceinline__ void add_entries(RowList& r, int m, int h, int C, int lane) {
  __syncwarp();
  const int i = (r.done + lane) % kTouchCap;
  const bool act = lane < m;
  const int cell = r.cells[i];
  const float v = r.vals[i];
  const uint32_t bit = 1u << (cell & 31);
  bool again = false;
  if (act) again = (atomicOr(r.bm + (cell >> 5), bit) & bit) != 0u;
  if (act && !again) {
    // the segments holding outputs cell - h .. cell + h of the valid range
    const int s0 = max(cell - h, h) / kSeg, s1 = min(cell + h, C - 1 - h) / kSeg;
    if (H > 0) {
      if (s1 >= s0) {  // at most (2H + 4) / 4 + 1 <= 10 segments: two words
        const unsigned long long mask = ((2ull << (s1 - s0)) - 1ull) << (s0 & 31);
        atomicOr(r.segbits + (s0 >> 5), (uint32_t)mask);
        if ((uint32_t)(mask >> 32)) atomicOr(r.segbits + (s0 >> 5) + 1, (uint32_t)(mask >> 32));
      }
    } else {
#pragma unroll 1
      for (int s = s0; s <= s1; s = (s | 31) + 1) {
        const uint32_t from = 0xffffffffu << (s & 31);
        const uint32_t to = (s1 | 31) == (s | 31) ? 0xffffffffu >> (31 - (s1 & 31)) : 0xffffffffu;
        atomicOr(r.segbits + (s >> 5), from & to);
      }
    }
  }
  const unsigned later = __ballot_sync(kFull, again);
  if ((later & (later - 1u)) == 0u) {
    if (act && !again) r.row[cell] = v;
    __syncwarp();
    if (again) r.row[cell] = __fadd_rn(r.row[cell], v);
  } else {
    add_grouped(act, cell, r.done, lane, r.row, r.vals);
  }
  r.done += m;
}

// Appends the lanes' entries marked `in`, in lane order.
template <int H>
__device__ __forceinline__ void append_entries(RowList& r, bool in, int cell, float v, int h, int C,
                                               int lane) {
  const unsigned act = __ballot_sync(kFull, in);
  if (in) {
    const int at = (r.n + __popc(act & ((1u << lane) - 1u))) % kTouchCap;
    r.cells[at] = (uint16_t)cell;
    r.vals[at] = v;
  }
  r.n += __popc(act);
  if (r.n - r.done >= 32) add_entries<H>(r, 32, h, C, lane);
}

// The same for two consecutive entries per lane.
template <int H>
__device__ __forceinline__ void append_pairs(RowList& r, bool in0, bool in1, int cell0, int cell1,
                                             float v0, float v1, int h, int C, int lane) {
  const unsigned lt = (1u << lane) - 1u;
  const unsigned act0 = __ballot_sync(kFull, in0), act1 = __ballot_sync(kFull, in1);
  const int at = r.n + __popc(act0 & lt) + __popc(act1 & lt);
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
  while (r.n - r.done >= 32) add_entries<H>(r, 32, h, C, lane);
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

// Is a range of n entries scanned (else binary-searched, or empty)?
__device__ __forceinline__ bool scans(const SearchArgs& a, uint32_t n) {
  return n - 1u < a.scan_thresh;
}

// The CSR ranges of a precursor's (fragment, window) pairs, fetched 32 at a time
// (lane q holds pair pb + q).
struct PairCursor {
  int pb = 0;
  int64_t q = 0;   // absolute position of the pair's first entry
  uint32_t n = 0;  // entries
};

// The pair in lane q of the cursor.
struct Pair {
  int64_t q;
  uint32_t n;
};
__device__ __forceinline__ Pair pair_of(const PairCursor& pc, int q, int lane) {
  return Pair{__shfl_sync(kFull, pc.q, q), from_lane(pc.n, q, lane)};
}

// Bins and window of pair pi of precursor p, read again where they are rarely needed (kept
// in registers they cost the hot loop five).
struct PairBins {
  uint32_t b0, b1;
  WinInfo w;
};
__device__ __forceinline__ PairBins pair_bins(const SearchArgs& a, int64_t p, int pi, int nwin) {
  const int f = pi / nwin;
  const int64_t fo = p * a.kf + f;
  return PairBins{a.blo[fo], a.bhi[fo], a.win[a.wins[p * a.maxw + (pi - f * nwin)]]};
}

// An entry at the window's first cycle counts only if it is the last of its bin there
// (where Rust's binary_search lands, src/quadrupole_observation/mod.rs:91-94): is the
// next entry, entry `tn` of the pair's n, in another bin or at another cycle?  Out of
// line: about one range in fifty holds such an entry.
static __device__ __noinline__ bool last_at_start(const SearchArgs& a, int64_t p, int pi, int nwin,
                                                  int64_t q, uint32_t tn, uint32_t n, int cs) {
  if (tn >= n) return true;
  const PairBins pb = pair_bins(a, p, pi, nwin);
  if (bin_starts_at(a.ss + pb.w.ss_off, pb.b0, pb.b1, (uint32_t)(q + tn - pb.w.base))) return true;
  return (int)__ldg(a.cyc + q + tn) != cs;
}

// The rare strategy of gather_pair, out of line: per bin, binary-search the first kept
// entry and the first entry at or past stop, then read only the kept entries.
struct SearchedPair {
  int n, done;           // of the row list
  unsigned read, offs;   // entries and offsets read
};
template <int H, bool FAST>
static __device__ __noinline__ SearchedPair gather_searched(const SearchArgs& a, int64_t p, int pi,
                                                            int nwin, int cs, int C, int lane,
                                                            RowList r, int h) {
  SearchedPair out{0, 0, 0, 0};
  const PairBins pb = pair_bins(a, p, pi, nwin);
  const uint32_t b0 = pb.b0, b1 = pb.b1;
  const int64_t wbase = pb.w.base;
  const uint32_t* ssw = a.ss + pb.w.ss_off;
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
      append_entries<H>(r, vt, c - cs, v, h, C, lane);
    }
  }
  out.n = r.n;
  out.done = r.done;
  return out;
}

// fill_xic_slice for the (fragment, window) pair pi of precursor p: its entries
// inside the RT window are listed, in CSR order.  Two exact strategies: scan, which reads
// every entry of the range and keeps start < cycle < stop plus, per bin, the last entry
// at cycle == start (`staged`: the range's first kStageEntries entries are already on
// their way); or, for long ranges, gather_searched.
template <int H, bool FAST, bool STATS>
__device__ __forceinline__ void gather_pair(const SearchArgs& a, int64_t p, int pi, int nwin,
                                            Pair pr, bool staged, int cs, int C, int lane,
                                            uint32_t stage, const unsigned char* stage_p,
                                            RowList& r, int h, Counters<STATS>& k) {
  if (staged) {
    k.read += pr.n;
#pragma unroll 1
    for (uint32_t q0 = 0; q0 < pr.n; q0 += kStageEntries) {
      const int m = (int)min(pr.n - q0, (uint32_t)kStageEntries);
      const int64_t q = pr.q + q0;
      if (q0 > 0) {
        __syncwarp();  // the area's previous entries have been read
        stage_entries<FAST>(a, q, m, stage, lane);
      }
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
#pragma unroll 1
          for (int e = 0; e < 2; ++e) {
            const bool ask = e == 0 ? in0 && cell0 == 0 : in1 && cell1 == 0;
            if (ask) {
              const bool keep = last_at_start(a, p, pi, nwin, pr.q, q0 + (uint32_t)(t + e) + 1,
                                              pr.n, cs);
              if (e == 0)
                in0 = keep;
              else
                in1 = keep;
            }
          }
        }
        append_pairs<H>(r, in0, in1, cell0, cell1, v.x, v.y, h, C, lane);
      }
    }
  } else {
    const SearchedPair sp = gather_searched<H, FAST>(a, p, pi, nwin, cs, C, lane, r, h);
    r.n = uniform(sp.n);
    r.done = uniform(sp.done);
    k.read += sp.read;
    k.off += sp.offs;
  }
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
template <bool FAST>
__device__ __forceinline__ float conv_at(const float* row, const float* kw_s, int h, int j) {
  float s = __fadd_rn(0.0f, __fmul_rn(row[j], kw_s[h]));
#pragma unroll 1
  for (int t = 0; t < h; ++t) {
    const float lr = __fadd_rn(row[j - h + t], row[j + h - t]);
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

// The score terms s + ln(c + 1) * w (src/score/scalar.rs:16-22) of the 32 * U listed outputs
// from lst[0]: one rounded operation at a time with the exact ln; FAST (BF16 storage) takes
// the hardware log2 and a fused multiply-add.  The slow path of the exact ln is behind one
// vote.
template <int U, bool FAST>
__device__ __forceinline__ void score_terms(const float2* lst, float* score, float w,
                                            const double2* lnt, const LnCoef& k, int lane) {
  float* at[U];
  float s[U], x[U], y[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const float2 e = lst[32 * u + lane];
    at[u] = score + __float_as_int(e.y);
    s[u] = *at[u];
    x[u] = e.x;
  }
  if (FAST) {
#pragma unroll
    for (int u = 0; u < U; ++u) s[u] = __fmaf_rn(ln1p_fast(x[u]), w, s[u]);
  } else {
    bool slow[U], any = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      x[u] = __fadd_rn(x[u], 1.0f);
      slow[u] = ln_table(x[u], lnt, k, &y[u]);
      any = any || slow[u];
    }
    if (__any_sync(kFull, any)) {
#pragma unroll
      for (int u = 0; u < U; ++u) y[u] = slow[u] ? ln_rn_slow(x[u]) : y[u];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) s[u] = __fadd_rn(s[u], __fmul_rn(y[u], w));
  }
#pragma unroll
  for (int u = 0; u < U; ++u) *at[u] = s[u];
}

// Stores the pair (v, at) where `on`, predicated (a branch around each store cost three
// times as much).
template <bool GROW>
__device__ __forceinline__ void put_if(bool on, float2* to, float v, int at) {
  if (GROW) {
    if (on) *to = make_float2(v, __int_as_float(at));
  } else {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.u32 q, %0, 0;\n @q st.shared.v2.b32 [%1], {%2, %3};\n}" ::"r"(
            (uint32_t)on),
        "r"((uint32_t)__cvta_generic_to_shared(to)), "r"(__float_as_uint(v)), "r"(at)
        : "memory");
  }
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
  pc.q = 0;
  pc.n = 0;
  if (pj < npairs) {
    const int fj = nwin == 1 ? pj : pj / nwin, wj = pj - fj * nwin;
    const int64_t fo = p * a.kf + fj;
    const uint32_t b0 = a.blo[fo], b1 = a.bhi[fo];
    const int wsel = a.wins[p * a.maxw + wj];
    if (b1 > b0) {
      const WinInfo w = a.win[wsel];
      const uint32_t rs = __ldg(a.ss + w.ss_off + b0);
      pc.q = w.base + rs;
      pc.n = __ldg(a.ss + w.ss_off + b1) - rs;
    }
  }
}

// Starts staging a pair's first entries (after the area's last ones have been read).
template <bool FAST>
__device__ __forceinline__ bool stage_pair(const SearchArgs& a, Pair pr, int lane, uint32_t stage) {
  const bool scan = scans(a, pr.n);
  if (scan) {
    __syncwarp();
    stage_entries<FAST>(a, pr.q, (int)min(pr.n, (uint32_t)kStageEntries), stage, lane);
  }
  return scan;
}

// The last gathered row's cells (and bitmap words) back to zero.
__device__ __forceinline__ void clear_row(RowList& r, float* row, const WarpPlan& P, int lane) {
  if (r.n > kTouchCap) {
    float4* r4 = reinterpret_cast<float4*>(row);
#pragma unroll 1
    for (int i = lane; i < P.row_words / 4; i += 32) r4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int i = lane; i < P.bw; i += 32) r.bm[i] = 0u;
  } else {
#pragma unroll 1
    for (int i = lane; i < r.n; i += 32) {
      const int c = r.cells[i];
      r.row[c] = 0.0f;
      r.bm[c >> 5] = 0u;
    }
  }
#pragma unroll 1
  for (int i = lane; i < P.sw; i += 32) r.segbits[i] = 0u;
  r.n = r.done = 0;
  __syncwarp();
}

// A row whose weight is not finite, out of line: ln(conv + 1) * w is NaN even where conv
// is zero, so every column takes its term, as in the reference.
template <bool FAST>
static __device__ __noinline__ void score_every_column(const SearchArgs& a, const float* row,
                                                       const float* kw_s, int h, int C, float wf,
                                                       float* score, const double2* lnt, int lane) {
#pragma unroll 1
  for (int j = lane; j < C; j += 32) {
    const float c = (j >= h && j < C - h) ? conv_at<FAST>(row, kw_s, h, j) : 0.0f;
    score_add<FAST>(score, j, c, wf, lnt, a.ln);
  }
}

// Strict 5-point local maxima of a precursor's scores (src/peak_group_selection/mod.rs:33-43),
// collected in cycle order, and the top K of them by (value descending, cycle
// ascending), the reference's stable sort (src/peak_group_selection/mod.rs:45-61),
// written to the candidate slots.  `score` is 16-byte aligned, with four readable words
// below cycle 0 and past the last multiple of 4.
__device__ __forceinline__ void pick_top_k(const SearchArgs& a, int64_t p, int cs, int C,
                                           const float* score, float* mval, int* midx, int mx,
                                           int lane) {
  const unsigned lt = (1u << lane) - 1u;
  int nmax = 0;
  // 4 consecutive cycles per lane; two maxima are at least 4 cycles apart, so a lane finds
  // at most one
#pragma unroll 1
  for (int c0 = 0; c0 < C; c0 += 128) {
    const int j0 = c0 + 4 * lane;
    int found = -1;
    if (j0 < C) {
      const float4* s4 = reinterpret_cast<const float4*>(score + j0);
      const float4 l = s4[-1], m = s4[0], h = s4[1];
      const float v[8] = {l.z, l.w, m.x, m.y, m.z, m.w, h.x, h.y};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int i = j0 + t;
        if (i >= 2 && i < C - 2 && v[t] < v[t + 1] && v[t + 1] < v[t + 2] && v[t + 2] > v[t + 3] &&
            v[t + 3] > v[t + 4])
          found = i;
      }
    }
    const unsigned b = __ballot_sync(kFull, found >= 0);
    const int pos = nmax + __popc(b & lt);
    if (found >= 0 && pos < mx) {
      mval[pos] = score[found];
      midx[pos] = found;
    }
    nmax += __popc(b);
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

// A warp's next precursor: its place in the work queue, its row and its header.  The place
// is taken before the last row of the precursor before is convolved and the header read
// before its maxima are picked: the two round trips, about 2 of the 50 us that a warp spends
// on 12 rows of 301 cycles, are no longer waited for (200,000 uneven precursors FP32 3.80 ->
// 3.77 ms, 500,000 BF16 7.88 -> 7.79).  Taken earlier, a place would be held by a warp that
// is still busy when others have run out.
struct Work {
  unsigned pw;
  int64_t p;
  int nf, cs, ce, nwin;
};
// (lane 0 holds the place, which load_work gives to every lane)
__device__ __forceinline__ unsigned take_index(const SearchArgs& a, int lane) {
  return lane == 0 ? (unsigned)min(atomicAdd(a.work, 1ull), 0xffffffffull) : 0u;
}
__device__ __forceinline__ Work load_work(const SearchArgs& a, unsigned taken, unsigned n_work) {
  Work w;
  w.pw = __reduce_max_sync(kFull, taken);
  w.p = 0;
  w.nf = w.cs = w.ce = w.nwin = 0;
  if (w.pw < n_work) {
    w.p = a.list ? (int64_t)uniform(a.list[w.pw]) : (int64_t)w.pw;
    w.nf = a.nf[w.p];
    w.cs = a.cs[w.p];
    w.ce = a.ce[w.p];
    w.nwin = a.nwin[w.p];
  }
  return w;
}
__device__ __forceinline__ Work take_work(const SearchArgs& a, int lane, unsigned n_work) {
  return load_work(a, take_index(a, lane), n_work);
}

// GROW: the warp's working set (row, bitmaps, scores, lists, maxima) lives in
// a global buffer of P.total words per warp (`a.grow`) instead of shared memory, for
// RT windows longer than kSmemMaxCycles; the code and every operation are the same.
// STATS: the statistics pass's work counters (compiled in only for it).
template <int H, bool FAST, bool GROW, bool STATS>
__global__ void __launch_bounds__(LaunchShape<GROW>::threads, LaunchShape<GROW>::blocks)
    search_kernel(const __grid_constant__ SearchArgs a) {
  extern __shared__ __align__(16) float smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = H > 0 ? H : a.h;
  const WarpPlan P = warp_plan(h, a.c_max);
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
  uint32_t* segbits = reinterpret_cast<uint32_t*>(wb + P.segbits);
  uint16_t* segs = reinterpret_cast<uint16_t*>(wb + P.segs);
  RowList r{row + P.off, bm, segbits, reinterpret_cast<uint16_t*>(wb + P.cells), wb + P.lst, 0, 0};
  {
    float4* r4 = reinterpret_cast<float4*>(row);
#pragma unroll 1
    for (int i = lane; i < P.row_words / 4; i += 32) r4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int i = lane; i < P.bw; i += 32) bm[i] = 0u;
#pragma unroll 1
    for (int i = lane; i < P.sw; i += 32) segbits[i] = 0u;
  }

#pragma unroll 1
  for (int i = threadIdx.x; i < kLnTableSize; i += blockDim.x) lnt[i] = a.ln_tab[i];
#pragma unroll 1
  for (int i = threadIdx.x; i <= a.h; i += blockDim.x) kw_s[i] = a.kw_dev ? a.kw_dev[i] : a.kw[i];
  __syncthreads();
  Counters<STATS> k;
  const unsigned lt = (1u << lane) - 1u;

  const unsigned n_work = a.list ? (unsigned)uniform((int)*a.list_len) : (unsigned)a.n_prec;
  Work next_p = take_work(a, lane, n_work);
#pragma unroll 1
  while (next_p.pw < n_work) {
    const int64_t p = next_p.p;
    const int F = uniform(next_p.nf);
    const int cs = uniform(next_p.cs);
    const int C = uniform(next_p.ce) - cs;
    const int nwin = uniform(next_p.nwin);
    if (F == 0 || C <= 0 || C > a.c_max) {
      if (lane == 0) {
        a.cand_n[p] = 0;
        if (F != 0 && C > a.c_max) atomicOr(a.err, 2);
      }
      next_p = take_work(a, lane, n_work);
      continue;
    }
    const int npairs = F * nwin;
    unsigned taken = npairs == 0 ? take_index(a, lane) : 0u;  // else with the last pair
    k.frag += F;
    // fragment weights, lane f holding fragment f's (fetched once per precursor)
    const float wf_lane = lane < F ? __ldg(a.fw + p * a.kf + lane) : 0.0f;
    PairCursor pc;
    load_pairs(a, p, 0, nwin, npairs, lane, pc);
    Pair next = pair_of(pc, 0, lane);
    bool staged = stage_pair<FAST>(a, next, lane, stage);
#pragma unroll 1
    for (int i = lane; i < C; i += 32) score[i] = 0.0f;
    int f = -1, wi = 0;
    // pairs in fragment, then window order (the reference's DenseXICObservation::new,
    // src/dense_xic_observation/mod.rs:30-64)
#pragma unroll 1
    for (int pi = 0; pi < npairs; ++pi) {
      // ---- 1. gather
      if (STATS) {
        const PairBins pb = pair_bins(a, p, pi, nwin);
        if (pb.b1 > pb.b0) {
          k.off += 2u;
          k.pairs += 1u;
          k.bins1 += pb.b1 - pb.b0 + 1;
        }
      }
      if (next.n > 0)
        gather_pair<H, FAST, STATS>(a, p, pi, nwin, next, staged, cs, C, lane, stage, stage_p, r, h, k);
      if (pi + 1 < npairs) {
        // the next pair's entries arrive while this row is convolved
        if (pi + 1 >= pc.pb + 32) load_pairs(a, p, pi + 1, nwin, npairs, lane, pc);
        next = pair_of(pc, pi + 1 - pc.pb, lane);
        staged = stage_pair<FAST>(a, next, lane, stage);
      } else {
        taken = take_index(a, lane);
      }
      if (++wi < nwin) continue;  // more windows hold this fragment
      wi = 0;
      ++f;
      k.acc += (unsigned int)r.n;
      if (r.done < r.n) add_entries<H>(r, r.n - r.done, h, C, lane);
      __syncwarp();
      float wf = __shfl_sync(kFull, wf_lane, f & 31);
      if (f >= 32) wf = __ldg(a.fw + p * a.kf + f);
      if (!isfinite(wf)) {
        score_every_column<FAST>(a, r.row, kw_s, h, C, wf, score, lnt, lane);
        __syncwarp();
        clear_row(r, row, P, lane);
        continue;
      }
      if (r.n == 0) continue;  // no entry accepted: every term is +0
      // ---- 2./3. convolution of the segments that a touched cycle reaches (every other
      // output is zero), one per lane, then the score terms of the non-zero outputs of the
      // valid range [h, C - h).  A zero output adds ln(1) * w = +0, which leaves a score
      // as it is, so only the others are listed and take a logarithm, 32 at a time.  Their
      // order within the row is free: each has its own cycle.
      const int n_seg = (C - h + kSeg - 1) / kSeg;
      int nact = 0;
#pragma unroll 1
      for (int w0 = 0; w0 < n_seg; w0 += 32) {
        const uint32_t x = segbits[w0 / 32];
        if ((x >> lane) & 1u) segs[nact + __popc(x & lt)] = (uint16_t)(w0 + lane);
        nact += __popc(x);
      }
      nact = uniform(nact);
      __syncwarp();
      int listed = 0;
#pragma unroll 1
      for (int a0 = 0; a0 < nact; a0 += 32) {
        const bool on = a0 + lane < nact;
        const int j0 = on ? (int)segs[a0 + lane] * kSeg : 0;  // (idle lanes: segment 0)
        const int rel = on ? j0 - h : -(1 << 20);             // of output 0 to the valid range
        float cv[kSeg];
        if (H > 0) {
          // cells j0 - OFF .. j0 + 3 + OFF; every output is formed in the reference's
          // order: 0 + x[j]*w[h], then + (x[j-d] + x[j+d]) * w[h-d] for d = h..1, two
          // outputs (m, m + 1) per packed instruction.  For odd d the pair sums straddle
          // the register pairs and are formed by two scalar adds.
          constexpr int OFF = (H + kSeg - 1) / kSeg * kSeg;
          constexpr int NX = kSeg + 2 * OFF;
          const float4* rb = reinterpret_cast<const float4*>(row + j0);
          float xv[NX];
#pragma unroll
          for (int q = 0; q < NX; q += 4) {
            const float4 v = rb[q / 4];
            xv[q] = v.x;
            xv[q + 1] = v.y;
            xv[q + 2] = v.z;
            xv[q + 3] = v.w;
          }
          f32x2 acc[kSeg / 2];
#pragma unroll
          for (int m = 0; m < kSeg; m += 2)
            acc[m / 2] = add2(a.zero2, fma2(pk2(xv[m + OFF], xv[m + 1 + OFF]), a.kw2[H], a.nzero2));
#pragma unroll
          for (int t = 0; t < H; ++t) {
            const int d = H - t;
#pragma unroll
            for (int m = 0; m < kSeg; m += 2) {
              const int l = m - d + OFF, u = m + d + OFF;
              f32x2 lr;
              if (d % 2 == 0)
                lr = add2(pk2(xv[l], xv[l + 1]), pk2(xv[u], xv[u + 1]));
              else
                lr = pk2(__fadd_rn(xv[l], xv[u]), __fadd_rn(xv[l + 1], xv[u + 1]));
              acc[m / 2] = FAST ? fma2(lr, a.kw2[t], acc[m / 2])
                                : add2(acc[m / 2], fma2(lr, a.kw2[t], a.nzero2));
            }
          }
#pragma unroll
          for (int m = 0; m < kSeg; m += 2) unpk2(acc[m / 2], cv[m], cv[m + 1]);
        } else {
#pragma unroll
          for (int m = 0; m < kSeg; ++m) {
            cv[m] = 0.0f;
            if ((unsigned)(rel + m) < (unsigned)(C - 2 * h)) cv[m] = conv_at<FAST>(r.row, kw_s, h, j0 + m);
          }
        }
#pragma unroll
        for (int m = 0; m < kSeg; ++m) {
          const bool ok = (unsigned)(rel + m) < (unsigned)(C - 2 * h) && cv[m] != 0.0f;
          const unsigned b = __ballot_sync(kFull, ok);
          put_if<GROW>(ok, lst + listed + __popc(b & lt), cv[m], j0 + m);
          listed += __popc(b);
        }
        if (a0 + 32 >= nact) {
          // the row's last round: idle entries up to a whole warp, which work on a word
          // below the scores
          lst[listed + lane] = make_float2(0.0f, __int_as_float(-4));
          listed = (listed + 31) & ~31;
        }
        __syncwarp();
#pragma unroll 1
        while (listed >= 32 * kTerms) {
          listed -= 32 * kTerms;
          score_terms<kTerms, FAST>(lst + listed, score, wf, lnt, a.ln, lane);
        }
#pragma unroll 1
        while (listed >= 32) {
          listed -= 32;
          score_terms<1, FAST>(lst + listed, score, wf, lnt, a.ln, lane);
        }
        __syncwarp();
      }
      clear_row(r, row, P, lane);
    }
    __syncwarp();
    // the next precursor was taken before the last row's convolution; its header arrives
    // while this one's maxima are picked
    next_p = load_work(a, taken, n_work);
    pick_top_k(a, p, cs, C, score, mval, midx, P.mx, lane);
  }
  flush_counters<STATS>(a, k, lane);
}
