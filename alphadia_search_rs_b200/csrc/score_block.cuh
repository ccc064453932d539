// The block kernel of scoring and quantification: a block of 2 warps takes up to kGroup
// candidates through the steps of score_kernel / quant_kernel with one thread per
// (candidate, fragment), per (candidate, cycle) or per candidate, whatever the step is
// made of, and everything in shared memory.  Included by score.cu inside namespace
// ads::{anonymous}; every f32 operation is that of the per-candidate kernels, in their
// order, through the same helpers.
//
// What bounds it: the gather's loads and the waits between steps (31 warps per SM issue on
// 48 % of the cycles with 15 of 32 lanes; 4.4 warps wait for memory and 4.4 at a barrier per
// issue).  A thread per candidate (score_kernel) ran 8 of 32 lanes per instruction on matrices
// in a global scratch, and walked every bin of every fragment with a binary search.  Here a
// row's whole range of entries is read 8 cycle indices at a time, and only an entry inside
// the window looks up its bin: 1.48 M candidates of 4-24 fragments scored 41.0 -> 10.2 ms,
// quantified 29.0 -> 7.8 ms.
constexpr int kGroup = 4;        // candidates of a block (at most)
// 2 warps for 4 candidates; for 2: scored 3.06 ms against 2.51 (295,000 candidates); 1 warp
// for 4: 2.76; 1 for 2: 2.47, but quantified 1.19 against 1.18.
constexpr int kBlockWarps = 2;
constexpr int kBlockThreads = 32 * kBlockWarps;
// A candidate's shared memory grows with fragments x cycles; beyond this many bytes a block
// the group is halved, and where not even 2 candidates fit the per-candidate kernels run.
constexpr size_t kBlockSmem = 64 * 1024;

// Vectors of one candidate, in words.
struct BlockPlan {
  int Fm, Cm;      // most kept fragments, most cycles
  int Fraw;        // most library fragments
  int cs;          // row stride of the profiles (odd: rows of consecutive lanes hit different banks)
  int fmz, fint, idf, tn, obs, corr;  // per fragment (mass error takes the m/z's place)
  int med, medf;   // per cycle
  int head;        // words of the vectors, all but the profiles
  int prof;        // profiles, before them the raw fragments, after them sort space
  int words;       // of one candidate (odd)
  int scratch;     // words of one thread's column or row buffer
};

__host__ __device__ inline BlockPlan block_plan(int Fm, int Fraw, int Cm) {
  BlockPlan b;
  b.Fm = Fm;
  b.Cm = Cm;
  b.Fraw = Fraw;
  b.cs = Cm | 1;
  int o = 0;
  b.fmz = o;
  o += Fm;
  b.fint = o;
  o += Fm;
  b.idf = o;
  o += Fm;
  b.tn = o;
  o += Fm;
  b.obs = o;
  o += Fm;
  b.corr = o;
  o += Fm;
  b.med = o;
  o += Cm;
  b.medf = o;
  o += Cm;
  b.head = o;
  b.prof = o;
  int pw = Fm * b.cs;
  if (pw < 3 * Fraw) pw = 3 * Fraw;
  if (pw < 2 * Fm) pw = 2 * Fm;
  o += pw;
  b.words = o | 1;
  b.scratch = Fm > Cm ? Fm : Cm;
  return b;
}

// What a block knows of a candidate.
struct BlockCand {
  int64_t q;       // its index
  int64_t fs;      // first library fragment
  int64_t prec;    // row of its precursor
  int nraw, F, cs, C;
  int woff, wlen;  // windows that hold its precursor m/z
  int nz;          // kept fragments whose profile is not all zero
  float pmz;
};

inline size_t block_smem_bytes(const BlockPlan& b, int group) {
  return (size_t)group * sizeof(BlockCand) + 4 * ((size_t)group * b.words + (size_t)kBlockThreads * b.scratch);
}

// Words of one candidate, for the shared helpers.
struct SmVec {
  typedef int I;
  static constexpr int kUnroll = 1;
  uint32_t* base;
  __device__ float f(int e) const { return __uint_as_float(base[e]); }
  __device__ void sf(int e, float v) const { base[e] = __float_as_uint(v); }
  __device__ uint32_t u(int e) const { return base[e]; }
  __device__ void su(int e, uint32_t v) const { base[e] = v; }
};
// One thread's buffer, interleaved across the block's threads.
struct ThreadVec {
  typedef int I;
  static constexpr int kUnroll = 1;
  uint32_t* base;  // of the thread
  __device__ float f(int e) const { return __uint_as_float(base[e * kBlockThreads]); }
  __device__ void sf(int e, float v) const { base[e * kBlockThreads] = __float_as_uint(v); }
  __device__ uint32_t u(int e) const { return base[e * kBlockThreads]; }
  __device__ void su(int e, uint32_t v) const { base[e * kBlockThreads] = v; }
};

// Bin of the window's entry at relative position q, searched in [b, b1).
__device__ __forceinline__ uint32_t bin_of(const uint32_t* ssw, uint32_t b, uint32_t b1, uint32_t q) {
  uint32_t lo = b, hi = b1;  // the last bin whose first entry is at or before q
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(ssw + mid) <= q)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// Bit 15 or 31 set where some 16-bit half of z is zero (perhaps also above a zero half).
__device__ __forceinline__ uint32_t zero_half(uint32_t z) { return (z - 0x00010001u) & ~z; }

// One fragment's row of gather_xic_mz: dense XIC (x) and intensity-weighted m/z (z) over
// cycles [cs, cs + C).
template <class X, class Z>
__device__ __forceinline__ void gather_one(const ScoreArgs& a, const X& x, int x0, const Z& z,
                                           float mz, int cs, int C, int woff, int wlen) {
#pragma unroll 1
  for (int j = 0; j < C; ++j) {
    x.sf(x0 + j, 0.0f);
    z.sf(j, 0.0f);
  }
  if (C <= 0 || cs > 0xffff) return;
  const float delta = __fmul_rn(__fmul_rn(mz, a.tol), 1e-6f);
  const uint32_t b0 = grid_lower_bound(a.g, __fsub_rn(mz, delta));
  const uint32_t b1 = max(b0, grid_upper_bound(a.g, __fadd_rn(mz, delta)));
  if (b1 <= b0) return;
  // (entries' cycles end at 65,535, a range may not: the RT index counts MS1 spectra)
  const uint32_t first2 = (uint32_t)cs * 0x10001u, last2 = (uint32_t)min(cs + C - 1, 0xffff) * 0x10001u;
  for (int w = 0; w < wlen; ++w) {
    const WinInfo wi = a.win[__ldg(a.wi.list + woff + w)];
    const uint32_t* ssw = a.ss + wi.ss_off;
    const uint32_t r0 = __ldg(ssw + b0), n = __ldg(ssw + b1) - r0;
    // 8 cycle indices at a time from the 16-byte boundary at or below the first entry
    // (the arrays are allocated kEntrySlack entries past the last one): position i of the
    // range is entry skip + i counted from there
    const int64_t q0 = wi.base + r0;
    const uint32_t skip = (uint32_t)(q0 & 7);
    const uint4* c8 = reinterpret_cast<const uint4*>(a.cyc + (q0 - skip));
    const uint16_t* cy = a.cyc + q0;
    const float* iy = a.inten + q0;
    uint32_t b = b0, b_end = 0;  // bin of the last entry and the bin's end
    float actual = 0.0f;
    for (uint32_t j = 0; j < skip + n; j += 8) {
      const uint4 v = __ldg(c8 + (j >> 3));
      // most groups of 8 hold none: a half of a word is in the window where clamping it
      // there changes nothing
      const uint32_t z0 = v.x ^ __vmaxu2(__vminu2(v.x, last2), first2);
      const uint32_t z1 = v.y ^ __vmaxu2(__vminu2(v.y, last2), first2);
      const uint32_t z2 = v.z ^ __vmaxu2(__vminu2(v.z, last2), first2);
      const uint32_t z3 = v.w ^ __vmaxu2(__vminu2(v.w, last2), first2);
      if (!((zero_half(z0) | zero_half(z1) | zero_half(z2) | zero_half(z3)) & 0x80008000u)) continue;
      uint32_t in = 0;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t word = h == 0 ? v.x : h == 1 ? v.y : h == 2 ? v.z : v.w;
        in |= (uint32_t)((unsigned)((int)(word & 0xffffu) - cs) < (unsigned)C) << (2 * h);
        in |= (uint32_t)((unsigned)((int)(word >> 16) - cs) < (unsigned)C) << (2 * h + 1);
      }
      if (j < skip) in &= 0xffu << skip;
      if (j + 8 > skip + n) in &= 0xffu >> (j + 8 - skip - n);
      while (in) {
        const uint32_t at = j + (uint32_t)__ffs(in) - 1u - skip;
        in &= in - 1;
        const float y = __ldg(iy + at);
        const int c = (int)__ldg(cy + at) - cs;
        if (r0 + at >= b_end) {  // (entries of one ion mostly share a bin)
          b = bin_of(ssw, b, b1, r0 + at);
          b_end = __ldg(ssw + b + 1);
          actual = __ldg(a.g.grid + b);
        }
        // Rust's binary_search lands on the last of a bin's entries at the first cycle
        if (c == 0 && r0 + at + 1 < b_end && (int)__ldg(cy + at + 1) == cs) continue;
        const float xs = __fadd_rn(x.f(x0 + c), y);
        x.sf(x0 + c, xs);
        if (y > 0.0f) {
          const float prev = __fsub_rn(xs, y);
          if (prev == 0.0f)
            z.sf(c, actual);
          else
            z.sf(c, __fdiv_rn(__fadd_rn(__fmul_rn(z.f(c), prev), __fmul_rn(actual, y)), xs));
        }
      }
    }
  }
}

// hyperscore over the fragments seen (observed intensity above 0); `inverse`: weighted by
// 1 / (|mass error| + 0.1).
__device__ float hyperscore_of(const SmVec& s, const BlockPlan& B, int v0, bool inverse, int n,
                               const Ln& ln) {
  HyperSums h;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    const float v = s.f(v0 + i);
    if (!(s.f(B.obs + i) > 0.0f) || v == 0.0f) continue;
    const float w = inverse ? __fdiv_rn(1.0f, __fadd_rn(fabsf(s.f(B.fmz + i)), 0.1f)) : 1.0f;
    h.add(s.u(B.tn + i) & 0xffu, __fmul_rn(v, w));
  }
  return h.value(ln);
}

// longest_series over the fragments seen, numbers sorted at etmp.
__device__ __forceinline__ uint32_t longest_series_of(const SmVec& s, const BlockPlan& B, int n,
                                                      uint32_t type, int etmp) {
  int m = 0;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    const uint32_t tn = s.u(B.tn + i);
    if (s.f(B.obs + i) > 0.0f && (tn & 0xffu) == type) s.su(etmp + m++, (tn >> 8) & 0xffu);
  }
  return longest_run(s, etmp, m);
}

// A kept fragment's word `tn`: type, number << 8, and these flags.  (Quantification has its
// library offset in `corr` and its observed m/z in `idf`.)
constexpr uint32_t kFlagNz = 1u << 16;   // profile not all zero
constexpr uint32_t kFlagTop = 1u << 17;  // among the six highest IDF values
constexpr int kFlagBand = 18;            // from this bit: intensity rank / 6 (4: rank 24 and on)

// Where the reference's binary search of the sorted precursor_idx ends: the last row at or
// below `pidx` (0 where there is none).  kRowLanes lanes of the warp per search, each
// testing the end of one of as many parts: 5 dependent loads in 500,000 rows instead of 19,
// which a block's other threads waited for (295,000 candidates of 4-24 fragments scored
// 2.55 -> 2.51 ms, 6000 of them 80.5 -> 78.8 us).  Whole warps call it, those without a search
// with no rows.
constexpr int kRowLanes = kBlockThreads / kGroup;
static_assert(kRowLanes <= 32 && 32 % kRowLanes == 0, "a search stays within a warp");
__device__ __forceinline__ int64_t find_row(const uint64_t* idx, int64_t n, uint64_t pidx, int lane) {
  const int sub = lane % kRowLanes;
  int64_t lo = 0;
  while (__any_sync(0xffffffffu, n > 0)) {
    const int64_t part = (n + kRowLanes - 1) / kRowLanes;
    const int64_t end = min((sub + 1) * part, n);
    const bool below = n > 0 && idx[lo + end - 1] <= pidx;
    const unsigned all = __ballot_sync(0xffffffffu, below) >> (lane - sub);
    const int parts = __popc(all & (unsigned)((1ull << kRowLanes) - 1ull));
    const int64_t from = min(parts * part, n);
    lo += from;
    n = max(min((parts + 1) * part, n) - 1 - from, (int64_t)0);
  }
  return max(lo - 1, (int64_t)0);
}

template <bool QUANT>
__global__ void __launch_bounds__(kBlockThreads) score_block_kernel(const __grid_constant__ QuantArgs qa,
                                                                    const __grid_constant__ BlockPlan B,
                                                                    int group) {
  const ScoreArgs& a = qa.s;
  extern __shared__ __align__(16) unsigned char block_smem[];
  BlockCand* cand = reinterpret_cast<BlockCand*>(block_smem);
  uint32_t* vec = reinterpret_cast<uint32_t*>(cand + group);
  uint32_t* thr = vec + (size_t)group * B.words;
  __shared__ int sh_max[3];  // of the group: raw fragments, kept fragments, cycles
  const int tid = threadIdx.x, lane = tid & 31;
  const ThreadVec own{thr + tid};
  const Ln ln{a.ln_tab, LnCoef()};
  const int64_t first = a.at + (int64_t)blockIdx.x * group, end = a.at + a.take;

  // ---- the candidates and their precursors
  __shared__ int64_t sh_row[kGroup];
  if (tid < 3) sh_max[tid] = 0;
  {
    const int c = tid / kRowLanes;
    const bool on = c < group && first + c < end;
    const int64_t q = on ? (a.order ? (int64_t)a.order[first + c] : first + c) : 0;
    const int64_t row = find_row(a.l_pidx, on ? a.P : 0, on ? a.c_pidx[q] : 0, lane);
    if (on && tid % kRowLanes == 0) sh_row[c] = row;
  }
  __syncthreads();
  if (tid < group) {
    BlockCand k;
    k.q = -1;
    k.fs = k.prec = 0;
    k.nraw = k.F = k.cs = k.C = k.woff = k.wlen = k.nz = 0;
    k.pmz = 0.0f;
    if (first + tid < end) {
      const int64_t q = a.order ? (int64_t)a.order[first + tid] : first + tid;
      const uint64_t pidx = a.c_pidx[q], cs64 = a.c_start[q], ce64 = a.c_stop[q], center = a.c_center[q];
      bool take = true;
      if (QUANT) {
        qa.o_nq[q] = 0;
        if (ce64 <= cs64 || center < cs64 || center >= ce64) {
          take = false;  // dropped, as in the reference
        } else if (ce64 > (uint64_t)a.n_rt || ce64 - cs64 > (uint64_t)B.Cm) {
          atomicOr(a.err, 1);
          take = false;
        }
      } else {
        a.o_found[q] = 0;
        if (cs64 > ce64 || ce64 > (uint64_t)a.n_rt || center >= (uint64_t)a.n_rt ||
            ce64 - cs64 > (uint64_t)B.Cm) {
          atomicOr(a.err, 1);
          take = false;
        }
      }
      if (take && a.P > 0) {
        // SpecLibFlat::get_precursor_by_idx_filtered: binary search of the sorted idx
        const int64_t base = sh_row[tid];
        if (a.l_pidx[base] == pidx) {  // else skipped, as in the reference
          const int64_t fs = (int64_t)a.l_fs[base], nraw = (int64_t)a.l_fe[base] - fs;
          if (nraw > B.Fraw) {
            atomicOr(a.err, 2);
          } else {
            k.q = q;
            k.fs = fs;
            k.prec = base;
            k.nraw = (int)nraw;
            k.cs = (int)cs64;
            k.C = (int)(ce64 - cs64);
            k.pmz = a.l_pmz[base];
            find_windows(a.wi, k.pmz, &k.woff, &k.wlen);
            atomicMax(sh_max + 0, k.nraw);
            atomicMax(sh_max + 2, k.C);
          }
        }
      }
    }
    cand[tid] = k;
  }
  __syncthreads();

  // ---- filter_sort_fragments (select_fragments): m/z key, intensity and keep mark ...
  const int RAWM = B.prof, RAWI = B.prof + B.Fraw, KEEP = B.prof + 2 * B.Fraw;
  const int nraw_max = sh_max[0];
  for (int t = tid; t < group * nraw_max; t += kBlockThreads) {
    const int c = t / nraw_max, r = t - c * nraw_max;
    const BlockCand& k = cand[c];
    if (r >= k.nraw) continue;
    const SmVec s{vec + c * B.words};
    const float I = a.l_fint[k.fs + r];
    s.sf(RAWM + r, mz_key(a.l_fmz[k.fs + r]));
    s.sf(RAWI + r, I);
    s.su(KEEP + r, I > 0.0f && !(a.l_ftype[k.fs + r] == 121 && a.l_fnum[k.fs + r] == 1) ? 1u : 0u);
  }
  __syncthreads();
  // ... the kept ones counted, and where they are too many the top_k by intensity marked
  // (ties to the lower position)
  if (tid < group) {
    const SmVec s{vec + tid * B.words};
    int nk = 0;
#pragma unroll 1
    for (int r = 0; r < cand[tid].nraw; ++r) nk += (int)s.u(KEEP + r);
    cand[tid].F = nk;
  }
  __syncthreads();
  const int top_k = (int)min(a.top_k, (int64_t)INT_MAX);
  for (int t = tid; t < group * nraw_max; t += kBlockThreads) {
    const int c = t / nraw_max, r = t - c * nraw_max;
    const BlockCand& k = cand[c];
    if (r >= k.nraw || k.F <= top_k) continue;
    const SmVec s{vec + c * B.words};
    if (!s.u(KEEP + r)) continue;
    const float I = s.f(RAWI + r);
    int rank = 0;
#pragma unroll 1
    for (int j = 0; j < r; ++j)
      if (s.u(KEEP + j)) rank += !(s.f(RAWI + j) < I);
#pragma unroll 1
    for (int j = r + 1; j < k.nraw; ++j)
      if (s.u(KEEP + j)) rank += s.f(RAWI + j) > I;
    if (rank < top_k) s.su(KEEP + r, 2u);  // (only told from 1 after the barrier)
  }
  __syncthreads();
  // ... and put in m/z order (ties keep library order)
  for (int t = tid; t < group * nraw_max; t += kBlockThreads) {
    const int c = t / nraw_max, r = t - c * nraw_max;
    const BlockCand& k = cand[c];
    if (r >= k.nraw) continue;
    const SmVec s{vec + c * B.words};
    const uint32_t need = k.F > top_k ? 2u : 1u;
    if (s.u(KEEP + r) < need) continue;
    const float key = s.f(RAWM + r), m = key < INFINITY ? key : a.l_fmz[k.fs + r];
    int pos = 0;
#pragma unroll 1
    for (int j = 0; j < r; ++j)
      if (s.u(KEEP + j) >= need) pos += s.f(RAWM + j) <= key;
#pragma unroll 1
    for (int j = r + 1; j < k.nraw; ++j)
      if (s.u(KEEP + j) >= need) pos += s.f(RAWM + j) < key;
    s.sf(B.fmz + pos, m);
    s.sf(B.fint + pos, s.f(RAWI + r));
    if (QUANT) {
      s.su(B.tn + pos, 0u);
      s.su(B.corr + pos, (uint32_t)r);
    } else {
      s.su(B.tn + pos, (uint32_t)a.l_ftype[k.fs + r] | (uint32_t)a.l_fnum[k.fs + r] << 8);
      float idf = 1.0f;
      if (a.idf_total != 0.0f) {
        const uint32_t cnt = a.idf_counts[grid_find_closest(a.g, a.l_fmzl[k.fs + r])];
        idf = ln(__fdiv_rn(a.idf_total, (float)max(cnt, 1u)));
      }
      s.sf(B.idf + pos, idf);
    }
  }
  __syncthreads();
  if (tid < group) {
    cand[tid].F = min(cand[tid].F, top_k);
    atomicMax(sh_max + 1, cand[tid].F);
  }
  __syncthreads();

  // ---- per fragment: XIC row, observed m/z and intensity, normalised profile
  const int F_max = sh_max[1], C_max = sh_max[2];
  for (int t = tid; t < group * F_max; t += kBlockThreads) {
    const int c = t / F_max, f = t - c * F_max;
    const BlockCand& k = cand[c];
    if (f >= k.F) continue;
    const SmVec s{vec + c * B.words};
    const int X = B.prof + f * B.cs, C = k.C;
    const float lib = s.f(B.fmz + f);
    gather_one(a, s, X, own, lib, k.cs, C, k.woff, k.wlen);
    s.sf(B.obs + f, ndarray_sum(s, X, C));
    float ws = 0.0f, wsum = 0.0f;
#pragma unroll 1
    for (int j = 0; j < C; ++j) {
      const float w = s.f(X + j);
      if (w > 0.0f) {
        ws = __fadd_rn(ws, __fmul_rn(own.f(j), w));
        wsum = __fadd_rn(wsum, w);
      }
    }
    const float o = wsum > 0.0f ? __fdiv_rn(ws, wsum) : 0.0f;
    s.sf(B.fmz + f, o > 0.0f ? __fmul_rn(__fdiv_rn(__fsub_rn(o, lib), lib), 1e6f) : 0.0f);
    if (QUANT) s.sf(B.idf + f, o);
    // normalize_profiles(xic, 1) (normalize_rows), in place
    const int cc = C / 2;
    const int c0 = cc > 1 ? cc - 1 : 0, c1 = cc + 2 < C ? cc + 2 : C;
    float sum = 0.0f;
    int count = 0;
#pragma unroll 1
    for (int j = c0; j < c1; ++j) {
      sum = __fadd_rn(sum, s.f(X + j));
      ++count;
    }
    const float mean = count > 0 ? __fdiv_rn(sum, (float)count) : 0.0f;
    uint32_t nz = 0;
#pragma unroll 1
    for (int j = 0; j < C; ++j) {
      const float v = mean > 0.0f ? __fdiv_rn(s.f(X + j), mean) : 0.0f;
      s.sf(X + j, v);
      nz |= v != 0.0f;
    }
    if (nz) {
      s.su(B.tn + f, s.u(B.tn + f) | kFlagNz);
      atomicAdd(&cand[c].nz, 1);
    }
  }
  __syncthreads();

  // ---- per cycle: median of all profiles and of those not all zero (zero when none)
  for (int t = tid; t < group * C_max; t += kBlockThreads) {
    const int c = t / C_max, j = t - c * C_max;
    const BlockCand& k = cand[c];
    if (j >= k.C) continue;
    const SmVec s{vec + c * B.words};
    const bool all_nz = k.nz == k.F;  // the two are then the median of the same values
#pragma unroll 1
    for (int pass = QUANT || all_nz ? 1 : 0; pass < 2; ++pass) {
      int R = 0;
#pragma unroll 1
      for (int f = 0; f < k.F; ++f)
        if (pass == 0 || (s.u(B.tn + f) & kFlagNz)) own.sf(R++, s.f(B.prof + f * B.cs + j));
      float med = 0.0f;
      if (R > 0) {
        sort_floats(own, 0, R);
        med = R % 2 == 0 ? __fdiv_rn(__fadd_rn(own.f(R / 2 - 1), own.f(R / 2)), 2.0f) : own.f(R / 2);
      }
      if (pass == 0 || all_nz) s.sf(B.med + j, med);
      if (pass == 1) s.sf(B.medf + j, med);
    }
  }
  __syncthreads();

  // ---- per fragment: correlation with the median of the non-zero profiles; ranks
  for (int t = tid; t < group * F_max; t += kBlockThreads) {
    const int c = t / F_max, f = t - c * F_max;
    const BlockCand& k = cand[c];
    if (f >= k.F) continue;
    const SmVec s{vec + c * B.words};
    if (QUANT && !(s.f(B.obs + f) > 0.0f)) continue;  // filter_fragments_by_intensity(0.0)
    const XStats xmed = x_stats(s, B.medf, k.C);
    const float corr = correlation_fixed_x(s, xmed, B.medf, B.prof + f * B.cs, k.C);
    if (QUANT) {
      int slot = 0;
#pragma unroll 1
      for (int j = 0; j < f; ++j) slot += s.f(B.obs + j) > 0.0f;
      const int64_t o = k.q * a.Fm + slot;
      qa.o_frow[o] = (uint64_t)k.fs + s.u(B.corr + f);
      qa.o_int[o] = s.f(B.obs + f);
      qa.o_mzo[o] = s.f(B.idf + f);
      qa.o_err[o] = s.f(B.fmz + f);
      qa.o_corr[o] = corr;
    } else {
      s.sf(B.corr + f, corr);
      // create_ranked_mask: earlier not below plus later above (ties to the lower index)
      const float v = s.f(B.fint + f), w = s.f(B.idf + f);
      int rank = 0, top = 0;
#pragma unroll 1
      for (int j = 0; j < f; ++j) {
        rank += !(s.f(B.fint + j) < v);
        top += !(s.f(B.idf + j) < w);
      }
#pragma unroll 1
      for (int j = f + 1; j < k.F; ++j) {
        rank += s.f(B.fint + j) > v;
        top += s.f(B.idf + j) > w;
      }
      s.su(B.tn + f, s.u(B.tn + f) | (top < 6 ? kFlagTop : 0u) |
                         (uint32_t)(rank < 24 ? rank / 6 : 4) << kFlagBand);
    }
  }
  __syncthreads();

  if (QUANT) {
    if (tid < group && cand[tid].q >= 0) {
      const BlockCand& k = cand[tid];
      const SmVec s{vec + tid * B.words};
      int nq = 0;
#pragma unroll 1
      for (int f = 0; f < k.F; ++f) nq += s.f(B.obs + f) > 0.0f;
      qa.o_nq[k.q] = nq;
      qa.o_prow[k.q] = qa.l_prow[k.prec];
      qa.o_rt[k.q] = a.rt[a.c_center[k.q]];
    }
    return;
  }

  // ---- what feature_kernel needs of them
  for (int t = tid; t < group * B.head; t += kBlockThreads) {
    const int c = t / B.head, j = t - c * B.head;
    if (cand[c].q >= 0) a.heads[(first - a.at + c) * B.head + j] = vec[c * B.words + j];
  }
  if (tid < group && first + tid < end) a.cands[first - a.at + tid] = cand[tid];
}

// The features of the candidates that score_block_kernel has been through, from their
// vectors: 32 candidates a block, a lane each, the features divided among the warps.  On its
// own because that kernel's blocks are small (few rows wait at each barrier for the one with
// most entries), where these steps would run on 8 of 32 lanes.
constexpr int kFeatureGroup = 32;
constexpr size_t kFeatureSmem = 128 * 1024;

inline size_t feature_smem_bytes(const BlockPlan& b) {
  return 4 * (size_t)kFeatureGroup * ((b.head + 2 * b.Fm) | 1);
}

__global__ void __launch_bounds__(128) feature_kernel(const __grid_constant__ QuantArgs qa,
                                                      const __grid_constant__ BlockPlan B) {
  const ScoreArgs& a = qa.s;
  extern __shared__ __align__(16) uint32_t feature_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t first = (int64_t)blockIdx.x * kFeatureGroup;  // of the launch's candidates
  const int here = (int)min((int64_t)kFeatureGroup, a.take - first);
  const int words = (B.head + 2 * B.Fm) | 1;
  const Ln ln{a.ln_tab, LnCoef()};
  for (int t = tid; t < here * B.head; t += 128) {
    const int c = t / B.head, j = t - c * B.head;
    feature_smem[c * words + j] = a.heads[(first + c) * B.head + j];
  }
  __syncthreads();
  if (lane >= here) return;
  const BlockCand k = a.cands[first + lane];
  if (k.q < 0) return;
  const SmVec s{feature_smem + lane * words};
  const int F = k.F, C = k.C;
  const int64_t n = a.n, q = k.q;
  float* o = a.o_feat + q;  // feature j at o[j * n]
  const int TMP = B.head + (warp >> 1) * B.Fm;  // (warps 0 and 2)
  if (warp == 0) {
    const float mean_corr = F > 0 ? __fdiv_rn(rust_sum(s, B.corr, F), (float)F) : 0.0f;
    o[0 * n] = a.c_score[q];
    o[1 * n] = mean_corr;
    o[2 * n] = median_of(s, B.corr, F, TMP);
    o[3 * n] = std_of(s, B.corr, F);
    o[4 * n] = correlation_safe(s, B.obs, B.fint, F);
    o[5 * n] = (float)F;
    o[6 * n] = (float)C;
    // count_values_above (src/utils/mod.rs:223-237), all in one pass
    int c95 = 0, c90 = 0, c80 = 0, c50 = 0, c0 = 0, t0 = 0, t50 = 0;
    int b0[4] = {0, 0, 0, 0}, b50[4] = {0, 0, 0, 0};
#pragma unroll 1
    for (int f = 0; f < F; ++f) {
      const float c = s.f(B.corr + f);
      const uint32_t flag = s.u(B.tn + f), band = flag >> kFlagBand;
      const bool top = (flag & kFlagTop) != 0u;
      c95 += c > 0.95f;
      c90 += c > 0.90f;
      c80 += c > 0.80f;
      c50 += c > 0.50f;
      c0 += c > 0.0f;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        b0[r] += band == (uint32_t)r && c > 0.0f;
        b50[r] += band == (uint32_t)r && c > 0.50f;
      }
      t0 += top && c > 0.0f;
      t50 += top && c > 0.50f;
    }
    o[7 * n] = (float)c95;
    o[8 * n] = (float)c90;
    o[9 * n] = (float)c80;
    o[10 * n] = (float)c50;
    o[11 * n] = (float)c0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      o[(12 + r) * n] = (float)b0[r];
      o[(16 + r) * n] = (float)b50[r];
    }
    o[39 * n] = (float)t0;
    o[40 * n] = (float)t50;
  } else if (warp == 1) {
    o[20 * n] = hyperscore_of(s, B, B.obs, false, F, ln);
    o[21 * n] = hyperscore_of(s, B, B.fint, false, F, ln);
    o[22 * n] = hyperscore_of(s, B, B.obs, true, F, ln);
    o[32 * n] = hyperscore_of(s, B, B.idf, false, F, ln);
  } else if (warp == 2) {
    o[25 * n] = (float)longest_series_of(s, B, F, 98, TMP);
    o[26 * n] = (float)longest_series_of(s, B, F, 121, TMP);
    float ib = 0.0f, iy = 0.0f, wmae_s = 0.0f, wmae_w = 0.0f;
#pragma unroll 1
    for (int f = 0; f < F; ++f) {
      const float v = s.f(B.obs + f);
      if (v > 0.0f) {
        const uint32_t type = s.u(B.tn + f) & 0xffu;
        if (type == 98) ib = __fadd_rn(ib, v);
        if (type == 121) iy = __fadd_rn(iy, v);
      }
      const float w = s.f(B.fint + f), e = s.f(B.fmz + f);
      if (w > 0.0f && e != 0.0f) {
        wmae_s = __fadd_rn(wmae_s, __fmul_rn(fabsf(e), w));
        wmae_w = __fadd_rn(wmae_w, w);
      }
    }
    o[28 * n] = wmae_w > 0.0f ? __fdiv_rn(wmae_s, wmae_w) : 0.0f;
    o[29 * n] = log10_rn(__fadd_rn(ib, 1e-8f));
    o[30 * n] = log10_rn(__fadd_rn(iy, 1e-8f));
  } else {
    const float med_sum = rust_sum(s, B.med, C), med_sum_f = rust_sum(s, B.medf, C);
    // calculate_fwhm_rt of the filtered median profile
    float fwhm = 0.0f;
    if (C > 0) {
      const int half = C / 2;
      const float cen = s.f(B.medf + half);
#pragma unroll 1
      for (int j = 0; j < half; ++j) {
        const float mean = __fdiv_rn(__fadd_rn(s.f(B.medf + half - j), s.f(B.medf + half + j)), 2.0f);
        if (mean <= __fdiv_rn(cen, 2.0f)) {
          fwhm = __fsub_rn(a.rt[k.cs + half + j], a.rt[k.cs + half - j]);
          break;
        }
      }
    }
    float idf_xic = -0.0f, idf_int = -0.0f;
#pragma unroll 1
    for (int f = 0; f < F; ++f) {
      idf_xic = __fadd_rn(idf_xic, __fmul_rn(s.f(B.idf + f), s.f(B.corr + f)));
      idf_int = __fadd_rn(idf_int, __fmul_rn(s.f(B.idf + f), s.f(B.obs + f)));
    }
    if (F == 0) idf_xic = idf_int = 0.0f;
    const float rt_obs = a.rt[a.c_center[q]];
    o[23 * n] = rt_obs;
    o[24 * n] = __fsub_rn(rt_obs, a.l_prt[k.prec]);
    o[27 * n] = (float)a.l_naa[k.prec];
    o[31 * n] = fwhm;
    o[33 * n] = idf_xic;
    o[34 * n] = log10_rn(__fadd_rn(idf_int, 1e-8f));
    o[35 * n] = med_sum;
    o[36 * n] = med_sum_f;
    o[37 * n] = (float)F;
    o[38 * n] = (float)k.nz;
    a.o_pidx[q] = a.c_pidx[q];
    a.o_rank[q] = a.c_rank[q];
    a.o_found[q] = 1;
  }
}
