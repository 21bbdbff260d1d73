// Pieces shared by the scan epilogues: per-gene / per-SNP window logic
// (include/eqtl/scan_common.hpp:58-69), the per-gene reduction state
// (n_tested, ACAT tan sum, best key) and candidate compaction.
#pragma once
#include "tdist.cuh"
#include "tile_gemm.cuh"

namespace eqtl {
namespace dev {

enum WinMode : int { kWinNone = 0, kWinExclude = 1, kWinInclude = 2 };

// high bit of a candidate's SNP field: its ACAT term is added on the host
constexpr uint32_t kCandDeferred = 0x80000000u;
constexpr uint32_t kCandTiny = 0x40000000u;  // deferred for 0 < |t| < tiny_t (kept SNP indices < 2^30)

struct GeneOut {
  double* acat_sum;            // [G] sum of tan((1/2 - p) pi)
  int* acat_used;              // [G]
  int* n_tested;               // [G]
  unsigned long long* best;    // [G] best_key (min)
  int2* cand;                  // (gene, kept snp | kCandDeferred) with |t| >= t_cand or a deferred ACAT term
  unsigned int* cand_count;
  unsigned int cand_cap;
};

struct Windows {
  int mode;
  const int32_t* gene_chrom;
  const int64_t* gene_lo;
  const int64_t* gene_hi;
  const int32_t* snp_chrom;  // padded as the blocks below
  const int64_t* snp_pos;
  // per block of 16 kept SNPs (b = s / 16, covering the padded tiles): the
  // block's chromosome (-1 where it mixes chromosomes or lies past the last
  // SNP) and its smallest and largest position
  const int32_t* blk_chrom;
  const int64_t* blk_lo;
  const int64_t* blk_hi;
};

// Per-thread (= per gene row) running state inside one tile.
struct GeneAcc {
  double acat = 0.0;
  int used = 0;
  int tested = 0;
  unsigned long long best = ~0ull;
  // no pair with u below this can be the gene's best (screen16_fast)
  float u_floor = 0.0f;
  int chrom = -1;
  int64_t lo = 0, hi = -1;

  __device__ __forceinline__ void reset() {
    acat = 0.0;
    used = 0;
    tested = 0;
    best = ~0ull;
  }
  // Starts from the best that any block has published for the gene (a stale
  // one is only a lower floor).
  __device__ __forceinline__ void load_best(const GeneOut& out, int g) {
    u_floor = __uint_as_float(~static_cast<uint32_t>(__ldcg(out.best + g) >> 32));
  }
  __device__ __forceinline__ void load_window(const Windows& w, int g) {
    if (w.mode != kWinNone) {
      chrom = w.gene_chrom[g];
      lo = w.gene_lo[g];
      hi = w.gene_hi[g];
    }
  }
  // true if no SNP of the 16-SNP block starting at s0 (a multiple of 16) can
  // lie in this gene's window: a gene without one, or a block on another
  // chromosome or wholly before or after it
  __device__ __forceinline__ bool chunk_clear(const Windows& w, int64_t s0) const {
    if (chrom < 0) return true;
    const int64_t b = s0 >> 4;
    const int32_t c = __ldg(w.blk_chrom + b);
    return c >= 0 && (c != chrom || __ldg(w.blk_hi + b) < lo || __ldg(w.blk_lo + b) > hi);
  }
  // true if every SNP of that block lies in this gene's window
  __device__ __forceinline__ bool chunk_inside(const Windows& w, int64_t s0) const {
    const int64_t b = s0 >> 4;
    return chrom >= 0 && __ldg(w.blk_chrom + b) == chrom && __ldg(w.blk_lo + b) >= lo && __ldg(w.blk_hi + b) <= hi;
  }
  // Bit j: SNP s0 + j of the block of 16 at s0 lies in this gene's window. The
  // positions come with eight 16-byte loads that do not wait for one another
  // (the arrays are padded to the block bounds' range); one at a time behind
  // the chromosome test, as the lanes' genes decide, they took thousands of
  // cycles a block.
  __device__ __forceinline__ uint32_t window_mask(const Windows& w, int64_t s0) const {
    const longlong2* p2 = reinterpret_cast<const longlong2*>(w.snp_pos + s0);
    const int4* c4 = reinterpret_cast<const int4*>(w.snp_chrom + s0);
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int4 c = __ldg(c4 + q);
      const longlong2 a = __ldg(p2 + 2 * q), b = __ldg(p2 + 2 * q + 1);
      m |= (c.x == chrom && a.x >= lo && a.x <= hi) ? 1u << (4 * q) : 0u;
      m |= (c.y == chrom && a.y >= lo && a.y <= hi) ? 2u << (4 * q) : 0u;
      m |= (c.z == chrom && b.x >= lo && b.x <= hi) ? 4u << (4 * q) : 0u;
      m |= (c.w == chrom && b.y >= lo && b.y <= hi) ? 8u << (4 * q) : 0u;
    }
    return chrom >= 0 ? m : 0u;
  }
  // Adds a chunk of 16 pairs: its counts, the FP32 sum of its ACAT terms (the
  // error is ~1e-6 of the chunk's largest term, below the screen's own) and its
  // best pair (score < 0: none). A chunk's best is its first pair with the
  // largest score; the 64-bit key breaks ties by SNP index across chunks.
  __device__ __forceinline__ void add_chunk(int n_tested, int n_used, float sum, float score, uint32_t snp) {
    tested += n_tested;
    used += n_used;
    acat += static_cast<double>(sum);
    if (score >= 0.0f) {
      const unsigned long long k = best_key(score, snp);
      best = k < best ? k : best;
    }
  }
  __device__ __forceinline__ void flush(const GeneOut& out, int g) const {
    if (tested == 0) return;
    atomicAdd(out.acat_sum + g, acat);
    atomicAdd(out.acat_used + g, used);
    atomicAdd(out.n_tested + g, tested);
    atomicMin(out.best + g, best);
  }
};

// 16 per-SNP flag bytes starting at a multiple of 16 (arrays padded to 16).
__device__ __forceinline__ void load_flags16(const uint8_t* p, uint32_t (&w)[4]) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  w[0] = v.x;
  w[1] = v.y;
  w[2] = v.z;
  w[3] = v.w;
}
__device__ __forceinline__ bool flag16(const uint32_t (&w)[4], int j) { return (w[j >> 2] >> (8 * (j & 3))) & 0xFFu; }

// 16 floats starting at a multiple of 16 of an array padded past its last
// tile (four 16-byte loads).
__device__ __forceinline__ void load16(const float* p, float (&v)[16]) {
  const float4* p4 = reinterpret_cast<const float4*>(p);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 x = __ldg(p4 + q);
    v[4 * q] = x.x;
    v[4 * q + 1] = x.y;
    v[4 * q + 2] = x.z;
    v[4 * q + 3] = x.w;
  }
}

__device__ __forceinline__ void emit_candidate(const GeneOut& out, int g, int64_t s, bool deferred, bool tiny) {
  const unsigned int idx = atomicAdd(out.cand_count, 1u);
  if (idx < out.cand_cap)
    out.cand[idx] = make_int2(g, static_cast<int>(static_cast<uint32_t>(s) | (deferred ? kCandDeferred : 0u) |
                                                  (tiny ? kCandTiny : 0u)));
}

// What a chunk of 16 pairs adds to its gene (GeneAcc::add_chunk).
struct ChunkSums {
  float sum, score;
  int tested, used, j;
};

// The ACAT screen of one gene's 16 pairs s0 .. s0 + 15, the general form: u =
// t^2 of each (0 outside the scan and where p = 1), the bits of `valid` mark
// the pairs that are tested. With u_tiny > 0:
//   tiny      0 < u < u_tiny         deferred   tiny or u >= u_defer
//   ACAT      u_tiny <= u < u_defer  candidate  u >= min(u_cand, u_defer) or tiny
// Candidates are emitted as they are found. Out of line: it serves the chunks
// that screen16_fast leaves, and inlined it cost the epilogues the registers that
// their common path needs. Unrolled, since a tile's accumulators are released by
// its slowest warp, so the latency of the rare chunk counts (a rolled loop here
// took the LM scan from 64 to 72 ms). tab: screen_tables (0: the tables in
// global memory).
__device__ __noinline__ inline ChunkSums screen16_general(const TTable& tt, uint32_t tab, const float* u,
                                                          uint32_t valid, float u_cand, const GeneOut& out, int gene,
                                                          int64_t s0) {
  ChunkSums r{0.0f, -1.0f, __popc(valid), 0, 0};
  const float uc = fminf(u_cand, tt.u_defer);
  if (tab) {
    const float u_tiny = tt.u_tiny, u_defer = tt.u_defer;
    float uv[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) uv[j] = u[j];
    auto screen = [&](auto&& term_of) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float uj = uv[j];
        const bool v = (valid >> j) & 1u;
        const float term = term_of(uj);
        const bool lo = uj < u_tiny;
        const bool use = v && !lo && uj < u_defer;
        r.sum += use ? term : 0.0f;
        r.used += use ? 1 : 0;
        const float key = v ? uj : -1.0f;
        r.j = key > r.score ? j : r.j;
        r.score = fmaxf(key, r.score);
      }
    };
    if (tt.lt_u) screen([&](float uj) { return cubic_term(uj, tt, tab); });
    else screen([&](float uj) { return node_term(uj, tt, tab); });
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const bool lo = uv[j] < u_tiny;
      if (((valid >> j) & 1u) && (uv[j] >= uc || (lo && uv[j] > 0.0f)))
        emit_candidate(out, gene, s0 + j, lo || uv[j] >= u_defer, lo);
    }
    return r;
  }
  for (int j = 0; j < 16; ++j) {
    if (!((valid >> j) & 1u)) continue;
    const float uj = u[j];
    const ScreenOut o = acat_screen_u(uj, tt);
    if (o.use_acat) {
      r.sum += o.term;
      ++r.used;
    }
    if (o.key > r.score) {
      r.score = o.key;
      r.j = j;
    }
    if (uj >= uc || o.deferred) emit_candidate(out, gene, s0 + j, o.deferred, o.tiny);
  }
  return r;
}

// Sum of the terms of 16 pairs from the node tables (long tails, df below about 29).
// Out of line for its registers, as screen16_general. Scan of 8e8 tests at n = 24
// (200,000 SNPs, 4,000 genes): LM 5.3 ms, LMM (p = 1) 6.8, p = 3 10.6; with these
// chunks left to the general form 6.3, 8.0, 12.8, and with the tables in global
// memory besides 9.9, 11.8, 16.4.
__device__ __noinline__ inline float node_sum16(const TTable& tt, uint32_t tab, const float* u) {
  float sum = 0.0f;
#pragma unroll
  for (int j = 0; j < 16; ++j) sum += node_term(u[j], tt, tab);
  return sum;
}

// The same screen of 16 pairs that are all tested (no SNP of the block gated,
// none out of scope), for tables in shared memory: u_of(j) gives u = t^2 of
// pair j, computed without the guards of the general form. Returns false,
// with acc untouched, unless every u lies in [u_tiny, u_defer): a pair near 0 or
// deferred, a NaN, and whatever the guards would have caught (a vanishing
// denominator gives u < 0, NaN or inf) are left to the general form. u_of is
// called twice for the pairs of a chunk with a candidate or with what may be the
// gene's best.
//
// The scans' epilogues are bound by instruction issue, and ~99 % of the
// 16-pair chunks hold nothing but ordinary pairs, so the per-pair flags, the
// candidate test, the counts and the best-SNP index leave the loop: the counts
// are 16, the extremes decide for the chunk, and the index is looked for only
// where the chunk's largest u reaches the best published for the gene. The
// terms and the order of their sum are those of the general form.
template <class U>
__device__ __forceinline__ bool screen16_fast(const TTable& tt, uint32_t tab, float u_cand, U&& u_of,
                                              const GeneOut& out, int gene, int64_t s0, GeneAcc& acc) {
  float sum = 0.0f, umin = INFINITY, umax = 0.0f;
  if (tt.lt_u) {  // uniform across the launch
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      const float ua = u_of(j), ub = u_of(j + 1);
      umin = min3(umin, ua, ub);
      umax = max3_nan(umax, ua, ub);
      sum += cubic_term(ua, tt, tab);
      sum += cubic_term(ub, tt, tab);
    }
  } else {
    float u[16];
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      u[j] = u_of(j);
      u[j + 1] = u_of(j + 1);
      umin = min3(umin, u[j], u[j + 1]);
      umax = max3_nan(umax, u[j], u[j + 1]);
    }
    sum = node_sum16(tt, tab, u);
  }
  if (!(umin >= tt.u_tiny && umax < tt.u_defer)) return false;
  float score = -1.0f;
  uint32_t bj = 0;
  if (umax >= fminf(acc.u_floor, u_cand)) {
#pragma unroll
    for (int j = 15; j >= 0; --j) {
      const float u = u_of(j);
      bj = u == umax ? j : bj;  // the first pair with the largest u
      if (u >= u_cand) emit_candidate(out, gene, s0 + j, false, false);
    }
    score = umax;
    acc.u_floor = fmaxf(acc.u_floor, umax);
  }
  acc.add_chunk(16, 16, sum, score, static_cast<uint32_t>(s0) + bj);
  return true;
}

// Whether all 16 flag bytes (0 or 1) are set.
__device__ __forceinline__ bool all_flags16(const uint32_t (&w)[4]) {
  return (w[0] & w[1] & w[2] & w[3]) == 0x01010101u;
}

// Scope of the block of 16 SNPs at s0 for the genes of the warp's active
// lanes (the vote keeps the warp on one path): kAll (a gw scan; a trans scan on
// a block clear of all their windows; a cis scan on a block inside all of them),
// kNone (the reverse) or kMixed (decided per pair).
enum ChunkScope : int { kScopeAll, kScopeNone, kScopeMixed };
__device__ __forceinline__ ChunkScope chunk_scope(const Windows& w, const GeneAcc& acc, int64_t s0) {
  if (w.mode == kWinNone) return kScopeAll;
  const uint32_t m = __activemask();
  const bool clear = __all_sync(m, acc.chunk_clear(w, s0));
  if (clear) return w.mode == kWinExclude ? kScopeAll : kScopeNone;
  const bool inside = __all_sync(m, acc.chunk_inside(w, s0));
  if (inside) return w.mode == kWinExclude ? kScopeNone : kScopeAll;
  return kScopeMixed;
}

// One chunk of 16 pairs through the two forms. ok: every SNP of the chunk is
// tested and the fast form's denominators are sound; tab: screen_tables of the
// tables in shared memory (0: none); u_fast(j): u without guards; u_gen(j, valid)
// sets whether pair j is tested (its scope aside) and gives u with guards, never
// NaN.
template <class UF, class UG>
__device__ __forceinline__ void screen_chunk(const TTable& tt, uint32_t tab, float u_cand, const Windows& win,
                                             const GeneOut& out, int gene, int64_t s0, bool ok, UF&& u_fast,
                                             UG&& u_gen, GeneAcc& acc) {
  const ChunkScope sc = chunk_scope(win, acc, s0);
  if (sc == kScopeNone) return;
  if (ok && sc == kScopeAll && tab && screen16_fast(tt, tab, u_cand, u_fast, out, gene, s0, acc))
    return;
  float u[16];
  uint32_t valid = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    bool v = true;
    u[j] = u_gen(j, v);
    valid |= v ? 1u << j : 0u;
  }
  if (sc == kScopeMixed) {
    const uint32_t in = acc.window_mask(win, s0);
    valid &= win.mode == kWinExclude ? ~in : in;
  }
  const ChunkSums r = screen16_general(tt, tab, u, valid, u_cand, out, gene, s0);
  acc.add_chunk(r.tested, r.used, r.sum, r.score, static_cast<uint32_t>(s0 + r.j));
}

}  // namespace dev
}  // namespace eqtl
