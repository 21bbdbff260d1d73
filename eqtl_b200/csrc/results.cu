// From a scan's candidate buffer to its results, on the device: the sorted list
// of pairs to refine, and after the refinement each gene's best pair, the pairs
// below the threshold in (snp, gene) order and the deferred ACAT p-values.
//
// The lists are sorted by 64-bit keys, either by one block (up to 4096 keys) or
// by a radix sort whose every pass is a histogram, a prefix sum and a stable
// scatter; the host sees only the final lists. Each kernel moves a few MB and is
// bound by its launch. The full LM scan (418,000 pairs refined, 216,000 kept,
// 213,000 deferred) spent 38 ms of 117 in host sorts, pageable copies of every
// refined pair and their page faults; now 10, of which the host's long-double terms
// are 5.
#include "block_sort.cuh"
#include "compact.cuh"
#include "host_par.hpp"
#include "scan_host.hpp"

namespace eqtl {
namespace dev {

constexpr int kRadixTile = 4096;  // keys per block and pass: 256 threads x 16

// hist[digit][block] of the digit at `shift`
__global__ void __launch_bounds__(256) radix_count_kernel(const uint64_t* __restrict__ key,
                                                          const unsigned* __restrict__ n_keys, int shift,
                                                          unsigned* __restrict__ hist) {
  __shared__ unsigned h[256];
  const int64_t n = *n_keys, base = static_cast<int64_t>(blockIdx.x) * kRadixTile;
  h[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll 4
  for (int r = 0; r < kRadixTile / 256; ++r) {
    const int64_t i = base + r * 256 + threadIdx.x;
    if (i < n) atomicAdd(&h[(key[i] >> shift) & 255], 1u);
  }
  __syncthreads();
  hist[static_cast<int64_t>(threadIdx.x) * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter by the digit at `shift`; hist: prefix sums of radix_count_kernel's.
__global__ void __launch_bounds__(256) radix_scatter_kernel(const uint64_t* __restrict__ key,
                                                            const unsigned* __restrict__ n_keys, int shift,
                                                            const unsigned* __restrict__ hist,
                                                            uint64_t* __restrict__ out) {
  constexpr int R = kRadixTile / 256;
  __shared__ unsigned at[8][256];  // per warp: keys of a digit so far, then their place
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t n = *n_keys;
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kRadixTile + w * (32 * R);  // the warp's keys, in order
#pragma unroll
  for (int i = 0; i < 8; ++i) at[i][threadIdx.x] = 0;
  __syncthreads();
  uint64_t k[R];
  unsigned rank[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t i = base + r * 32 + lane;
    const bool valid = i < n;
    k[r] = valid ? key[i] : 0;
    const int d = valid ? static_cast<int>((k[r] >> shift) & 255) : 256;
    const unsigned same = __match_any_sync(0xffffffffu, d);
    const unsigned before = __popc(same & ((1u << lane) - 1));
    const unsigned c = valid ? at[w][d] : 0;
    __syncwarp();
    if (valid && before == 0) at[w][d] = c + __popc(same);
    __syncwarp();
    rank[r] = c + before;
  }
  __syncthreads();
  unsigned s = hist[static_cast<int64_t>(threadIdx.x) * gridDim.x + blockIdx.x];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const unsigned c = at[i][threadIdx.x];
    at[i][threadIdx.x] = s;
    s += c;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (base + r * 32 + lane < n) out[at[w][(k[r] >> shift) & 255] + rank[r]] = k[r];
}

// ------------------------------------------------ the pairs to refine
// Key of a pair: (gene, snp, 0 if its ACAT term is deferred else 1), so that a
// pair listed twice (a candidate that is its gene's best) comes first as deferred.
__device__ __forceinline__ uint64_t pair_key(int gene, uint32_t snp, int snp_bits, bool deferred) {
  return (((static_cast<uint64_t>(static_cast<uint32_t>(gene)) << snp_bits) | snp) << 1) | (deferred ? 0 : 1);
}

struct CollectArgs {
  const int2* cand;
  int64_t n_cand;
  const int* tested;
  const unsigned long long* best;
  int G, snp_bits;
  bool split_tiny;  // pairs deferred only for their small |t| go to `tiny`
  int2* tiny;
  unsigned* n_tiny;
  // item i < n_cand + G: its key, or ~0 (none); tiny pairs are appended here
  __device__ __forceinline__ uint64_t key(int64_t i) const {
    if (i < n_cand) {
      const int2 q = cand[i];
      const uint32_t s = static_cast<uint32_t>(q.y), snp = s & ~(kCandDeferred | kCandTiny);
      if (split_tiny && (s & kCandTiny)) {
        tiny[atomicAdd(n_tiny, 1u)] = make_int2(q.x, static_cast<int>(snp));
        return ~0ull;
      }
      return pair_key(q.x, snp, snp_bits, (s & kCandDeferred) != 0);
    }
    const int g = static_cast<int>(i - n_cand);
    if (tested[g] <= 0 || best[g] == ~0ull) return ~0ull;
    return pair_key(g, static_cast<uint32_t>(best[g]), snp_bits, false);
  }
};

__global__ void __launch_bounds__(256) collect_keys_kernel(CollectArgs a, uint64_t* key, unsigned* n_key) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t k = i < a.n_cand + a.G ? a.key(i) : ~0ull;
  const unsigned has = __ballot_sync(0xffffffffu, k != ~0ull);
  const int lane = threadIdx.x & 31;
  unsigned at = 0;
  if (lane == 0 && has) at = atomicAdd(n_key, __popc(has));
  at = __shfl_sync(0xffffffffu, at, 0) + __popc(has & ((1u << lane) - 1));
  if (k != ~0ull) key[at] = k;
}

// sorted keys -> distinct pairs and the places of the deferred ones among them
struct UniquePairs {
  const uint64_t* key;
  const unsigned* n;
  int snp_bits;
  int2* pairs;
  int* deferred;
  __device__ int64_t size() const { return *n; }
  __device__ uint64_t test(int64_t i) const {
    const uint64_t k = key[i];
    if (i > 0 && (key[i - 1] >> 1) == (k >> 1)) return 0;
    return (k & 1) ? 1ull : (1ull << 32) | 1ull;
  }
  __device__ void emit(int64_t i, uint64_t t, uint64_t at) const {
    const uint64_t k = key[i] >> 1;
    const unsigned p = static_cast<unsigned>(at);
    pairs[p] = make_int2(static_cast<int>(k >> snp_bits), static_cast<int>(k & ((1ull << snp_bits) - 1)));
    if (t >> 32) deferred[at >> 32] = static_cast<int>(p);
  }
};

// the same in one block, for n_cand + G <= 4 T
template <int T>
__global__ void __launch_bounds__(T) collect_block_kernel(CollectArgs a, int2* pairs, int* deferred,
                                                          uint64_t* total) {
  extern __shared__ uint64_t key[];  // 4 T
  __shared__ uint64_t sm[33];
  uint64_t k[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t i = r * T + threadIdx.x;
    k[r] = i < a.n_cand + a.G ? a.key(i) : ~0ull;
  }
  block_sort_u64<T>(k, key);
  const unsigned n = 4 * T;
  const UniquePairs u{key, &n, a.snp_bits, pairs, deferred};
  uint64_t t[4], s = 0, all;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = 4 * threadIdx.x + r;
    t[r] = key[i] != ~0ull ? u.test(i) : 0;
    s += t[r];
  }
  uint64_t at = block_prefix(s, sm, all);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    if (t[r]) u.emit(4 * threadIdx.x + r, t[r], at);
    at += t[r];
  }
  if (threadIdx.x == 0) *total = all;
}

// ------------------------------------------------ distinct SNPs of the pairs
__global__ void mark_snps_kernel(const int2* __restrict__ pairs, int n, int* __restrict__ mark) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) mark[pairs[i].y] = 1;
}
struct MarkedSnps {
  int64_t m;
  int* mark;  // 1: listed; becomes the SNP's place
  int* snps;
  __device__ int64_t size() const { return m; }
  __device__ uint64_t test(int64_t i) const { return mark[i] != 0 ? 1 : 0; }
  __device__ void emit(int64_t i, uint64_t, uint64_t at) const {
    snps[at] = static_cast<int>(i);
    mark[i] = static_cast<int>(at);
  }
};
__global__ void snp_place_kernel(const int2* __restrict__ pairs, int n, const int* __restrict__ mark,
                                 int* __restrict__ col) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) col[i] = mark[pairs[i].y];
}

// ------------------------------------------------ after the refinement
// One warp per gene: the counts of the scan and the gene's best refined pair
// (smallest p, then lowest SNP; the gene's first pair where that one's p is NaN,
// as the sequential comparison leaves it).
__global__ void __launch_bounds__(256) gene_results_kernel(const double* __restrict__ acat,
                                                           const int* __restrict__ used,
                                                           const int* __restrict__ tested, int G,
                                                           const eqtl_pair* __restrict__ refined, int n,
                                                           eqtl_gene_result* __restrict__ out) {
  const int lane = threadIdx.x & 31, g = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (g >= G) return;
  auto lower = [&](int gene) {  // first refined pair of a gene >= `gene`
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (refined[mid].gene < gene) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  const int lo = lower(g), hi = lower(g + 1);
  int bi = hi;
  double bp = 0.0;
  for (int i = lo + lane; i < hi; i += 32) {
    const double p = refined[i].p;
    if (!isnan(p) && (bi == hi || p < bp)) {
      bp = p;
      bi = i;
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const double p = __shfl_xor_sync(0xffffffffu, bp, o);
    const int i = __shfl_xor_sync(0xffffffffu, bi, o);
    if (i < hi && (bi == hi || p < bp || (p == bp && i < bi))) {
      bp = p;
      bi = i;
    }
  }
  if (lane != 0) return;
  if (lo < hi && isnan(refined[lo].p)) bi = lo;
  eqtl_gene_result r;
  r.n_tested = tested[g];
  r.acat_used = used[g];
  r.acat_tan_sum = acat[g];
  if (r.n_tested > 0 && lo < hi) {
    const eqtl_pair& q = refined[bi];
    r.best_snp = q.snp;
    r.best_p = q.p;
    r.best_beta = q.beta;
    r.best_se = q.se;
    r.best_t = q.t;
    r.best_r2 = q.r2;
  } else {
    r.best_snp = -1;
    r.best_p = 2.0;
    r.best_beta = r.best_se = r.best_t = r.best_r2 = 0.0;
  }
  out[g] = r;
}

// pairs with p <= pthr (key: snp, place) and candidates with finite p < perm_thr
struct SelectPairs {
  const eqtl_pair* refined;
  int64_t n;
  double pthr, perm_thr;
  uint64_t* key;
  int* cand;
  __device__ int64_t size() const { return n; }
  __device__ uint64_t test(int64_t i) const {
    const double p = refined[i].p;
    return (p <= pthr ? 1ull : 0ull) | (perm_thr > 0 && isfinite(p) && p < perm_thr ? 1ull << 32 : 0ull);
  }
  __device__ void emit(int64_t i, uint64_t t, uint64_t at) const {
    if (t & 1) key[static_cast<uint32_t>(at)] = (static_cast<uint64_t>(refined[i].snp) << 32) | static_cast<uint32_t>(i);
    if (t >> 32) cand[at >> 32] = static_cast<int>(i);
  }
};

// the selection and the pairs' sort in one block, for n <= 4 T
template <int T>
__global__ void __launch_bounds__(T) select_block_kernel(SelectPairs f, uint64_t* total) {
  extern __shared__ uint64_t key[];  // 4 T
  __shared__ uint64_t sm[33];
  uint64_t t[4], k[4], s = 0, all;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = 4 * threadIdx.x + r;
    t[r] = i < f.n ? f.test(i) : 0;
    k[r] = (t[r] & 1) ? (static_cast<uint64_t>(f.refined[i].snp) << 32) | static_cast<uint32_t>(i) : ~0ull;
    s += t[r];
  }
  uint64_t at = block_prefix(s, sm, all);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    if (t[r] >> 32) f.cand[at >> 32] = 4 * threadIdx.x + r;
    at += t[r];
  }
  block_sort_u64<T>(k, key);
  const int n = static_cast<int>(static_cast<uint32_t>(all));
  for (int i = threadIdx.x; i < n; i += T) f.key[i] = key[i];
  if (threadIdx.x == 0) *total = all;
}

// The candidates, listed by gene and SNP, into the order gene, p, SNP: a candidate's
// place among its gene's is the number of those before it. Quadratic in the gene's
// candidates, of which there are a few; a gene with more than kCandRankMax sets
// *big and the host sorts.
constexpr int kCandRankMax = 2048;
__global__ void cand_place_kernel(const eqtl_pair* __restrict__ refined, const int* __restrict__ cand, int n,
                                  int* __restrict__ placed, unsigned* big) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int ci = cand[i], g = refined[ci].gene;
  auto lower = [&](int gene) {
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (refined[cand[mid]].gene < gene) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  const int lo = lower(g), hi = lower(g + 1);
  if (hi - lo > kCandRankMax) {
    placed[i] = ci;
    *big = 1;
    return;
  }
  const double p = refined[ci].p;
  int rank = 0;
  for (int j = lo; j < hi; ++j) {
    const double q = refined[cand[j]].p;
    rank += q < p || (q == p && j < i) ? 1 : 0;
  }
  placed[lo + rank] = ci;
}

// out: rows [first, end) of the list of the n_pairs selected pairs in key order, then
// the candidates; a thread per 8-byte word
__global__ void gather_pairs_kernel(const eqtl_pair* __restrict__ refined, const uint64_t* __restrict__ key,
                                    int64_t n_pairs, const int* __restrict__ cand, int64_t first, int64_t end,
                                    eqtl_pair* __restrict__ out) {
  constexpr int W = sizeof(eqtl_pair) / 8;
  static_assert(sizeof(eqtl_pair) % 8 == 0 && alignof(eqtl_pair) == 8, "eqtl_pair words");
  const uint64_t* src = reinterpret_cast<const uint64_t*>(refined);
  uint64_t* dst = reinterpret_cast<uint64_t*>(out);
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < (end - first) * W;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t j = first + t / W;
    const int64_t i = j < n_pairs ? static_cast<int64_t>(static_cast<uint32_t>(key[j])) : cand[j - n_pairs];
    dst[t] = src[i * W + t % W];
  }
}

__global__ void deferred_p_kernel(const eqtl_pair* __restrict__ refined, const int* __restrict__ idx, int n,
                                  double* __restrict__ p, int* __restrict__ gene) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const eqtl_pair& q = refined[idx[i]];
  p[i] = q.p;
  gene[i] = q.gene;
}

}  // namespace dev

using namespace dev;

namespace {

int bits_of(int64_t values) {  // bits that hold 0 .. values - 1
  int b = 1;
  while (b < 62 && (int64_t(1) << b) < values) ++b;
  return b;
}

// Sorts *n_dev <= n_max keys by bits [lo, hi); a, b: buffers that hold n_max.
// Returns the one with the result.
uint64_t* radix_sort(eqtl_ctx* ctx, uint64_t* a, uint64_t* b, const unsigned* n_dev, int64_t n_max, int lo, int hi) {
  const unsigned nb = blocks(n_max, kRadixTile);
  DevBuf<unsigned>& hist = ctx->ws.res_hist;
  hist.alloc(static_cast<size_t>(nb) * 256);
  for (int shift = lo; shift < hi; shift += 8) {
    ctx->launches += 3;
    radix_count_kernel<<<nb, 256, 0, ctx->stream>>>(a, n_dev, shift, hist.p);
    prefix_kernel<unsigned><<<1, 1024, 0, ctx->stream>>>(hist.p, static_cast<int64_t>(nb) * 256, nullptr);
    radix_scatter_kernel<<<nb, 256, 0, ctx->stream>>>(a, n_dev, shift, hist.p, b);
    EQTL_CUDA(cudaGetLastError());
    std::swap(a, b);
  }
  return a;
}

// res_count: [0] keys, [1] tiny pairs, [2, 3] totals of a compaction
uint64_t* total_of(Workspace& ws) { return reinterpret_cast<uint64_t*>(ws.res_count.p + 2); }

// The reference's long-double ACAT terms of p[i] added to gene[i]
// (src/stats_extra.cpp:16-22; p <= 0 -> 1e-300), on every host thread, then summed
// in list order (the sums do not depend on the thread count).
template <class GeneOf>
void add_terms(eqtl_gene_result* genes, const std::vector<double>& ps, GeneOf gene_of) {
  const long double kPiL = 3.14159265358979323846L;
  std::vector<double> term(ps.size());
  std::vector<uint8_t> use(ps.size());
  parallel_for(ps.size(), [&](size_t i) {
    double p = ps[i];
    use[i] = !(!std::isfinite(p) || p < 0.0 || p >= 1.0 - 1e-12);  // AcatAcc::add guards
    if (!use[i]) return;
    if (p <= 0.0) p = 1e-300;
    term[i] = static_cast<double>(std::tan((0.5L - static_cast<long double>(p)) * kPiL));
  });
  for (size_t i = 0; i < ps.size(); ++i) {
    if (!use[i]) continue;
    eqtl_gene_result& g = genes[gene_of(i)];
    g.acat_tan_sum += term[i];
    ++g.acat_used;
  }
}

}  // namespace

void ScanOutputs::collect(bool split_tiny) {
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  const int64_t n_max = static_cast<int64_t>(n_cand) + G;
  ws.res_count.alloc(4);
  ws.res_count.zero(st);
  ws.ref_pairs.alloc(static_cast<size_t>(n_max));
  ws.res_deferred.alloc(static_cast<size_t>(n_max));
  if (split_tiny) ws.tiny_pairs.alloc(std::max<size_t>(n_cand, 1));
  const int snp_bits = bits_of(m);
  const CollectArgs a{cand.p, n_cand, tested.p, best.p, G, snp_bits, split_tiny, ws.tiny_pairs.p, ws.res_count.p + 1};
  // One block sorts what it holds (4096 keys in about 20 us); the radix sort
  // takes about 70 us however few the keys.
  if (n_max <= kBlockSortMax) {
    with_sort_block(static_cast<int>(n_max), [&](auto t) {
      constexpr int T = decltype(t)::value;
      ++ctx->launches;
      collect_block_kernel<T><<<1, T, 4 * T * sizeof(uint64_t), st>>>(a, ws.ref_pairs.p, ws.res_deferred.p,
                                                                      total_of(ws));
    });
    EQTL_CUDA(cudaGetLastError());
  } else {
    ws.res_key[0].alloc(static_cast<size_t>(n_max));
    ws.res_key[1].alloc(static_cast<size_t>(n_max));
    ++ctx->launches;
    collect_keys_kernel<<<blocks(n_max, 256), 256, 0, st>>>(a, ws.res_key[0].p, ws.res_count.p);
    EQTL_CUDA(cudaGetLastError());
    const uint64_t* key = radix_sort(ctx, ws.res_key[0].p, ws.res_key[1].p, ws.res_count.p, n_max, 0,
                                     bits_of(G) + snp_bits + 1);
    compact(ctx, UniquePairs{key, ws.res_count.p, snp_bits, ws.ref_pairs.p, ws.res_deferred.p}, n_max, total_of(ws));
  }
  unsigned c[4];
  ws.res_count.download(c, 4, st);
  EQTL_CUDA(cudaStreamSynchronize(st));
  n_tiny = static_cast<int>(c[1]);
  n_todo = static_cast<int>(c[2]);
  n_deferred = static_cast<int>(c[3]);
}

void ScanOutputs::finish(const eqtl_scan_params* prm, eqtl_gene_result* genes, PairList& pairs, PairList& cands) {
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  const int64_t n = n_todo;
  const eqtl_pair* refined = ws.refined.p;
  ws.res_genes.alloc(static_cast<size_t>(G));
  ++ctx->launches;
  gene_results_kernel<<<blocks(G, 8), 256, 0, st>>>(acat.p, used.p, tested.p, G, refined, n_todo, ws.res_genes.p);
  EQTL_CUDA(cudaGetLastError());
  std::vector<double> dp(static_cast<size_t>(n_deferred));
  std::vector<int> dg(static_cast<size_t>(n_deferred));
  if (n_deferred > 0) {
    ws.res_dp.alloc(dp.size());
    ws.res_dg.alloc(dg.size());
    ++ctx->launches;
    deferred_p_kernel<<<blocks(n_deferred, 256), 256, 0, st>>>(refined, ws.res_deferred.p, n_deferred, ws.res_dp.p,
                                                               ws.res_dg.p);
    EQTL_CUDA(cudaGetLastError());
  }
  uint64_t total = 0;
  const uint64_t* key = nullptr;
  if (n > 0) {
    ws.res_key[0].alloc(static_cast<size_t>(n));
    ws.res_cand.alloc(static_cast<size_t>(n));
    const SelectPairs f{refined, n, prm->pthr, prm->perm_thr, ws.res_key[0].p, ws.res_cand.p};
    key = ws.res_key[0].p;
    if (n <= kBlockSortMax) {
      with_sort_block(n_todo, [&](auto t) {
        constexpr int T = decltype(t)::value;
        ++ctx->launches;
        select_block_kernel<T><<<1, T, 4 * T * sizeof(uint64_t), st>>>(f, total_of(ws));
      });
      EQTL_CUDA(cudaGetLastError());
    } else {
      ws.res_key[1].alloc(static_cast<size_t>(n));
      compact(ctx, f, n, total_of(ws));
      // the low half of the total is the number of keys; in place order already,
      // so only the SNP has to be sorted
      key = radix_sort(ctx, ws.res_key[0].p, ws.res_key[1].p, ws.res_count.p + 2, n, 32, 32 + bits_of(m));
    }
    EQTL_CUDA(cudaMemcpyAsync(&total, total_of(ws), sizeof(total), cudaMemcpyDeviceToHost, st));
  }
  ws.res_genes.download(genes, static_cast<size_t>(G), st);
  ws.res_dp.download(dp.data(), dp.size(), st);
  ws.res_dg.download(dg.data(), dg.size(), st);
  EQTL_CUDA(cudaStreamSynchronize(st));
  const int64_t np = static_cast<int64_t>(total & 0xFFFFFFFFull), nc = static_cast<int64_t>(total >> 32);
  pairs.n = np;
  cands.n = nc;
  unsigned big = 0;  // some gene has too many candidates for cand_place_kernel
  if (np + nc > 0 && np <= pairs.cap && nc <= cands.cap) {
    if (nc > 0) {
      ws.res_placed.alloc(static_cast<size_t>(nc));
      EQTL_CUDA(cudaMemsetAsync(ws.res_count.p, 0, sizeof(unsigned), st));
      ++ctx->launches;
      cand_place_kernel<<<blocks(nc, 128), 128, 0, st>>>(refined, ws.res_cand.p, static_cast<int>(nc),
                                                         ws.res_placed.p, ws.res_count.p);
      ws.res_count.download(&big, 1, st);
    }
    // in pieces of 56 MB, however long the lists
    constexpr int64_t kPiece = 1 << 20;
    ws.res_pairs.alloc(static_cast<size_t>(std::min(kPiece, np + nc)));
    for (int64_t first = 0; first < np + nc; first += kPiece) {
      const int64_t end = std::min(np + nc, first + kPiece), split = std::min(std::max(first, np), end);
      ++ctx->launches;
      gather_pairs_kernel<<<static_cast<unsigned>(std::min<int64_t>(blocks((end - first) * 7, 256), 4096)), 256, 0, st>>>(
          refined, key, np, ws.res_placed.p, first, end, ws.res_pairs.p);
      EQTL_CUDA(cudaGetLastError());
      if (split > first) ws.res_pairs.download(pairs.p + first, static_cast<size_t>(split - first), st);
      if (end > split)
        EQTL_CUDA(cudaMemcpyAsync(cands.p + (split - np), ws.res_pairs.p + (split - first),
                                  sizeof(eqtl_pair) * (end - split), cudaMemcpyDeviceToHost, st));
    }
  }
  add_terms(genes, dp, [&](size_t i) { return dg[i]; });
  EQTL_CUDA(cudaStreamSynchronize(st));
  if (big)
    std::sort(cands.p, cands.p + nc, [](const eqtl_pair& a, const eqtl_pair& b) {
      if (a.gene != b.gene) return a.gene < b.gene;
      if (a.p != b.p) return a.p < b.p;
      return a.snp < b.snp;
    });
}

void add_acat_terms(eqtl_gene_result* genes, const std::vector<int2>& pairs, const std::vector<double>& p_pairs) {
  add_terms(genes, p_pairs, [&](size_t i) { return pairs[i].x; });
}

std::vector<int> distinct_snps(eqtl_ctx* ctx, const int2* pairs, int n_pairs, int64_t m) {
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  ws.ref_mark.alloc(static_cast<size_t>(m));
  ws.ref_mark.zero(st);
  ws.ref_snps.alloc(static_cast<size_t>(std::min<int64_t>(m, n_pairs)));
  ws.ref_col.alloc(static_cast<size_t>(n_pairs));
  ws.res_count.alloc(4);
  ctx->launches += 2;
  mark_snps_kernel<<<blocks(n_pairs, 256), 256, 0, st>>>(pairs, n_pairs, ws.ref_mark.p);
  compact(ctx, MarkedSnps{m, ws.ref_mark.p, ws.ref_snps.p}, m, total_of(ws));
  snp_place_kernel<<<blocks(n_pairs, 256), 256, 0, st>>>(pairs, n_pairs, ws.ref_mark.p, ws.ref_col.p);
  EQTL_CUDA(cudaGetLastError());
  uint64_t u = 0;
  EQTL_CUDA(cudaMemcpyAsync(&u, total_of(ws), sizeof(u), cudaMemcpyDeviceToHost, st));
  EQTL_CUDA(cudaStreamSynchronize(st));
  std::vector<int> snps(static_cast<size_t>(u));
  ws.ref_snps.download(snps.data(), snps.size(), st);
  EQTL_CUDA(cudaStreamSynchronize(st));
  return snps;
}

}  // namespace eqtl
