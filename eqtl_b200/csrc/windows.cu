// The scans' windows: their upload with the bounds of every 16-SNP block, the order
// of the genes, and the banded tile list of a cis scan.
//
// The block bounds and the tile list are made on the device from the uploaded
// windows and positions; each kernel is bound by its launch. On the host the SNPs'
// chromosome blocks, the block bounds and the genes' binary searches took a quarter
// of a cis LM call over 20,000 SNPs and 1,000 genes (1.03 -> 0.89 ms) and a third of
// one over 45,000 SNPs and 32,000 permuted columns (5.0 -> 3.5 ms).
#include <algorithm>
#include <vector>

#include "compact.cuh"
#include "scan_host.hpp"

namespace eqtl {
namespace dev {

// Bounds of 16-SNP blocks: the SNPs' chromosome (-1: several), least and greatest
// position; blocks past the SNPs get an empty range.
__global__ void win_blocks_kernel(const int32_t* __restrict__ chrom, const int64_t* __restrict__ pos, int64_t m,
                                  int64_t n_blocks, int32_t* __restrict__ bc, int64_t* __restrict__ blo,
                                  int64_t* __restrict__ bhi) {
  const int64_t b = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (b >= n_blocks) return;
  int32_t c = -1;
  int64_t lo = 0, hi = -1;
  const int64_t s0 = b * 16, s1 = min(m, s0 + 16);
  for (int64_t s = s0; s < s1; ++s) {
    const int32_t cs = chrom[s];
    const int64_t p = pos[s];
    c = s == s0 || cs == c ? cs : -1;
    lo = s == s0 || p < lo ? p : lo;
    hi = s == s0 || p > hi ? p : hi;
  }
  bc[b] = c;
  blo[b] = lo;
  bhi[b] = hi;
}

// First SNP of every run of one chromosome.
struct ChromRuns {
  const int32_t* chrom;
  int64_t m;
  int* start;
  __device__ int64_t size() const { return m; }
  __device__ uint64_t test(int64_t k) const { return k == 0 || chrom[k] != chrom[k - 1] ? 1 : 0; }
  __device__ void emit(int64_t k, uint64_t, uint64_t at) const { start[at] = static_cast<int>(k); }
};
// Whether the positions of some run decrease.
__global__ void win_sorted_kernel(const int32_t* __restrict__ chrom, const int64_t* __restrict__ pos, int64_t m,
                                  unsigned* unsorted) {
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k > 0 && k < m && chrom[k] == chrom[k - 1] && pos[k] < pos[k - 1]) *unsorted = 1;
}

// The runs by chromosome: a table of chromosome << 32 | run with open addressing, at
// most half full. A genome has tens of runs, a draft assembly tens of thousands, SNPs
// in no order as many as SNPs.
constexpr unsigned long long kNoRun = ~0ull;
__host__ __device__ __forceinline__ uint32_t run_slots(uint32_t n_runs) {  // power of two in [2 n, 4 n]
  uint32_t s = 2;
  while (s < 2 * n_runs) s *= 2;
  return s;
}
__device__ __forceinline__ uint32_t run_slot(int32_t chrom, uint32_t slots) {
  const uint32_t h = static_cast<uint32_t>(chrom) * 0x9E3779B1u;
  return (h ^ (h >> 16)) & (slots - 1);
}

// Fills the table; a chromosome with two runs: the SNPs are not grouped. One block.
// Cis LM call of 20,000 genes over 200,000 SNPs: 3.1 ms on 16,000 chromosomes as on
// 100,000, against 14.1 with all runs compared with one another and searched in a row,
// and 23.5 on the whole masked grid.
__global__ void __launch_bounds__(1024)
    win_runs_kernel(const int32_t* __restrict__ chrom, const int* __restrict__ start,
                    const uint64_t* __restrict__ n_runs, unsigned long long* table, unsigned* unsorted) {
  __shared__ unsigned stop;
  const uint32_t n = static_cast<uint32_t>(*n_runs), slots = run_slots(n);
  if (threadIdx.x == 0) stop = *unsorted;
  __syncthreads();
  if (stop) return;
  for (uint32_t i = threadIdx.x; i < slots; i += blockDim.x) table[i] = kNoRun;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n && !*static_cast<volatile unsigned*>(&stop); i += blockDim.x) {
    const int32_t c = chrom[start[i]];
    const unsigned long long entry = static_cast<unsigned long long>(static_cast<uint32_t>(c)) << 32 | i;
    for (uint32_t h = run_slot(c, slots), k = 0; k < slots; h = (h + 1) & (slots - 1), ++k) {
      const unsigned long long old = atomicCAS(table + h, kNoRun, entry);
      if (old == kNoRun) break;
      if (static_cast<int32_t>(old >> 32) == c) {
        stop = 1;
        *unsorted = 1;
        break;
      }
    }
  }
}
// The run of a chromosome, or -1.
__device__ __forceinline__ int64_t find_run(const unsigned long long* __restrict__ table, uint32_t slots,
                                            int32_t chrom) {
  for (uint32_t h = run_slot(chrom, slots), k = 0; k < slots; h = (h + 1) & (slots - 1), ++k) {
    const unsigned long long e = table[h];
    if (e == kNoRun) return -1;
    if (static_cast<int32_t>(e >> 32) == chrom) return static_cast<int64_t>(e & 0xFFFFFFFFu);
  }
  return -1;
}

// Marks the tiles (128 operand rows, NT SNPs) that hold some gene's window.
__global__ void win_mark_kernel(Windows w, int G, int64_t m, const int* __restrict__ gene_row,
                                const int* __restrict__ start, const uint64_t* __restrict__ n_runs,
                                const unsigned long long* __restrict__ table, const unsigned* __restrict__ unsorted,
                                int NT, int64_t tiles_b,
                                uint8_t* __restrict__ mark) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= G || *unsorted) return;
  const int32_t c = w.gene_chrom[g];
  if (c < 0) return;
  const int64_t n = static_cast<int64_t>(*n_runs);
  const int64_t run = find_run(table, run_slots(static_cast<uint32_t>(n)), c);
  if (run < 0) return;
  const int64_t beg = start[run], end = run + 1 < n ? start[run + 1] : m;
  auto first = [&](int64_t bound) {  // first SNP of the run at `bound` or after it
    int64_t lo = beg, hi = end;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (w.snp_pos[mid] < bound) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  const int64_t glo = w.gene_lo[g], ghi = w.gene_hi[g];
  const int64_t k_lo = first(glo), k_hi = ghi == INT64_MAX ? end : first(ghi + 1);  // k_hi exclusive
  if (k_hi <= k_lo) return;
  const int r = gene_row ? gene_row[g] : g;
  uint8_t* row = mark + static_cast<int64_t>(r / kTileM) * tiles_b;
  for (int64_t tb = k_lo / NT; tb <= (k_hi - 1) / NT; ++tb) row[tb] = 1;
}

struct MarkedTiles {
  const uint8_t* mark;
  int64_t n, tiles_b;
  int2* list;
  __device__ int64_t size() const { return n; }
  __device__ uint64_t test(int64_t i) const { return mark[i]; }
  __device__ void emit(int64_t i, uint64_t, uint64_t at) const {
    list[at] = make_int2(static_cast<int>(i / tiles_b), static_cast<int>(i % tiles_b));
  }
};

}  // namespace dev

using namespace dev;

dev::Windows upload_windows(eqtl_ctx* ctx, const eqtl_scan_params* prm, int64_t m, int mode) {
  dev::Windows w{};
  w.mode = dev::kWinNone;
  if (mode == dev::kWinNone || !prm->gene_chrom || !prm->gene_lo || !prm->gene_hi || !prm->snp_chrom ||
      !prm->snp_pos)
    return w;
  Workspace& ws = ctx->ws;
  ws.win_gc.upload(prm->gene_chrom, prm->n_genes, ctx->stream);
  ws.win_glo.upload(prm->gene_lo, prm->n_genes, ctx->stream);
  ws.win_ghi.upload(prm->gene_hi, prm->n_genes, ctx->stream);
  // 16-SNP blocks, up to one 256-SNP tile past the last padded tile; the
  // padding's values are not used (its SNPs are not tested)
  const int64_t nb = ((m + 255) / 256 + 1) * 16;
  ws.win_sc.alloc(static_cast<size_t>(nb * 16));
  ws.win_sp.alloc(static_cast<size_t>(nb * 16));
  ws.win_sc.upload(prm->snp_chrom, m, ctx->stream);
  ws.win_sp.upload(prm->snp_pos, m, ctx->stream);
  w.mode = mode;
  w.gene_chrom = ws.win_gc.p;
  w.gene_lo = ws.win_glo.p;
  w.gene_hi = ws.win_ghi.p;
  w.snp_chrom = ws.win_sc.p;
  w.snp_pos = ws.win_sp.p;
  ws.win_bc.alloc(static_cast<size_t>(nb));
  ws.win_blo.alloc(static_cast<size_t>(nb));
  ws.win_bhi.alloc(static_cast<size_t>(nb));
  ++ctx->launches;
  win_blocks_kernel<<<blocks(nb, 128), 128, 0, ctx->stream>>>(ws.win_sc.p, ws.win_sp.p, m, nb, ws.win_bc.p,
                                                              ws.win_blo.p, ws.win_bhi.p);
  EQTL_CUDA(cudaGetLastError());
  w.blk_chrom = ws.win_bc.p;
  w.blk_lo = ws.win_blo.p;
  w.blk_hi = ws.win_bhi.p;
  return w;
}

// Scans with windows (trans, cis) lay their genes out by window position, so
// that the 32 genes of a warp and the 128 of a tile have windows close together:
// a warp's 16-SNP blocks are then mostly in or out for all of its genes
// (chunk_scope), and a cis tile's band covers few SNP tiles. In the caller's
// order the windows of 32 genes scattered over the genome make over a quarter of
// the blocks mixed, and the bands of 128 cover nearly every SNP. Consecutive
// genes with the same window (permuted columns) stay together. Scans of genes in
// random order, before and after: cis LMM (p = 16, 500 genes, 45,000 SNPs) 2.07 ->
// 0.74 ms, cis LM (1,000 genes, 20,000 SNPs) 0.156 -> 0.093 ms, trans LM on dosages
// (1.8e8 tests) 1.13 -> 0.79 ms. The order changes no pair's arithmetic.
GeneOrder gene_order(eqtl_ctx* ctx, const eqtl_scan_params* prm) {
  GeneOrder go;
  const int G = prm->n_genes;
  if (prm->exclude_cis == 0 || !prm->gene_chrom || !prm->gene_lo || !prm->gene_hi || !prm->snp_chrom ||
      !prm->snp_pos)
    return go;
  struct Run {
    uint32_t chrom;  // genes without a location (-1) last
    int64_t lo;
    int first, count;
  };
  std::vector<Run> runs;
  for (int g = 0; g < G; ++g) {
    const uint32_t c = static_cast<uint32_t>(prm->gene_chrom[g]);
    if (g > 0 && prm->gene_chrom[g] == prm->gene_chrom[g - 1] && prm->gene_lo[g] == prm->gene_lo[g - 1] &&
        prm->gene_hi[g] == prm->gene_hi[g - 1])
      ++runs.back().count;
    else
      runs.push_back({c, prm->gene_lo[g], g, 1});
  }
  auto before = [](const Run& a, const Run& b) {
    if (a.chrom != b.chrom) return a.chrom < b.chrom;
    if (a.lo != b.lo) return a.lo < b.lo;
    return a.first < b.first;
  };
  if (std::is_sorted(runs.begin(), runs.end(), before)) return go;
  std::sort(runs.begin(), runs.end(), before);
  Workspace& ws = ctx->ws;
  std::vector<int> gene(static_cast<size_t>(G)), row(static_cast<size_t>(G));
  int r = 0;
  for (const Run& run : runs)
    for (int k = 0; k < run.count; ++k, ++r) {
      gene[static_cast<size_t>(r)] = run.first + k;
      row[static_cast<size_t>(run.first + k)] = r;
    }
  ws.row_gene.upload(gene.data(), gene.size(), ctx->stream);
  ws.gene_row.upload(row.data(), row.size(), ctx->stream);
  go.row = ws.gene_row.p;
  go.gene = ws.row_gene.p;
  return go;
}

// Banded tile list of a cis scan (scope 2): for every tile of 128 operand rows, the
// SNP tiles of NT kept SNPs that hold some gene's window. Needs the kept
// SNPs grouped by chromosome in position order (as in a sorted .bim); returns
// false otherwise, and the caller runs the full grid masked to the windows.
bool cis_tile_list(eqtl_ctx* ctx, const dev::Windows& w, int G, const GeneOrder& go, int64_t m, int NT,
                   const int2*& list, int& n_list) {
  list = nullptr;
  n_list = 0;
  if (w.mode != dev::kWinInclude || m == 0) return false;
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  const int tiles_a = (G + dev::kTileM - 1) / dev::kTileM;
  const int64_t tiles_b = (m + NT - 1) / NT, n_tiles = tiles_a * tiles_b;
  ws.win_count.alloc(3);  // runs, listed tiles, unsorted
  ws.win_count.zero(st);
  uint64_t* count = ws.win_count.p;
  unsigned* unsorted = reinterpret_cast<unsigned*>(count + 2);
  ws.win_runs.alloc(static_cast<size_t>(m));
  ws.win_mark.alloc(static_cast<size_t>(n_tiles));
  ws.win_mark.zero(st);
  ws.tile_list.alloc(static_cast<size_t>(n_tiles));
  ctx->launches += 3;
  win_sorted_kernel<<<blocks(m, 256), 256, 0, st>>>(w.snp_chrom, w.snp_pos, m, unsorted);
  compact(ctx, ChromRuns{w.snp_chrom, m, ws.win_runs.p}, m, count);
  ws.win_table.alloc(run_slots(static_cast<uint32_t>(m)));
  win_runs_kernel<<<1, 1024, 0, st>>>(w.snp_chrom, ws.win_runs.p, count, ws.win_table.p, unsorted);
  win_mark_kernel<<<blocks(G, 128), 128, 0, st>>>(w, G, m, go.row, ws.win_runs.p, count, ws.win_table.p, unsorted, NT,
                                                  tiles_b, ws.win_mark.p);
  EQTL_CUDA(cudaGetLastError());
  compact(ctx, MarkedTiles{ws.win_mark.p, n_tiles, tiles_b, ws.tile_list.p}, n_tiles, count + 1);
  uint64_t c[3];
  ws.win_count.download(c, 3, st);
  EQTL_CUDA(cudaStreamSynchronize(st));
  if (c[2]) return false;
  n_list = static_cast<int>(c[1]);
  list = ws.tile_list.p;
  return true;
}

}  // namespace eqtl
