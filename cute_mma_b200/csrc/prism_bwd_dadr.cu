// Prism backward, input and rotation gradients: second-level reductions, launch plan and launcher of
// prism_bwd_dadr_kernel (prism_bwd_dadr_kernel.cuh; its instances live in prism_bwd_dadr_f16.cu and
// prism_bwd_dadr_bf16.cu).
#include "prism_bwd_dadr_kernel.cuh"

namespace prism {

// The sums over CTAs that end the dA+dR call, in one launch: blocks [0, dr_blocks) form dR, the next d_ib_blocks the
// internal-bias gradient, the rest dA (where the groups were split into parts).  A launch each cost 2 to 3 us of
// device time, and more of host time where that is what a short step waits for.
struct DadrReduce {
  const float* partial;      // dR: see DadrParams
  const float* partial_x;
  void* dR;
  long long lddr;
  const float* partial_ib;   // d_ib: see DadrExtra
  const float* partial_ib_x;
  uint16_t* d_ib;
  const float* partial_da;   // dA of the group parts [parts][M][K]
  uint16_t* dA;
  long long ldda;
  int M, G, rs, E, K, runs, n_ft, n_main, n_extra, steal, slots, parts;
  int k_blocks;              // blocks per row: 1024 columns each
  unsigned dr_blocks, ib_blocks;
  float scale, da_scale;
};

// Four neighbouring columns k.. of the sum over CTAs of `rows`-row buffers of K (main CTAs, in increasing order) and of 128
// columns (for every run, the slabs of the extra pair that helped the main pair (run, column of k)).
__device__ __forceinline__ float4 dadr_sum4(const DadrReduce& p, const float* main, const float* extra, long long rows,
                                            long long row, int k) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  auto add = [&](const float* src) {
    const float4 v = *reinterpret_cast<const float4*>(src);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  };
  for (int r = 0; r < 2 * p.runs; ++r) add(main + ((long long)r * rows + row) * p.K + k);
  if (p.steal > 0) {
    const int fx = k >> 7, kk = k & 127;
    for (int run = 0; run < p.runs; ++run) {
      const int m = run * p.n_ft + fx;
      const int e = ((m + 1) * p.n_extra - 1) / p.n_main;   // the extra pair that helps main pair m
      const int mi = m - e * p.n_main / p.n_extra;
      for (int rank = 0; rank < 2; ++rank) add(extra + (((long long)(e * 2 + rank) * p.slots + mi) * rows + row) * 128 + kk);
    }
  }
  return acc;
}

// dR[g*rs + i, k] = cast( scale * sum of the CTAs' partial sums ), in a fixed order.  For rs = 8 two neighbouring blocks
// share one 16-row group of the partial buffers: the block in the upper 8 columns of each 16-column pair sits in rows
// 8..15.  d_ib[g, k]: the CTAs' column sums of dS in the same order.  dA[m, k]: the parts' sums in part order.
// One row, 1024 columns and four columns per thread (K is a multiple of 8).
template <int DT, bool F32OUT>
__global__ void __launch_bounds__(256) dadr_reduce_kernel(const DadrReduce p) {
  unsigned blk = blockIdx.x;
  const bool is_dr = blk < p.dr_blocks;
  if (!is_dr) blk -= p.dr_blocks;
  const bool is_ib = !is_dr && blk < p.ib_blocks;
  if (!is_dr && !is_ib) blk -= p.ib_blocks;
  const int row = (int)(blk / p.k_blocks);
  const int k = (int)(blk - (unsigned)row * p.k_blocks) * 1024 + threadIdx.x * 4;
  if (k >= p.K) return;
  float4 v;
  float scale = p.scale;
  uint16_t* dst;
  if (is_dr) {
    const int g = row / p.rs, i = row - g * p.rs;
    const int ip = (p.rs == 8 && (k & 8)) ? i + 8 : i;
    v = dadr_sum4(p, p.partial, p.partial_x, (long long)p.G * p.E, (long long)g * p.E + ip, k);
    if (F32OUT) {   // the fp32 sums leave as they are (mixed-precision optimisers)
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.dR) + (long long)row * p.lddr + k) =
          make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
      return;
    }
    dst = reinterpret_cast<uint16_t*>(p.dR) + (long long)row * p.lddr + k;
  } else if (is_ib) {
    v = dadr_sum4(p, p.partial_ib, p.partial_ib_x, p.G, row, k);
    dst = p.d_ib + (long long)row * p.K + k;
  } else {
    const float4* src = reinterpret_cast<const float4*>(p.partial_da + (long long)row * p.K + k);
    const long long step = (long long)p.M * p.K / 4;
    v = __ldg(src);
    for (int s = 1; s < p.parts; ++s) {
      const float4 w = __ldg(src + s * step);
      v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    scale = p.da_scale;
    dst = p.dA + (long long)row * p.ldda + k;
  }
  const uint2 o = make_uint2(Elem<DT>::pack(v.x * scale, v.y * scale), Elem<DT>::pack(v.z * scale, v.w * scale));
  if (is_ib && (reinterpret_cast<uintptr_t>(dst) & 7) != 0) {   // d_ib comes from the caller with no more than its own alignment
    dst[0] = (uint16_t)o.x; dst[1] = (uint16_t)(o.x >> 16); dst[2] = (uint16_t)o.y; dst[3] = (uint16_t)(o.y >> 16);
  } else {
    *reinterpret_cast<uint2*>(dst) = o;
  }
}

// Grid of the dA+dR kernel.  runs: the number of main CTA pairs that share one feature column (each
// walks every runs-th 256-token tile).  When the main pairs leave SM pairs idle and have enough
// tiles each, the idle pairs become extra pairs and every main pair leaves its last `steal` tiles
// to them (see DadrUnit): measured faster than many short runs, with a quarter of the workspace.
// cfg (or null): {runs, steal, n_extra}; 0 = default; steal < 0 = no extra pairs.
void dadr_plan_grid(int M, int K, int G, int gs, int num_sms, const int* cfg, DadrGrid* gr) {
  const int n_ft = (K + 127) / 128;
  const int n_mp = (M + 255) / 256;
  const int slots_sm = num_sms / 2 > 0 ? num_sms / 2 : 1;
  int runs = (cfg && cfg[0] > 0) ? cfg[0] : 0;
  if (runs <= 0) {
    runs = 1;
    if (n_ft <= slots_sm) {
      // one wave: the count that leaves the fewest tiles per pair (ties: fewer pairs, less workspace);
      // the SM pairs that stay idle become extra pairs below
      int best_tiles = n_mp;
      for (int r = 2; r <= n_mp && n_ft * r <= slots_sm; ++r) {
        const int tiles = (n_mp + r - 1) / r;
        if (tiles < best_tiles) { best_tiles = tiles; runs = r; }
      }
    } else {
      // more columns than SM pairs: minimise (waves of pairs) x (tiles per pair)
      long long best_cost = -1;
      for (int r = 1; r <= n_mp && r <= 32; ++r) {
        const long long waves = ((long long)n_ft * r + slots_sm - 1) / slots_sm;
        const long long cost = waves * ((n_mp + r - 1) / r);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; runs = r; }
      }
    }
  }
  if (runs > n_mp) runs = n_mp;
  if (runs < 1) runs = 1;
  gr->runs = runs;
  gr->n_ft = n_ft;
  gr->n_main = n_ft * runs;
  gr->n_extra = 0; gr->steal = 0; gr->slots = 0;
  gr->g_per = G; gr->parts = 1;
  if (!cfg || (cfg[0] <= 0 && cfg[1] == 0 && cfg[2] <= 0)) {   // the default plan: no extra pairs beside group parts
    gr->g_per = dadr_groups_per_part(M, K, G, gs, gr->n_main, slots_sm);
    gr->parts = (G + gr->g_per - 1) / gr->g_per;
    if (gr->parts > 1) return;
  }
  const int t_min = n_mp / runs, t_max = (n_mp + runs - 1) / runs;   // tiles of the shortest / longest run
  int steal = cfg ? cfg[1] : 0;
  int n_extra = (cfg && cfg[2] > 0) ? cfg[2] : (slots_sm - gr->n_main);
  if (steal < 0 || n_extra < 1) return;
  if (n_extra > gr->n_main) n_extra = gr->n_main;
  const int cnt_max = (gr->n_main + n_extra - 1) / n_extra;          // main pairs per extra pair
  if (steal == 0) {
    steal = (t_max * n_extra + (gr->n_main + n_extra) / 2) / (gr->n_main + n_extra);
    while (steal > 0 && cnt_max * steal > t_max - steal) --steal;   // an extra pair must not become the longest
  }
  if (steal > t_min - 1) steal = t_min - 1;                           // every main pair keeps a tile
  if (steal < 1) return;
  gr->n_extra = n_extra; gr->steal = steal; gr->slots = cnt_max;
}

template <int E>
static int dadr_plan(DadrParams& p, int& smem_bytes, bool ib) {
  using St = dadr::Stage<E>;
  p.rr_tile_bytes = ((E / 2 * 128) + 1023) / 1024 * 1024;
  p.rd_tile_bytes = ((E * 128) + 1023) / 1024 * 1024;
  p.rb = (E <= 16) ? 4 : 2;
  const int fixed = 6 * dadr::kTile + p.rb * 2 * (p.rr_tile_bytes + p.rd_tile_bytes) + (int)sizeof(DadrBarriers) + 1024 +
                    (ib ? 8192 : 0);
  int ns = (227 * 1024 - 256 - fixed) / St::kBytes;
  if (ns > dadr::kMaxStages) ns = dadr::kMaxStages;
  if (ns < 2) return fail(PRISM_ERR_UNSUPPORTED, "bwd_dadr does not fit shared memory (E=%d)", E);
  p.ns = ns;
  smem_bytes = fixed + ns * St::kBytes;
  return PRISM_OK;
}

int launch_bwd_dadr(const DadrArgs& a) {
  DadrParams p;
  p.M = a.M; p.N = a.N; p.K = a.K; p.gs = a.gs; p.E = a.E; p.G = a.N / a.gs;
  p.n_mtiles = (a.M + 127) / 128;
  p.runs = a.grid.runs;
  p.n_ft = a.grid.n_ft; p.n_main = a.grid.n_main;
  p.n_extra = a.grid.n_extra; p.steal = a.grid.steal; p.slots = a.grid.slots;
  p.partial_x = a.partial_x;
  p.scale = a.scale;
  p.dA = a.dA; p.ldda = a.ldda; p.partial = a.partial; p.err = a.err;
  int smem_bytes = 0;
  const bool ib = a.ib != nullptr && a.gate != GATE_NONE;
  DadrExtra x;
  x.g_per = a.grid.g_per; x.partial_da = a.partial_da;
  x.ib = ib ? a.ib : nullptr; x.partial_ib = a.partial_ib; x.partial_ib_x = a.partial_ib_x;
  int rc = (a.E == 16) ? dadr_plan<16>(p, smem_bytes, ib) : (a.E == 32) ? dadr_plan<32>(p, smem_bytes, ib) : dadr_plan<64>(p, smem_bytes, ib);
  if (rc) return rc;
  const int stage_out = 64;

  CUtensorMap tmA, tmRr, tmRd, tmdC, tmB;
  if ((rc = make_tmap_2d(&tmA, a.dtype, a.A, a.M, a.K, a.lda, 128, 64, true))) return rc;
  if ((rc = make_tmap_2d(&tmRr, a.dtype, a.R_eff, (uint64_t)p.G * a.E, a.K, a.ldr, a.E / 2, 64, true))) return rc;
  if ((rc = make_tmap_2d(&tmRd, a.dtype, a.R_eff, (uint64_t)p.G * a.E, a.K, a.ldr, a.E, 64, true))) return rc;
  if ((rc = make_tmap_2d(&tmdC, a.dtype, a.dC, a.M, a.N, a.lddc, 128, 64, true))) return rc;
  if ((rc = make_tmap_2d(&tmB, a.dtype, a.B, a.N, a.K, a.ldb, stage_out, 64, true))) return rc;

  const bool drop = a.drop_seeds != nullptr && a.drop_p > 0.f && a.gate != GATE_NONE;
  if (drop && a.E != 16) return fail(PRISM_ERR_UNSUPPORTED, "bwd_dadr: dropout needs reconn_sz 8 or 16");
  x.drop_seeds = a.drop_seeds; x.drop_thr = drop_threshold(a.drop_p); x.drop_mask = a.drop_mask; x.drop_inv_keep = drop ? 1.f / (1.f - a.drop_p) : 1.f;
  const bool parts = a.grid.parts > 1 || (dadr_sigmoid16(a.dtype, a.gate, a.E, ib, drop) && !dadr_whole(a.gs));
  DadrKernel kern = (a.dtype == DT_BF16) ? dadr_kernel_bf16(a.gate, a.E, ib, drop, parts) : dadr_kernel_f16(a.gate, a.E, ib, drop, parts);
  if ((rc = set_max_dynamic_smem(reinterpret_cast<const void*>(kern), smem_bytes, "bwd_dadr"))) return rc;
  dim3 grid(2 * (p.n_main + p.n_extra), a.grid.parts, 1);   // the two CTAs of a pair are neighbours
  kern<<<grid, dadr::kThreads, smem_bytes, a.stream>>>(tmA, tmRr, tmRd, tmdC, tmB, p, x);
  if ((rc = check_launch("prism_bwd_dadr"))) return rc;
  DadrReduce r;
  r.partial = a.partial; r.partial_x = a.partial_x; r.dR = a.dR; r.lddr = a.lddr;
  r.partial_ib = a.partial_ib; r.partial_ib_x = a.partial_ib_x; r.d_ib = reinterpret_cast<uint16_t*>(a.d_ib);
  r.partial_da = a.partial_da; r.dA = reinterpret_cast<uint16_t*>(a.dA); r.ldda = a.ldda;
  r.M = a.M; r.G = p.G; r.rs = a.rs; r.E = a.E; r.K = a.K; r.runs = p.runs; r.n_ft = p.n_ft; r.n_main = p.n_main;
  r.n_extra = p.n_extra; r.steal = p.steal; r.slots = p.slots; r.parts = a.grid.parts;
  // gated mode: the kernel formed 2 dS against the halved R tiles, so the dR partials are doubled
  r.scale = (a.gate != GATE_NONE) ? 0.5f * a.scale : a.scale;
  r.da_scale = a.scale;
  r.k_blocks = (a.K + 1023) / 1024;
  const long long dr_blocks = (long long)p.G * a.rs * r.k_blocks, ib_blocks = ib ? (long long)p.G * r.k_blocks : 0;
  const long long blocks = dr_blocks + ib_blocks + (a.grid.parts > 1 ? (long long)a.M * r.k_blocks : 0);
  if (blocks > 0x7fffffffll) return fail(PRISM_ERR_UNSUPPORTED, "bwd_dadr: too many rows to reduce (%lld blocks)", blocks);
  r.dr_blocks = (unsigned)dr_blocks; r.ib_blocks = (unsigned)ib_blocks;
  const int threads = a.K >= 1024 ? 256 : ((a.K >> 2) + 31) / 32 * 32;
#define PRISM_DADR_REDUCE(DT_, F32_) dadr_reduce_kernel<DT_, F32_><<<(unsigned)blocks, threads, 0, a.stream>>>(r)
  if (a.dtype == DT_BF16) { if (a.dr_f32) PRISM_DADR_REDUCE(DT_BF16, true); else PRISM_DADR_REDUCE(DT_BF16, false); }
  else { if (a.dr_f32) PRISM_DADR_REDUCE(DT_F16, true); else PRISM_DADR_REDUCE(DT_F16, false); }
#undef PRISM_DADR_REDUCE
  return check_launch("prism_bwd_dadr reduce");
}

}  // namespace prism
