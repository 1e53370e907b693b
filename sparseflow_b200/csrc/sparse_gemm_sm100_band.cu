// 2:4-sparse GEMM for sm_100a between decode and prefill: CTA-pair tiles of any token width, optionally with K split over
// a cluster of pairs.
//
// Operand formats, tensor-memory layout and MMA are those of sparse_gemm_sm100_2cta.cu (256 weight rows per SM pair,
// tcgen05.mma.sp.cta_group::2).  What bounds a K step of such a tile is the shared-memory port: per CTA and 128-wide step
// TMA writes 18 KB of weight + 128 B per token column and the MMAs read 16 KB + 128 B per column, at 128 B/clk
// = 0.145 us + 1.02 ns * T for T tokens (the pair tiles of 192 ... 256 tokens measure 0.159 us + 1.02 ns * T).  A single
// CTA would read every token column itself, twice that per column.  So below prefill the time of a GEMM is
// (K steps in series) x (that step), and what is to be won is fewer steps in series with all pairs at work:
//   * the token tile is a run-time multiple of 16 (the ring gets as many stages as fit), so a tile is not wider
//     than the tokens there are.  Above 256 and up to 400 tokens it is two MMAs over one weight tile: 18 KB less to write per
//     step than two tiles, a quarter less L2 traffic, and less energy, which is what counts at the power limit;
//   * split 1: persistent pairs.  Tiles that fill whole passes over the pairs run at full width; those left over (fewer
//     than pairs) are cut into token slices, as many as the idle pairs allow, so the last pass is short.  A slice packs as
//     many K steps into a ring stage as a whole tile's stage has room for: with one, the three stages of a 304-token
//     ring kept 78 KB of a slice in flight and its step took 0.4 us of latency (22016 x 4096 at 300 tokens 40.3 us, now 36.9);
//   * split 2, 3 or 4 (few row tiles): a cluster of that many pairs shares one tile, each pair streaming a slice of K.  The fp32
//     accumulators are summed through distributed shared memory: pair p owns the 16-token chunks c with c % split == p,
//     the others store theirs into its shared memory (the drained operand ring) as register fragments, 512 contiguous
//     bytes per store instruction, and the owner adds them in pair order.  No scratch in global memory, no
//     atomics, the same bits on every run.
//
// Measured (B200, steady load at the power limit, fixed tiles before -> now): 4096 x 11008 at 150 / 300 / 400 tokens 33.6 / 34.0 /
// 35.9 -> 17.8 / 23.6 / 28.2 us; 22016 x 4096 (SiLU.mul) at 72 / 150 / 300 / 400 tokens 28.3 / 33.0 / 47.3 / 50.1 -> 24.8 / 28.8 /
// 38.4 / 43.3 us; 8192 x 8192 at 520 tokens 56.2 -> 42.5 us; 57344 x 8192 at 300 tokens 211 -> 171 us.  90 registers, no spills.  Evict-last token loads and
// evict-first stores are 3-10 % of that.  Split 3 against split 2: 4096 x 11008 at 96 / 150 tokens 18.3 / 19.2 -> 16.0 / 17.6 us.
//
// Warps: warp 0 = TMA producer, warp 1 = MMA issuer / tensor-memory owner, warps 2 ... 17 = epilogue.
// All loads are plain per-CTA TMA copies.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

#include "kernels.h"
#include "launch.h"
#include "sm100_pair.cuh"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

namespace sfb200 {

namespace {

constexpr int kEpiWarps = 16;
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kABytes = 128 * 128;             // 128 rows x 64 kept values per CTA and step
constexpr int kEBytes = 2048;                  // their metadata tile
constexpr int kStagingBytes = 16 * 64;         // per epilogue warp: 16 tokens x 32 rows of 16-bit outputs
constexpr int kBarBytes = 256;
constexpr int kRingBytes = 232448 - 1024 - kBarBytes - kEpiWarps * kStagingBytes;
constexpr int kMaxStages = 8;

__host__ __device__ constexpr int stage_bytes(int t) { return kABytes + kEBytes + 128 * t; }
__host__ __device__ constexpr int ring_stages(int t) {
  return kRingBytes / stage_bytes(t) < kMaxStages ? kRingBytes / stage_bytes(t) : kMaxStages;
}
constexpr int kMaxTile = 400;
static_assert(ring_stages(256) >= 4 && ring_stages(kMaxTile) >= 3, "the widest tiles keep three stages");
static_assert(8 * (2 * kMaxStages + 4) + 16 <= kBarBytes, "barrier area");

struct BandParams {
  const void* bias;       // as SparseGemmArgs
  const void* bias_up;
  void* y;
  int* status;
  int n_out, m_tok, ldy;
  int k_tiles128;
  int split;              // pairs per cluster = K slices
  int t_full, t_tail;     // tokens of a full item / of a slice of a left-over tile
  int n0_full;            // columns of a full item's first MMA (the rest, if any, is a second one over the same weights)
  int ks_tail;            // K steps per ring stage of a slice
  int stage_stride;       // bytes of a ring stage: one K step of a whole tile, ks_tail of a slice
  int tail_col;           // > 0: slices accumulate in columns of their own, from this one on
  int num_n_blks;         // token blocks of t_full
  int n_full;             // items [0, n_full) are whole tiles, the rest slices of the tiles from n_full on
  int slices;             // slices per left-over tile
  int n_tail;             // slices in all (at most one per cluster)
  int stages, acc_bufs, tmem_cols;
  int fmt, act;
};

struct Item {
  int m_blk, tok0, tok_end, n;
  int n0;         // columns [0, n0) and [n0, n) are one MMA each
  int ks;         // K steps per ring stage
  bool tail;
};
// The i-th item of cluster c: whole tiles c, c + clusters, ..., then at most one slice of a left-over tile, slice c.
// (Half of the clusters taking their slice first, so that a pass bound by HBM runs beside one bound by shared memory, was
// measured slower from 150 tokens -- 22016 x 4096: 26.9 -> 28.0 us at 150 tokens, 34.8 -> 37.1 at 300 -- because
// the pairs that share weight or token tiles no longer read them at the same time.)
__device__ __forceinline__ int item_count(int c, int clusters, const BandParams& p) {
  return (p.n_full - c + clusters - 1) / clusters + (c < p.n_tail ? 1 : 0);
}
// Item: a 256-row tile and a token range; false = nothing to do (a slice beyond the last token).
__device__ __forceinline__ bool get_item(int i, int c, int clusters, const BandParams& p, Item& it) {
  int tile = c + i * clusters, off = 0;
  it.tail = tile >= p.n_full;
  it.n = p.t_full;
  it.n0 = p.n0_full;
  it.ks = 1;
  if (it.tail) {
    tile = p.n_full + c / p.slices;
    off = (c % p.slices) * p.t_tail;
    it.n = it.n0 = p.t_tail;
    it.ks = p.ks_tail;
  }
  it.m_blk = tile / p.num_n_blks;
  const int t0 = (tile - it.m_blk * p.num_n_blks) * p.t_full;
  it.tok0 = t0 + off;
  it.tok_end = t0 + p.t_full < p.m_tok ? t0 + p.t_full : p.m_tok;
  return it.tok0 < it.tok_end;
}

// Accumulator of the next item: barrier index, its use count so far and first column.  `done` counts the items before it that
// use the common set(s).
__device__ __forceinline__ void next_acc(const BandParams& p, const Item& it, uint32_t& done, uint32_t& as, uint32_t& use,
                                         uint32_t& col) {
  if (it.tail && p.tail_col > 0) {      // at most one per pair
    as = 1;
    use = 0;
    col = p.tail_col;
    return;
  }
  as = p.acc_bufs == 2 ? (done & 1u) : 0u;
  use = p.acc_bufs == 2 ? (done >> 1) : done;
  col = as * p.t_full;
  ++done;
}

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, const uint32_t* r) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void add_f32(uint32_t& a, uint32_t b) { a = __float_as_uint(__uint_as_float(a) + __uint_as_float(b)); }

template <int EPI>
__global__ void __launch_bounds__(kThreads, 1)
sparse_gemm_band_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                        const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmBt,
                        const __grid_constant__ CUtensorMap tmE,
                        const BandParams p) {
  extern __shared__ uint8_t smem_raw[];
  // the same offset in every CTA of the cluster: the dynamic shared memory base is identical
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t st_bytes = static_cast<uint32_t>(p.stage_stride);
  const uint32_t staging = sbase + p.stages * st_bytes;
  const uint32_t bar_full = staging + kEpiWarps * kStagingBytes;   // used in the even CTA of the pair only
  const uint32_t bar_empty = bar_full + 8 * kMaxStages;            // both CTAs
  const uint32_t bar_accf = bar_empty + 8 * kMaxStages;            // both CTAs, one per accumulator set
  const uint32_t bar_acce = bar_accf + 16;                         // even CTA only, one per accumulator set
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + (bar_acce + 16 - sbase));
  volatile int* err = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank();
  const uint32_t rank = crank & 1;          // within the pair
  const uint32_t even = crank & ~1u;        // cluster rank of the pair's even CTA
  const int kpart = static_cast<int>(crank >> 1);   // this pair's K slice
  const bool leader = rank == 0;
  const int ctas = 2 * p.split;
  const int cluster_id = blockIdx.x / ctas;
  const int num_clusters = gridDim.x / ctas;
  const int items = item_count(cluster_id, num_clusters, p);
  // K slice in 128-wide tiles
  const int kbase = p.k_tiles128 / p.split, kextra = p.k_tiles128 % p.split;
  const int k_begin = kpart * kbase + (kpart < kextra ? kpart : kextra);
  const int k_end = k_begin + kbase + (kpart < kextra ? 1 : 0);

  if (threadIdx.x == 0) {
    *err = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_accf + 8 * b, 1);
      mbar_init(bar_acce + 8 * b, 2 * kEpiWarps);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmB);
    if (p.n0_full < p.t_full) tma_prefetch_desc(&tmB1);
    if (p.n_tail > 0) tma_prefetch_desc(&tmBt);
  }
  if (threadIdx.x == 64) {      // the first ring of weight tiles into L2, under the previous kernel's tail
    Item it;
    if (items > 0 && get_item(0, cluster_id, num_clusters, p, it)) {
      const int row0 = it.m_blk * 256 + static_cast<int>(rank) * 128, e_row = (row0 >> 7) * p.k_tiles128;
      for (int kt = k_begin; row0 < p.n_out && kt < k_end && kt < k_begin + p.stages; ++kt) {
        prefetch_l2_2d(&tmA, kt * 64, row0);
        prefetch_l2_1d_tensor(&tmE, (e_row + kt) * 256);
      }
    }
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), p.tmem_cols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // every CTA's barriers are initialised before anything remote touches them
  tc_fence_after();
  dependency_wait();
  dependency_trigger();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      const uint32_t pair_full0 = mapa_u32(bar_full, even);
      const uint64_t pol_keep = l2_policy_evict_last();     // every row tile reads the activations again
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int i = 0; i < items && ok; ++i) {
        Item it;
        if (!get_item(i, cluster_id, num_clusters, p, it)) continue;
        const CUtensorMap* tb = it.tail ? &tmBt : &tmB;
        const int n1 = it.n - it.n0;
        const uint32_t b0 = 64u * it.n0, b1 = 64u * n1;          // bytes of one 64-wide K half of this CTA's tokens
        const int row0 = it.m_blk * 256 + static_cast<int>(rank) * 128;
        const int tok = it.tok0 + static_cast<int>(rank) * (it.n0 / 2), tok1 = it.tok0 + it.n0 + static_cast<int>(rank) * (n1 / 2);
        const int e_row = (row0 >> 7) * p.k_tiles128;
        const uint32_t step = stage_bytes(it.n);                 // weights, tokens, metadata of one K step
        const uint32_t tx = 2u * (kABytes + kEBytes + 2u * (b0 + b1));   // bytes of BOTH CTAs land on the even CTA's barrier
        for (int kt = k_begin; kt < k_end; kt += it.ks) {
          ok = mbar_wait(bar_empty + 8 * s, ph ^ 1, err, p.status, 1);
          if (!ok) break;
          const uint32_t full = pair_full0 + 8 * s;
          const int nk = kt + it.ks < k_end ? it.ks : k_end - kt;
          if (leader) mbar_arrive_expect_tx(bar_full + 8 * s, nk * tx);
          uint32_t st = sbase + s * st_bytes;
          for (int k = kt; k < kt + nk; ++k, st += step) {
            tma_load_2d_pair(st, &tmA, k * 64, row0, full);
            tma_load_2d_pair_hint(st + kABytes, tb, k * 128, tok, full, pol_keep);
            tma_load_2d_pair_hint(st + kABytes + b0, tb, k * 128 + 64, tok, full, pol_keep);
            if (n1 > 0) {
              tma_load_2d_pair_hint(st + kABytes + 2 * b0, &tmB1, k * 128, tok1, full, pol_keep);
              tma_load_2d_pair_hint(st + kABytes + 2 * b0 + b1, &tmB1, k * 128 + 64, tok1, full, pol_keep);
            }
            tma_load_1d_pair(st + step - kEBytes, &tmE, (e_row + k) * 256, full);
          }
          if (++s == p.stages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (even CTA of each pair)
    if (leader && elect_one()) {
      const uint16_t both = static_cast<uint16_t>(3u << even);
      // metadata columns start after the accumulators
      const uint32_t e_col0 = tmem_base + (p.tail_col > 0 ? p.tail_col + p.t_tail : p.acc_bufs * p.t_full);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      uint32_t done = 0;
      for (int i = 0; i < items && ok; ++i) {
        Item it;
        if (!get_item(i, cluster_id, num_clusters, p, it)) continue;
        uint32_t as, use, col;
        next_acc(p, it, done, as, use, col);
        const int n1 = it.n - it.n0;
        const uint32_t idesc = make_idesc_f16(256, it.n0, p.fmt, true), idesc1 = make_idesc_f16(256, n1, p.fmt, true);
        const uint32_t d = tmem_base + col;
        const uint32_t b0 = 64u * it.n0, b1 = 64u * n1, step = stage_bytes(it.n);
        ok = mbar_wait(bar_acce + 8 * as, (use & 1u) ^ 1u, err, p.status, 3);
        if (!ok) break;
        tc_fence_after();
        for (int kt = k_begin; kt < k_end; kt += it.ks) {
          ok = mbar_wait(bar_full + 8 * s, ph, err, p.status, 2);
          if (!ok) break;
          tc_fence_after();
          const int nk = kt + it.ks < k_end ? it.ks : k_end - kt;
          uint32_t st = sbase + s * st_bytes, e_cols = e_col0 + 4 * p.ks_tail * s;
          for (int k = kt; k < kt + nk; ++k, st += step, e_cols += 4) {
            tc_cp_128x128b_pair(e_cols, make_smem_desc(st + step - kEBytes, 0, 128, kSwNone));
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
              const uint64_t adesc = make_smem_desc(st + kb * 32, 16, 1024, kSw128);
              const uint64_t bdesc = make_smem_desc(st + kABytes + (kb >> 1) * b0 + (kb & 1) * 64, 16, 1024, kSw128);
              const uint32_t accumulate = (k > k_begin || kb > 0) ? 1u : 0u;
              tc_mma_sp_f16_pair(d, adesc, bdesc, e_cols + (kb & ~1), idesc | (kb & 1), accumulate);
              if (n1 > 0) {
                const uint64_t bdesc1 = make_smem_desc(st + kABytes + 2 * b0 + (kb >> 1) * b1 + (kb & 1) * 64, 16, 1024, kSw128);
                tc_mma_sp_f16_pair(d + it.n0, adesc, bdesc1, e_cols + (kb & ~1), idesc1 | (kb & 1), accumulate);
              }
            }
          }
          tc_commit_pair(bar_empty + 8 * s, both);
          if (++s == p.stages) { s = 0; ph ^= 1; }
        }
        if (!ok) break;
        tc_commit_pair(bar_accf + 8 * as, both);
      }
    }
  }
  if (warp < 2) {
    __syncwarp();
    if (p.split > 1) {   // the two barriers of the reduction
      cluster_sync_all();
      cluster_sync_all();
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2 ... 17, both CTAs)
    const int q = warp & 3;                   // lane quadrant
    const int part = (warp - 2) >> 2;         // the warps of a quadrant take its 16-token chunks in turn
    const int g = lane >> 2;
    constexpr int kRowBytes = (EPI == kEpiSwiGLU) ? 32 : 64;
    const uint32_t stage = staging + (warp - 2) * kStagingBytes;
    // stmatrix row address of this lane: matrix = lane / 8, row in matrix = lane % 8
    const uint32_t st_off = static_cast<uint32_t>(((lane & 7) + 8 * (lane >> 4)) * kRowBytes + 16 * ((lane >> 3) & 1));
    const int out_cols = (EPI == kEpiSwiGLU) ? p.n_out / 2 : p.n_out;
    const uint32_t even_acce0 = mapa_u32(bar_acce, even);
    const uint64_t pol_stream = l2_policy_evict_first();
    bool ok = true;
    uint32_t done = 0;
    for (int i = 0; i < items && ok; ++i) {
      Item it;
      if (!get_item(i, cluster_id, num_clusters, p, it)) continue;
      uint32_t as, use, col;
      next_acc(p, it, done, as, use, col);
      ok = __all_sync(0xffffffffu, mbar_wait(bar_accf + 8 * as, use & 1u, err, p.status, 4));
      if (!ok && p.split == 1) break;
      tc_fence_after();
      const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + col;
      const int row_w = it.m_blk * 256 + static_cast<int>(rank) * 128 + q * 32;
      const int chunks = (it.tok_end - it.tok0 + 15) / 16 < it.n / 16 ? (it.tok_end - it.tok0 + 15) / 16 : it.n / 16;
      auto load_chunk = [&](int c, uint32_t (&r)[16]) {
        tmem_ld_16x256b_x2(t_acc + 16 * c, *reinterpret_cast<uint32_t(*)[8]>(&r[0]));                                       // lanes 0..15
        tmem_ld_16x256b_x2(t_acc + 16 * c + (16u << 16), *reinterpret_cast<uint32_t(*)[8]>(&r[8]));   // lanes 16..31
        tmem_ld_wait();
      };
      float b0 = 0.f, b1 = 0.f, b2 = 0.f, b3 = 0.f;   // bias of rows g, g+8, 16+g, 24+g
      if (EPI == kEpiStore && p.bias != nullptr) {
        if (row_w + g < p.n_out) b0 = bias_at(p.bias, row_w + g, p.fmt);
        if (row_w + g + 8 < p.n_out) b1 = bias_at(p.bias, row_w + g + 8, p.fmt);
        if (row_w + g + 16 < p.n_out) b2 = bias_at(p.bias, row_w + g + 16, p.fmt);
        if (row_w + g + 24 < p.n_out) b3 = bias_at(p.bias, row_w + g + 24, p.fmt);
      }
      if (EPI == kEpiSwiGLU) load_gate_up_bias(p.bias, p.bias_up, row_w, g, p.n_out, p.fmt, b0, b1, b2, b3);
      // one chunk: activation / SiLU.mul, transpose through the staging tile, 16-byte stores
      auto store_chunk = [&](const uint32_t (&r)[16], int t0) {
        const uint32_t* a = &r[0];
        const uint32_t* b = &r[8];
        __syncwarp();                                 // every lane has read the tile's previous contents
        if (EPI == kEpiSwiGLU) {
          auto emit = [&](auto f, const int of) {
            stmatrix_x4_trans(stage + st_off, pack16(f(a[0], b[0], b0, b2), f(a[1], b[1], b0, b2), of),
                              pack16(f(a[2], b[2], b1, b3), f(a[3], b[3], b1, b3), of),
                              pack16(f(a[4], b[4], b0, b2), f(a[5], b[5], b0, b2), of),
                              pack16(f(a[6], b[6], b1, b3), f(a[7], b[7], b1, b3), of));
          };
          auto plain = [](uint32_t gate, uint32_t up, float, float) { return silu_mul(gate, up); };
          if (p.bias != nullptr || p.bias_up != nullptr) emit(silu_mul_bias, p.fmt);
          else if (p.fmt == 1) emit(plain, 1);
          else emit(plain, 0);
        } else {
          auto emit = [&](auto f, const int of) {
            stmatrix_x4_trans(stage + st_off, pack16(f(a[0], b0), f(a[1], b0), of), pack16(f(a[2], b1), f(a[3], b1), of),
                              pack16(f(a[4], b0), f(a[5], b0), of), pack16(f(a[6], b1), f(a[7], b1), of));
            stmatrix_x4_trans(stage + st_off + 32, pack16(f(b[0], b2), f(b[1], b2), of), pack16(f(b[2], b3), f(b[3], b3), of),
                              pack16(f(b[4], b2), f(b[5], b2), of), pack16(f(b[6], b3), f(b[7], b3), of));
          };
          auto plain = [](uint32_t v, float bias) { return __uint_as_float(v) + bias; };
          if (p.act != kActNone) emit([&](uint32_t v, float bias) { return act_fn(__uint_as_float(v) + bias, p.act); }, p.fmt);
          else if (p.fmt == 1) emit(plain, 1);
          else emit(plain, 0);
        }
        __syncwarp();
        constexpr int kUnits = kRowBytes / 16, kRounds = kUnits / 2, kTokRound = 32 / kUnits;
        const int tk = lane / kUnits, unit = lane % kUnits;
        const int col = (EPI == kEpiSwiGLU ? row_w / 2 : row_w) + unit * 8;
        uint16_t* dst = static_cast<uint16_t*>(p.y) + static_cast<size_t>(t0 + tk) * p.ldy + col;
#pragma unroll
        for (int j = 0; j < kRounds; ++j)
          if (t0 + tk + j * kTokRound < it.tok_end && col < out_cols) {
            const uint4 v = ld_shared_v4(stage + (tk + j * kTokRound) * kRowBytes + unit * 16);
            asm volatile("st.global.L2::cache_hint.v4.b32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(
                             dst + static_cast<size_t>(j * kTokRound) * p.ldy),
                         "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "l"(pol_stream)
                         : "memory");
          }
      };
      auto release_acc = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(even_acce0 + 8 * as);
      };

      uint32_t r[16];
      if (p.split == 1) {
        if (part >= chunks) release_acc();
#pragma unroll 1
        for (int c = part; c < chunks; c += 4) {
          load_chunk(c, r);
          if (c + 4 >= chunks) release_acc();         // this warp's last chunk is in registers
          store_chunk(r, it.tok0 + c * 16);
        }
      } else {
        // slot of each other pair for own chunk oc, quadrant q: 2 KB of fragments, [register / 4][lane] 16 bytes each
        const int own_max = (p.t_full / 16 + p.split - 1) / p.split;
        const uint32_t slot_q = static_cast<uint32_t>(q * 2048 + lane * 16);
        __syncwarp();
        cluster_sync_all();      // every pair's MMAs have read their operands: the rings are free
        if (ok) {
#pragma unroll 1
          for (int c = part; c < chunks; c += 4) {
            const int owner = c % p.split;
            if (owner == kpart) continue;
            load_chunk(c, r);
            const uint32_t dst = mapa_u32(sbase, 2 * owner + rank) + slot_q +
                                 static_cast<uint32_t>(((kpart - (kpart > owner ? 1 : 0)) * own_max + c / p.split) * 8192);
#pragma unroll
            for (int j = 0; j < 4; ++j) st_cluster_v4(dst + j * 512, &r[4 * j]);
          }
        }
        __syncwarp();
        cluster_sync_all();      // all partial sums have landed in their owners' shared memory
        if (ok && *err == 0) {
#pragma unroll 1
          for (int oc = part; oc * p.split + kpart < chunks; oc += 4) {
            const int c = oc * p.split + kpart;
            uint32_t own[16];
            load_chunk(c, own);
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = 0u;
            for (int src = 0; src < p.split; ++src) {
              if (src == kpart) {
#pragma unroll
                for (int j = 0; j < 16; ++j) add_f32(r[j], own[j]);
              } else {
                const uint32_t slot = sbase + slot_q + static_cast<uint32_t>(((src - (src > kpart ? 1 : 0)) * own_max + oc) * 8192);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const uint4 v = ld_shared_v4(slot + j * 512);
                  add_f32(r[4 * j], v.x);
                  add_f32(r[4 * j + 1], v.y);
                  add_f32(r[4 * j + 2], v.z);
                  add_f32(r[4 * j + 3], v.w);
                }
              }
            }
            store_chunk(r, it.tok0 + c * 16);
          }
        }
      }
    }
  }

  // ------------------------------------------------------------ teardown
  __syncwarp();
  if (*err) {
    // give copies that may still be in flight time to land before shared memory is released
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer may still be signalling this CTA's barriers until here
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, p.tmem_cols);
  }
}

int round16(int v) { return (v + 15) & ~15; }

// Ring geometry.  A slice packs ks K steps into a stage; the stage is made larger than a whole tile's K step where that
// puts more bytes of a slice in flight without taking the ring below four stages (three for tiles above 256 tokens).  At one
// step per stage the slices of a 160-token ring (5 x 22 KB in flight) ran at 0.30 us a step, bound by latency.
struct Ring {
  int stages, ks, stride;
};
Ring plan_ring(int t, int t_tail, bool slices) {
  Ring best{ring_stages(t), 1, stage_bytes(t)};
  if (!slices) return best;
  int most = best.stages * stage_bytes(t_tail);
  for (int ks = 2; ks <= 4; ++ks) {
    const int need = ks * stage_bytes(t_tail), stride = need > stage_bytes(t) ? need : stage_bytes(t);
    int stages = kRingBytes / stride < kMaxStages ? kRingBytes / stride : kMaxStages;
    if (stages < (t > 256 ? 3 : 4)) break;
    if (stages * need > most) {
      most = stages * need;
      best = Ring{stages, ks, stride};
    }
  }
  return best;
}

// Work items of a split-1 launch: tiles that fill whole passes over the pairs, then the left-over tiles cut into
// token slices so that one more, shorter pass covers them.
struct ItemPlan {
  int n_full, slices, t_tail, n_tail;
};
ItemPlan plan_items(int tiles, int t, int pairs) {
  ItemPlan q{tiles, 1, t, 0};
  const int left = tiles % pairs;
  if (left == 0 || left * 2 > pairs) return q;          // the last pass has no room for slices
  int sl = pairs / left;
  if (sl > t / 16) sl = t / 16;
  q.t_tail = round16((t + sl - 1) / sl);
  q.slices = (t + q.t_tail - 1) / q.t_tail;
  q.n_full = tiles - left;
  q.n_tail = left * q.slices;
  return q;
}

template <int EPI>
int launch_band(const SparseGemmArgs& a, int split, int t, cudaStream_t stream) {
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  constexpr int kSmemBytes = 232448;
  if (dev < 16 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(sparse_gemm_band_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess)
      return kErrCuda;
    attr_set[dev] = true;
  }
  BandParams p;
  p.bias = a.bias;
  p.bias_up = a.bias_up;
  p.y = a.y;
  p.status = a.status;
  p.n_out = a.n_out;
  p.m_tok = a.m_tok;
  p.ldy = a.ldy;
  p.k_tiles128 = (a.K + 127) / 128;
  p.split = split;
  p.t_full = t;
  p.num_n_blks = (a.m_tok + t - 1) / t;
  p.fmt = a.fmt;
  p.act = a.act;
  const int tiles = ((a.n_out + 255) / 256) * p.num_n_blks;
  const int pairs = a.num_sms / 2 > 0 ? a.num_sms / 2 : 1;
  const ItemPlan q = split == 1 ? plan_items(tiles, t, pairs) : ItemPlan{tiles, 1, t, 0};
  p.t_tail = q.t_tail;
  p.n_full = q.n_full;
  p.slices = q.slices;
  p.n_tail = q.n_tail;
  p.n0_full = t <= 256 ? t : round16(t / 2);
  const Ring ring = plan_ring(t, p.t_tail, p.n_tail > 0);
  p.stages = ring.stages;
  p.ks_tail = ring.ks;
  p.stage_stride = ring.stride;
  p.acc_bufs = (split == 1 && 2 * t + 4 * p.stages <= 512) ? 2 : 1;
  const bool tail_own = p.acc_bufs == 1 && p.n_tail > 0 && t + p.t_tail + 4 * p.stages <= 512;
  p.tail_col = tail_own ? t : 0;
  const int acc_cols = tail_own ? t + p.t_tail : p.acc_bufs * t;
  while (p.ks_tail > 1 && acc_cols + 4 * p.stages * p.ks_tail > 512) --p.ks_tail;   // metadata columns of every step in flight
  const int used = acc_cols + 4 * p.stages * p.ks_tail;
  p.tmem_cols = 32;
  while (p.tmem_cols < used) p.tmem_cols *= 2;

  CUtensorMap tmA, tmB, tmB1, tmBt, tmE;
  const uint64_t kc = static_cast<uint64_t>(a.K) / 2;
  if (!make_map_2d(&tmA, a.values, a.n_out, kc, kc * 2, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B, a.fmt)) return kErrTensorMap;
  const uint64_t pitch = static_cast<uint64_t>(a.ldx) * 2;
  if (!make_map_2d(&tmB, a.x, a.m_tok, a.K, pitch, p.n0_full / 2, 64, CU_TENSOR_MAP_SWIZZLE_128B, a.fmt)) return kErrTensorMap;
  tmBt = tmB1 = tmB;
  if (p.n0_full < t &&
      !make_map_2d(&tmB1, a.x, a.m_tok, a.K, pitch, (t - p.n0_full) / 2, 64, CU_TENSOR_MAP_SWIZZLE_128B, a.fmt))
    return kErrTensorMap;
  if (p.n_tail > 0 && !make_map_2d(&tmBt, a.x, a.m_tok, a.K, pitch, p.t_tail / 2, 64, CU_TENSOR_MAP_SWIZZLE_128B, a.fmt))
    return kErrTensorMap;
  if (!make_map_1d_u64(&tmE, a.meta, meta_bytes(a.n_out, a.K) / 8, 256)) return kErrTensorMap;

  // split > 1: one cluster per tile; split 1: persistent pairs (a plan with slices fills whole passes before them)
  const int work = p.n_full > 0 ? p.n_full : p.n_tail;
  const int clusters = (split > 1 || work < pairs) ? work : pairs;
  const size_t smem = 1024 + static_cast<size_t>(p.stages) * p.stage_stride + kEpiWarps * kStagingBytes + kBarBytes;
  return launch_dependent(sparse_gemm_band_kernel<EPI>, clusters * 2 * split, kThreads, smem, 2 * split, stream, tmA, tmB, tmB1,
                          tmBt, tmE, p);
}

// Clusters of 2 * split CTAs that are resident at once: a cluster does not straddle the GPU's processor groups, and on the 148
// SMs of a B200 74, 33, 22 and 15 fit (cudaOccupancyMaxActiveClusters).
int clusters_resident(int split, int num_sms) {
  const int of148[5] = {0, 74, 33, 22, 15};
  const int n = num_sms * of148[split] / 148;
  return n > 0 ? n : 1;
}

// Estimated time in us of one (split, token tile) on a GPU with num_sms SMs; constants measured on B200.
//   K step of a t-token tile: 0.15 + 0.00102 t us (the shared-memory port, see the top of this file), wide tiles up to 12 %
//     more where K is long (the pair kernel's factor);
//   weights from HBM at 6.6 TB/s; the passes' K loops and that stream overlap only in part, a third of the shorter one adds;
//   two MMAs over one weight tile (t > 256) read it from shared memory twice, 0.065 us;
//   a tile with a single accumulator set (t > 240) exposes its drain between whole tiles, 2 us;
//   split K: the exchange costs 0.4 us + 10 ns per token column; with more than three quarters of the pairs at work on the few row tiles
//     of such a shape a step takes 15 % longer (one partly filled pass of split 1: 7 %).
double band_cost(int m_tok, int n_out, int K, int num_sms, int split, int t) {
  const int k = (K + 127) / 128, pairs = num_sms / 2 > 0 ? num_sms / 2 : 1;
  const int tiles = ((n_out + 255) / 256) * ((m_tok + t - 1) / t);
  const double ks = (k + split - 1) / split, dbl = ks > 32 ? std::log2(ks / 32.0) : 0.0, fk = 1.0 + 0.08 * (dbl < 1.5 ? dbl : 1.5);
  auto step = [&](int n) { return (0.15 + 0.00102 * n) * (n > 160 ? fk : 1.0) + (n > 256 ? 0.065 : 0.0); };
  const double hbm = static_cast<double>(n_out) * K * 1.125 / 6.6e6;
  double comp, extra;
  if (split == 1) {
    const ItemPlan q = plan_items(tiles, t, pairs);
    const int passes = (q.n_full + pairs - 1) / pairs;
    const double crowd = (tiles <= pairs && 4 * tiles > 3 * pairs) ? 1.07 : 1.0;
    comp = k * (passes * step(t) + (q.n_tail ? step(q.t_tail) : 0.0)) * crowd;
    const int ring = 4 * ring_stages(t);
    const bool two_sets = 2 * t + ring <= 512, tail_own = q.n_tail > 0 && t + q.t_tail + ring <= 512;
    extra = 0.004 * t + (two_sets ? 0.0 : 2.0 * (passes - 1 + (q.n_tail > 0 && !tail_own ? 1 : 0)));
  } else {
    const int resident = clusters_resident(split, num_sms), waves = (tiles + resident - 1) / resident;
    const double crowd = 4 * tiles * split > 3 * pairs ? 1.15 : 1.0;
    comp = waves * ks * step(t) * crowd;
    extra = 0.4 + 0.010 * t + (waves - 1) * 5.0;
  }
  const double lo = comp < hbm ? comp : hbm, hi = comp < hbm ? hbm : comp;
  return 4.6 + hi + lo / 3.0 + extra;
}

}  // namespace

// Cheapest form for a shape: split 1 ... 4 and the token tile that cuts the tokens into equal blocks.
int pick_band_variant(int m_tok, int n_out, int K, int num_sms, double* cost_us) {
  constexpr int kForm[5] = {0, 6000, 7000, 9000, 8000};
  double best = 1e300;
  int pick = 0;
  const int pairs = num_sms / 2 > 0 ? num_sms / 2 : 1;
  for (int nb = (m_tok + kMaxTile - 1) / kMaxTile; nb <= (m_tok + 63) / 64; ++nb) {
    const int t = round16((m_tok + nb - 1) / nb);
    const int tiles = ((n_out + 255) / 256) * ((m_tok + t - 1) / t);
    for (int split = 1; split <= 4; ++split) {
      if (split > 1 && (K + 127) / 128 < 4 * split) continue;      // at least K = 512 per slice
      // fewer tiles than half the pairs: more, narrower token blocks do what slicing every tile would, with a deeper ring
      if (split == 1 && 2 * tiles <= pairs && t > 64) continue;
      const double c = band_cost(m_tok, n_out, K, num_sms, split, t);
      if (c < best) {
        best = c;
        pick = kForm[split] + t;
      }
    }
  }
  if (cost_us) *cost_us = best;
  return pick;
}

bool band_has_slices(int m_tok, int n_out, int num_sms, int variant) {
  const int t = variant % 1000, pairs = num_sms / 2 > 0 ? num_sms / 2 : 1;
  return variant < 7000 && t > 0 && plan_items(((n_out + 255) / 256) * ((m_tok + t - 1) / t), t, pairs).n_tail > 0;
}

int launch_sparse_gemm_band(const SparseGemmArgs& a, cudaStream_t stream) {
  const int split = a.force_bn >= 9000 ? 3 : a.force_bn >= 8000 ? 4 : a.force_bn >= 7000 ? 2 : 1, t = a.force_bn % 1000;
  if (a.K % 64 != 0 || a.K <= 0 || a.m_tok <= 0 || a.n_out <= 0) return kErrInvalid;
  if (a.n_out % 8 != 0 || a.ldx % 8 != 0 || a.ldy % 8 != 0) return kErrInvalid;
  if ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.values) | reinterpret_cast<uintptr_t>(a.meta) |
       reinterpret_cast<uintptr_t>(a.y)) & 15)
    return kErrInvalid;
  if (a.out_f32 || a.peer_y != nullptr) return kErrInvalid;
  if (t < 16 || t > kMaxTile || t % 16 != 0 || (a.K + 127) / 128 < split) return kErrInvalid;
  if (a.epi == kEpiSwiGLU) {
    if (a.n_out % 32 != 0 || (a.n_out / 2) % 8 != 0) return kErrInvalid;
    return launch_band<kEpiSwiGLU>(a, split, t, stream);
  }
  return launch_band<kEpiStore>(a, split, t, stream);
}

}  // namespace sfb200
