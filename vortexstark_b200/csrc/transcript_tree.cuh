// Committed trees followed by their Fiat-Shamir step on the device, for provers whose next
// challenge depends on the root: the launch that finishes a tree also mixes its root and
// draws the challenge, and the last FRI layers run in one launch. Trees of several equal
// jobs share the launches (batch_prover.cu); a single transcript is a batch of one.
#pragma once
#include <algorithm>
#include <cstdint>

#include "channel_dev.cuh"
#include "fri_impl.cuh"
#include "merkle.h"
#include "prover.h"

namespace vs {

// What a job's channel does with a finished tree: mix the root (copied into the job's
// arena) and, when alpha_off >= 0, draw a challenge into the job's alpha slots.
struct ChannelStep {
  ChanDev* ch;
  int reset;
  uint32_t* arena;
  uint64_t words, arena_off;
  uint32_t* alpha;
  uint32_t astride;
  int alpha_off;
};
// One block into the chaining state h; h (8 words) and m (16 words) in shared memory.
// Out of line: the few compressions of a channel step share one copy of the code.
static __device__ __noinline__ void channel_compress(uint32_t* h, const uint32_t* m, uint32_t t, bool last) {
  uint32_t hh[8], mm[16];
#pragma unroll
  for (int i = 0; i < 8; i++) hh[i] = h[i];
#pragma unroll
  for (int i = 0; i < 16; i++) mm[i] = m[i];
  b2s_compress(hh, mm, t, last);
#pragma unroll
  for (int i = 0; i < 8; i++) h[i] = hh[i];
}
// Mixes `root` into the state in blk[0..8) and, with `draw`, leaves a challenge in h[0..4).
// Run by one thread on shared memory: root and h 8 words, blk 16. Returns the draws made,
// 0 when 64 were not enough.
__device__ __forceinline__ uint32_t channel_mix_draw(uint32_t* blk, uint32_t* h, const uint32_t* root, bool draw) {
#pragma unroll
  for (int i = 0; i < 8; i++) blk[8 + i] = root[i];
  b2s_init(h);
  channel_compress(h, blk, 64u, true);  // state || digest
#pragma unroll
  for (int i = 0; i < 8; i++) blk[i] = h[i];
  if (!draw) return 0;
#pragma unroll
  for (int i = 9; i < 16; i++) blk[i] = 0;
  for (uint32_t draws = 1; draws <= 64; draws++) {  // until all words are below 2p
    blk[8] = draws - 1;
    b2s_init(h);
    channel_compress(h, blk, 37u, true);  // state || counter || 0x00
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 8; i++) ok = ok && h[i] < 2u * VS_P;
    if (!ok) continue;
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] %= VS_P;
    return draws;
  }
#pragma unroll
  for (int i = 0; i < 4; i++) h[i] = 0;
  return 0;
}
// Run by one thread; the root (8 words) and 24 words of scratch are in shared memory.
__device__ __forceinline__ void channel_step(const ChannelStep& s, uint32_t j, const uint32_t* root, uint32_t* scratch) {
  uint32_t *blk = scratch, *h = scratch + 16;
  ChanDev* c = s.ch + j;
  uint32_t* ar = s.arena + (uint64_t)j * s.words + s.arena_off;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    ar[i] = root[i];
    blk[i] = s.reset ? 0u : c->state[i];
  }
  const bool draw = s.alpha_off >= 0;
  const uint32_t draws = channel_mix_draw(blk, h, root, draw);
#pragma unroll
  for (int i = 0; i < 8; i++) c->state[i] = blk[i];
  for (int i = 0; draw && i < 4; i++) s.alpha[(uint64_t)j * s.astride + s.alpha_off + i] = h[i];
  c->n_draws = draws;
  if (s.reset) c->error = 0;
  if (draw && !draws) c->error = 1;
}

// One CTA per tile of 2^TL hashes of tree level k (leaves: k = 0): every kept level
// above, up to the tile's root. When the tile is a whole tree (tile = job), its channel
// step follows in the same launch.
template <class Leaf>
__global__ void __launch_bounds__(MK_THREADS) channel_tile_kernel(Leaf leaf, TreeLevels t, uint32_t k, uint32_t TL,
                                                                 ChannelStep step) {
  extern __shared__ uint32_t mk_sm[];
  const uint64_t base = (uint64_t)blockIdx.x << TL;
  uint32_t* root = merkle_tile_reduce(leaf, TL, base, ~0ull, 1, mk_sm, KeepLevels{t, blockIdx.x, k + TL});
  if (k + TL == t.m && threadIdx.x == 0) channel_step(step, blockIdx.x, root, root + 8);
}

// The last FRI layers (2^TAIL_LOG values and fewer), one CTA per job: folds from shared
// memory, trees and challenges without leaving the SM. As separate launches each of these
// layers took about 12 us.
// Layer l has 2^(log_eval-1-l) values; its challenge is at alpha0 + 4 l of the job's slots.
constexpr uint32_t TAIL_LOG = 9;
constexpr int TAIL_MAXF = 28;
constexpr uint32_t TAIL_TILE_WORDS = 12u << TAIL_LOG;  // merkle_smem_bytes(TAIL_LOG) / 4
struct FriTail {
  uint32_t first, nf, log_eval;        // layers first .. nf - 1
  uint32_t alpha0;
  const uint32_t* tw[TAIL_MAXF];
  const uint32_t* in[4];               // what layer first folds: planes [jobs][2^(log_eval-first)]
  uint32_t* fri[TAIL_MAXF][4];         // planes [jobs][2^(log_eval-1-l)]
  TreeLevels tree[TAIL_MAXF];
  ChannelStep step;                    // of layer first
  uint64_t a_last, a_q;                // QUERIES: last layer and query indices in the arena
  uint32_t* qidx;
};
// QUERIES: the last layer (eight values) is committed and mixed, and the queries drawn;
// otherwise it is only folded.
template <bool QUERIES>
__global__ void __launch_bounds__(MK_THREADS, 2) fri_tail_kernel(FriTail p) {
  extern __shared__ __align__(16) uint32_t tail_sm[];
  uint32_t(*val)[4][1 << TAIL_LOG] = reinterpret_cast<uint32_t(*)[4][1 << TAIL_LOG]>(tail_sm);
  uint32_t* sm = tail_sm + 2 * 4 * (1 << TAIL_LOG);
  uint32_t *blk = sm + TAIL_TILE_WORDS, *h = blk + 48;  // the channel's blocks and digest
  const uint32_t j = blockIdx.x;
  // the channel state stays in shared memory between layers; a layer's challenge is h
  ChanDev* c = p.step.ch + j;
  uint32_t* al = p.step.alpha + (uint64_t)j * p.step.astride + p.alpha0;
  uint32_t* ar = p.step.arena + (uint64_t)j * p.step.words;
  if (threadIdx.x < 8) blk[threadIdx.x] = c->state[threadIdx.x];
  if (threadIdx.x < 4) h[threadIdx.x] = al[4 * p.first + threadIdx.x];
  __syncthreads();
  for (uint32_t l = p.first; l < p.nf; l++) {
    const uint32_t m = p.log_eval - 1 - l, half = 1u << m;
    const qm31 alpha{{h[0], h[1], h[2], h[3]}};
    auto fold = [&](uint32_t i, uint32_t w[4]) {
      qm31 f0, f1;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint2 x = l == p.first ? ld2(p.in[k] + 2 * ((uint64_t)j * half + i))
                                     : *reinterpret_cast<const uint2*>(&val[(l + 1) & 1][k][2 * i]);
        f0.v[k] = x.x;
        f1.v[k] = x.y;
      }
      const qm31 r = fold_pair(f0, f1, alpha, __ldg(p.tw[l] + i));
#pragma unroll
      for (int k = 0; k < 4; k++) {
        val[l & 1][k][i] = w[k] = r.v[k];
        p.fri[l][k][(uint64_t)j * half + i] = r.v[k];
      }
    };
    if (!QUERIES && l + 1 == p.nf) {
      uint32_t w[4];
      if (threadIdx.x < half) fold(threadIdx.x, w);
      return;
    }
    uint32_t* root = merkle_tile_reduce(
        [&](uint64_t i, uint32_t h[8]) {
          uint32_t w[16] = {0};
          fold((uint32_t)i, w);
          b2s_single(h, w, 4);
        },
        m, 0, half, 1, sm, KeepLevels{p.tree[l], j, m});
    if (threadIdx.x == 0) {  // mix the root; the next layer's challenge
      const bool draw = l + 1 < p.nf;
      const uint32_t draws = channel_mix_draw(blk, h, root, draw);
      for (int i = 0; i < 8; i++) ar[p.step.arena_off + 8 * (l - p.first) + i] = root[i];
      for (int i = 0; draw && i < 4; i++) al[4 * (l + 1) + i] = h[i];
      for (int i = 0; i < 8; i++) c->state[i] = blk[i];
      c->n_draws = draws;
      if (draw && !draws) c->error = 1;
    }
    __syncthreads();  // challenge before the next layer
  }
  // mix_felts(last layer): state || 8 values, 160 bytes
  uint32_t(*v)[1 << TAIL_LOG] = val[(p.nf - 1) & 1];
  if (threadIdx.x >= 8 && threadIdx.x < 48) {
    const uint32_t w = threadIdx.x;
    blk[w] = w < 40 ? v[(w - 8) & 3][(w - 8) >> 2] : 0u;
  }
  if (threadIdx.x < 32) ar[p.a_last + threadIdx.x] = v[threadIdx.x & 3][threadIdx.x >> 2];
  __syncthreads();
  if (threadIdx.x == 0) {
    b2s_init(h);
    for (uint32_t b = 0; b < 3; b++) channel_compress(h, blk + 16 * b, b < 2 ? 64u * (b + 1) : 160u, b == 2);
    for (int i = 0; i < 8; i++) c->state[i] = h[i];
    c->n_draws = N_QUERIES;
  }
  __syncthreads();
  // the q-th draw after the mix squeezes with counter q
  if (threadIdx.x < N_QUERIES) {
    ChanDev d;
#pragma unroll
    for (int i = 0; i < 8; i++) d.state[i] = h[i];
    d.n_draws = threadIdx.x;
    const uint32_t q = ch_draw_pow2(d, p.log_eval);
    p.qidx[j * N_QUERIES + threadIdx.x] = q;
    ar[p.a_q + threadIdx.x] = q;
  }
}

template <class Leaf>
int channel_tiles(const Leaf& leaf, const TreeLevels& t, uint32_t k, uint32_t TL, uint32_t jobs, const ChannelStep& c,
                  cudaStream_t st) {
  // the channel step's 24 words follow the root, wherever the levels left it
  const unsigned smem = std::max(merkle_smem_bytes(TL), (8u << TL) * 4 + 128);
  channel_tile_kernel<Leaf><<<jobs << (t.m - k - TL), merkle_tile_threads(TL), smem, st>>>(leaf, t, k, TL, c);
  VS_LAUNCHED("channel_tile_kernel");
  return VS_OK;
}
// The levels above level k (kept), then the jobs' channel steps.
inline int channel_levels(const TreeLevels& t, uint32_t k, uint32_t jobs, const ChannelStep& c, cudaStream_t st) {
  while (k < t.m) {
    const uint32_t TL = std::min<uint32_t>(MK_MAX_TL, t.m - k);
    VS_TRY(channel_tiles(LeafHashes{t.level(k)}, t, k, TL, jobs, c, st));
    k += TL;
  }
  return VS_OK;
}
// First level a launch over the leaves of trees of 2^m leaves leaves to the next one
// (2^all leaves in all, below 2^MK_WIDE): enough tiles for the SMs, and at most 2^10 a
// tree, so that one more launch ends it; small trees end in the first.
inline uint32_t channel_leaf_tile(uint32_t m, uint32_t all) {
  if (m <= TAIL_LOG) return m;
  return std::max(merkle_tile(std::min(all, 17u), false, 0).TL, m - std::min<uint32_t>(m, MK_MAX_TL));
}
// `jobs` trees from their leaves: every kept level, then the channel steps.
template <class Leaf>
int commit_with_channel(const Leaf& leaf, const TreeLevels& t, uint32_t jobs, const ChannelStep& c, cudaStream_t st) {
  const uint32_t m = t.m, all = ilog2(jobs) + m;
  uint32_t k;
  if (all >= MK_WIDE) {  // bound by the rate of compressions: tiles stop at the lowest kept level
    const uint32_t TL = std::min<uint32_t>(MK_MAX_TL, m);
    VS_TRY(merkle_tile_roots(leaf, (uint64_t)jobs << m, TL, t.level(t.s), st, TL - t.s));
    k = t.s;
  } else {
    k = channel_leaf_tile(m, all);
    VS_TRY(channel_tiles(leaf, t, 0, k, jobs, c, st));
  }
  return channel_levels(t, k, jobs, c, st);
}
template <bool QUERIES>
int launch_fri_tail(FriTail& p, uint32_t jobs, cudaStream_t st) {
  for (int k = 0; k < 4 && !p.in[k]; k++) p.in[k] = p.fri[p.first - 1][k];
  const unsigned smem = 4 * (TAIL_TILE_WORDS + 2 * 4 * (1u << TAIL_LOG) + 56);  // 40 KiB: no opt-in needed
  fri_tail_kernel<QUERIES><<<jobs, MK_THREADS, smem, st>>>(p);
  VS_LAUNCHED("fri_tail_kernel");
  return VS_OK;
}

}  // namespace vs
