// Host-side Merkle helpers over the generic subtree kernel (merkle_impl.cuh).
// Templates live here so other translation units can commit with fused leaf
// functors (FRI folds, constraint quotients).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "merkle_impl.cuh"
#include "vs_common.cuh"

namespace vs {

// One level of parents: parents[i] = Blake2s(children[2i] || children[2i+1]).
int launch_hash_nodes(const uint32_t* children, uint32_t* parents, uint64_t n_parents, cudaStream_t st);

// Threads of a tile that is reduced to its root: one a leaf, at most MK_THREADS (the
// kernels' loops step by MK_THREADS, so a smaller block must cover the tile at once). The
// 2^10 tiles of 128 hashes behind a 2^20-leaf tile-root tree are then resident together.
inline unsigned merkle_tile_threads(uint32_t TL) { return std::min<unsigned>(MK_THREADS, std::max<unsigned>(32, 1u << TL)); }

// stop_log (<= TL): 2^stop_log roots per tile instead of one (merkle_subtree_kernel).
template <class Leaf>
int merkle_tile_roots(const Leaf& leaf, uint64_t n_leaves, uint32_t TL, uint32_t* roots, cudaStream_t st,
                      uint32_t stop_log = 0) {
  const unsigned smem = merkle_smem_bytes(TL);  // at most 48 KiB (TL <= 10): no opt-in needed
  const uint64_t tiles = (n_leaves + (1ull << TL) - 1) >> TL;
  if (stop_log > TL) stop_log = TL;
  const unsigned threads = stop_log ? MK_THREADS : merkle_tile_threads(TL);
  merkle_subtree_kernel<Leaf><<<(unsigned)tiles, threads, smem, st>>>(leaf, TL, n_leaves, roots, stop_log);
  VS_LAUNCHED("merkle_subtree_kernel");
  return VS_OK;
}

// Largest split a caller may set (vs_merkle_split_set): 2^8 roots left per 1024-leaf
// tile, the level where all 256 threads of a CTA still have a node.
constexpr uint32_t MK_MAX_SPLIT = 8;
// Process-wide split (vs_merkle_split_set); 0 leaves the choice to merkle_root_split.
uint32_t merkle_split();

// From 2^MK_WIDE leaves on, the rate of compressions bounds a root-only tree: its
// 1024-leaf tiles stop at 2^split roots, where a level still fills warps, and the next
// level takes them over. Below, the chain of dependent compressions does (log2(n)
// levels): tiles are smaller, so that every SM has some and a thread hashes one or two
// leaves in a row and not four.
constexpr uint32_t MK_WIDE = 20;
// Split of a wide tree of 2^L leaves when none is set: 7, the fastest (row-packed root
// of 34 x 2^26: 11.90 / 11.64 / 11.30 / 11.42 ms at 5 / 6 / 7 / 8), less where its
// roots would take more than 256 MB of scratch.
inline uint32_t merkle_default_split(uint32_t L) { return L <= 26 ? 7u : 33u - L; }
inline uint32_t merkle_root_split(uint32_t L) {
  const uint32_t s = merkle_split();
  return s ? s : merkle_default_split(L);
}
// Tile of a reduction level over 2^L leaves, or over 2^L hashes of the level before:
// 2^TL of them, reduced to 2^stop. Measured on whole roots (us, one 1024-leaf tile a CTA
// and one root a tile, then this rule; 34 / 16 columns): 2^12 leaves 43 -> 23 / 31 -> 23,
// 2^16 46 -> 33 / 36 -> 29, 2^18 74 -> 68 / 51 -> 47, 2^19 132 -> 109 / 84 -> 70. One CTA
// ends trees of up to 2^9 leaves (14.4 us with one column, 22.5 with 34; tiles of 2^7 and a
// second launch 18.5 and 22.5) and of 2^10 hashes (14.9; 16.4).
// Split 0, for callers with little scratch, leaves one root a tile from 2^18 on;
// MK_LEAST does at every size, which takes the least scratch (none up to 2^10 leaves).
constexpr uint32_t MK_LEAST = MK_MAX_SPLIT + 1;
struct MerkleTile {
  uint32_t TL, stop;
};
inline MerkleTile merkle_tile(uint32_t L, bool hashes, uint32_t split) {
  if (split == MK_LEAST) return {std::min<uint32_t>(L, MK_MAX_TL), 0};
  if (L <= (hashes ? 10u : 9u)) return {L, 0};
  if (L <= 14) return {7, 0};
  if (L <= 17) return {L - 7, 0};
  if (L < MK_WIDE) return split ? MerkleTile{L - 10, 7} : MerkleTile{MK_MAX_TL, 0};
  return {MK_MAX_TL, split};
}

// A forest's CTAs for tiles of at most 2^TL leaves; trees are added largest first.
inline void merkle_forest_add(MerkleForest& f, uint32_t TL, uint32_t log_n, const uint32_t* src, uint32_t* out) {
  f.log_n[f.n] = log_n;
  f.src[f.n] = src;
  f.out[f.n] = out;
  f.start[f.n + 1] = f.start[f.n] + (1u << (log_n - std::min(TL, log_n)));
  f.n++;
}
template <class Leaf>
int merkle_forest(const MerkleForest& f, uint32_t TL, cudaStream_t st) {
  if (!f.n) return VS_OK;
  merkle_forest_kernel<Leaf><<<f.start[f.n], MK_THREADS, merkle_smem_bytes(TL), st>>>(f, TL);
  VS_LAUNCHED("merkle_forest_kernel");
  return VS_OK;
}

// Words of scratch merkle_root needs for n_leaves leaves with split `split` (0 when
// one CTA does): the sum of the hash levels it writes, in the order it writes them
// (merkle_root follows the same sequence). hashes: the leaves are hashes already.
inline uint64_t merkle_scratch_words(uint64_t n_leaves, uint32_t split = 0, bool hashes = false) {
  uint64_t words = 0;
  uint32_t L = ilog2(n_leaves);
  for (;; hashes = true) {
    const MerkleTile t = merkle_tile(L, hashes, split);
    if (t.TL == L && !t.stop) return words;
    L -= t.TL - t.stop;
    words += 8ull << L;
  }
}
// Trees that keep their 1024-leaf tile roots: from 2^20 leaves the tiles stop at 2^sp
// roots and one launch over those brings them up to the tile roots. sp is the split set,
// or 7 (one 2^20-leaf tree of 16 columns 140 -> 119 us), and at most `most`: a prover
// that holds its scratch takes 5 (32 hashes a tile).
constexpr uint32_t MK_TILE_SPLIT_MAX = 5;
inline uint32_t merkle_tile_split(uint64_t n_leaves, uint32_t most = MK_TILE_SPLIT_MAX) {
  const uint32_t s = merkle_split();
  return n_leaves >= (1ull << 20) ? std::min<uint32_t>(s ? s : 7, most) : 0u;
}
// Subroot scratch of a tile-root tree of n_leaves leaves at split sp (0: none).
inline uint64_t merkle_tile_scratch_bytes(uint64_t n_leaves, uint32_t sp) {
  return sp ? ((n_leaves >> MK_MAX_TL) << sp) * 32 : 0;
}
// Tile roots of a 2^TL-leaf tiling through 2^sp subtree roots per tile, in `sub`
// (sp = 0: none). Same tile roots as merkle_tile_roots(leaf, n, TL, roots).
template <class Leaf>
int merkle_tile_roots_split(const Leaf& leaf, uint64_t n_leaves, uint32_t TL, uint32_t sp, uint32_t* roots,
                            uint32_t* sub, cudaStream_t st) {
  if (!sp) return merkle_tile_roots(leaf, n_leaves, TL, roots, st);
  VS_TRY(merkle_tile_roots(leaf, n_leaves, TL, sub, st, sp));
  // A tile's 2^sp subroots alone leave most lanes of its levels idle; while 2^10 CTAs
  // remain, one takes those of several tiles (graph proof of 2^24 rows 19.0 -> 18.1 ms,
  // of 2^26 70.2 -> 66.5).
  const uint32_t log_sub = ilog2((n_leaves >> TL) << sp);
  const uint32_t T = std::min<uint32_t>(MK_MAX_TL, std::max(sp, log_sub - std::min(log_sub, 10u)));
  return merkle_tile_roots(LeafHashes{sub}, 1ull << log_sub, T, roots, st, T - sp);
}

// Scratch that serves merkle_root at every split 0..MK_MAX_SPLIT.
inline uint64_t merkle_scratch_words_any(uint64_t n_leaves) {
  uint64_t w = 0;
  for (uint32_t sp = 0; sp <= MK_MAX_SPLIT; sp++) w = std::max(w, merkle_scratch_words(n_leaves, sp));
  return w;
}

// Root of a power-of-two tree whose leaves come from `leaf`. Intermediate tile
// roots go to `scratch` (merkle_scratch_words(n_leaves, split) words; when null it
// is allocated stream-ordered for the call; where that fails the tree is built with
// MK_LEAST instead). Each reduction level is written after the previous one, never in place. Levels of 2^MK_WIDE and more stop at 2^split roots
// per 1024-leaf tile (split <= MK_MAX_SPLIT); the root is the same for every split.
template <class Leaf>
int merkle_root(const Leaf& leaf, uint64_t n_leaves, uint32_t* d_root, cudaStream_t st, uint32_t* scratch = nullptr,
                uint32_t split = 0) {
  if (!is_pow2(n_leaves)) return set_error(VS_ERR_INVALID, "merkle: leaf count %llu is not a power of two",
                                           (unsigned long long)n_leaves);
  if (split > MK_MAX_SPLIT) return set_error(VS_ERR_INVALID, "merkle: split %u above %u", split, MK_MAX_SPLIT);
  constexpr bool hashes = std::is_same_v<Leaf, LeafHashes>;
  // A capture of a tree of one tile stays free of memory nodes, so that its graph may be
  // instantiated and launched more than once.
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (!scratch && n_leaves <= (1ull << MK_MAX_TL) && cudaStreamIsCapturing(st, &capture) != cudaSuccess) cudaGetLastError();
  if (capture != cudaStreamCaptureStatusNone) split = MK_LEAST;
  uint64_t words = merkle_scratch_words(n_leaves, split, hashes);
  uint32_t *level = scratch, *buf = nullptr;
  if (words && !scratch) {
    cudaError_t e = cudaMallocAsync((void**)&buf, words * 4, st);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();  // the refused allocation's error
      buf = nullptr;
      split = MK_LEAST;
      words = merkle_scratch_words(n_leaves, split, hashes);
      e = words ? cudaMallocAsync((void**)&buf, words * 4, st) : cudaSuccess;
    }
    VS_TRY(check_cuda(e, "merkle scratch"));
    level = buf;
  }
  uint32_t L = ilog2(n_leaves);
  MerkleTile t = merkle_tile(L, hashes, split);
  bool last = t.TL == L && !t.stop;
  int rc = merkle_tile_roots(leaf, n_leaves, t.TL, last ? d_root : level, st, t.stop);
  while (rc == VS_OK && !last) {
    L -= t.TL - t.stop;
    t = merkle_tile(L, true, split);
    last = t.TL == L && !t.stop;
    uint32_t* next = level + (8ull << L);
    rc = merkle_tile_roots(LeafHashes{level}, 1ull << L, t.TL, last ? d_root : next, st, t.stop);
    level = next;
  }
  if (buf) {
    cudaError_t e = cudaFreeAsync(buf, st);
    if (rc == VS_OK) rc = check_cuda(e, "merkle scratch free");
  }
  return rc;
}

}  // namespace vs
