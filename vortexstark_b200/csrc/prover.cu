// Fibonacci Circle-STARK prover entry point (src/prover.rs:192-233; the proof itself is
// batch_prover.cu's, as a batch of one), and the decommitment of trees that keep their
// 1024-leaf tile roots.
#include <algorithm>
#include <vector>

#include "batch_prover.h"
#include "fri_impl.cuh"
#include "host_math.h"
#include "merkle.h"
#include "prover.h"
#include "vs_common.cuh"

namespace vs {

// Recompute queried tiles and emit each query's TL intra-tile siblings.
template <class Leaf>
__global__ void __launch_bounds__(256) tile_paths_kernel(Leaf leaf, uint32_t TL, const uint64_t* __restrict__ tiles,
                                                         const uint64_t* __restrict__ q, uint32_t nq,
                                                         uint32_t* __restrict__ out) {
  extern __shared__ uint32_t tp_sm[];  // levels 0..TL, row-major hashes
  const uint64_t tile = tiles[blockIdx.x];
  const uint32_t n0 = 1u << TL;
  for (uint32_t i = threadIdx.x; i < n0; i += blockDim.x) {
    uint32_t hh[8];
    leaf((tile << TL) + i, hh);
    for (int w = 0; w < 8; w++) tp_sm[8 * i + w] = hh[w];
  }
  __syncthreads();
  uint32_t off = 0, cnt = n0;
  for (uint32_t k = 1; k <= TL; k++) {
    const uint32_t* prev = tp_sm + 8 * off;
    uint32_t* cur = tp_sm + 8 * (off + cnt);
    for (uint32_t i = threadIdx.x; i < cnt / 2; i += blockDim.x) {
      uint32_t hh[8];
      b2s_node(hh, prev + 16 * i, prev + 16 * i + 8);
      for (int w = 0; w < 8; w++) cur[8 * i + w] = hh[w];
    }
    off += cnt;
    cnt >>= 1;
    __syncthreads();
  }
  for (uint32_t qi = threadIdx.x; qi < nq; qi += blockDim.x) {
    if ((q[qi] >> TL) != tile) continue;
    uint32_t intra = (uint32_t)(q[qi] & (n0 - 1));
    uint32_t lo = 0, lc = n0;
    for (uint32_t k = 0; k < TL; k++) {
      uint32_t sib = (intra >> k) ^ 1;
      for (int w = 0; w < 8; w++) out[((uint64_t)qi * TL + k) * 8 + w] = tp_sm[8 * (lo + sib) + w];
      lo += lc;
      lc >>= 1;
    }
  }
}

// Siblings above the tile level from the resident layers.
__global__ void upper_paths_kernel(const uint32_t* const* __restrict__ layers, uint32_t n_up,
                                   const uint64_t* __restrict__ q, uint32_t nq, uint32_t TL,
                                   uint32_t* __restrict__ out) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nq * n_up) return;
  uint32_t qi = t / n_up, k = t % n_up;
  uint64_t sib = ((q[qi] >> TL) >> k) ^ 1;
  for (int w = 0; w < 8; w++) out[((uint64_t)qi * n_up + k) * 8 + w] = layers[k][8 * sib + w];
}

// ------------------------------------------------------------------ host helpers
// Stream-ordered device allocations released together.
struct DevMem {
  cudaStream_t st;
  std::vector<void*> ptrs;
  explicit DevMem(cudaStream_t s) : st(s) {}
  ~DevMem() { for (void* p : ptrs) cudaFreeAsync(p, st); }
  template <class T>
  int alloc(T** out, uint64_t count) {
    void* p = nullptr;
    cudaError_t e = cudaMallocAsync(&p, std::max<uint64_t>(count, 1) * sizeof(T), st);
    if (e != cudaSuccess) return set_error(VS_ERR_OOM, "device allocation of %llu bytes: %s",
                                           (unsigned long long)(count * sizeof(T)), cudaGetErrorString(e));
    ptrs.push_back(p);
    *out = (T*)p;
    return VS_OK;
  }
};

struct DevTree {
  uint64_t n = 0;
  uint32_t TL = 0;
  std::vector<uint32_t*> layers;  // [0] tile roots ... back() = root
};

template <class Leaf>
static int tree_paths(const Leaf& leaf, const DevTree& t, const std::vector<uint64_t>& idx,
                      std::vector<std::vector<h::Hash>>& paths, DevMem& mem, cudaStream_t st) {
  const uint32_t nq = (uint32_t)idx.size();
  std::vector<uint64_t> tiles;
  for (uint64_t i : idx) tiles.push_back(i >> t.TL);
  std::sort(tiles.begin(), tiles.end());
  tiles.erase(std::unique(tiles.begin(), tiles.end()), tiles.end());
  const uint32_t n_up = (uint32_t)t.layers.size() - 1;
  uint64_t *d_q, *d_tiles;
  uint32_t *d_tp, *d_up;
  const uint32_t** d_layers;
  VS_TRY(mem.alloc(&d_q, nq));
  VS_TRY(mem.alloc(&d_tiles, tiles.size()));
  VS_TRY(mem.alloc(&d_tp, (uint64_t)nq * t.TL * 8));
  VS_TRY(mem.alloc(&d_up, (uint64_t)nq * n_up * 8));
  VS_TRY(mem.alloc(&d_layers, t.layers.size()));
  VS_CUDA(cudaMemcpyAsync(d_q, idx.data(), nq * 8, cudaMemcpyHostToDevice, st));
  VS_CUDA(cudaMemcpyAsync(d_tiles, tiles.data(), tiles.size() * 8, cudaMemcpyHostToDevice, st));
  VS_CUDA(cudaMemcpyAsync(d_layers, t.layers.data(), t.layers.size() * sizeof(void*), cudaMemcpyHostToDevice, st));
  if (t.TL > 0) {
    const unsigned smem = (unsigned)(((2u << t.TL) - 1) * 32);
    if (smem > 48 * 1024)
      VS_CUDA(cudaFuncSetAttribute(tile_paths_kernel<Leaf>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    tile_paths_kernel<Leaf><<<(unsigned)tiles.size(), 256, smem, st>>>(leaf, t.TL, d_tiles, d_q, nq, d_tp);
    VS_LAUNCHED("tile_paths_kernel");
  }
  if (n_up) {
    upper_paths_kernel<<<blocks_for((uint64_t)nq * n_up, 128), 128, 0, st>>>(d_layers, n_up, d_q, nq, t.TL, d_up);
    VS_LAUNCHED("upper_paths_kernel");
  }
  std::vector<uint32_t> htp((uint64_t)nq * t.TL * 8), hup((uint64_t)nq * n_up * 8);
  if (!htp.empty()) VS_CUDA(cudaMemcpyAsync(htp.data(), d_tp, htp.size() * 4, cudaMemcpyDeviceToHost, st));
  if (!hup.empty()) VS_CUDA(cudaMemcpyAsync(hup.data(), d_up, hup.size() * 4, cudaMemcpyDeviceToHost, st));
  VS_CUDA(cudaStreamSynchronize(st));
  paths.assign(nq, {});
  for (uint32_t q = 0; q < nq; q++) {
    auto& p = paths[q];
    for (uint32_t k = 0; k < t.TL; k++) { h::Hash x; std::copy_n(&htp[((uint64_t)q * t.TL + k) * 8], 8, x.begin()); p.push_back(x); }
    for (uint32_t k = 0; k < n_up; k++) { h::Hash x; std::copy_n(&hup[((uint64_t)q * n_up + k) * 8], 8, x.begin()); p.push_back(x); }
  }
  return VS_OK;
}

}  // namespace vs

using namespace vs;

extern "C" int vs_prove_fib(uint32_t a, uint32_t b, uint32_t log_n, uint8_t* h_out, uint64_t cap, uint64_t* out_len,
                            vs_stream_t stream) {
  clear_error();
  if (log_n < 4 || log_n + BLOWUP_BITS > 30) return set_error(VS_ERR_INVALID, "log_n %u outside [4, 28]", log_n);
  if (a >= h::P || b >= h::P) return set_error(VS_ERR_INVALID, "public inputs must be canonical M31");
  return BatchProver::prove_once(a, b, log_n, h_out, cap, out_len, (cudaStream_t)stream);
}

// ------------------------------------------------------------------ decommitment of tile-rooted trees
namespace vs {
// out[q * n_cols + c] = cols[c][idx[q]]
__global__ void gather_cols_kernel(const uint32_t* const* __restrict__ cols, uint32_t n_cols,
                                   const uint64_t* __restrict__ idx, uint32_t nq, uint32_t* __restrict__ out) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nq * n_cols) return;
  const uint32_t q = t / n_cols, c = t % n_cols;
  out[t] = cols[c][idx[q]];
}

// Auth paths of a tree whose 1024-leaf tile roots are resident: the levels above
// the tiles are rebuilt from the tile roots, the queried tiles from their leaves.
template <class Leaf>
static int tile_tree_paths(const Leaf& leaf, uint32_t log_n, const uint32_t* d_tile_roots,
                           const std::vector<uint64_t>& idx, std::vector<std::vector<h::Hash>>& paths, DevMem& mem,
                           cudaStream_t st) {
  DevTree t;
  t.n = 1ull << log_n;
  t.TL = std::min<uint32_t>(MK_MAX_TL, log_n);
  uint64_t cnt = t.n >> t.TL;
  t.layers.push_back(const_cast<uint32_t*>(d_tile_roots));
  while (cnt > 1) {
    uint32_t* par = nullptr;
    VS_TRY(mem.alloc(&par, (cnt / 2) * 8));
    VS_TRY(launch_hash_nodes(t.layers.back(), par, cnt / 2, st));
    t.layers.push_back(par);
    cnt /= 2;
  }
  return tree_paths(leaf, t, idx, paths, mem, st);
}
}  // namespace vs

extern "C" int vs_tile_tree_paths(uint32_t leaf_kind, const uint32_t* const* h_cols, uint32_t n_cols,
                                  uint32_t log_n_leaves, const uint32_t* d_tile_roots, const uint64_t* h_indices,
                                  uint32_t n_indices, uint32_t* h_values, uint32_t* h_paths, vs_stream_t stream) {
  clear_error();
  cudaStream_t st = (cudaStream_t)stream;
  if (!h_cols || !d_tile_roots || (n_indices && (!h_indices || !h_paths)))
    return set_error(VS_ERR_INVALID, "vs_tile_tree_paths: null argument");
  if (leaf_kind == VS_LEAF_SOA4 ? n_cols != 4 : (leaf_kind != VS_LEAF_CAPPED || n_cols == 0 || n_cols > 16))
    return set_error(VS_ERR_INVALID, "vs_tile_tree_paths: leaf kind %u with %u columns", leaf_kind, n_cols);
  if (log_n_leaves > 30) return set_error(VS_ERR_INVALID, "vs_tile_tree_paths: log_n_leaves %u", log_n_leaves);
  for (uint32_t c = 0; c < n_cols; c++)
    if (!h_cols[c]) return set_error(VS_ERR_INVALID, "vs_tile_tree_paths: null column %u", c);
  const uint64_t n = 1ull << log_n_leaves;
  std::vector<uint64_t> idx(h_indices, h_indices + n_indices);
  for (uint64_t i : idx)
    if (i >= n) return set_error(VS_ERR_INVALID, "vs_tile_tree_paths: index %llu >= %llu", (unsigned long long)i,
                                 (unsigned long long)n);
  if (!n_indices) return VS_OK;
  DevMem mem(st);
  const uint32_t** d_cols = nullptr;
  VS_TRY(mem.alloc(&d_cols, n_cols));
  VS_CUDA(cudaMemcpyAsync(d_cols, h_cols, n_cols * sizeof(void*), cudaMemcpyHostToDevice, st));
  std::vector<std::vector<h::Hash>> paths;
  if (leaf_kind == VS_LEAF_SOA4)
    VS_TRY(tile_tree_paths(LeafSoa4{h_cols[0], h_cols[1], h_cols[2], h_cols[3]}, log_n_leaves, d_tile_roots, idx,
                           paths, mem, st));
  else
    VS_TRY(tile_tree_paths(LeafCapped{d_cols, nullptr, 0, n_cols}, log_n_leaves, d_tile_roots, idx, paths, mem, st));
  for (uint32_t q = 0; q < n_indices; q++)
    for (uint32_t k = 0; k < log_n_leaves; k++)
      std::copy_n(paths[q][k].data(), 8, h_paths + ((uint64_t)q * log_n_leaves + k) * 8);
  if (h_values) {
    uint64_t* d_idx;
    uint32_t* d_out;
    VS_TRY(mem.alloc(&d_idx, n_indices));
    VS_TRY(mem.alloc(&d_out, (uint64_t)n_indices * n_cols));
    VS_CUDA(cudaMemcpyAsync(d_idx, idx.data(), n_indices * 8, cudaMemcpyHostToDevice, st));
    gather_cols_kernel<<<blocks_for((uint64_t)n_indices * n_cols, 128), 128, 0, st>>>(d_cols, n_cols, d_idx, n_indices,
                                                                                   d_out);
    VS_LAUNCHED("gather_cols_kernel");
    VS_CUDA(cudaMemcpyAsync(h_values, d_out, (uint64_t)n_indices * n_cols * 4, cudaMemcpyDeviceToHost, st));
    VS_CUDA(cudaStreamSynchronize(st));
  }
  return VS_OK;
}
