// FRI folds (drop-in for cuda/fri.cu) and the fused fold -> commit chain.
//
// A fold layer is one pass: each leaf of the new layer's Merkle tree is the
// folded value itself, so the fold runs inside the Merkle subtree kernel's leaf
// functor (it writes the folded value and hashes it in registers) and the layer
// is never re-read for its commitment.
#include <algorithm>

#include "fri_impl.cuh"
#include "merkle.h"
#include "twiddles.h"
#include "vs_field.cuh"

namespace vs {

// FRI layers of at most 2^fri_forest_log values take the shared launches of
// vs_fri_fold_commit. Measured (us, layers from 2^19 / 2^20 / 2^21 down): chains of 2^21
// 251 / 244 / 244, of 2^22 435 / 445 / 466, of 2^24 1496 / 1506 / 1524.
inline uint32_t fri_forest_log(uint32_t log_n) { return log_n <= 21 ? 20 : 19; }

__global__ void fold_line_kernel(Soa4Ptrs in, const uint32_t* __restrict__ tw, Soa4Out out, qm31 alpha,
                                 uint32_t half_n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= half_n) return;
  qm31 f0 = load_q(in.c, 2 * (uint64_t)i), f1 = load_q(in.c, 2 * (uint64_t)i + 1);
  qm31 r = fold_pair(f0, f1, alpha, tw[i]);
#pragma unroll
  for (int k = 0; k < 4; k++) out.c[k][i] = r.v[k];
}
__global__ void fold_circle_kernel(Soa4Out dst, Soa4Ptrs src, const uint32_t* __restrict__ tw, qm31 alpha, qm31 alpha_sq,
                                   uint32_t half_n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= half_n) return;
  qm31 f0 = load_q(src.c, 2 * (uint64_t)i), f1 = load_q(src.c, 2 * (uint64_t)i + 1);
  qm31 fp = fold_pair(f0, f1, alpha, tw[i]);
  qm31 prev{{dst.c[0][i], dst.c[1][i], dst.c[2][i], dst.c[3][i]}};
  qm31 r = qadd(qmul(prev, alpha_sq), fp);
#pragma unroll
  for (int k = 0; k < 4; k++) dst.c[k][i] = r.v[k];
}

// Several folds in one launch, for layers whose challenges are known: a CTA folds its
// 2^c consecutive values c times (or down to the last layer), the later folds from
// shared memory, and writes every layer's values. Layer l of the launch has
// 2^(log_in - 1 - l) values, planes that far apart at dst[l].
constexpr int FOLD_CHAIN = 10;
struct FoldChain {
  const uint32_t* src[4];
  uint32_t log_in, n, c;
  const uint32_t* tw[FOLD_CHAIN];
  qm31 alpha[FOLD_CHAIN];
  uint32_t* dst[FOLD_CHAIN];
  uint32_t* last;  // 8 values of the chain's end, limbs together (or null)
};
__global__ void __launch_bounds__(256) fold_chain_kernel(FoldChain p) {
  __shared__ __align__(8) uint32_t sm[2][4][1 << (FOLD_CHAIN - 1)];
  // a thread's first twiddle of a layer, fetched a layer ahead
  uint32_t tw_next = 0;
  auto fetch_tw = [&](uint32_t l) {
    if (l >= p.n) return;
    const uint32_t cnt = 1u << (p.c - 1 - l);
    if (threadIdx.x < cnt) tw_next = __ldg(p.tw[l] + (uint64_t)blockIdx.x * cnt + threadIdx.x);
  };
  fetch_tw(0);
  for (uint32_t l = 0; l < p.n; l++) {
    const uint32_t tw_first = tw_next;
    fetch_tw(l + 1);
    const uint32_t cnt = 1u << (p.c - 1 - l);              // this CTA's values of layer l
    const uint64_t base = (uint64_t)blockIdx.x * cnt, size = 1ull << (p.log_in - 1 - l);
    const uint32_t(*in)[1 << (FOLD_CHAIN - 1)] = sm[(l + 1) & 1];
    for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) {
      qm31 f0, f1;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint2 w = l == 0 ? ld2(p.src[k] + 2 * (base + i)) : *reinterpret_cast<const uint2*>(&in[k][2 * i]);
        f0.v[k] = w.x;
        f1.v[k] = w.y;
      }
      const qm31 r = fold_pair(f0, f1, p.alpha[l], i == threadIdx.x ? tw_first : __ldg(p.tw[l] + base + i));
#pragma unroll
      for (int k = 0; k < 4; k++) {
        sm[l & 1][k][i] = r.v[k];
        p.dst[l][k * size + base + i] = r.v[k];
        if (p.last && l + 1 == p.n) p.last[4 * (base + i) + k] = r.v[k];
      }
    }
    __syncthreads();
  }
}

}  // namespace vs

using namespace vs;

extern "C" {

void cuda_fold_line_soa(const uint32_t* in0, const uint32_t* in1, const uint32_t* in2, const uint32_t* in3,
                        const uint32_t* tw, uint32_t* out0, uint32_t* out1, uint32_t* out2, uint32_t* out3,
                        const uint32_t* alpha, uint32_t half_n) {
  if (!half_n) return;
  fold_line_kernel<<<blocks_for(half_n, 256), 256>>>(Soa4Ptrs{{in0, in1, in2, in3}}, tw, Soa4Out{{out0, out1, out2, out3}},
                                                     qm31{{alpha[0], alpha[1], alpha[2], alpha[3]}}, half_n);
  check_cuda(cudaGetLastError(), "cuda_fold_line_soa");
}

void cuda_fold_circle_into_line_soa(uint32_t* dst0, uint32_t* dst1, uint32_t* dst2, uint32_t* dst3,
                                    const uint32_t* src0, const uint32_t* src1, const uint32_t* src2,
                                    const uint32_t* src3, const uint32_t* tw, const uint32_t* alpha,
                                    const uint32_t* alpha_sq, uint32_t half_n) {
  if (!half_n) return;
  fold_circle_kernel<<<blocks_for(half_n, 256), 256>>>(Soa4Out{{dst0, dst1, dst2, dst3}}, Soa4Ptrs{{src0, src1, src2, src3}},
                                                       tw, qm31{{alpha[0], alpha[1], alpha[2], alpha[3]}},
                                                       qm31{{alpha_sq[0], alpha_sq[1], alpha_sq[2], alpha_sq[3]}}, half_n);
  check_cuda(cudaGetLastError(), "cuda_fold_circle_into_line_soa");
}

int vs_fri_fold_commit(const uint32_t* d_src, uint32_t log_n, const uint32_t* h_alphas, uint32_t* d_work,
                       uint32_t* d_roots, uint32_t* d_last, vs_stream_t stream) {
  clear_error();
  cudaStream_t st = (cudaStream_t)stream;
  if (!d_src || !h_alphas || !d_work || !d_roots || !d_last) return set_error(VS_ERR_INVALID, "vs_fri_fold_commit: null");
  if (log_n < 4 || log_n > 30) return set_error(VS_ERR_INVALID, "vs_fri_fold_commit: log_n %u out of range", log_n);
  const uint64_t N = 1ull << log_n;
  const uint32_t layers = log_n - 3;
  // Large layers: each fold is fused with the hashing of its tiles (the folded values
  // are not read again). Small ones: their challenges are known, so their folds run
  // first, several to a launch, and their trees share launches, as do the upper
  // levels of all trees. Taken alone, a small layer is two launches that leave the
  // chip idle (about 30 us at any size below 2^17).
  const uint32_t n_big = log_n - 1 > fri_forest_log(log_n) ? log_n - 1 - fri_forest_log(log_n) : 0;
  const uint32_t split = std::min<uint32_t>(merkle_root_split(log_n), 5);
  const uint32_t small_log = log_n - 1 - n_big;  // log2 of the first small layer
  const uint32_t TL = small_log <= 9 ? 9 : std::min<uint32_t>(MK_MAX_TL, std::max<uint32_t>(8, small_log - 8));
  // hash levels of each tree: its tile roots, then the roots of every 1024 of those
  uint64_t words = 0, at[MK_FOREST][3];
  uint32_t tile_log[MK_FOREST];
  for (uint32_t l = 0; l < layers; l++) {
    const uint32_t L = log_n - 1 - l;
    tile_log[l] = l < n_big ? L - MK_MAX_TL + split : L - std::min(TL, L);
    uint32_t log = tile_log[l];
    for (int k = 0; k < 3 && log; k++, log = log > MK_MAX_TL ? log - MK_MAX_TL : 0) {
      at[l][k] = words;
      words += 8ull << log;
    }
  }
  uint32_t* h = nullptr;
  VS_CUDA(cudaMallocAsync((void**)&h, words * 4, st));
  auto run = [&]() -> int {
    const uint32_t* src[4] = {d_src, d_src + N, d_src + 2 * N, d_src + 3 * N};
    uint32_t* val[MK_FOREST];  // layer l's values: 4 planes of 2^(log_n-1-l) words, one layer after the other
    const uint32_t* tw[MK_FOREST];
    for (uint32_t l = 0; l < layers; l++) {
      val[l] = l ? val[l - 1] + (4ull << (log_n - l)) : d_work;
      VS_TRY(get_fold_twiddles(l == 0 ? COSET_HALF_COSET : COSET_HALF_ODDS, log_n - l, &tw[l], st));
    }
    auto alpha = [&](uint32_t l) { return qm31{{h_alphas[4 * l], h_alphas[4 * l + 1], h_alphas[4 * l + 2], h_alphas[4 * l + 3]}}; };
    for (uint32_t l = 0; l < n_big; l++) {
      const uint64_t half = N >> (l + 1);
      LeafFold leaf{};
      for (int k = 0; k < 4; k++) { leaf.src.c[k] = src[k]; leaf.dst.c[k] = val[l] + k * half; src[k] = leaf.dst.c[k]; }
      leaf.tw = tw[l];
      leaf.alpha = alpha(l);
      VS_TRY(merkle_tile_roots(leaf, half, MK_MAX_TL, h + at[l][0], st, split));
    }
    for (uint32_t l = n_big; l < layers;) {
      FoldChain p{};
      for (int k = 0; k < 4; k++) p.src[k] = src[k];
      p.log_in = log_n - l;
      p.c = std::min<uint32_t>(FOLD_CHAIN, p.log_in);
      p.n = std::min(p.c, layers - l);
      for (uint32_t i = 0; i < p.n; i++) { p.tw[i] = tw[l + i]; p.alpha[i] = alpha(l + i); p.dst[i] = val[l + i]; }
      l += p.n;
      if (l == layers) p.last = d_last;
      fold_chain_kernel<<<1u << (p.log_in - p.c), 256, 0, st>>>(p);
      VS_LAUNCHED("fold_chain_kernel");
      for (int k = 0; k < 4; k++) src[k] = val[l - 1] + (uint64_t)k * (N >> l);
    }
    MerkleForest leaves{};
    for (uint32_t l = n_big; l < layers; l++)
      merkle_forest_add(leaves, TL, log_n - 1 - l, val[l], tile_log[l] ? h + at[l][0] : d_roots + 8 * l);
    VS_TRY(merkle_forest<LeafSoa4>(leaves, TL, st));
    // trees of more than 1024 hashes first lose ten levels, then all end together
    uint32_t log[MK_FOREST], most = 0;
    int k_of[MK_FOREST] = {};
    for (uint32_t l = 0; l < layers; l++) most = std::max(most, log[l] = tile_log[l]);
    for (; most > MK_MAX_TL; most -= MK_MAX_TL) {
      MerkleForest mid{};
      for (uint32_t l = 0; l < layers; l++) {
        if (log[l] <= MK_MAX_TL) continue;
        merkle_forest_add(mid, MK_MAX_TL, log[l], h + at[l][k_of[l]], h + at[l][k_of[l] + 1]);
        k_of[l]++;
        log[l] -= MK_MAX_TL;
      }
      VS_TRY(merkle_forest<LeafHashes>(mid, MK_MAX_TL, st));
    }
    MerkleForest top{};
    for (uint32_t l = 0; l < layers; l++)
      if (log[l]) merkle_forest_add(top, MK_MAX_TL, log[l], h + at[l][k_of[l]], d_roots + 8 * l);
    return merkle_forest<LeafHashes>(top, MK_MAX_TL, st);
  };
  int rc = run();
  cudaError_t e = cudaFreeAsync(h, st);
  if (rc == VS_OK) rc = check_cuda(e, "fri scratch free");
  return rc;
}

}  // extern "C"
