// Batched Fibonacci prover: many independent proofs of one trace size run as one
// CUDA graph in which every stage is a single kernel launch over all of them.
//
// The reference proves a batch one proof after another (ProverPipeline::prove_batch,
// src/prover.rs:2265-2270), and the graph-captured prover (prover_graph.cu) still
// issues one chain of small launches per proof. Here job j's buffers are the j-th
// slices of batch-wide arrays, so one launch covers every job:
//
//   * trace: blockIdx.y selects the job's public inputs;
//   * LDE: the jobs' traces are the columns of one multi-column native LDE;
//   * Merkle trees: job j's 2^m leaves are leaves [j 2^m, (j+1) 2^m) of one leaf
//     range, so tiles never straddle jobs and each stored level is the
//     concatenation of the jobs' levels (parents never straddle jobs either);
//   * fused quotient / fold leaves: the leaf functors split a global leaf index
//     into (job, index) and read the job's own challenges;
//   * Fiat-Shamir channel: the launch that ends a tree mixes its root and draws the
//     next challenge, one thread a job (transcript_tree.cuh);
//   * the FRI layers of 2^9 values and fewer, and the query draw (whose squeezes are
//     independent given the state): one launch, a CTA a job;
//   * decommitment: one launch over all trees, one warp per (job, query) gathers its
//     authentication path.
//
// Trees keep every level from level 3 up (eight-leaf groups; 6 in the trees of single
// proofs above 2^22 leaves): an authentication path is a gather of the stored
// siblings plus the recomputation of one group, instead of one 1024-leaf tile per
// query and tree as in the tile-root provers (the reference keeps whole trees at these sizes too,
// MerkleTree::commit, src/prover.rs:1764-1766). The arithmetic, transcript and
// proof layout are the graph prover's: every proof is byte-identical to
// vs_prove_fib's for the same (a, b, log_n).
#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "batch_prover.h"
#include "channel_dev.cuh"
#include "fri_impl.cuh"
#include "merkle.h"
#include "ntt.h"
#include "prover.h"
#include "prover_graph.h"
#include "transcript_tree.cuh"
#include "twiddles.h"
#include "vs_common.cuh"

namespace vs {

namespace {

constexpr int BMAXF = 28;  // FRI layers for log_eval <= 30
// Lowest kept level of a tree of 2^m leaves: an opened leaf's group of 2^s is hashed again.
// Eight-leaf groups cost 8 bytes a leaf; trees above 2^22 leaves keep 64-leaf groups (1
// byte a leaf), which one warp hashes in two steps.
constexpr uint32_t BGROUP_MAX = 6;
constexpr uint32_t group_log(uint32_t m) { return m > 22 ? BGROUP_MAX : (m < 3 ? m : 3); }
// 64-leaf groups in every tree, where the device has no room for more levels.
constexpr uint32_t group_most(uint32_t m) { return std::min(m, BGROUP_MAX); }

// ------------------------------------------------------------------ batched leaf functors
// Global leaf g of a batch of trees with 2^log_len leaves each: job g >> log_len,
// index g & (2^log_len - 1).
struct LeafFibQuotB {
  const uint32_t* e;      // [jobs][N] evaluations
  uint32_t log_n;         // log N
  const uint32_t* alpha;  // job j's quotient challenge at alpha + j * astride
  uint32_t astride;
  __device__ __forceinline__ qm31 q(uint64_t g) const {
    const uint64_t mask = (1ull << log_n) - 1, j = g >> log_n, i = g & mask;
    const uint32_t* ej = e + (j << log_n);
    const uint32_t* a = alpha + j * astride;
    const qm31 av{{__ldg(a), __ldg(a + 1), __ldg(a + 2), __ldg(a + 3)}};
    return qscale(av, sub(ej[(i + 2) & mask], add(ej[(i + 1) & mask], ej[i])));
  }
  __device__ __forceinline__ void operator()(uint64_t g, uint32_t out[8]) const {
    const qm31 r = q(g);
    uint32_t m[16] = {0};
    m[0] = r.v[0]; m[1] = r.v[1]; m[2] = r.v[2]; m[3] = r.v[3];
    b2s_single(out, m, 4);
  }
};

// Circle fold of the quotient (never materialised) into FRI layer 0.
struct LeafFoldQuotB {
  LeafFibQuotB quot;
  const uint32_t* tw;     // 2^log_half fold twiddles, shared by the jobs
  uint32_t log_half;
  const uint32_t* alpha;  // job j's fold challenge at alpha + j * astride
  uint32_t astride;
  uint32_t* dst[4];       // planes [jobs][2^log_half]
  __device__ __forceinline__ void operator()(uint64_t g, uint32_t out[8]) const {
    const uint64_t j = g >> log_half, i = g & ((1ull << log_half) - 1);
    const uint32_t* a = alpha + j * astride;
    const qm31 av{{__ldg(a), __ldg(a + 1), __ldg(a + 2), __ldg(a + 3)}};
    // 2g = j * 2^(log_half+1) + 2i: the job's own quotient values 2i and 2i + 1
    const qm31 r = fold_pair(quot.q(2 * g), quot.q(2 * g + 1), av, __ldg(tw + i));
#pragma unroll
    for (int k = 0; k < 4; k++) dst[k][g] = r.v[k];
    uint32_t m[16] = {0};
    m[0] = r.v[0]; m[1] = r.v[1]; m[2] = r.v[2]; m[3] = r.v[3];
    b2s_single(out, m, 4);
  }
};

// Line fold of FRI layer l - 1 (planes [jobs][2^(log_half+1)]) into layer l.
struct LeafFoldB {
  const uint32_t* src[4];
  uint32_t* dst[4];
  const uint32_t* tw;
  uint32_t log_half;
  const uint32_t* alpha;
  uint32_t astride;
  __device__ __forceinline__ void operator()(uint64_t g, uint32_t out[8]) const {
    const uint64_t j = g >> log_half, i = g & ((1ull << log_half) - 1);
    const uint32_t* a = alpha + j * astride;
    const qm31 av{{__ldg(a), __ldg(a + 1), __ldg(a + 2), __ldg(a + 3)}};
    const uint2 s0 = *reinterpret_cast<const uint2*>(src[0] + 2 * g);
    const uint2 s1 = *reinterpret_cast<const uint2*>(src[1] + 2 * g);
    const uint2 s2 = *reinterpret_cast<const uint2*>(src[2] + 2 * g);
    const uint2 s3 = *reinterpret_cast<const uint2*>(src[3] + 2 * g);
    const qm31 r = fold_pair(qm31{{s0.x, s1.x, s2.x, s3.x}}, qm31{{s0.y, s1.y, s2.y, s3.y}}, av, __ldg(tw + i));
#pragma unroll
    for (int k = 0; k < 4; k++) dst[k][g] = r.v[k];
    uint32_t m[16] = {0};
    m[0] = r.v[0]; m[1] = r.v[1]; m[2] = r.v[2]; m[3] = r.v[3];
    b2s_single(out, m, 4);
  }
};

// ------------------------------------------------------------------ kernels
// Decommitment of every tree in one launch: blockIdx.y is the tree (trace, quotient, FRI
// layers), a warp takes one (job, query): the opened values and the authentication paths
// of leaf f (the query, or q >> (l+1) in FRI layer l) and of its sibling f ^ 1. Levels
// below s come from recomputing f's 2^s-leaf group, levels s..m-1 from the kept ones.
struct BDecommit {
  const uint32_t* eval;
  uint32_t log_eval, nf, jobs;
  const uint32_t* alpha;
  uint32_t astride;
  const uint32_t* qidx;
  uint32_t* arena;
  uint64_t words, a_tv, a_qv, a_fv[BMAXF], a_tree[2 + BMAXF];
  const uint32_t* fri[BMAXF][4];  // plane k of layer l: [jobs][2^(log_eval-1-l)]
  TreeLevels tree[2 + BMAXF];
};
__global__ void __launch_bounds__(256) batch_decommit_kernel(BDecommit p) {
  __shared__ __align__(16) uint32_t sm[8][(2 << BGROUP_MAX) * 8];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, y = blockIdx.y;
  const uint32_t wi = blockIdx.x * 8 + warp;
  if (wi >= p.jobs * N_QUERIES) return;  // uniform per warp
  const uint32_t j = wi / N_QUERIES, qi = wi % N_QUERIES;
  const TreeLevels t = p.tree[y];
  const uint32_t s = t.s, m = t.m, g = 1u << s;
  const uint32_t f = p.qidx[j * N_QUERIES + qi] >> (y < 2 ? 0 : y - 1);
  const uint32_t* al = p.alpha + (uint64_t)j * p.astride;
  // the words of leaf i of this job's tree
  auto words = [&](uint32_t i, uint32_t w[4]) {
    if (y == 0) {
      w[0] = p.eval[((uint64_t)j << m) + i];
      w[1] = w[2] = w[3] = 0;
    } else if (y == 1) {
      const uint32_t* e = p.eval + ((uint64_t)j << m);
      const uint32_t mask = (1u << m) - 1;
      const qm31 q = qscale(qm31{{al[0], al[1], al[2], al[3]}}, sub(e[(i + 2) & mask], add(e[(i + 1) & mask], e[i])));
#pragma unroll
      for (int k = 0; k < 4; k++) w[k] = q.v[k];
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) w[k] = p.fri[y - 2][k][((uint64_t)j << m) + i];
    }
  };
  uint32_t* ar = p.arena + (uint64_t)j * p.words;
  uint32_t* S = sm[warp];
  for (uint32_t x = lane; x < g; x += 32) {
    const uint32_t i = ((f >> s) << s) + x;
    uint32_t w[4], h[8], msg[16] = {0};
    words(i, w);
    if ((i ^ f) <= 1) {  // the query's leaf or its sibling: an opened value
      const uint32_t at = ((i ^ f) & 1 ? N_QUERIES : 0) + qi;
      if (y == 0) {
        ar[p.a_tv + at] = w[0];
      } else {
        uint32_t* o = ar + (y == 1 ? p.a_qv : p.a_fv[y - 2]) + 4 * at;
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = w[k];
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) msg[k] = w[k];
    b2s_single(h, msg, y == 0 ? 1 : 4);
#pragma unroll
    for (int k = 0; k < 8; k++) S[8 * x + k] = h[k];
  }
  __syncwarp();
  uint32_t lo = 0, cnt = g;
  for (uint32_t k = 1; k < s; k++) {
    if (lane < cnt / 2) {  // at most 32 nodes
      uint32_t h[8];
      b2s_node(h, S + 8 * (lo + 2 * lane), S + 8 * (lo + 2 * lane + 1));
#pragma unroll
      for (int w = 0; w < 8; w++) S[8 * (lo + cnt + lane) + w] = h[w];
    }
    __syncwarp();
    lo += cnt;
    cnt >>= 1;
  }
  uint32_t* out = ar + p.a_tree[y];
  // a lane copies one word: eight lanes a hash
  for (uint32_t x = lane >> 3; x < 2 * m; x += 4) {
    const uint32_t sd = x / m, k = x % m, i = f ^ sd;
    const uint32_t* src;
    if (k < s) src = S + 8 * (2 * g - (2 * g >> k) + (((i & (g - 1)) >> k) ^ 1));
    else src = t.level(k) + (((uint64_t)j << (m - k)) + ((i >> k) ^ 1)) * 8;
    uint32_t* path = out + (uint64_t)(sd * N_QUERIES + qi) * (1 + 8 * m);
    if (k == 0 && (lane & 7) == 0) path[0] = m;
    path[1 + 8 * k + (lane & 7)] = src[lane & 7];
  }
}

uint64_t align256(uint64_t b) { return (b + 255) & ~255ull; }

}  // namespace

// ------------------------------------------------------------------ the prover
struct BatchProver::Impl {
  uint32_t log_n = 0, log_eval = 0, nf = 0, cap = 0, astride = 0;
  uint64_t n = 0, N = 0, total = 0;
  uint32_t (*group)(uint32_t) = group_log;
  int device = 0;
  cudaStream_t st = nullptr, running = nullptr;
  uint32_t count = 0;  // jobs of the batch in flight
  uint8_t* mem = nullptr;
  uint32_t *h_ab = nullptr, *h_arena = nullptr;
  uint32_t *d_ab = nullptr, *d_trace = nullptr, *d_eval = nullptr, *d_alpha = nullptr, *d_qidx = nullptr,
           *d_arena = nullptr;
  ChanDev* d_ch = nullptr;
  TreeLevels trace_t{}, quot_t{}, fri_t[BMAXF] = {};
  uint32_t* fri[BMAXF][4] = {};
  ArenaLayout lay;
  std::map<uint32_t, cudaGraphExec_t> exec;  // per batch size

  ~Impl() {
    if (running) cudaStreamSynchronize(running);
    if (st) cudaStreamSynchronize(st);
    for (auto& kv : exec) cudaGraphExecDestroy(kv.second);
    if (mem) cudaFree(mem);
    if (h_arena) cudaFreeHost(h_arena);
    if (h_ab) cudaFreeHost(h_ab);
    if (st) cudaStreamDestroy(st);
  }

  // Assigns every device buffer inside one allocation at `base` (sizes only when
  // null); returns the bytes used.
  uint64_t carve(uint8_t* base) {
    uint64_t off = 0;
    auto take = [&](uint64_t bytes) -> uint8_t* {
      uint8_t* p = base ? base + off : nullptr;
      off += align256(std::max<uint64_t>(bytes, 4));
      return p;
    };
    d_ab = (uint32_t*)take(8ull * cap);
    d_trace = (uint32_t*)take(4 * n * cap);
    d_eval = (uint32_t*)take(4 * N * cap);
    d_alpha = (uint32_t*)take(4ull * astride * cap);
    d_qidx = (uint32_t*)take(4ull * N_QUERIES * cap);
    d_ch = (ChanDev*)take(sizeof(ChanDev) * cap);
    d_arena = (uint32_t*)take(4ull * lay.words * cap);
    for (uint32_t l = 0; l < nf; l++) {
      const uint64_t half = N >> (l + 1);
      for (int k = 0; k < 4; k++) fri[l][k] = (uint32_t*)take(4 * half * cap);
    }
    auto tree = [&](TreeLevels& t, uint32_t m) {
      t = TreeLevels{nullptr, cap, group(m), m};
      t.base = (uint32_t*)take(TreeLevels::bytes(cap, t.s, m));
    };
    tree(trace_t, log_eval);
    tree(quot_t, log_eval);
    for (uint32_t l = 0; l < nf; l++) tree(fri_t[l], log_eval - 1 - l);
    return off;
  }

  void plan(uint32_t ln, uint32_t c) {
    log_n = ln;
    log_eval = ln + BLOWUP_BITS;
    n = 1ull << ln;
    N = 1ull << log_eval;
    nf = log_eval - LOG_LAST_LAYER;
    cap = c;
    astride = 4 * (2 + nf);
    lay.plan(ln);
    total = carve(nullptr);
  }

  ChannelStep step(int reset, uint64_t arena_off, int alpha_off) const {
    return {d_ch, reset, d_arena, lay.words, arena_off, d_alpha, astride, alpha_off};
  }
  // The whole batch of b proofs, stream-ordered on st, from the public inputs in h_ab
  // to the arenas in h_arena.
  int enqueue(uint32_t b) {
    VS_CUDA(cudaMemcpyAsync(d_ab, h_ab, 8ull * b, cudaMemcpyHostToDevice, st));
    fib_trace_params_kernel<<<dim3(blocks_for(n, 256 * 32), b), 256, 0, st>>>(d_ab, d_trace, n);
    VS_LAUNCHED("fib_trace_params_kernel");
    VS_TRY(lde_cached(TW_NATIVE, d_trace, n, d_eval, N, b, log_n, BLOWUP_BITS, st));
    VS_TRY(commit_with_channel(LeafOne{d_eval}, trace_t, b, step(1, lay.root(0), 0), st));
    const LeafFibQuotB quot{d_eval, log_eval, d_alpha, astride};
    VS_TRY(commit_with_channel(quot, quot_t, b, step(0, lay.root(1), 4), st));
    FriTail tail{};
    for (uint32_t l = 0; l < nf; l++) {
      const uint32_t cur = log_eval - l;
      const uint32_t* tw = nullptr;
      VS_TRY(get_fold_twiddles(l == 0 ? COSET_HALF_COSET : COSET_HALF_ODDS, cur, &tw, st));
      const ChannelStep c = step(0, lay.root(2 + l), l + 1 < nf ? (int)(4 * (2 + l)) : -1);
      if (l == 0) {
        LeafFoldQuotB leaf{quot, tw, cur - 1, d_alpha + 4, astride, {fri[0][0], fri[0][1], fri[0][2], fri[0][3]}};
        VS_TRY(commit_with_channel(leaf, fri_t[0], b, c, st));
      } else if (cur - 1 > TAIL_LOG) {
        LeafFoldB leaf{{fri[l - 1][0], fri[l - 1][1], fri[l - 1][2], fri[l - 1][3]},
                       {fri[l][0], fri[l][1], fri[l][2], fri[l][3]}, tw, cur - 1, d_alpha + 4 * (1 + l), astride};
        VS_TRY(commit_with_channel(leaf, fri_t[l], b, c, st));
      } else if (!tail.first) {
        tail.first = l;
        tail.step = c;
      }
      tail.tw[l] = tw;
      tail.tree[l] = fri_t[l];
      for (int k = 0; k < 4; k++) tail.fri[l][k] = fri[l][k];
    }
    tail.nf = nf;
    tail.log_eval = log_eval;
    tail.a_last = lay.last;
    tail.a_q = lay.q;
    tail.qidx = d_qidx;
    tail.alpha0 = 4;
    VS_TRY(launch_fri_tail<true>(tail, b, st));
    BDecommit dp{};
    dp.eval = d_eval;
    dp.log_eval = log_eval;
    dp.nf = nf;
    dp.jobs = b;
    dp.alpha = d_alpha;
    dp.astride = astride;
    dp.qidx = d_qidx;
    dp.arena = d_arena;
    dp.words = lay.words;
    dp.a_tv = lay.tv;
    dp.a_qv = lay.qv;
    dp.tree[0] = trace_t;
    dp.tree[1] = quot_t;
    for (uint32_t y = 0; y < 2 + nf; y++) dp.a_tree[y] = lay.tree[y];
    for (uint32_t l = 0; l < nf; l++) {
      dp.tree[2 + l] = fri_t[l];
      dp.a_fv[l] = lay.fv[l];
      for (int k = 0; k < 4; k++) dp.fri[l][k] = fri[l][k];
    }
    batch_decommit_kernel<<<dim3(blocks_for((uint64_t)b * N_QUERIES, 8), 2 + nf), 256, 0, st>>>(dp);
    VS_LAUNCHED("batch_decommit_kernel");
    VS_CUDA(cudaMemcpyAsync(h_arena, d_arena, 4ull * lay.words * b, cudaMemcpyDeviceToHost, st));
    return VS_OK;
  }

  int graph_for(uint32_t b, cudaGraphExec_t* out) {
    auto it = exec.find(b);
    if (it != exec.end()) { *out = it->second; return VS_OK; }
    cudaGraph_t g = nullptr;
    VS_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    int rc = enqueue(b);
    cudaError_t e = cudaStreamEndCapture(st, &g);
    if (rc != VS_OK) { if (g) cudaGraphDestroy(g); return rc; }
    VS_CUDA(e);
    cudaGraphExec_t x = nullptr;
    e = cudaGraphInstantiate(&x, g, 0);
    cudaGraphDestroy(g);
    VS_CUDA(e);
    exec[b] = x;
    *out = x;
    return VS_OK;
  }

  int setup(uint32_t ln, uint32_t c) {
    plan(ln, c);
    VS_CUDA(cudaGetDevice(&device));
    VS_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    cudaError_t e = cudaMalloc((void**)&mem, total);
    if (e != cudaSuccess) {
      mem = nullptr;
      return set_error(VS_ERR_OOM, "batch prover workspace (%llu bytes): %s", (unsigned long long)total,
                       cudaGetErrorString(e));
    }
    carve(mem);
    VS_CUDA(cudaMallocHost((void**)&h_ab, 8ull * cap));
    VS_CUDA(cudaMallocHost((void**)&h_arena, 4ull * lay.words * cap));
    for (uint32_t i = 0; i < 2 * cap; i++) h_ab[i] = 1;
    // twiddles and fold twiddles are built (and cached) outside the capture
    const TwiddleSet* tw = nullptr;
    VS_TRY(get_twiddles(TW_NATIVE, log_n, &tw, st));
    VS_TRY(get_twiddles(TW_NATIVE, log_eval, &tw, st));
    for (uint32_t l = 0; l < nf; l++) {
      const uint32_t* ft = nullptr;
      VS_TRY(get_fold_twiddles(l == 0 ? COSET_HALF_COSET : COSET_HALF_ODDS, log_eval - l, &ft, st));
    }
    VS_CUDA(cudaStreamSynchronize(st));
    // one plain run of a full batch sets kernel attributes before any capture;
    // then the graphs of every batch size a launch may use
    VS_TRY(enqueue(cap));
    VS_CUDA(cudaStreamSynchronize(st));
    for (uint32_t b = 1;; b = std::min(2 * b, cap)) {
      cudaGraphExec_t x = nullptr;
      VS_TRY(graph_for(b, &x));
      if (b == cap) break;
    }
    return VS_OK;
  }
  // Batch size a launch of `count` proofs runs at: the next power of two (at most
  // the capacity), so a workspace needs only log2(capacity) + 1 graphs; the
  // padding jobs prove (1, 1) and are not returned.
  uint32_t padded(uint32_t count) const {
    uint32_t b = 1;
    while (b < count) b *= 2;
    return std::min(b, cap);
  }
};

int BatchProver::prove_once(uint32_t a, uint32_t b, uint32_t log_n, uint8_t* out, uint64_t cap, uint64_t* out_len,
                            cudaStream_t st) {
  Impl p;
  p.plan(log_n, 1);
  if (out_len) *out_len = p.lay.bytes();
  if (!out || cap < p.lay.bytes())
    return set_error(VS_ERR_INVALID, "proof needs %llu bytes, buffer has %llu", (unsigned long long)p.lay.bytes(),
                     (unsigned long long)cap);
  uint8_t* mem = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&mem, p.total, st);
  if (e == cudaErrorMemoryAllocation) {  // 96 bytes a row instead of 100 to 180
    cudaGetLastError();
    p.group = group_most;
    p.plan(log_n, 1);
    e = cudaMallocAsync((void**)&mem, p.total, st);
  }
  if (e != cudaSuccess)
    return set_error(VS_ERR_OOM, "proof workspace (%llu bytes): %s", (unsigned long long)p.total, cudaGetErrorString(e));
  p.carve(mem);
  uint32_t ab[2] = {a, b};
  p.st = st;
  p.h_ab = ab;
  p.h_arena = reinterpret_cast<uint32_t*>(out);  // only the copy's destination
  int rc = p.enqueue(1);
  p.st = nullptr;  // the caller's stream and buffer are not the workspace's to release
  p.h_ab = p.h_arena = nullptr;
  cudaFreeAsync(mem, st);
  e = cudaStreamSynchronize(st);
  VS_TRY(rc);
  VS_CUDA(e);
  p.lay.finish(out, a, b);
  return VS_OK;
}

BatchProver::BatchProver() : impl(new Impl) {}
BatchProver::~BatchProver() = default;

uint32_t BatchProver::default_capacity(uint32_t log_n) {
  return log_n <= 16 ? 64u : std::max<uint32_t>(1u, 64u >> std::min<uint32_t>(log_n - 16, 6));
}

uint64_t BatchProver::bytes_for(uint32_t log_n, uint32_t capacity) {
  Impl p;
  p.plan(log_n, capacity);
  return p.total;
}

int BatchProver::init(uint32_t log_n, uint32_t capacity) {
  if (log_n < 4 || log_n > BATCH_MAX_LOG_N)
    return set_error(VS_ERR_INVALID, "batch prover: log_n %u outside [4, %u]", log_n, BATCH_MAX_LOG_N);
  if (capacity == 0 || capacity > 1024) return set_error(VS_ERR_INVALID, "batch prover: capacity %u", capacity);
  return impl->setup(log_n, capacity);
}

int BatchProver::launch(const uint32_t* ab, uint32_t count, cudaStream_t on) {
  if (count == 0 || count > impl->cap)
    return set_error(VS_ERR_INVALID, "batch of %u proofs (capacity %u)", count, impl->cap);
  for (uint32_t i = 0; i < 2 * count; i++)
    if (ab[i] >= h::P) return set_error(VS_ERR_INVALID, "public inputs must be canonical M31");
  const uint32_t b = impl->padded(count);
  cudaGraphExec_t x = nullptr;
  VS_TRY(impl->graph_for(b, &x));
  std::copy(ab, ab + 2 * count, impl->h_ab);
  std::fill(impl->h_ab + 2 * count, impl->h_ab + 2 * b, 1u);
  impl->count = count;
  impl->running = on ? on : impl->st;
  VS_CUDA(cudaGraphLaunch(x, impl->running));
  return VS_OK;
}

int BatchProver::finish(std::vector<std::vector<uint8_t>>& out) {
  VS_CUDA(cudaStreamSynchronize(impl->running ? impl->running : impl->st));
  impl->running = nullptr;  // the launch stream may be reused for other work from here on
  const uint32_t count = impl->count;
  out.resize(count);
  for (uint32_t j = 0; j < count; j++) {
    uint8_t* proof = reinterpret_cast<uint8_t*>(impl->h_arena + (uint64_t)j * impl->lay.words);
    impl->lay.finish(proof, impl->h_ab[2 * j], impl->h_ab[2 * j + 1]);
  }
  // copied out on up to 8 host threads
  auto take = [&](uint32_t j0, uint32_t step) {
    for (uint32_t j = j0; j < count; j += step) {
      const uint8_t* proof = reinterpret_cast<const uint8_t*>(impl->h_arena + (uint64_t)j * impl->lay.words);
      out[j].assign(proof, proof + impl->lay.bytes());
    }
  };
  const uint32_t nt = std::min<uint32_t>(8, count / 4);
  std::vector<std::thread> th;
  for (uint32_t t = 1; t < nt; t++) th.emplace_back(take, t, nt);
  take(0, std::max<uint32_t>(nt, 1));
  for (auto& x : th) x.join();
  return VS_OK;
}

uint32_t BatchProver::log_n() const { return impl->log_n; }
uint32_t BatchProver::capacity() const { return impl->cap; }
uint64_t BatchProver::device_bytes() const { return impl->total; }

}  // namespace vs
