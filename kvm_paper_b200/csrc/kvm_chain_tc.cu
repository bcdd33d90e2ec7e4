// The memory chain of the prefill for head_dim 128 and blocks of 128 or 256 tokens, organised for the latency of
// one update (the updates of a kv row are strictly sequential: block m routes against the memory block m-1 left).
//
// Follows the reference's eager update (model/kvm_mixer.py:250-340) with the fp32 merge routing of
// model/kvm_fp32_routing_reference.py:24-49; what the reference does with 3-5 host-issued launches per block
// (model/kernels/kvm_triton_training_kernels.py:1606-1747) is one resident step here.
//
// Split of the work
//   kvm_chain_tc_kernel   routing and the KEY side of the memory: a cluster of 1..8 CTAs per kv row walks all
//                         updates.  Memory row r belongs to CTA r % nc, which keeps the attention view of its
//                         rows (k_attn) RESIDENT in shared memory in the tensor-core operand layout, so a routing
//                         pass loads nothing.  Per update, in the common case of few appended rows:
//                           1. logits pass    S = gk x k_attn^T against the memory as it is (tcgen05, accumulators
//                                             in tensor memory), running fp32 first-argmax per token (sink rows
//                                             excluded), then the novelty pass S = pk x k_attn^T, running maximum
//                                             per token; both partial results exchanged between the CTAs in one
//                                             go (st.async into the peers' shared memory); the n_append tokens of
//                                             lowest bf16-rounded novelty are appended (LayerNorm by one warp per
//                                             row) and scored against every token (warp-level MMAs, a token warp its
//                                             own 32 tokens); a new row wins a token only with a strictly larger logit
//                                             (with many appended rows: novelty pass, appends, then one logits pass
//                                             against the memory after the appends)
//                           2. scatter        delta[rows x D] = onehot[rows x tokens] x gk[tokens x D] on the
//                                             tensor cores (touched rows compacted onto the 128 accumulator
//                                             lanes; a row's first token stands for it: it names its accumulator lane and
//                                             its pool row; the one-hot operand lives in the buffer of the prepared
//                                             keys, cleared by the copy engine; products are exact, the accumulation
//                                             order is the hardware's and fixed), then row = bf16(row + bf16(delta)),
//                                             LayerNorm refresh of the touched rows into shared memory and into the
//                                             row pool, staged so that global memory sees whole rows
//                         What only a token needs (exchange, selection, new rows, routing table, one-hot) runs on the
//                         C / 32 warps whose threads stand for the tokens, with barriers of just those.
//                         Prepared keys pk and gated keys gk = bf16(pk * gate) of every token come from a parallel
//                         pre-pass and arrive by tiled TMA, issued as soon as the buffers are free (prepared keys only
//                         for blocks that append rows).
//                         CTAs of the launch beyond the routing's (whole clusters on the SMs it leaves free) work on
//                         the value side meanwhile: see kvm_vdelta.cuh.
//   value side            which no later update reads: value deltas per (kv row, update) on the tensor cores
//                         (kvm_vdelta.cuh), then one warp per memory row (kvm_vpass.cu); kvm_vpass_kernel below is
//                         the variant for a chain of which only the final memory is wanted (no versions): one warp
//                         per memory row walks the routing decisions of all updates and accumulates the gated
//                         values routed to its row in token order.
// The code of an update is walked through once per update by warps that wait for one another, so instruction fetch is part of
// its latency: what an update touches is kept small enough to stay in the SM's instruction cache (rolled loops, the loops of
// waits and the read-back of accumulators not inlined, shifts instead of divisions by the cluster size).
// Every wait is bounded; a wait that runs out sets the status word, all roles and all CTAs of the cluster leave
// through the common exit, tensor memory is freed.
#include <algorithm>
#include <mutex>

#include "kvm_common.cuh"
#include "kvm_tc.cuh"
#include "kvm_tma_host.cuh"
#include "kvm_vdelta.cuh"

namespace kvm {
namespace chain {

constexpr int HD = 128;
constexpr int kWorkerWarps = 16;
constexpr int kWorkers = kWorkerWarps * 32;   // threads that do everything but issuing copies and MMAs
constexpr int kIssuers = 2;                   // issuing threads (one warp each): issuing an MMA costs its thread about as much
                                              // as the tensor core needs to execute it, so each token tile has its own
constexpr int kThreads = kWorkers + kIssuers * 32;
constexpr int kChunk = 256;                   // memory rows per MMA instruction and per tensor-memory chunk (the N limit)
constexpr int kRowPad = 64;                   // granularity of the resident rows per CTA
constexpr int kNewRows = 16;                  // up to this many appended rows per update take the logits-first order
constexpr int kTokenBits = 9;                 // bits of a token's place inside its block
constexpr uint32_t kTmemCols = 512;
constexpr int kMaxSmem = 226 * 1024;          // dynamic part; the kernel also holds 1 KB of static shared memory

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Shared-memory carve-up (byte offsets from a 1024-byte aligned base).
struct Layout {
  int Rcap;  // resident memory rows per CTA (multiple of 64)
  uint32_t R, P, G, xbuf, part, tok, rowi, tloc, stat, bars, total;
  __host__ __device__ Layout(int C, int s_max, int nc) {
    Rcap = ceil_div(ceil_div(s_max, nc), kRowPad) * kRowPad;
    uint32_t off = 0;
    R = off;    off += 2u * Rcap * 128u;                 // [2 halves of D][Rcap][64] bf16, 128-byte swizzle
    P = off;    off += (uint32_t)C * 256u;               // prepared keys of the block; then the one-hot operand; then the staged sums
    G = off;    off += (uint32_t)C * 256u;               // gated keys of the block
    xbuf = off; off += 2u * nc * C * 8u;                 // [parity][source CTA][token] {value, row | novelty}
    part = off; off += (2u * C * 8u > 4096u ? 2u * C * 8u : 4096u);  // [column half][token]: the two halves of a chunk; small operand of the appended rows
    tok = off;  off += 2u * C * 4u;                      // nov[C] f32, list[C]
    const uint32_t sp = (uint32_t)((s_max + 63) & ~31);  // padded row count: every region below stays 16-byte aligned
    rowi = off; off += sp * 4u + (uint32_t)Rcap * 8u;    // lead[sp] i32; cur[Rcap], lci[Rcap] i32 (by local row)
    tloc = off; off += (4u * C + 15u) & ~15u;            // touched rows of this CTA by accumulator lane
    stat = part;                                         // LayerNorm partial sums of the scatter epilogue (the routing partials are dead by then)
    bars = off; off += 448u;
    total = (off + 15u) & ~15u;
  }
};

struct Bars {
  uint64_t full_p, full_g;              // TMA arrivals of the block's prepared / gated keys
  // MMAs of a chunk complete, per tile of 128 tokens / ... and read back.  With at most 128 resident rows per CTA the
  // 256 accumulator columns of a token tile hold two chunks: consecutive passes alternate between the halves (first
  // index), so that a pass is issued while the workers still read the one before it
  uint64_t tm_full[2][2];
  uint64_t tm_empty[2][2];
  uint64_t w2i;                         // all worker warps -> issuer: the resident rows are final for the next pass
  uint64_t t2i;                         // token warps -> issuer: prepared keys dead / one-hot operand ready
  uint64_t idle;                        // all worker warps (and the second issuer) -> issuer: the update is in global memory,
                                        // its staging buffer free
  uint64_t sc_done;                     // scatter MMAs complete
  uint64_t xbar[2];                     // arrivals of the peers' partial results (two in flight)
  uint64_t zero_done;                   // the copy engine has cleared the one-hot operand
  uint32_t tmem_base;
  int abort;                            // somebody in the cluster gave up
  int n_loc;                            // touched rows of this CTA in the current update
  float red_v[16];
  int red_t[32];
};

static_assert(sizeof(Bars) <= 448, "the barrier block outgrew its shared-memory region");

struct Args {
  LayerDev L;
  const kvm_update_plan* plan;
  int n_plan;
  int nc, lg;            // CTAs per kv row (a power of two) and its logarithm
  int s_max;             // final number of memory rows
  long long n_tok;       // tokens per kv row in pk_all / gk_all
  bf16* k_sum;           // [rows][capacity][D]
  bf16* k_attn;          // [rows][capacity][D] final view
  int capacity;
  bf16* pool_k;          // [rows][pool_rows][D] or null (no versions kept)
  long long pool_rows;
  int* ver_idx;          // [rows][ver_rows] or null
  long long ver_rows;
  int* route;            // [rows][n_plan][C]
  int* born;             // [rows][s_max] token that created each memory row, or null
  int* progress;         // [rows][nc] last update whose routes and version table are published (for the value-delta jobs
                         // that spare CTAs of this launch work on meanwhile), or null
  int* chain_done;       // CTAs of the routing that have finished
  int chain_ctas;        // CTAs of the routing (the CTAs behind them take value-delta jobs)
  int* status;
  uint32_t wait_limit;
  uint32_t test_flags;   // bit 0: the issuer withholds one commit (exercises the timeout path)
};

// Source of the copy that clears the one-hot operand of the scatter (64 KB of zeros, resident in L2).
__device__ __align__(128) unsigned char g_zeros[256 * 256];

// ------------------------------------------------------------------------------------------------ primitives
__device__ __forceinline__ void wsync() { asm volatile("bar.sync 1, %0;" ::"n"(kWorkers) : "memory"); }
// barrier of the first `n` worker threads (one per token of the block)
__device__ __forceinline__ void tsync(int n) { asm volatile("bar.sync 2, %0;" ::"r"(n) : "memory"); }
// barrier of the four warps that share an accumulator lane quarter
__device__ __forceinline__ void qsync(int quarter) { asm volatile("bar.sync %0, 128;" ::"r"(3 + quarter) : "memory"); }
// uniform AND over the worker threads
__device__ __forceinline__ bool wvote(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 1, %2, p;\n\t"
      "selp.b32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)ok), "n"(kWorkers)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ bool try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(tc::smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait; also gives up when somebody else has.  The first attempt is inlined, the loop is not: the code an update
// walks through has to stay small (see above).
template <bool CLUSTER>
__device__ __noinline__ bool wait_loop(uint64_t* bar, uint32_t parity, uint32_t limit, volatile int* abort) {
  for (uint32_t i = 0; i < limit; ++i) {
    if (CLUSTER ? try_wait_cluster(bar, parity) : tc::mbar_try_wait(bar, parity)) return true;
    if ((i & 63) == 63) {  // try_wait suspends the thread for a while by itself; look at the abort flag now and then
      if (*abort) return false;
      if (i >= 4096) __nanosleep(100);
    }
  }
  return false;
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity, uint32_t limit, volatile int* abort) {
  if (CLUSTER ? try_wait_cluster(bar, parity) : tc::mbar_try_wait(bar, parity)) return true;
  return wait_loop<CLUSTER>(bar, parity, limit, abort);
}
__device__ __forceinline__ uint32_t peer_addr(const void* local, int peer) {
  uint32_t a = tc::smem_u32(local), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(peer));
  return r;
}
// 8-byte store into a peer's shared memory that completes 8 bytes of the transaction count of the peer's barrier:
// the data is visible to whoever has waited for that barrier phase (no fence, no separate arrival)
__device__ __forceinline__ void st_async_v2(uint32_t addr, float v, int i, uint32_t bar_addr) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "r"(__float_as_uint(v)), "r"(i), "r"(bar_addr)
               : "memory");
}
__device__ __forceinline__ void st_peer_b32(uint32_t addr, int v) {
  asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 16-byte piece c (elements 8c..8c+7) of row r of an operand stored as [2 halves][rows][64] in the 128-byte swizzle
__device__ __forceinline__ uint32_t piece(int rows, int r, int c) {
  return (uint32_t)((c >> 3) * rows * 128 + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}

// rows r < S owned by CTA `rank` of 2^lg (r % 2^lg == rank)
__device__ __forceinline__ int n_local(int S, int lg, int rank) { return S > rank ? (S - rank + (1 << lg) - 1) >> lg : 0; }

// One thread's share of a routing pass: `groups` groups of 16 accumulator columns from tensor-memory address `at`, column 0
// = local row l0; rows outside [l_min, n_rows) do not count.  ARG: first maximum {value, local row or -1}; otherwise the
// maximum.  (Not inlined: three call sites.)
template <bool ARG>
__device__ __noinline__ float2 read_columns(uint32_t at, int groups, int l0, int l_min, int n_rows) {
  float best = -INFINITY;
  int where = -1;
#pragma unroll 1
  for (; groups > 0; --groups, at += 16, l0 += 16) {
    uint32_t r[16];
    tc::tmem_ld16(at, r);
    tc::tmem_ld_wait();
    if (l0 < l_min || l0 + 16 > n_rows) {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (l0 + j < l_min || l0 + j >= n_rows) r[j] = 0xff800000u;  // -inf
    }
    if (ARG) {
      // two runs of eight, each with its first maximum; strictly greater replaces, so the first of equal values stays
      float v0 = -INFINITY, v1 = -INFINITY;
      int j0 = -1, j1 = -1;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float x0 = __uint_as_float(r[j]), x1 = __uint_as_float(r[8 + j]);
        if (x0 > v0) { v0 = x0; j0 = j; }
        if (x1 > v1) { v1 = x1; j1 = 8 + j; }
      }
      if (v1 > v0) { v0 = v1; j0 = j1; }
      if (v0 > best) { best = v0; where = l0 + j0; }
    } else {
#pragma unroll
      for (int j = 0; j < 16; j += 2) best = fmaxf(best, fmaxf(__uint_as_float(r[j]), __uint_as_float(r[j + 1])));
    }
  }
  return make_float2(best, __int_as_float(where));
}

// ------------------------------------------------------------------------------------------------ the issuer
// One thread per token tile: the MMAs of that tile's routing passes.  The first also issues all copies and the scatter.
struct Issuer {
  const Args& a;
  unsigned char* smem;
  const Layout& lay;
  Bars* bars;
  uint32_t tmem;
  int crank, row;
  const CUtensorMap* map_pk;
  const CUtensorMap* map_gk;
  int which;             // 0: token tile 0, all copies, the scatter; 1: token tile 1 of the routing passes only
  uint32_t g = 0;        // chunks issued so far
  uint32_t n_w2i = 0, n_t2i = 0, n_idle = 0, n_sc = 0, n_g = 0, n_p = 0, n_zero = 0;
  volatile int* abort;
  // accumulator half and per-barrier phase of chunk number gg (see Bars::tm_full): with at most 128 resident rows per
  // CTA consecutive chunks alternate between the halves of a token tile's 256 columns
  __device__ __forceinline__ int acc_half(uint32_t gg) const { return lay.Rcap <= 128 ? (int)(gg & 1u) : 0; }
  __device__ __forceinline__ int acc_phase(uint32_t gg) const { return lay.Rcap <= 128 ? (int)(gg >> 1) : (int)gg; }

  __device__ __forceinline__ bool wait_on(uint64_t* bar, uint32_t& n) {
    const bool ok = wait(bar, n & 1, a.wait_limit, abort);
    ++n;
    tc::tc_fence_after_sync();
    return ok;
  }
  // Update u of this CTA's rows is complete in global memory (routes, version table): tell the CTAs that work on the
  // value side.  Called behind a wait for all worker warps, whose writes this thread's fence makes visible with the flag.
  __device__ __forceinline__ void publish(int u) {
    if (a.progress == nullptr) return;
    __threadfence();
    *reinterpret_cast<volatile int*>(a.progress + (size_t)row * a.nc + crank) = u;
  }
  __device__ __forceinline__ int block_row(int u) const { return (int)((long long)row * a.n_tok + (long long)u * a.L.C); }
  // warm L2 with a later block (the copy into shared memory then does not wait for DRAM)
  __device__ __forceinline__ void prefetch(const CUtensorMap* map, int u) {
    const int y = block_row(u);
#pragma unroll
    for (int x = 0; x < 128; x += 64)
      asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
  }
  __device__ __forceinline__ void load(const CUtensorMap* map, uint32_t off, uint64_t* bar, int u) {
    const int C = a.L.C, y = block_row(u);
    tc::mbar_arrive_expect_tx(bar, (uint32_t)C * 256u);
    tc::tma_load_2d(smem + off, map, 0, y, bar);
    tc::tma_load_2d(smem + off + C * 128, map, 64, y, bar);
  }
  // Operand descriptors and strides that never change, built once (the per-update code of this thread stays short: it
  // runs alone, so every instruction-cache line it touches for the first time in an update is a wait of its own).
  uint64_t d_p, d_g, d_r, d_gmn;         // prepared keys / one-hot (K-major), gated keys (K-major), resident rows, gated keys (MN-major)
  uint32_t a_half, r_half;               // second 64-element half of an operand, in descriptor units (16 bytes)
  __device__ __forceinline__ void setup() {
    const int C = a.L.C;
    d_p = tc::make_desc(tc::smem_u32(smem + lay.P), 16, 1024);
    d_g = tc::make_desc(tc::smem_u32(smem + lay.G), 16, 1024);
    d_r = tc::make_desc(tc::smem_u32(smem + lay.R), 16, 1024);
    d_gmn = tc::make_desc(tc::smem_u32(smem + lay.G), (uint32_t)C * 128u, 1024);
    a_half = (uint32_t)(C * 128) >> 4;
    r_half = (uint32_t)(lay.Rcap * 128) >> 4;
  }
  // S[tokens x rows] = A[tokens x D] * R[rows x D]^T over the first n_rows local rows, up to 256 rows per chunk: one
  // MMA per token tile and k-step covers the whole chunk (issuing an MMA costs about as much as executing a small
  // one), the accumulators of token tile m live in tensor-memory columns [256 m, 256 m + N).  One commit per token
  // tile, so that the first tile is read back while the second is computed.  The loops are kept rolled on purpose.
  __device__ __forceinline__ bool pass(uint64_t da_base, int n_rows, bool withhold_first_commit) {
    const int n_mt = a.L.C / 128;
    const int n_chunks = ceil_div(n_rows, kChunk);
    for (int c = 0; c < n_chunks; ++c, ++g) {
      const int n = min(kChunk, n_rows - c * kChunk);
      const uint32_t idesc = tc::make_idesc(128, (n + 15) & ~15, 0, 0);
      const uint64_t db0 = d_r + (uint64_t)((uint32_t)(c * kChunk * 128) >> 4);
      for (int m = which; m < n_mt; m += kIssuers) {
        const int hb = acc_half(g), ph = acc_phase(g);
        if (ph >= 1 && !wait(&bars->tm_empty[hb][m], (ph - 1) & 1, a.wait_limit, abort)) return false;
        tc::tc_fence_after_sync();
        const uint64_t da0 = da_base + (uint64_t)((uint32_t)(m * 128 * 128) >> 4);
        const uint32_t d = tmem + (uint32_t)(m * kChunk + hb * 128);
#pragma unroll 1
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t lo = (uint32_t)(ks & 3) * 2u;
          tc::mma_ss(d, da0 + (uint64_t)(((ks >> 2) ? a_half : 0u) + lo), db0 + (uint64_t)(((ks >> 2) ? r_half : 0u) + lo), idesc, ks > 0);
        }
        if (!(withhold_first_commit && c == 0 && m == 0)) tc::mma_commit_own_cta(&bars->tm_full[hb][m]);
      }
    }
    return true;
  }
  // delta[128 compacted rows x D] = onehot[rows x C tokens] * gk[C tokens x D]
  // (one-hot: K-major [C/64][128][64] in the buffer of the prepared keys; gated keys: MN-major)
  __device__ __forceinline__ void scatter() {
    constexpr uint32_t idesc = tc::make_idesc(128, HD, 0, 1);
    const int n_ks = a.L.C / 16;
#pragma unroll 1
    for (int ks = 0; ks < n_ks; ++ks)
      tc::mma_ss(tmem, d_p + (uint64_t)((uint32_t)(ks >> 2) * (128u * 128u >> 4) + (uint32_t)(ks & 3) * 2u), d_gmn + (uint64_t)((uint32_t)ks * (2048u >> 4)), idesc, ks > 0);
    tc::mma_commit_own_cta(&bars->sc_done);
  }
  __device__ __forceinline__ void clear_onehot() {
    tc::mbar_arrive_expect_tx(&bars->zero_done, (uint32_t)a.L.C * 256u);
    tc::bulk_g2s(smem + lay.P, g_zeros, (uint32_t)a.L.C * 256u, &bars->zero_done);
  }

  __device__ bool run() {
    const int C = a.L.C, nc = a.nc;
    const bool primary = which == 0;
    if (which >= C / 128) return true;
    setup();
    if (primary) {  // block 0 (the initial memory): prepared keys, or the gated ones where the layer gates the initial memory
      load(map_pk, lay.P, &bars->full_p, 0);
      load(map_gk, lay.G, &bars->full_g, 0);
    }
    ++n_p; ++n_g;
    kvm_update_plan pl_next = a.plan[0];  // fetched one update ahead: the table lives in global memory
    bool g_late = true;                   // the gated keys of the next block are asked for at the head of its update
    for (int u = 0; u < a.n_plan; ++u) {
      const kvm_update_plan pl = pl_next;
      if (u + 1 < a.n_plan) pl_next = a.plan[u + 1];
      const int S0 = pl.state_before, na = pl.n_append, S1 = S0 + na, nm = C - na;
      const bool fast = na <= kNewRows, has_nov = na > 0 && nm > 0;
      if (u > 0) {
        if (!wait_on(&bars->w2i, n_w2i)) return false;  // the resident rows of the previous update are final
        if (!primary) tc::mbar_arrive(&bars->idle);     // (no worker runs two updates ahead of this thread)
        if (primary && g_late) load(map_gk, lay.G, &bars->full_g, u);
        const bool withhold = (a.test_flags & 1u) && u == 1;
        // (A block that is appended as a whole asks nothing of the second issuer, so nothing would keep the barrier from
        // completing the next block's phase before it has looked: it does not look.  The workers do, ahead of their w2i.)
        if ((primary || nm > 0) && !wait(&bars->full_g, n_g & 1, a.wait_limit, abort)) return false;
        ++n_g;
        // Few appended rows: the logits against the OLD memory do not depend on them, so they go first and the novelty
        // follows behind; many: the novelty first, then the logits against the memory after the appends.
        for (int k = 0; k < 2; ++k) {
          const bool logits = (k == 0) == fast;
          if (!logits) {
            if (primary) {
              if (!wait_on(&bars->idle, n_idle)) return false;  // the previous update is in global memory, its staging buffer free
              publish(u - 1);
              if (na > 0) load(map_pk, lay.P, &bars->full_p, u);
              else clear_onehot();
            }
            if (na > 0) {
              if (has_nov && !wait(&bars->full_p, n_p & 1, a.wait_limit, abort)) return false;
              ++n_p;
            }
          } else if (!fast && nm > 0 && !wait_on(&bars->w2i, n_w2i)) {  // the appended rows are in the resident memory
            return false;
          }
          if ((logits ? nm > 0 : has_nov) &&
              !pass(logits ? d_g : d_p, n_local(logits && !fast ? S1 : S0, a.lg, crank), withhold && logits)) return false;
        }
        if (primary && fast && na > 0) {
          // nobody reads the prepared keys any more (novelty read back, appended rows stored): their buffer is cleared by
          // the copy engine and becomes the one-hot operand of the scatter while the workers score the new rows
          if (!wait_on(&bars->t2i, n_t2i)) return false;
          clear_onehot();
        }
        if (primary && nm > 0) {
          // scatter passes (their number is known once the routing is final)
          if (!wait_on(&bars->t2i, n_t2i)) return false;
          const int n_pass = ceil_div(*reinterpret_cast<volatile int*>(&bars->n_loc), 128);
          for (int p = 0; p < n_pass; ++p) {
            if (p > 0 && !wait_on(&bars->t2i, n_t2i)) return false;
            scatter();
            if (!wait(&bars->sc_done, n_sc & 1, a.wait_limit, abort)) return false;
            ++n_sc;
          }
        }
      }
      // Every routing pass was read back before the scatter was asked for: the gated keys of this block are dead.  A block
      // that is appended as a whole has no scatter: the workers may be taking its rows from the buffer until they have
      // signalled w2i, which is waited for at the head of the next update.
      g_late = u == 0 || nm == 0;
      if (primary && !g_late && u + 1 < a.n_plan) load(map_gk, lay.G, &bars->full_g, u + 1);
      if (primary && u + 2 < a.n_plan && crank == (u & (nc - 1))) {  // one CTA of the cluster asks, all profit
        prefetch(map_gk, u + 2);
        if (a.plan[u + 2].n_append > 0) prefetch(map_pk, u + 2);
      }
    }
    if (!primary) tc::mbar_arrive(&bars->idle);
    if (primary && a.n_plan > 1) {
      if (!wait_on(&bars->idle, n_idle)) return false;
      publish(a.n_plan - 1);
    }
    return true;
  }
};

// ------------------------------------------------------------------------------------------------ the workers
struct Workers {
  const Args& a;
  unsigned char* smem;
  const Layout& lay;
  Bars* bars;
  uint32_t tmem;
  int crank, row;
  const float* ln_w;
  const float* ln_b;
  volatile int* abort;
  int tid, warp, lane;
  uint32_t g = 0, n_sc = 0, n_x = 0, n_p = 0, n_zero = 0;
  // accumulator half and per-barrier phase of chunk number gg (see Issuer)
  __device__ __forceinline__ int acc_half(uint32_t gg) const { return lay.Rcap <= 128 ? (int)(gg & 1u) : 0; }
  __device__ __forceinline__ int acc_phase(uint32_t gg) const { return lay.Rcap <= 128 ? (int)(gg >> 1) : (int)gg; }

  __device__ __forceinline__ float* nov() const { return reinterpret_cast<float*>(smem + lay.tok); }
  __device__ __forceinline__ int* list() const { return reinterpret_cast<int*>(smem + lay.tok) + a.L.C; }
  // per memory row: (update that last touched it) << kTokenBits | (its first token in that update, counted from the end);
  // the maximum over an update's tokens wins, later updates win over earlier ones, nothing is ever cleared
  __device__ __forceinline__ int* lead() const { return reinterpret_cast<int*>(smem + lay.rowi); }
  __device__ __forceinline__ int* cur() const { return lead() + ((a.s_max + 63) & ~31); }  // [local row] pool row of the current view
  __device__ __forceinline__ int* lci() const { return cur() + lay.Rcap; }                 // [local row] accumulator lane in this update
  __device__ __forceinline__ int* tloc() const { return reinterpret_cast<int*>(smem + lay.tloc); }
  __device__ __forceinline__ float2* part(int half) const { return reinterpret_cast<float2*>(smem + lay.part) + half * a.L.C; }
  __device__ __forceinline__ float2* xb(int parity, int src) const { return reinterpret_cast<float2*>(smem + lay.xbuf) + (size_t)(parity * a.nc + src) * a.L.C; }
  __device__ __forceinline__ float* stat(int which) const { return reinterpret_cast<float*>(smem + lay.stat) + which * 4 * 128; }

  // this warp's shared-memory writes are visible to the tensor core and the copy engine; it arrives on `bar`
  __device__ __forceinline__ void signal(uint64_t* bar) {
    tc::fence_proxy_async();
    tc::tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(bar);
  }

  // Read back the chunks of a routing pass: maximum (ARG = false: novelty) or first maximum over rows >= `protected_rows`
  // (true), the thread's result (value; global row or -1) left in registers.  Warp w reads token tile (w / 4) % 2, lanes
  // 32 (w % 4).., and one half of the chunk's 16-column groups.
  template <bool ARG>
  __device__ __forceinline__ bool read_regs(int n_rows, int protected_rows, float& v_out, int& i_out) {
    const int half = warp >> 3, mt = (warp >> 2) & 1;
    const int n_chunks = ceil_div(n_rows, kChunk);
    // first local row that counts: global row l * nc + crank >= protected_rows
    const int l_min = ARG ? n_local(protected_rows, a.lg, crank) : 0;
    float best = -INFINITY;
    int where = -1;
    bool ok = true;
#pragma unroll 1
    for (int c = 0; c < n_chunks; ++c, ++g) {
      if (mt * 128 >= a.L.C) continue;
      const int hb = acc_half(g), ph = acc_phase(g);
      ok = ok && wait(&bars->tm_full[hb][mt], ph & 1, a.wait_limit, abort);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;  // the caller aborts
      tc::tc_fence_after_sync();
      const int n_groups = ceil_div(min(kChunk, n_rows - c * kChunk), 16), g_half = (n_groups + 1) / 2;
      const int g_begin = half ? g_half : 0, n_mine = half ? n_groups - g_half : g_half;
      const float2 f = read_columns<ARG>(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(mt * kChunk + hb * 128 + g_begin * 16), n_mine,
                                         c * kChunk + g_begin * 16, l_min, n_rows);
      if (f.x > best) { best = f.x; where = __float_as_int(f.y); }
      tc::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bars->tm_empty[hb][mt]);
    }
    v_out = best;
    i_out = where >= 0 ? (where << a.lg) + crank : -1;
    return ok;
  }
  // This thread's share of the routing results of its token -> shared memory.  {best logit over the old rows, row (16
  // bits, 0xffff = none) | novelty maximum as bf16 << 16}; the bf16 rounding of the novelty commutes with the maximum.
  __device__ __forceinline__ void store_part(float v, int i, float nv) {
    const int mt = (warp >> 2) & 1;
    if (mt * 128 < a.L.C) {
      const unsigned packed = ((unsigned)i & 0xffffu) | ((unsigned)__bfloat16_as_ushort(__float2bfloat16_rn(nv)) << 16);
      part(warp >> 3)[mt * 128 + (warp & 3) * 32 + lane] = make_float2(v, __uint_as_float(packed));
    }
  }
  // Token threads: merge the two column halves, exchange the CTA's partial result with the peers, combine.
  __device__ __forceinline__ bool exchange(float& best_v, int& best_i, float& novelty) {
    const int C = a.L.C, nc = 1 << a.lg;
    const int parity = n_x & 1;
    float v = -INFINITY, nv = -INFINITY;
    int i = -1;
    auto take = [&](float2 p) {
      const unsigned w = __float_as_uint(p.y);
      const int pi = (w & 0xffffu) == 0xffffu ? -1 : (int)(w & 0xffffu);
      nv = fmaxf(nv, __uint_as_float(w & 0xffff0000u));
      if (pi >= 0 && (i < 0 || p.x > v || (p.x == v && pi < i))) { v = p.x; i = pi; }
    };
    take(part(0)[tid]);
    take(part(1)[tid]);
    bool ok = true;
    if (nc > 1) {
      // every token's partial result goes to the same token's slot in every peer; this CTA expects the peers' bytes
      if (tid == 0) tc::mbar_arrive_expect_tx(&bars->xbar[parity], (uint32_t)((nc - 1) * C * 8));
      const float2* slot = &xb(parity, crank)[tid];
      const int packed = (int)(((unsigned)i & 0xffffu) | (__float_as_uint(nv) & 0xffff0000u));
#pragma unroll 1
      for (int p = 0; p < nc; ++p)
        if (p != crank) st_async_v2(peer_addr(slot, p), v, packed, peer_addr(&bars->xbar[parity], p));
      ok = wait<true>(&bars->xbar[parity], (n_x >> 1) & 1, a.wait_limit, abort);
      if (ok)
#pragma unroll 1
        for (int p = 0; p < nc; ++p)
          if (p != crank) take(xb(parity, p)[tid]);
    }
    best_v = v;
    best_i = i;
    novelty = nv;
    return ok;
  }

  // the 16 elements of lane gl of row t of a block operand (prepared or gated keys)
  __device__ __forceinline__ void load_block_row(RowVec<HD, 8>& x, uint32_t off, int t, int gl) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 u = *reinterpret_cast<const uint4*>(smem + off + piece(a.L.C, t, 2 * gl + h));
      const float2 p0 = unpack_bf16(u.x), p1 = unpack_bf16(u.y), p2 = unpack_bf16(u.z), p3 = unpack_bf16(u.w);
      x.x[h * 8 + 0] = p0.x; x.x[h * 8 + 1] = p0.y; x.x[h * 8 + 2] = p1.x; x.x[h * 8 + 3] = p1.y;
      x.x[h * 8 + 4] = p2.x; x.x[h * 8 + 5] = p2.y; x.x[h * 8 + 6] = p3.x; x.x[h * 8 + 7] = p3.y;
    }
  }
  // Rows [S0, S0 + na) from the tokens list()[0..na), all warps, eight lanes per row: carried sums, resident view, pool
  // row (a row lives in the pool row of its token).  `src_off`: operand holding what is stored (prepared or gated keys).
  __device__ __forceinline__ void append_rows(int S0, int na, uint32_t src_off, int u) {
    const int gl = tid & 7, grp = tid >> 3;
#pragma unroll 1
    for (int base = 0; base < na; base += kWorkers / 8) {  // whole warps stay together: the LayerNorm uses group shuffles
      const int p = base + grp;
      const bool mine = p < na && ((S0 + p) & (a.nc - 1)) == crank;
      if (!__any_sync(0xffffffffu, mine)) continue;  // nothing for this warp to store
      const int r = S0 + (p < na ? p : 0), t = list()[p < na ? p : 0];
      RowVec<HD, 8> x;
      load_block_row(x, src_off, t, gl);
      if (mine) store_row<HD, 8>(x, a.k_sum + ((size_t)row * a.capacity + r) * HD, gl);
      layer_norm_row<HD, 8>(x, ln_w, ln_b, a.L.ln_eps, gl);
      if (mine) {
        uint4 u0, u1;
        u0.x = pack_bf16(x.x[0], x.x[1]); u0.y = pack_bf16(x.x[2], x.x[3]); u0.z = pack_bf16(x.x[4], x.x[5]); u0.w = pack_bf16(x.x[6], x.x[7]);
        u1.x = pack_bf16(x.x[8], x.x[9]); u1.y = pack_bf16(x.x[10], x.x[11]); u1.z = pack_bf16(x.x[12], x.x[13]); u1.w = pack_bf16(x.x[14], x.x[15]);
        const int l = r >> a.lg;
        *reinterpret_cast<uint4*>(smem + lay.R + piece(lay.Rcap, l, 2 * gl)) = u0;
        *reinterpret_cast<uint4*>(smem + lay.R + piece(lay.Rcap, l, 2 * gl + 1)) = u1;
        if (a.pool_k) {
          bf16* dst = a.pool_k + ((size_t)row * a.pool_rows + (size_t)u * a.L.C + t) * HD + gl * 16;
          *reinterpret_cast<uint4*>(dst) = u0;
          *reinterpret_cast<uint4*>(dst + 8) = u1;
        }
        if (gl == 0) {
          cur()[l] = u * a.L.C + t;
          if (a.born) a.born[(size_t)row * a.s_max + r] = u * a.L.C + t;
        }
      }
    }
  }
  // The same for at most kNewRows rows by the token warps, one warp per row and four elements per lane, every CTA keeping
  // the rows' view in its small operand of new rows: the few warps that store rows run alone, and what they wait for is
  // mostly their own instructions, so the code is kept short.
  __device__ __forceinline__ void append_rows_warp(int S0, int na, uint32_t src_off, int u) {
#pragma unroll 1
    for (int p = warp; p < na; p += a.L.C / 32) {
      const int r = S0 + p, t = list()[p], pc = lane >> 1;
      const uint32_t sub = (uint32_t)(lane & 1) * 8u;  // which half of a 16-byte piece
      const uint2 raw = *reinterpret_cast<const uint2*>(smem + src_off + piece(a.L.C, t, pc) + sub);
      RowVec<HD, 32> x;
      const float2 e0 = unpack_bf16(raw.x), e1 = unpack_bf16(raw.y);
      x.x[0] = e0.x; x.x[1] = e0.y; x.x[2] = e1.x; x.x[3] = e1.y;
      const bool mine = (r & (a.nc - 1)) == crank;
      if (mine) *reinterpret_cast<uint2*>(a.k_sum + ((size_t)row * a.capacity + r) * HD + lane * 4) = raw;  // the carried sum is the token's row
      layer_norm_row<HD, 32>(x, ln_w, ln_b, a.L.ln_eps, lane);
      uint2 o;
      o.x = pack_bf16(x.x[0], x.x[1]);
      o.y = pack_bf16(x.x[2], x.x[3]);
      *reinterpret_cast<uint2*>(smem + lay.part + piece(kNewRows, p, pc) + sub) = o;
      if (mine) {
        *reinterpret_cast<uint2*>(smem + lay.R + piece(lay.Rcap, r >> a.lg, pc) + sub) = o;
        if (a.pool_k) *reinterpret_cast<uint2*>(a.pool_k + ((size_t)row * a.pool_rows + (size_t)u * a.L.C + t) * HD + lane * 4) = o;
        if (lane == 0) {
          cur()[r >> a.lg] = u * a.L.C + t;
          if (a.born) a.born[(size_t)row * a.s_max + r] = u * a.L.C + t;
        }
      }
    }
  }
  // A token warp: logits of its 32 tokens against the rows that were just appended (the small operand), warp-level MMAs;
  // a new row has a higher index than every old one, it wins only with a strictly larger logit.
  __device__ __forceinline__ void score_new_rows(int S0, int na, int protected_rows, float& best_v, int& best_i) {
    const int gq = lane >> 2, tq = lane & 3;
    for (int n0 = 0; n0 < na; n0 += 8) {
      float acc[2][4];
#pragma unroll
      for (int m = 0; m < 2; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
#pragma unroll 2
      for (int ks = 0; ks < HD / 16; ++ks) {
        const unsigned char* nb = smem + lay.part;
        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(nb + piece(kNewRows, n0 + gq, ks * 2) + tq * 4);
        const uint32_t b1 = *reinterpret_cast<const uint32_t*>(nb + piece(kNewRows, n0 + gq, ks * 2 + 1) + tq * 4);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          uint32_t ka[4];
          ldmatrix_x4(ka, smem + lay.G + piece(a.L.C, warp * 32 + m * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, ks * 2 + (lane >> 4)));
          mma_bf16_16816(acc[m], ka, b0, b1);
        }
      }
      const int src = (lane & 7) * 4, e_mine = lane >> 3;  // a token's own lane = tile * 16 + upper half * 8 + quad
      if (na == 1) {  // column 0 only
        float x = -INFINITY;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float sv = __shfl_sync(0xffffffffu, acc[k >> 1][(k & 1) * 2], src);
          if (k == e_mine) x = sv;
        }
        if (S0 >= protected_rows && (x > best_v || best_i < 0)) { best_v = x; best_i = S0; }
        return;
      }
      // first maximum over the new rows: this thread's columns 2 tq, 2 tq + 1, then the quad; tokens gq and gq + 8 of a tile
      float v[4];
      int j[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {  // e = tile * 2 + upper half
        const int c = n0 + tq * 2;
        const float x0 = acc[e >> 1][(e & 1) * 2], x1 = acc[e >> 1][(e & 1) * 2 + 1];
        const bool ok0 = c < na && S0 + c >= protected_rows, ok1 = c + 1 < na && S0 + c + 1 >= protected_rows;
        v[e] = ok0 ? x0 : -INFINITY;
        j[e] = ok0 ? c : -1;
        if (ok1 && (j[e] < 0 || x1 > v[e])) { v[e] = x1; j[e] = c + 1; }
#pragma unroll
        for (int off = 1; off <= 2; off <<= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, v[e], off);
          const int oj = __shfl_xor_sync(0xffffffffu, j[e], off);
          if (oj >= 0 && (j[e] < 0 || ov > v[e] || (ov == v[e] && oj < j[e]))) { v[e] = ov; j[e] = oj; }
        }
      }
      float tv = -INFINITY;
      int tj = -1;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float sv = __shfl_sync(0xffffffffu, v[k], src);
        const int sj = __shfl_sync(0xffffffffu, j[k], src);
        if (k == e_mine) { tv = sv; tj = sj; }
      }
      if (tj >= 0 && (tv > best_v || best_i < 0)) { best_v = tv; best_i = S0 + tj; }
    }
  }
  // Token threads: the na tokens of lowest novelty, lowest index among equals; returns this token's place in the append
  // list (token order) or -1, fills list().
  __device__ __forceinline__ int select(float novelty, int na) {
    const int C = a.L.C, n_warps = C / 32;
    if (na == 1) {
      float bv = novelty;
      int bt = tid;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
        const int ot = __shfl_xor_sync(0xffffffffu, bt, off);
        if (ov < bv || (ov == bv && ot < bt)) { bv = ov; bt = ot; }
      }
      if (lane == 0) { bars->red_v[warp] = bv; bars->red_t[warp] = bt; }
      tsync(C);
      bv = bars->red_v[lane & (n_warps - 1)];
      bt = bars->red_t[lane & (n_warps - 1)];
#pragma unroll
      for (int off = 4; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
        const int ot = __shfl_xor_sync(0xffffffffu, bt, off);
        if (ov < bv || (ov == bv && ot < bt)) { bv = ov; bt = ot; }
      }
      if (tid == 0) list()[0] = bt;
      return tid == bt ? 0 : -1;
    }
    nov()[tid] = novelty;
    tsync(C);
    int rank = 0;
#pragma unroll 4
    for (int u0 = 0; u0 < C; u0 += 4) {  // stable rank of the novelty scores
      const float4 q = *reinterpret_cast<const float4*>(nov() + u0);
      rank += (q.x < novelty || (q.x == novelty && u0 + 0 < tid)) ? 1 : 0;
      rank += (q.y < novelty || (q.y == novelty && u0 + 1 < tid)) ? 1 : 0;
      rank += (q.z < novelty || (q.z == novelty && u0 + 2 < tid)) ? 1 : 0;
      rank += (q.w < novelty || (q.w == novelty && u0 + 3 < tid)) ? 1 : 0;
    }
    const bool f = rank < na;
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (lane == 0) bars->red_t[warp] = __popc(bal);
    tsync(C);
    int p = __popc(bal & ((1u << lane) - 1u));
#pragma unroll 1
    for (int w = 0; w < warp; ++w) p += bars->red_t[w];
    if (f) list()[p] = tid;
    return f ? p : -1;
  }

  // The 128 touched rows of scatter pass p: carried sums, LayerNorm refresh into the resident memory and the row pool.
  // The four warps of an accumulator lane quarter work on its 32 rows by themselves (qsync).  Rows are scattered over the
  // carried sums and the pool, so they travel between global memory and a staging buffer (the one-hot operand's, dead
  // by now) as whole rows, while the arithmetic runs one row per thread and 32 columns per warp, as tensor memory has
  // them: row per lane straight to global memory touches 32 lines per instruction, which alone took 6 000 cycles.
  // `last`: the resident rows are final behind this pass, the next update's routing may start.
  __device__ __forceinline__ bool epilogue(int p, int n_loc, bool last) {
    const int quarter = warp & 3, colq = warp >> 2;
    // whole rows: sixteen threads per row, this one the piece pc of the quarter's rows r8, r8 + 8, ..
    constexpr int kPieces = HD / 8, kShare = 32 * kPieces / 128;
    const int qt = colq * 32 + lane, pc = qt % kPieces, r8 = quarter * 32 + qt / kPieces;
    unsigned char* stage = smem + lay.P;
    unsigned char* const mine = stage + piece(128, r8, pc);   // (+ 1024 bytes per further row: the swizzle repeats every 8 rows)
    const int* const rows = tloc() + p * 128 + r8;
    const int n_share = ceil_div(n_loc - p * 128 - r8, 8);    // how many of them are live
    bf16* const sums = a.k_sum + (size_t)row * a.capacity * HD + pc * 8;
    uint4 old[kShare];
#pragma unroll
    for (int k = 0; k < kShare; ++k)
      if (k < n_share) old[k] = *reinterpret_cast<const uint4*>(sums + (size_t)rows[k * 8] * HD);
    const bool ok = wait(&bars->sc_done, n_sc & 1, a.wait_limit, abort);
    ++n_sc;
    tc::tc_fence_after_sync();
#pragma unroll
    for (int k = 0; k < kShare; ++k)
      if (k < n_share) *reinterpret_cast<uint4*>(mine + k * 1024) = old[k];
    const int ci = quarter * 32 + lane;
    const bool act = p * 128 + ci < n_loc;
    const int l = act ? tloc()[p * 128 + ci] >> a.lg : 0;
    // Three short sweeps over this thread's 32 columns, the row's new sum (bf16, exact) kept in the staging buffer between
    // them: row = bf16(row + bf16(delta)) on packed pairs (the sum of two bf16 numbers rounded once), variance, output
    unsigned char* const at0 = stage + (colq >> 1) * (128 * 128) + ci * 128;
    auto at = [&](int j) { return reinterpret_cast<uint4*>(at0 + ((((colq & 1) * 4 + j) ^ (ci & 7)) << 4)); };
    qsync(quarter);
    float s1 = 0.f;
#pragma unroll 1
    for (int j = 0; j < 4; j += 2) {
      uint32_t d[16];
      tc::tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(colq * 32 + j * 8), d);
      tc::tmem_ld_wait();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint4 o4 = *at(j + h);
        uint32_t* w = reinterpret_cast<uint32_t*>(&o4);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = h * 8 + e * 2;
          const __nv_bfloat162 dl = __floats2bfloat162_rn(__uint_as_float(d[c]), __uint_as_float(d[c + 1]));
          const __nv_bfloat162 sum = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&w[e]), dl);
          w[e] = *reinterpret_cast<const uint32_t*>(&sum);
          const float2 f2 = __bfloat1622float2(sum);
          s1 += f2.x + f2.y;
        }
        *at(j + h) = o4;
      }
    }
    tc::tc_fence_before_sync();
    stat(0)[colq * 128 + ci] = s1;
    qsync(quarter);
    const float mean = (stat(0)[ci] + stat(0)[128 + ci] + stat(0)[256 + ci] + stat(0)[384 + ci]) * (1.0f / HD);
    float s2 = 0.f;
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      const uint4 o4 = *at(j);
      const uint32_t w[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f2 = unpack_bf16(w[e]);
        const float x0 = f2.x - mean, x1 = f2.y - mean;
        s2 += x0 * x0;
        s2 += x1 * x1;
      }
    }
    stat(1)[colq * 128 + ci] = s2;
    qsync(quarter);
    const float var = (stat(1)[ci] + stat(1)[128 + ci] + stat(1)[256 + ci] + stat(1)[384 + ci]) * (1.0f / HD);
    const float rstd = 1.0f / sqrtf(var + a.L.ln_eps);
    if (act) {
      unsigned char* const dst = smem + lay.R + (colq >> 1) * lay.Rcap * 128 + l * 128;
#pragma unroll 1
      for (int j = 0; j < 4; ++j) {
        const uint4 o4 = *at(j);
        const uint32_t w[4] = {o4.x, o4.y, o4.z, o4.w};
        uint32_t y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f2 = unpack_bf16(w[e]);
          const float2 lw = *reinterpret_cast<const float2*>(ln_w + colq * 32 + j * 8 + e * 2), lb = *reinterpret_cast<const float2*>(ln_b + colq * 32 + j * 8 + e * 2);
          y[e] = pack_bf16((f2.x - mean) * rstd * lw.x + lb.x, (f2.y - mean) * rstd * lw.y + lb.y);
        }
        *reinterpret_cast<uint4*>(dst + ((((colq & 1) * 4 + j) ^ (l & 7)) << 4)) = make_uint4(y[0], y[1], y[2], y[3]);
      }
    }
    if (last) signal(&bars->w2i);  // behind this the next update's routing reads the resident memory
    qsync(quarter);
    // out to global memory, whole rows again
#pragma unroll 1
    for (int k = 0; k < kShare && k < n_share; ++k) {
      const int r = rows[k * 8], lr = r >> a.lg;
      *reinterpret_cast<uint4*>(sums + (size_t)r * HD) = *reinterpret_cast<const uint4*>(mine + k * 1024);
      if (a.pool_k)
        *reinterpret_cast<uint4*>(a.pool_k + ((size_t)row * a.pool_rows + cur()[lr]) * HD + pc * 8) =
            *reinterpret_cast<const uint4*>(smem + lay.R + piece(lay.Rcap, lr, pc));
    }
    return ok;
  }

  __device__ bool run() {
    const int C = a.L.C, nc = a.nc;
    const bool token = tid < C;  // (whole warps)
    int* route_row = a.route + (size_t)row * a.n_plan * C;
    kvm_update_plan pl_next = a.plan[0];  // fetched one update ahead
    // (a wait that ran out shows in `ok` and ends the walk at the next vote: nobody leaves a barrier of the others alone)
    bool ok = true;
    for (int u = 0; u < a.n_plan; ++u) {
      const kvm_update_plan pl = pl_next;
      if (u + 1 < a.n_plan) pl_next = a.plan[u + 1];
      const int S0 = pl.state_before, na = pl.n_append, S1 = S0 + na, nm = C - na;
      int* ver = (a.ver_idx && pl.version_row >= 0) ? a.ver_idx + (size_t)row * a.ver_rows + pl.version_row : nullptr;
      if (u == 0 || nm == 0) {
        // ---- the block becomes memory rows token by token: the initial memory (model/kvm_mixer.py:434-447), or a block
        // that is appended as a whole
        ok = ok && wait(&bars->full_p, n_p & 1, a.wait_limit, abort) && wait(&bars->full_g, u & 1, a.wait_limit, abort);
        ++n_p;
        if (token) list()[tid] = tid;
        if (!wvote(ok)) return false;
        append_rows(S0, na, ((u == 0 ? a.L.gate_initial : a.L.gate_appends) && a.L.gate_keys) ? lay.G : lay.P, u);
        if (crank == 0)
#pragma unroll 1
          for (int i = tid; i < C; i += kWorkers) route_row[(size_t)u * C + i] = i < na ? -(1 + S0 + i) : 0;
        signal(&bars->w2i);
        wsync();
      } else {
        const int protected_rows = min(a.L.sink_len, S1);
        // few appended rows: logits against the old memory first, the novelty behind them, both exchanged together, the
        // logits against the new rows last (see the issuer); many: novelty, appends, then all logits
        const bool fast = na <= kNewRows;
        // ---- 1. routing passes, partial results of the CTAs, appended rows
        float best_v = -INFINITY, novelty = -INFINITY;  // this token's best logit and row so far
        int best_i = -1, app = -1;                      // ... and its place among the appended ones
        {
          float vl = -INFINITY, vn = -INFINITY;
          int il = -1, unused;
          if (fast) ok = read_regs<true>(n_local(S0, a.lg, crank), protected_rows, vl, il) && ok;
          if (na > 0) ok = read_regs<false>(n_local(S0, a.lg, crank), 0, vn, unused) && ok;
          store_part(vl, il, vn);
        }
        wsync();
        if (token) {
          ok = exchange(best_v, best_i, novelty) && ok;
          if (na > 0) {
            app = select(novelty, na);
            tsync(C);
          }
        }
        ++n_x;
        if (na > 0) {
          ++n_p;
          const uint32_t src = (a.L.gate_appends && a.L.gate_keys) ? lay.G : lay.P;
          if (fast) {
            if (token) {
              append_rows_warp(S0, na, src, u);
              signal(&bars->t2i);  // the prepared keys are dead: the copy engine may clear their buffer
              tsync(C);
              score_new_rows(S0, na, protected_rows, best_v, best_i);
            }
          } else {
            wsync();
            append_rows(S0, na, src, u);
            signal(&bars->w2i);  // the appended rows are in place: the pass against them may start
            wsync();             // ... and the prepared keys dead: cleared while the tensor core works on the logits
            uint4* o = reinterpret_cast<uint4*>(smem + lay.P);
#pragma unroll 1
            for (int i = tid; i < C * 16; i += kWorkers) o[i] = make_uint4(0, 0, 0, 0);
            tc::fence_proxy_async();
            float vl;
            int il;
            ok = read_regs<true>(n_local(S1, a.lg, crank), protected_rows, vl, il) && ok;
            store_part(vl, il, -INFINITY);
            wsync();
            if (token) {
              float unused;
              ok = exchange(best_v, best_i, unused) && ok;
            }
            ++n_x;
          }
        }
        // ---- 2. routing table; touched rows of this CTA, an accumulator lane and a pool row for each
        const int my = app >= 0 ? -1 : best_i;
        if (token) {
          if (crank == 0) route_row[(size_t)u * C + tid] = app >= 0 ? -(1 + S0 + app) : my;
          const int key = (u << kTokenBits) | ((1 << kTokenBits) - 1 - tid);
          if (my >= 0) atomicMax(lead() + my, key);
          tsync(C);
          const bool mine = my >= 0 && (my & (a.nc - 1)) == crank;
          const bool leads = mine && lead()[my] == key;
          const unsigned bal = __ballot_sync(0xffffffffu, leads);
          if (lane == 0) bars->red_t[16 + warp] = __popc(bal);
          tsync(C);
          int before = 0, total = 0;
#pragma unroll 1
          for (int w = 0; w < C / 32; ++w) {
            const int c = bars->red_t[16 + w];
            if (w < warp) before += c;
            total += c;
          }
          if (leads) {
            const int ll = before + __popc(bal & ((1u << lane) - 1u)), l = my >> a.lg;
            lci()[l] = ll;
            tloc()[ll] = my;
            cur()[l] = u * C + tid;  // the row moves to the pool row of its first token
          }
          if (tid == 0) bars->n_loc = total;
          tsync(C);
          // one-hot operand [C/64][128 rows][64 tokens] of the first 128 touched rows, in the cleared buffer
          if (fast) ok = wait(&bars->zero_done, n_zero & 1, a.wait_limit, abort) && ok;
          if (ok && mine) {
            const int ll = lci()[my >> a.lg];
            if (ll < 128)
              *reinterpret_cast<unsigned short*>(smem + lay.P + (uint32_t)(tid >> 6) * (128u * 128u) + tc::sw128_offset(ll, tid & 63)) = 0x3F80;  // bf16 1.0
          }
          signal(&bars->t2i);
        }
        if (fast) ++n_zero;
        if (!wvote(ok)) return false;
        // ---- 3. scatter: delta of the touched rows on the tensor cores, 128 rows per pass
        const int n_loc = bars->n_loc, n_pass = ceil_div(n_loc, 128);
        if (n_pass == 0) signal(&bars->w2i);
#pragma unroll 1
        for (int p = 0; p < n_pass; ++p) {
          if (p > 0) {  // a further pass: the buffer holds staged sums, clear it and set the next rows
            wsync();
            uint4* o = reinterpret_cast<uint4*>(smem + lay.P);
#pragma unroll 1
            for (int i = tid; i < C * 16; i += kWorkers) o[i] = make_uint4(0, 0, 0, 0);
            tc::fence_proxy_async();
            wsync();
            if (token) {
              if (my >= 0 && (my & (a.nc - 1)) == crank) {
                const int ll = lci()[my >> a.lg] - p * 128;
                if (ll >= 0 && ll < 128)
                  *reinterpret_cast<unsigned short*>(smem + lay.P + (uint32_t)(tid >> 6) * (128u * 128u) + tc::sw128_offset(ll, tid & 63)) = 0x3F80;
              }
              signal(&bars->t2i);
            }
          }
          ok = epilogue(p, n_loc, p == n_pass - 1) && ok;
        }
        if (!ok) *abort = 1;
      }
      // ---- 4. the version: pool rows of this CTA's memory rows
      if (ver)
#pragma unroll 1
        for (int l = tid; l < n_local(S1, a.lg, crank); l += kWorkers) ver[(l << a.lg) + crank] = cur()[l];
      signal(&bars->idle);
    }
    // final attention view of the keys, row order, for whoever continues from this memory (the decode cache)
    {
      const kvm_update_plan pl = a.plan[a.n_plan - 1];
      const int S = pl.state_before + pl.n_append;
      if (!wvote(ok)) return false;
#pragma unroll 1
      for (int i = tid; i < n_local(S, a.lg, crank) * 16; i += kWorkers) {
        const int l = i >> 4, c = i & 15;
        const int r = (l << a.lg) + crank;
        *reinterpret_cast<uint4*>(a.k_attn + ((size_t)row * a.capacity + r) * HD + c * 8) =
            *reinterpret_cast<const uint4*>(smem + lay.R + piece(lay.Rcap, l, c));
      }
    }
    return true;
  }
};

struct Maps {
  CUtensorMap pk, gk;  // [rows * n_tok][D] bf16, boxes of 64 elements x C tokens
};

__global__ void __launch_bounds__(kThreads, 1)
kvm_chain_tc_kernel(const __grid_constant__ Args a, const __grid_constant__ Maps maps, const __grid_constant__ vside::DeltaArgs va,
                    const __grid_constant__ vside::Maps vmaps) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(16) float ln_s[2 * HD];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((int)blockIdx.x >= a.chain_ctas) {
    // A spare CTA of the launch (whole clusters of them): it works on the value side of the updates the routing has
    // published so far, until the routing is over; what is left then is taken by the kernel behind this one.
    if (tid < vside::kThreads) vside::delta_jobs(va, vmaps, smem, tid);
    return;
  }
  const int nc = a.nc;
  const int row = blockIdx.x / nc, crank = blockIdx.x % nc;
  const Layout lay(a.L.C, a.s_max, nc);
  Bars* bars = reinterpret_cast<Bars*>(smem + lay.bars);
  const bool aligned = (tc::smem_u32(smem) & 1023u) == 0;  // operand tiles need 1024-byte alignment (uniform over the grid)
  if (!aligned) {
    if (tid == 0) {
      atomicExch(a.status, KVM_ERR_UNSUPPORTED);
      if (a.chain_done) atomicAdd(a.chain_done, 1);
    }
    return;
  }
  for (int i = tid; i < HD; i += kThreads) {
    ln_s[i] = a.L.ln_w[i];
    ln_s[HD + i] = a.L.ln_b[i];
  }
  {  // resident memory starts as zeros: rows past the live ones feed the MMAs, too (their scores are masked)
    uint4* r4 = reinterpret_cast<uint4*>(smem + lay.R);
    for (int i = tid; i < lay.Rcap * 16; i += kThreads) r4[i] = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < a.s_max; i += kThreads) reinterpret_cast<int*>(smem + lay.rowi)[i] = 0;  // update numbers start at 1
  }
  if (tid == 0) {
    tc::mbar_init(&bars->full_p, 1);
    tc::mbar_init(&bars->full_g, 1);
    for (int i = 0; i < 2; ++i) {
      for (int hb = 0; hb < 2; ++hb) {
        tc::mbar_init(&bars->tm_full[hb][i], 1);
        tc::mbar_init(&bars->tm_empty[hb][i], 8);  // the eight warps that read a token tile
      }
    }
    tc::mbar_init(&bars->w2i, kWorkerWarps);
    tc::mbar_init(&bars->t2i, a.L.C / 32);
    tc::mbar_init(&bars->idle, kWorkerWarps + (a.L.C > 128 ? 1 : 0));  // ... and the second issuer
    tc::mbar_init(&bars->sc_done, 1);
    tc::mbar_init(&bars->xbar[0], 1);  // one local arrival that states the bytes the peers will store
    tc::mbar_init(&bars->xbar[1], 1);
    tc::mbar_init(&bars->zero_done, 1);
    bars->abort = 0;
    bars->n_loc = 0;
    tc::fence_barrier_init();
  }
  if (warp == kWorkerWarps) tc::tmem_alloc(&bars->tmem_base, kTmemCols);
  tc::fence_proxy_async();
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  if (nc > 1) cluster_barrier();  // the peers' barriers exist before anybody arrives on them
  const uint32_t tmem = bars->tmem_base;
  volatile int* abort = &bars->abort;

  bool ok = true;
  if (warp >= kWorkerWarps) {
    if (lane == 0) {
      Issuer is{a, smem, lay, bars, tmem, crank, row, &maps.pk, &maps.gk, warp - kWorkerWarps};
      is.abort = abort;
      ok = is.run();
    }
  } else {
    Workers w{a, smem, lay, bars, tmem, crank, row, ln_s, ln_s + HD, abort, tid, warp, lane};
    ok = w.run();
  }
  if (!ok) {
    // report, tell everybody in the cluster, then leave through the common exit
    atomicExch(a.status, KVM_ERR_DEVICE_TIMEOUT);
    *abort = 1;
    if (nc > 1 && lane == 0)
      for (int p = 0; p < nc; ++p)
        if (p != crank) st_peer_b32(peer_addr(&bars->abort, p), 1);
  }
  __syncwarp();
  __syncthreads();
  if (*abort) {
    // copies and MMAs of this CTA may still be in flight: they complete on their own within microseconds
    for (int k2 = 0; k2 < 64; ++k2) __nanosleep(1000);
  }
  tc::tc_fence_before_sync();
  __syncthreads();
  if (warp == kWorkerWarps) tc::tmem_dealloc(tmem, kTmemCols);
  if (tid == 0 && a.chain_done) {  // (the spare CTAs stop taking value-delta jobs when every routing CTA has got here)
    __threadfence();
    atomicAdd(a.chain_done, 1);
  }
  if (nc > 1) cluster_barrier();  // nobody leaves while a peer may still write into its shared memory
}

// ------------------------------------------------------------------------------------------------ value side
constexpr int kVpWarps = 16;
constexpr int kVpQueue = 4;  // routed tokens of a row whose value rows are fetched together

// One warp per memory row.  route: [rows][n_plan][C] (>= 0: merged into that row, -(1+r): appended as row r).
// The warp walks the decisions of all updates (a tile of them at a time in shared memory), queues the tokens that
// concern its row and fetches their value rows kVpQueue at a time (the loads are independent, the sums are formed
// afterwards in token order), so that the walk is bound by throughput and not by the latency of one row.
__global__ void __launch_bounds__(kVpWarps * 32, 2)
kvm_vpass_kernel(LayerDev L, Tensor4 v, Tensor4 gate, const kvm_update_plan* __restrict__ plan, int n_plan,
                 const int* __restrict__ route, MemoryDev mem, bf16* __restrict__ pool_v, long long pool_rows,
                 const int* __restrict__ ver_idx, long long ver_rows, int s_final, int tile_updates,
                 const int* __restrict__ status) {
  if (*status != 0) return;  // the chain gave up: its routing decisions and version tables are not to be trusted
  extern __shared__ __align__(16) unsigned char vsm[];
  short* rt = reinterpret_cast<short*>(vsm);                                        // [tile_updates][C] decisions of the tile
  int* vrow = reinterpret_cast<int*>(vsm + (size_t)tile_updates * L.C * 2);         // [n_plan] version_row of every update
  const int C = L.C, EPL = C / 32;            // EPL tokens per lane: 4 or 8
  const int log2c = C == 256 ? 8 : 7;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = blockIdx.y;
  const int b = row / L.Hkv, h = row % L.Hkv;
  const int r = blockIdx.x * kVpWarps + warp;  // this warp's memory row
  const bool live = r < s_final;
  const bool versions = pool_v != nullptr && ver_idx != nullptr;
  const int* route_row = route + (size_t)row * n_plan * C;
  const int* ver_row = ver_idx + (size_t)row * ver_rows + r;
  const bf16* v_base = v.row(b, h, 0) + lane * 4;
  const bf16* g_base = gate.row(b, h, 0);
  bf16* pool_row = pool_v + (size_t)row * pool_rows * HD + lane * 4;
  const bool gate_values = L.gate_values != 0;
  float x[4] = {0.f, 0.f, 0.f, 0.f};           // carried value sum of the row (bf16 values), elements 4*lane..
  float acc[4] = {0.f, 0.f, 0.f, 0.f};         // sum of the gated values of the update being collected
  float vl = 0.f;
  int acc_u = -1, acc_slot = -1, nq = 0;
  int q0 = 0, q1 = 0, q2 = 0, q3 = 0;          // queued tokens (bit 30: appended); the same in every lane
  bool born = false;
  for (int i = tid; i < n_plan; i += kVpWarps * 32) vrow[i] = plan[i].version_row;

  // the value view of the row after the update being collected: normalize(sum) * magnitude, into the pool row of that version
  auto finalize = [&]() {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[i] = bf16_round(x[i] + bf16_round(acc[i]));
      acc[i] = 0.f;
    }
    if (acc_slot >= 0) {
      const float n2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
      const float nrm = fmaxf(sqrtf(warp_sum(n2)), 1e-12f);
      float y[4] = {x[0], x[1], x[2], x[3]};
      divide_by(y, nrm);
      uint2 o;
      o.x = pack_bf16(y[0] * vl, y[1] * vl);
      o.y = pack_bf16(y[2] * vl, y[3] * vl);
      *reinterpret_cast<uint2*>(pool_row + (size_t)acc_slot * HD) = o;
    }
    acc_u = -1;
  };
  // fetch the queued tokens' value rows (and gates, and the pool slots of their updates) together, then apply in order
  auto flush = [&]() {
    const int item[kVpQueue] = {q0, q1, q2, q3};
    uint2 raw[kVpQueue];
    bf16 g[kVpQueue];
    int slot[kVpQueue];
#pragma unroll
    for (int i = 0; i < kVpQueue; ++i) {
      if (i < nq) {
        const int t = item[i] & 0x3fffffff;
        raw[i] = *reinterpret_cast<const uint2*>(v_base + (long long)t * v.st);
        g[i] = g_base[(long long)t * gate.st];
        const int vr = vrow[t >> log2c];
        slot[i] = (versions && vr >= 0) ? ver_row[vr] : -1;
      }
    }
#pragma unroll
    for (int i = 0; i < kVpQueue; ++i) {
      if (i < nq) {
        const int u = (item[i] & 0x3fffffff) >> log2c;
        if (acc_u >= 0 && acc_u != u) finalize();
        const float2 p0 = unpack_bf16(raw[i].x), p1 = unpack_bf16(raw[i].y);
        float o[4] = {p0.x, p0.y, p1.x, p1.y};
        const float gf = __bfloat162float(g[i]);
        if (item[i] & 0x40000000) {
          // the row is born from this token: value (gated where the layer says so) and magnitude
          const bool gated = u == 0 ? (L.gate_initial != 0) : (L.gate_appends != 0 && gate_values);
          if (u > 0 && gated) {
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = bf16_round(o[e] * gf);
          }
          vl = sqrtf(warp_sum(o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3]));  // initial rows: of the ungated value
#pragma unroll
          for (int e = 0; e < 4; ++e) x[e] = (u == 0 && gated) ? bf16_round(o[e] * gf) : o[e];
          born = true;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[e] += gate_values ? bf16_round(o[e] * gf) : o[e];
        }
        acc_u = u;
        acc_slot = slot[i];
      }
    }
    nq = 0;
  };
  auto push = [&](int item) {
    if (nq == 0) q0 = item;
    else if (nq == 1) q1 = item;
    else if (nq == 2) q2 = item;
    else q3 = item;
    if (++nq == kVpQueue) flush();
  };

  for (int u0 = 0; u0 < n_plan; u0 += tile_updates) {
    const int nu = min(tile_updates, n_plan - u0);
    __syncthreads();
    for (int i = tid; i < nu * C; i += kVpWarps * 32) rt[i] = (short)route_row[(size_t)u0 * C + i];
    __syncthreads();
    if (!live) continue;
    const unsigned want_m = (unsigned)(r & 0xffff) * 0x10001u, want_a = (unsigned)((-(1 + r)) & 0xffff) * 0x10001u;
    for (int uu = 0; uu < nu; ++uu) {
      const int u = u0 + uu;
      // two decisions per 32-bit word; token 2j of this lane's share in the low half of word j
      const unsigned* w = reinterpret_cast<const unsigned*>(rt + uu * C + lane * EPL);
      unsigned e4[4];
      if (EPL == 8) {
        const uint4 q4 = *reinterpret_cast<const uint4*>(w);
        e4[0] = q4.x; e4[1] = q4.y; e4[2] = q4.z; e4[3] = q4.w;
      } else {
        const uint2 q2w = *reinterpret_cast<const uint2*>(w);
        e4[0] = q2w.x; e4[1] = q2w.y;
        e4[2] = e4[3] = 0x80008000u;  // matches no row
      }
      // bit j: token 2j, bit 16 + j: token 2j + 1
      unsigned m_app = 0, m_mrg = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        m_app |= (__vcmpeq2(e4[j], want_a) & 0x00010001u) << j;
        m_mrg |= (__vcmpeq2(e4[j], want_m) & 0x00010001u) << j;
      }
      if (u == 0) m_mrg = 0;
      unsigned any = __ballot_sync(0xffffffffu, (m_app | m_mrg) != 0);
      while (any) {  // lanes in order = tokens in order
        const int src = __ffs(any) - 1;
        any &= any - 1;
        const unsigned ma = __shfl_sync(0xffffffffu, m_app, src);
        unsigned mm = __shfl_sync(0xffffffffu, m_mrg, src) | ma;
        const int t0 = (u << log2c) + src * EPL;
        while (mm) {  // next token of the lane: the lower of (2 * first low bit, 2 * first high bit + 1)
          const unsigned lo = mm & 0xffffu, hi = mm >> 16;
          const int jl = lo ? 2 * (__ffs(lo) - 1) : 64, jh = hi ? 2 * (__ffs(hi) - 1) + 1 : 64;
          const int j = min(jl, jh);
          const unsigned bit = 1u << ((j >> 1) + ((j & 1) << 4));
          mm &= ~bit;
          push((t0 + j) | ((ma & bit) ? 0x40000000 : 0));
        }
      }
    }
  }
  if (live) {
    flush();
    if (acc_u >= 0) finalize();
  }
  if (live && born) {  // the carried state and its final view
    const size_t off = ((size_t)row * mem.capacity + r) * HD + lane * 4;
    uint2 s;
    s.x = pack_bf16(x[0], x[1]);
    s.y = pack_bf16(x[2], x[3]);
    *reinterpret_cast<uint2*>(mem.v_sum + off) = s;
    if (lane == 0) mem.vlen[(size_t)row * mem.capacity + r] = vl;
    const float n2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
    const float nrm = fmaxf(sqrtf(warp_sum(n2)), 1e-12f);
    float y[4] = {x[0], x[1], x[2], x[3]};
    divide_by(y, nrm);
    uint2 o;
    o.x = pack_bf16(y[0] * vl, y[1] * vl);
    o.y = pack_bf16(y[2] * vl, y[3] * vl);
    *reinterpret_cast<uint2*>(mem.v_attn + off) = o;
  }
}

}  // namespace chain

// ------------------------------------------------------------------------------------------------ host side
// Cluster size for `rows` kv rows: the largest size (<= 8) that fits shared memory and whose clusters are all
// resident at once; if none is, the smallest that fits (the rows then run in waves).  0: the shape does not fit.
static int chain_tc_cluster_size(int C, int s_max, int rows) {
  using namespace chain;
  static std::mutex mu;
  static int fit[64][4][2];      // [device][log2 nc][C == 256]: co-resident clusters, 0 = not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int smallest = 0, best = 0;
  for (int lg = 0; lg <= 3; ++lg) {
    const int nc = 1 << lg;
    const Layout lay(C, s_max, nc);
    if (lay.total > (uint32_t)kMaxSmem) continue;
    if (!smallest) smallest = nc;
    int n_clusters;
    {
      std::lock_guard<std::mutex> lock(mu);
      n_clusters = fit[dev][lg][C == 256];
    }
    if (n_clusters == 0) {
      // the answer depends on the shared-memory size only through "one CTA per SM": ask with the largest size
      cudaLaunchConfig_t cfg = {};
      cfg.blockDim = dim3(kThreads);
      cfg.gridDim = dim3(nc * 64);
      cfg.dynamicSmemBytes = 200 * 1024;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = nc;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (cudaFuncSetAttribute(kvm_chain_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&n_clusters, kvm_chain_tc_kernel, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        n_clusters = -1;
      }
      if (n_clusters == 0) n_clusters = -1;
      std::lock_guard<std::mutex> lock(mu);
      fit[dev][lg][C == 256] = n_clusters;
    }
    if (n_clusters >= rows) best = nc;
  }
  return best ? best : smallest;
}

bool chain_tc_supported(int D, const LayerDev& L, int n_plan, int s_max, int rows) {
  if (D != 128 || (L.C != 128 && L.C != 256) || n_plan < 2 || s_max >= 32000) return false;
  if (L.gate_initial && !L.gate_keys) return false;  // the pre-pass only writes gated keys for layers that gate keys
  return chain_tc_cluster_size(L.C, s_max, rows) > 0;
}

// The chain for one batch: routing + key side, then the value side.  pk_all / gk_all: [rows][n_plan*C][D] from the
// pre-pass; route: [rows][n_plan][C].
bool vside_setup(const LayerDev& L, int batch, long long T, Tensor4 v, Tensor4 gate, const kvm_update_plan* plan_dev, int n_plan,
                 int s_max, bf16* pool_v, long long pool_rows, const int* ver_idx, long long ver_rows, const int* route,
                 unsigned* tbits, int* status, uint32_t wait_limit, vside::DeltaArgs* a, vside::Maps* maps);
size_t vside_smem_bytes(int C, int s_max);
cudaError_t launch_vside(vside::DeltaArgs a, const vside::Maps& maps, Tensor4 v, MemoryDev mem, const int* born, cudaStream_t stream);

cudaError_t launch_chain_tc(const LayerDev& L, int batch, long long T, Tensor4 v, Tensor4 gate, const kvm_update_plan* plan_dev,
                            int n_plan, int s_max, MemoryDev mem, bf16* pool_k, bf16* pool_v, long long pool_rows, int* ver_idx,
                            long long ver_rows, const bf16* pk_all, const bf16* gk_all, int* route, int* born, unsigned* tbits,
                            int* status, uint32_t wait_limit, uint32_t test_flags, cudaStream_t stream) {
  using namespace chain;
  const int rows = batch * L.Hkv, C = L.C;
  const int nc = chain_tc_cluster_size(C, s_max, rows);
  if (nc <= 0) return cudaErrorInvalidConfiguration;
  const Layout lay(C, s_max, nc);
  const long long n_tok = (long long)n_plan * C;
  Maps maps;
  {
    const cuuint64_t dims[2] = {(cuuint64_t)HD, (cuuint64_t)((long long)rows * n_tok)};
    const cuuint64_t strides[1] = {(cuuint64_t)HD * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)C};
    if (!encode_bf16_map(&maps.pk, pk_all, 2, dims, strides, box) || !encode_bf16_map(&maps.gk, gk_all, 2, dims, strides, box))
      return cudaErrorInvalidValue;
  }
  Args a;
  a.L = L; a.plan = plan_dev; a.n_plan = n_plan; a.nc = nc; a.lg = nc == 8 ? 3 : nc == 4 ? 2 : nc == 2 ? 1 : 0; a.s_max = s_max; a.n_tok = n_tok;
  a.k_sum = mem.k_sum; a.k_attn = mem.k_attn; a.capacity = mem.capacity;
  a.pool_k = ver_idx ? pool_k : nullptr; a.pool_rows = pool_rows; a.ver_idx = ver_idx; a.ver_rows = ver_rows;
  a.route = route; a.born = born; a.status = status; a.wait_limit = wait_limit; a.test_flags = test_flags;
  a.progress = nullptr; a.chain_done = nullptr; a.chain_ctas = rows * nc;
  // The value side (with versions): deltas of every (kv row, update) on the tensor cores, then one warp per memory row.
  // SMs the routing leaves free take value-delta jobs inside the same launch, as whole clusters behind the routing's,
  // following the routing through a flag per (kv row, CTA); three control words and the flags live behind the bit table.
  const bool vside_on = ver_idx && pool_v;
  vside::DeltaArgs va = {};
  vside::Maps vmaps = {};
  int spare = 0;
  size_t smem_bytes = lay.total;
  cudaError_t e;
  if (vside_on) {
    if (!vside_setup(L, batch, T, v, gate, plan_dev, n_plan, s_max, pool_v, pool_rows, ver_idx, ver_rows, route, tbits, status,
                     wait_limit, &va, &vmaps))
      return cudaErrorInvalidValue;
    // control words: job counter, finished routing CTAs, given-back jobs (count, taken), then the progress flags and
    // the list of given-back jobs (one per spare CTA at most)
    int* ctrl = reinterpret_cast<int*>(tbits + (size_t)rows * n_plan * va.words);
    e = cudaMemsetAsync(ctrl, 0, (size_t)(4 + rows * nc) * sizeof(int), stream);
    if (e != cudaSuccess) return e;
    va.queue = ctrl;
    int dev = 0, n_sm = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    spare = std::max(0, (n_sm - rows * nc) / nc) * nc;
    if (vside_smem_bytes(C, s_max) > (size_t)kMaxSmem) spare = 0;
    if (spare > 0) {
      a.chain_done = ctrl + 1;
      a.progress = ctrl + 4;
      va.n_given_back = ctrl + 2;
      va.given_back_taken = ctrl + 3;
      va.given_back = ctrl + 4 + rows * nc;
      va.chain_done = a.chain_done;
      va.progress = a.progress;
      va.nc = nc;
      va.chain_ctas = rows * nc;
      smem_bytes = std::max(smem_bytes, vside_smem_bytes(C, s_max));
    }
  }
  e = cudaFuncSetAttribute(kvm_chain_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.gridDim = dim3(rows * nc + spare);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = nc;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kvm_chain_tc_kernel, a, maps, va, vmaps);
  if (e != cudaSuccess) return e;
  if (vside_on) return launch_vside(va, vmaps, v, mem, born, stream);
  // Without (only the final memory is wanted): one warp per memory row walks the routing decisions itself, as many
  // updates as fit 64 KB per tile
  const int tile_updates = std::max(1, std::min(n_plan, (64 * 1024) / (C * 2)));
  const size_t vsmem = (size_t)tile_updates * C * 2 + (size_t)((n_plan + 3) & ~3) * 4;
  e = cudaFuncSetAttribute(kvm_vpass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)vsmem);
  if (e != cudaSuccess) return e;
  dim3 vgrid((unsigned)ceil_div(s_max, kVpWarps), rows);
  kvm_vpass_kernel<<<vgrid, kVpWarps * 32, vsmem, stream>>>(L, v, gate, plan_dev, n_plan, route, mem, ver_idx ? pool_v : nullptr,
                                                            pool_rows, ver_idx, ver_rows, s_max, tile_updates, status);
  return cudaGetLastError();
}

}  // namespace kvm
