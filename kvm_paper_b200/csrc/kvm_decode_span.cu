// Several decode tokens per sequence in one pass over the keys, for tokens whose inputs are all on the device
// (teacher-forced decoding).  Between two memory updates of a sequence the tokens attend to the same memory and to
// windows that begin at the same token, so a kv row's keys and values are streamed once for all of them: the tokens
// of a span are columns of the score MMAs next to the query heads of the kv head.  Follows model/kvm_mixer.py:572-713
// (single-token steps) token by token: same chunks, same order of every sum.
//   kvm_span_write_kernel   the span's keys, values and gates into the rings (and, inside the first block, the memory)
//   kvm_span_attn_kernel    attention of all tokens of the spans, persistent
// 64 sequences x 16 heads x 128, 1024 + ~400 rows each, 32 tokens: 740 MB are read once instead of 32 times.
#include <mutex>
#include <type_traits>

#include "kvm_decode.cuh"

namespace kvm {

// Rows that a token of the span must not see have probability 0 for it, but 0 * inf is not 0.  So the infinities and NaN among
// the values of the span's own tokens (older ones are everybody's) are taken out of the products and added to the sums of
// the tokens that see them: whatever their weight, the sum is what they make of it.  The write kernel marks a launch that has
// any, in the launch counter, and only such launches go through it.  64 sequences, 16 heads x 128, 32 tokens: 492.5 us without
// any of it, 496.5 with it, 504 with a look at every value in the attention kernel's loop.
constexpr int kOddMark = 1 << 30;
// Two bf16 values: an infinity or NaN among them / 0 in the place of those.
__device__ __forceinline__ bool not_finite2(uint32_t w) { return (w & 0x7f80u) == 0x7f80u || (w & 0x7f800000u) == 0x7f800000u; }
__device__ __forceinline__ uint32_t finite2(uint32_t w) {
  return ((w & 0x7f80u) == 0x7f80u ? 0u : w & 0xffffu) | ((w & 0x7f800000u) == 0x7f800000u ? 0u : w & 0xffff0000u);
}

// Rows [r0, r1) of a chunk's values without them (one warp).
template <int D>
__device__ __forceinline__ void clear_odd_values(unsigned char* sV, int r0, int r1, int lane) {
#pragma unroll 1
  for (int p = r0 * (D / 8) + lane; p < r1 * (D / 8); p += 32) {
    uint4* at = reinterpret_cast<uint4*>(sV + dec_piece<D>(p / (D / 8), p % (D / 8)));
    const uint4 u = *at;
    *at = make_uint4(finite2(u.x), finite2(u.y), finite2(u.z), finite2(u.w));
  }
  tc::fence_proxy_async();
  __syncwarp();
}

// One warp per (token of the span, kv row).
template <int D>
__global__ void __launch_bounds__(256)
kvm_span_write_kernel(LayerDev L, DecodeCacheDev cache, Tensor4 k, Tensor4 v, Tensor4 gate, long long kv_step, long long gate_step,
                      const __grid_constant__ SpanSet spans, int rows, int* __restrict__ done_counter) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= rows) return;
  const int b = row / L.Hkv, h = row % L.Hkv, i = blockIdx.y;
  if (i >= spans.count[b]) return;
  const int past = cache.total_len[b];
  const bool direct = past < L.C && cache.state_len[b] == past;  // (then so is every token of the span: it ends with the block)
  const long long at = spans.first[b] + i;
  k.ptr += at * kv_step;
  v.ptr += at * kv_step;
  gate.ptr += at * gate_step;
  const uint4 u = write_new_token<D>(L, cache, k, v, gate, b, h, past + i, direct, lane);
  const bool odd = lane >= D / 8 && (not_finite2(u.x) || not_finite2(u.y) || not_finite2(u.z) || not_finite2(u.w));
  if (__any_sync(0xffffffffu, odd) && lane == 0) atomicOr(done_counter, kOddMark);
}

// Shared-memory layout (byte offsets); NH = tiles of 8 columns, a column = (token of the span, query head of the kv head)
struct SpanSmem {
  size_t stages, stage_bytes, qst, ored, wred, meta, bars, temps, seq, total;
  __host__ __device__ SpanSmem(int D, int NH, int Hq, int nb, int ST) {
    size_t off = 0;
    stage_bytes = (size_t)2 * kDecChunk * D * 2;
    stages = off; off += (size_t)ST * stage_bytes;
    qst = off;    off += (size_t)ST * NH * 8 * (D + 8) * 2;             // [slot][column][padded D] bf16
    ored = off;   off += (size_t)kDecConsumers * 8 * (D + 4) * 4;       // [warp][column of a tile][padded D] fp32
    wred = off;   off += (size_t)2 * kDecConsumers * 8 * 4;             // per-warp running max / sum of a tile
    meta = off;   off += (size_t)ST * 48;                               // per-stage chunk description (12 ints)
    bars = off;   off += (size_t)(2 * ST + 1) * 8;
    temps = off;  off += (size_t)2 * Hq * 4;
    seq = off;    off += (size_t)(3 * nb + 4) * 4;                      // per sequence: S, total, chunk prefix
    total = (off + 15) & ~(size_t)15;
  }
};

// Threads: two warpgroups of math warps and one whose first warp is the producer (the others only take part in the
// set-up).  At D = 128 with four column tiles a math thread's running output alone is 128 registers: the math warpgroups
// take the registers the producer's warpgroup does not need (2 x 128 x 216 + 128 x 72 = 384 x 168, the launch's total).
constexpr int kSpanThreads = kDecConsumers * 32 + 128;
__device__ __forceinline__ void registers_for_math() { asm volatile("setmaxnreg.inc.sync.aligned.u32 216;"); }
__device__ __forceinline__ void registers_for_copies() { asm volatile("setmaxnreg.dec.sync.aligned.u32 72;"); }

// The structure is kvm_decode_attn_kernel's: one CTA per SM takes an equal contiguous range of all (sequence, kv head,
// chunk) triples, a producer warp streams it through ST stages, eight math warps own 16 keys of every chunk each.  What
// differs: NH tiles of 8 columns (the query fragments are read from shared memory at every chunk, registers hold the
// running output), a causal limit per token in the window's last chunks, the merge of the warps one tile at a time, and
// partial results of cut rows by CTA (a CTA cuts at most its first and its last row), so that they do not grow with the
// batch.
template <int D, int ST, int NH>
__global__ void __launch_bounds__(kSpanThreads, 1)
kvm_span_attn_kernel(LayerDev L, DecodeCacheDev cache, Tensor4 q, long long q_step, const __grid_constant__ SpanSet spans,
                     const __grid_constant__ UpdateSet upd, float* __restrict__ partial, int* __restrict__ row_counters,
                     int* __restrict__ done_counter, int* __restrict__ status, bf16* __restrict__ out, long long out_step,
                     float sm_scale, int nb, const __grid_constant__ DecMaps maps) {
  constexpr int STRQ = D + 8, STRO = D + 4;
  constexpr int KS = D / 16, DT16 = D / 16;
  constexpr int CH = kDecChunk, NW = kDecConsumers, NC = NH * 8;
  constexpr int CPR = D / 8;
  constexpr int BOXW = D >= 64 ? 64 : D;
  constexpr int NBLK = D / BOXW;
  constexpr uint32_t kBoxBytes = (uint32_t)kDecBoxRows * BOXW * 2;
  extern __shared__ __align__(1024) unsigned char span_smem[];
  const int G = L.Hq / L.Hkv, Hkv = L.Hkv;
  const SpanSmem lay(D, NH, L.Hq, nb, ST);
  unsigned char* stage0 = span_smem + lay.stages;
  bf16* qst = reinterpret_cast<bf16*>(span_smem + lay.qst);
  float* ored = reinterpret_cast<float*>(span_smem + lay.ored);
  float* wmax = reinterpret_cast<float*>(span_smem + lay.wred);
  float* wsum = wmax + NW * 8;
  int* meta = reinterpret_cast<int*>(span_smem + lay.meta);
  uint64_t* full = reinterpret_cast<uint64_t*>(span_smem + lay.bars);
  uint64_t* empty = full + ST;
  uint64_t* fbar = empty + ST;
  float* temp_mem = reinterpret_cast<float*>(span_smem + lay.temps);
  float* temp_win = temp_mem + L.Hq;
  int* sq_S = reinterpret_cast<int*>(span_smem + lay.seq);
  int* sq_tot = sq_S + nb;
  int* cpre = sq_tot + nb;
  __shared__ int s_flag, s_abort, s_odd;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int C = L.C, W = L.W, WC = L.W * L.C;
  const int cap = cache.mem.capacity;

  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < ST; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], NW);
    }
    tc::mbar_init(fbar, NW);
    tc::fence_barrier_init();
    s_abort = 0;
    cpre[0] = 0;
  }
  for (int h = tid; h < L.Hq; h += kSpanThreads) {
    temp_mem[h] = sm_scale * L.state_temp[h] * kLog2e;
    temp_win[h] = sm_scale * L.front_temp[h] * kLog2e;
  }
  // Columns past the last token of a span hold zeros, or what an earlier, longer span of the launch left in the slot; their
  // results are dropped (c >= n_col below).
  for (int i = tid; i < ST * NC * STRQ / 2; i += kSpanThreads) reinterpret_cast<uint32_t*>(qst)[i] = 0u;
  pdl_wait();
  if (tid == kSpanThreads - 1) s_odd = __ldcg(done_counter) & kOddMark;  // (ahead of this CTA's own count)
  for (int b = tid; b < nb; b += kSpanThreads) {
    const int n = spans.count[b];
    int cnt = 0, S = 0, total = 0;
    if (n > 0) {
      const int past = cache.total_len[b], n_app = upd.appended(b);
      S = cache.state_len[b] + (n_app > 0 ? n_app : 0);
      if (past < C && S == past) S += n;  // the tokens become memory rows directly
      total = past + n;
      cnt = dec_geometry(S, total, C, W).chunks();
    }
    sq_S[b] = S;
    sq_tot[b] = total;
    cpre[b + 1] = cnt;
  }
  tc::fence_proxy_async();  // the zeroed query slots -> before the copies into them
  __syncthreads();
  if (warp == 0) {  // inclusive scan of cpre[1..nb]
    int carry = 0;
    for (int base = 0; base < nb; base += 32) {
      const int i = base + lane;
      int x = i < nb ? cpre[i + 1] : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
      }
      if (i < nb) cpre[i + 1] = x + carry;
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
  }
  __syncthreads();
  const int total_f = cpre[nb] * Hkv;
  // (at least two chunks per CTA, as in the single-token kernel, which has no more partial results to give away)
  const int per = max(2, (total_f + (int)gridDim.x - 1) / (int)gridDim.x);
  const int cta = blockIdx.x;
  const bool has_work = cta * per < total_f;
  const int f_begin = has_work ? cta * per : 0, f_end = has_work ? min(total_f, f_begin + per) : 0;
  const int nloc = f_end - f_begin;
  volatile int* abort_flag = &s_abort;
  // every CTA has read the lengths once it has counted itself; the last one advances them (see kvm_decode_attn_kernel)
  if (warp == NW - 1) {
    int is_last = 0;
    if (lane == 0) {
      __threadfence();
      is_last = (atomicAdd(done_counter, 1) & ~kOddMark) == (int)gridDim.x - 1;
    }
    if (__shfl_sync(0xffffffffu, is_last, 0)) {
      for (int b = lane; b < nb; b += 32) {
        if (cpre[b + 1] != cpre[b]) {
          cache.total_len[b] = sq_tot[b];
          cache.state_len[b] = sq_S[b];
        }
      }
      if (lane == 0) *done_counter = 0;
    }
  }

  constexpr bool kSplitRegisters = NH == 4 && D == 128;
  if (!has_work) {
    // nothing to stream
  } else if (warp >= NW) {
    if constexpr (kSplitRegisters) registers_for_copies();
    if (warp == NW) {
    // =============================================================== producer warp (lanes in lockstep)
    int pb, ph, pc, pcb, slot = -1;
    DecGeo pg;
    {
      int lo = 0, hi = nb - 1;  // last b with cpre[b] * Hkv <= f_begin: its chunk range holds f_begin
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (cpre[mid] * Hkv <= f_begin) lo = mid; else hi = mid - 1;
      }
      pb = lo;
      pcb = cpre[pb + 1] - cpre[pb];
      const int rem = f_begin - cpre[pb] * Hkv;
      ph = rem / pcb;
      pc = rem - ph * pcb;
      pg = dec_geometry(sq_S[pb], sq_tot[pb], C, W);
    }
    for (int i = 0; i < nloc; ++i) {
      const int s = i % ST;
      if (i >= ST) {
        const bool ok = dec_wait(&empty[s], (uint32_t)((i / ST - 1) & 1), abort_flag);
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) {
            s_abort = 1;
            atomicExch(status, KVM_ERR_DEVICE_TIMEOUT);
          }
          break;
        }
      }
      const int row = pb * Hkv + ph;
      int n, y0, w_base = 0;  // rows of the chunk, first of them in its array, its window index
      const bool is_mem = pc < pg.c_mem;
      if (is_mem) {
        n = min(CH, pg.S_act - pc * CH);
        y0 = row * cap + pc * CH;
      } else if (pc < pg.c_mem + pg.c_a) {
        w_base = (pc - pg.c_mem) * CH;
        n = min(CH, pg.len_a - w_base);
        y0 = row * WC + pg.slot0 + w_base;
      } else {
        const int c = (pc - pg.c_mem - pg.c_a) * CH;
        n = min(CH, pg.len_b - c);
        y0 = row * WC + c;
        w_base = pg.len_a + c;
      }
      const int n_tok = spans.count[pb];
      const bool first = i == 0 || pc == 0;
      const bool last = i == nloc - 1 || pc == pcb - 1;
      // the queries of a row stay in their slot while the row is being worked on: at most ST rows are (every row has a
      // chunk of its own among the ST stages)
      if (first) slot = (slot + 1) % ST;
      const int groups = (n + kDecBoxRows - 1) / kDecBoxRows;
      if (lane == 0) {
        int seg = 0, nsegs = 1, first_cta = cta;
        if (last) {
          const int row_f = cpre[pb] * Hkv + ph * pcb;
          first_cta = row_f / per;
          seg = cta - first_cta;
          nsegs = (row_f + pcb - 1) / per - first_cta + 1;
        }
        int* m = meta + s * 12;
        m[0] = n | (is_mem ? 1 << 16 : 0) | (first ? 1 << 17 : 0) | (last ? 1 << 18 : 0) | (ph << 20);
        m[1] = pb;
        m[2] = seg;
        m[3] = nsegs;
        m[4] = w_base;
        m[5] = sq_tot[pb] - n_tok + 1 - bswa_begin_dev(sq_tot[pb], C, W);  // window rows the first token of the span sees
        m[6] = n_tok | (slot << 16);
        m[7] = first_cta;
        tc::mbar_arrive_expect_tx(&full[s], (uint32_t)groups * 2u * NBLK * kBoxBytes + (first ? (uint32_t)(n_tok * G * D * 2) : 0u));
      }
      __syncwarp();
      if (lane < groups) {
        const CUtensorMap* mk = is_mem ? &maps.mem_k : &maps.ring_k;
        const CUtensorMap* mv = is_mem ? &maps.mem_v : &maps.ring_v;
        unsigned char* dk = stage0 + (size_t)s * lay.stage_bytes + (size_t)lane * kDecBoxRows * (BOXW * 2);
        unsigned char* dv = dk + (size_t)CH * D * 2;
        const int y = y0 + lane * kDecBoxRows;
#pragma unroll
        for (int blk = 0; blk < NBLK; ++blk) {
          tc::tma_load_2d(dk + (size_t)blk * CH * 128, mk, blk * 64, y, &full[s]);
          tc::tma_load_2d(dv + (size_t)blk * CH * 128, mv, blk * 64, y, &full[s]);
        }
      }
      if (first)
        for (int c = lane; c < n_tok * G; c += 32)  // column c: token c / G, query head c % G of the kv head
          tc::bulk_g2s(qst + ((size_t)slot * NC + c) * STRQ,
                       q.row(pb, ph * G + c % G, 0) + (long long)(spans.first[pb] + c / G) * q_step, D * 2, &full[s]);
      if (++pc == pcb) {
        pc = 0;
        if (++ph == Hkv) {
          ph = 0;
          ++pb;
          while (pb < nb && cpre[pb + 1] == cpre[pb]) ++pb;
          if (pb < nb) {
            pcb = cpre[pb + 1] - cpre[pb];
            pg = dec_geometry(sq_S[pb], sq_tot[pb], C, W);
          }
        }
      }
    }
    }
  } else {
    // ==================================================================================== math warps
    if constexpr (kSplitRegisters) registers_for_math();
    // (layouts as in kvm_decode_attn_kernel: keys on M, columns on N; thread (g, t) holds keys g, g+8, columns 2t, 2t+1)
    float m_run[NH][2], l_run[NH][2];
    float o[NH][DT16][4];
    int col_tok[NH][2];   // token of this thread's accumulator columns
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
      for (int j = 0; j < 2; ++j) col_tok[h][j] = (h * 8 + t * 2 + j) / G;
    const int krow = warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
    const int vrow = warp * 16 + (lane & 7) + (lane >> 4) * 8;
    uint32_t fphase = 0;
    bool alive = true;
    const bool odd = s_odd != 0;
    auto rendezvous = [&]() -> bool {
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(fbar);
      const bool ok = dec_wait(fbar, fphase & 1, abort_flag);
      ++fphase;
      return __all_sync(0xffffffffu, ok);
    };

    for (int i = 0; i < nloc && alive; ++i) {
      const int s = i % ST;
      if (!__all_sync(0xffffffffu, dec_wait(&full[s], (uint32_t)((i / ST) & 1), abort_flag))) {
        alive = false;
        break;
      }
      const int4 md = *reinterpret_cast<const int4*>(meta + s * 12), md2 = *reinterpret_cast<const int4*>(meta + s * 12 + 4);
      const int n = md.x & 0xffff, hkv = md.x >> 20;
      const bool is_mem = (md.x >> 16) & 1, first = (md.x >> 17) & 1, last = (md.x >> 18) & 1;
      const int n_tok = md2.z & 0xffff;
      const bf16* qs = qst + (size_t)(md2.z >> 16) * NC * STRQ;
      if (first) {
#pragma unroll
        for (int h = 0; h < NH; ++h) {
          m_run[h][0] = m_run[h][1] = -INFINITY;
          l_run[h][0] = l_run[h][1] = 0.f;
#pragma unroll
          for (int dt = 0; dt < DT16; ++dt) o[h][dt][0] = o[h][dt][1] = o[h][dt][2] = o[h][dt][3] = 0.f;
        }
      }
      if (warp * 16 < n) {
        unsigned char* sK = stage0 + (size_t)s * lay.stage_bytes;
        unsigned char* sV = sK + (size_t)CH * D * 2;
        if (n < warp * 16 + 16) {
          // ragged end of the run inside this warp's rows: values are zeroed (0 * garbage must stay finite)
          const int cnt = (warp * 16 + 16 - n) * CPR;
          for (int p = lane; p < cnt; p += 32) {
            const int r = n + p / CPR, j = p % CPR;
            *reinterpret_cast<uint4*>(sV + dec_piece<D>(r, j)) = make_uint4(0, 0, 0, 0);
          }
          tc::fence_proxy_async();
          __syncwarp();
        }
        // rows of the chunk that the first token sees; token i sees i more (memory rows: everybody sees all)
        const int lim = is_mem ? CH : md2.y - md2.x;
        if (odd && lim < warp * 16 + 16)  // (rows that not every token sees)
          clear_odd_values<D>(sV, max(lim, warp * 16), min(n, warp * 16 + 16), lane);
        float sacc[NH][4];
#pragma unroll
        for (int h = 0; h < NH; ++h) sacc[h][0] = sacc[h][1] = sacc[h][2] = sacc[h][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          uint32_t ka[4];
          ldmatrix_x4(ka, sK + dec_piece<D>(krow, ks * 2 + (lane >> 4)));
#pragma unroll
          for (int h = 0; h < NH; ++h) {
            const bf16* qp = qs + (size_t)(h * 8 + g) * STRQ + ks * 16 + t * 2;
            mma_bf16_16816(sacc[h], ka, *reinterpret_cast<const uint32_t*>(qp), *reinterpret_cast<const uint32_t*>(qp + 8));
          }
        }
        const int r_lo = warp * 16 + g, r_hi = r_lo + 8;
        const float* temp = is_mem ? temp_mem : temp_win;
        uint32_t pb[NH][2];
#pragma unroll
        for (int h = 0; h < NH; ++h) {
          float mx[2], f[2];
          bool grew = false;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int tok = col_tok[h][j];
            const float sc = temp[hkv * G + (h * 8 + t * 2 + j) - tok * G];
            const int vis = min(n, lim + (is_mem ? 0 : tok));
            sacc[h][j] = r_lo < vis ? sacc[h][j] * sc : -INFINITY;
            sacc[h][2 + j] = r_hi < vis ? sacc[h][2 + j] * sc : -INFINITY;
            float x = fmaxf(sacc[h][j], sacc[h][2 + j]);
            x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 4));
            x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 8));
            x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 16));
            mx[j] = x;
            grew = grew || x > m_run[h][j];
          }
          if (__any_sync(0xffffffffu, grew)) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const float mn = fmaxf(m_run[h][j], mx[j]);
              f[j] = m_run[h][j] == -INFINITY ? 0.f : exp2f(m_run[h][j] - mn);
              m_run[h][j] = mn;
              l_run[h][j] *= f[j];
            }
#pragma unroll
            for (int dt = 0; dt < DT16; ++dt) {
              o[h][dt][0] *= f[0];
              o[h][dt][1] *= f[1];
              o[h][dt][2] *= f[0];
              o[h][dt][3] *= f[1];
            }
          }
          const float mu0 = m_run[h][0] == -INFINITY ? 0.f : m_run[h][0];
          const float mu1 = m_run[h][1] == -INFINITY ? 0.f : m_run[h][1];
          const float p0 = exp2f(sacc[h][0] - mu0), p1 = exp2f(sacc[h][1] - mu1);
          const float p2 = exp2f(sacc[h][2] - mu0), p3 = exp2f(sacc[h][3] - mu1);
          l_run[h][0] += p0 + p2;
          l_run[h][1] += p1 + p3;
          pb[h][0] = movmatrix_trans(pack_bf16(p0, p1));
          pb[h][1] = movmatrix_trans(pack_bf16(p2, p3));
        }
#pragma unroll
        for (int dt = 0; dt < DT16; ++dt) {
          uint32_t va[4];
          ldmatrix_x4_trans(va, sV + dec_piece<D>(vrow, dt * 2 + ((lane >> 3) & 1)));
#pragma unroll
          for (int h = 0; h < NH; ++h) mma_bf16_16816(o[h][dt], va, pb[h][0], pb[h][1]);
        }
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&empty[s]);  // this warp is done with the stage (and with the row's queries, if the row ends)
      if (!last) continue;

      // ---- the CTA leaves this kv row: merge the warps' running states, a tile of 8 columns at a time
      const int b = md.y, seg = md.z, nsegs = md.w, first_cta = md2.w;
      const int n_col = n_tok * G;
      const int row = b * Hkv + hkv;
      bf16* out_row = out + (long long)spans.first[b] * out_step + (size_t)b * L.Hq * D + (size_t)hkv * G * D;
      // this CTA's slot for a row that it shares: the row it begins with, or the one it ends with
      float* my_part = partial + (size_t)(cta * 2 + (seg == 0 ? 1 : 0)) * NC * (D + 2);
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        if (h * 8 >= n_col) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float l = l_run[h][j];
          l += __shfl_xor_sync(0xffffffffu, l, 4);
          l += __shfl_xor_sync(0xffffffffu, l, 8);
          l += __shfl_xor_sync(0xffffffffu, l, 16);
          const int cc = t * 2 + j;
          if (g == 0) {
            wmax[warp * 8 + cc] = m_run[h][j];
            wsum[warp * 8 + cc] = l;
          }
          float* dst = ored + ((size_t)warp * 8 + cc) * STRO + g;
#pragma unroll
          for (int dt = 0; dt < DT16; ++dt) {
            dst[dt * 16] = o[h][dt][j];
            dst[dt * 16 + 8] = o[h][dt][2 + j];
          }
        }
        alive = alive && rendezvous();
        if (alive) {
          for (int e = tid; e < 8 * D; e += NW * 32) {  // whole warps stay on one column
            const int cc = e / D, d = e % D, c = h * 8 + cc;
            if (c >= n_col) break;
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < NW; ++w) M = fmaxf(M, wmax[w * 8 + cc]);
            float lsum = 0.f, acc = 0.f;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
              const float f = wmax[w * 8 + cc] == -INFINITY ? 0.f : exp2f(wmax[w * 8 + cc] - M);
              lsum += f * wsum[w * 8 + cc];
              acc += f * ored[((size_t)w * 8 + cc) * STRO + d];
            }
            if (nsegs == 1) {
              out_row[(long long)(c / G) * out_step + (c % G) * D + d] = __float2bfloat16_rn(lsum > 0.f ? acc / lsum : 0.f);
            } else {
              float* pout = my_part + (size_t)c * (D + 2);
              pout[2 + d] = acc;
              if (d == 0) {
                pout[0] = M;
                pout[1] = lsum;
              }
            }
          }
          if (nsegs > 1) __threadfence();
          alive = rendezvous();  // the merge buffers are free again (and the partial results fenced)
        }
      }
      if (!alive) break;
      bool combine = false;
      if (nsegs > 1) {  // the last CTA of this kv row combines the partial results
        if (tid == 0) s_flag = atomicAdd(&row_counters[row], 1) == nsegs - 1;
        if (!rendezvous()) {
          alive = false;
          break;
        }
        combine = s_flag != 0;
        if (combine) {
          __threadfence();
          for (int e = tid; e < n_col * D; e += NW * 32) {
            const int c = e / D, d = e % D;
            // segment s2 lies with CTA first_cta + s2: as the row it ends with (s2 = 0) or begins with
            auto part = [&](int s2) { return partial + ((size_t)((first_cta + s2) * 2 + (s2 == 0 ? 1 : 0)) * NC + c) * (D + 2); };
            float M = -INFINITY;
            for (int s2 = 0; s2 < nsegs; ++s2) M = fmaxf(M, __ldcg(part(s2)));
            float Lsum = 0.f, a = 0.f;
            for (int s2 = 0; s2 < nsegs; ++s2) {
              const float ms = __ldcg(part(s2));
              const float w = ms == -INFINITY ? 0.f : exp2f(ms - M);
              Lsum += w * __ldcg(part(s2) + 1);
              a += w * __ldcg(part(s2) + 2 + d);
            }
            out_row[(long long)(c / G) * out_step + (c % G) * D + d] = __float2bfloat16_rn(Lsum > 0.f ? a / Lsum : 0.f);
          }
          if (tid == 0) row_counters[row] = 0;
        }
        if (!rendezvous()) {  // the flag may be set for another row again
          alive = false;
          break;
        }
      }
      if (odd && (nsegs == 1 || combine)) {  // the values that were taken out, to the results of the tokens that see them
#pragma unroll 1
        for (int e = tid; e < n_col * D; e += NW * 32) {
          const int c = e / D, d = e % D;
          float sum = 0.f;
#pragma unroll 1
          for (int i = 0; i <= c / G; ++i) {
            const float x = __bfloat162float(cache.ring_v[((size_t)row * WC + (sq_tot[b] - n_tok + i) % WC) * D + d]);
            if (!(fabsf(x) < INFINITY)) sum += x;
          }
          bf16* y = &out_row[(long long)(c / G) * out_step + (c % G) * D + d];
          *y = __float2bfloat16_rn(__bfloat162float(*y) + sum);
        }
      }
    }
    if (!alive && lane == 0) {
      s_abort = 1;
      atomicExch(status, KVM_ERR_DEVICE_TIMEOUT);
    }
  }
  if (*abort_flag) {
    // somebody gave up: copies of this CTA may still be in flight, give them a bounded time to land
    for (int k2 = 0; k2 < 1000; ++k2) __nanosleep(1000);
  }
}

// ------------------------------------------------------------------------------------- host side
template <int D, int ST, int NH>
static cudaError_t launch_span_attn(const LayerDev& L, int batch, const DecodeCacheDev& cache, Tensor4 q, long long q_step,
                                    const SpanSet& spans, const UpdateSet& upd, float* partial, int* counters, bf16* out,
                                    long long out_step, int n_sm, const DecMaps& maps, cudaStream_t stream) {
  const SpanSmem lay(D, NH, L.Hq, batch, ST);
  auto kern = kvm_span_attn_kernel<D, ST, NH>;
  static size_t smem_set[kMaxDevices] = {0};  // largest dynamic shared memory enabled so far, per device
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (lay.total > smem_set[dev]) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lay.total);
      if (e != cudaSuccess) return e;
      smem_set[dev] = lay.total;
    }
  }
  const int rows = batch * L.Hkv;
  kern<<<n_sm, kSpanThreads, lay.total, stream>>>(L, cache, q, q_step, spans, upd, partial, counters, counters + rows, counters + rows + batch,
                                                 out, out_step, 1.0f / sqrtf((float)D), batch, maps);
  return cudaGetLastError();
}

template <int D>
static cudaError_t launch_span(const LayerDev& L, int batch, const DecodeCacheDev& cache, Tensor4 q, Tensor4 k, Tensor4 v, Tensor4 gate,
                               long long q_step, long long kv_step, long long gate_step, const SpanSet& spans, int max_count,
                               const UpdateSet& upd, bf16* pk_scr, float* partial, int* counters, bf16* out, long long out_step,
                               cudaStream_t stream) {
  const int rows = batch * L.Hkv, n_sm = device_sm_count();
  DecMaps maps;
  if (!decode_maps(cache, (uint64_t)rows, cache.mem.capacity, L.W * L.C, D, &maps)) return cudaErrorInvalidValue;
  cudaError_t e;
  if (upd.n > 0 && (e = decode_update(D, L, batch, cache, upd, pk_scr, stream)) != cudaSuccess) return e;
  kvm_span_write_kernel<D><<<dim3((rows + 7) / 8, max_count), 256, 0, stream>>>(L, cache, k, v, gate, kv_step, gate_step, spans, rows, counters + rows);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  // stages: as many chunks of keys and values as fit next to the merge buffers (two of 64 KB at D = 128)
  constexpr int ST = D == 128 ? 2 : 4;
  const int cols = max_count * (L.Hq / L.Hkv);
  auto run = [&](auto nh) {
    return launch_span_attn<D, ST, decltype(nh)::value>(L, batch, cache, q, q_step, spans, upd, partial, counters, out, out_step, n_sm,
                                                        maps, stream);
  };
  if (cols <= 8) return run(std::integral_constant<int, 1>());
  if (cols <= 16) return run(std::integral_constant<int, 2>());
  return run(std::integral_constant<int, 4>());
}

cudaError_t span_dispatch(int D, const LayerDev& L, int batch, const DecodeCacheDev& cache, Tensor4 q, Tensor4 k, Tensor4 v, Tensor4 gate,
                          long long q_step, long long kv_step, long long gate_step, const SpanSet& spans, int max_count,
                          const UpdateSet& upd, bf16* pk_scr, float* partial, int* counters, bf16* out, long long out_step,
                          cudaStream_t stream) {
  switch (D) {
    case 32: return launch_span<32>(L, batch, cache, q, k, v, gate, q_step, kv_step, gate_step, spans, max_count, upd, pk_scr, partial, counters, out, out_step, stream);
    case 64: return launch_span<64>(L, batch, cache, q, k, v, gate, q_step, kv_step, gate_step, spans, max_count, upd, pk_scr, partial, counters, out, out_step, stream);
    case 128: return launch_span<128>(L, batch, cache, q, k, v, gate, q_step, kv_step, gate_step, spans, max_count, upd, pk_scr, partial, counters, out, out_step, stream);
  }
  return cudaErrorInvalidValue;
}
size_t span_partial_bytes(int D) { return (size_t)device_sm_count() * 2 * kSpanColumns * (D + 2) * sizeof(float); }

}  // namespace kvm
