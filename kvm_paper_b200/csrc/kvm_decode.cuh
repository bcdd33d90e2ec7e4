// What the decode kernels share: geometry of a sequence's key rows, the shared-memory layout of a chunk, the write of a
// new token, programmatic launches.
#pragma once

#include <cuda.h>

#include "kvm_pdl.cuh"
#include "kvm_tc.cuh"
#include "kvm_tma_host.cuh"

namespace kvm {

__device__ __forceinline__ int bswa_begin_dev(int total, int C, int W) {
  const int end = ((total + C - 1) / C) * C;
  return max(0, end - W * C);
}

// Writes of this thread (also to global memory) -> visible to its later asynchronous copies.
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// One box of a 2-D tensor into L2 (a hint: nothing is waited for).
__device__ __forceinline__ void prefetch_2d(const CUtensorMap* m, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(m), "r"(x), "r"(y) : "memory");
}

// The new token of one kv row, written by one warp: its ring slot and, while the sequence is still inside its first
// block, memory row `past` directly (model/kvm_mixer.py:623-638; no gating on this path).  Returns what this lane wrote to the
// ring: 16 bytes of the key (the first D / 8 lanes) or of the value (the next D / 8).
template <int D>
__device__ __forceinline__ uint4 write_new_token(const LayerDev& L, const DecodeCacheDev& cache, const Tensor4& k, const Tensor4& v,
                                                const Tensor4& gate, int b, int h, int past, bool direct, int lane) {
  const int row = b * L.Hkv + h, WC = L.W * L.C, slot = past % WC, cap = cache.mem.capacity;
  const bf16* kp = k.row(b, h, 0);
  const bf16* vp = v.row(b, h, 0);
  constexpr int PPR = D / 8;  // 16-byte pieces per row: keys on the first lanes, values on the next
  uint4 piece = make_uint4(0, 0, 0, 0);
  if (lane < 2 * PPR) {
    const bool is_v = lane >= PPR;
    const int pc = is_v ? lane - PPR : lane;
    bf16* dst = (is_v ? cache.ring_v : cache.ring_k) + ((size_t)row * WC + slot) * D;
    piece = *reinterpret_cast<const uint4*>((is_v ? vp : kp) + pc * 8);
    *reinterpret_cast<uint4*>(dst + pc * 8) = piece;
  }
  if (lane == 0) cache.ring_g[(size_t)row * WC + slot] = *gate.row(b, h, 0);
  if (direct && past < cap) {
    RowVec<D> pk, vr;
    prepare_key_row<D>(L, pk, kp, lane);
    load_row<D>(vr, vp, lane);
    const float vl = row_norm<D>(vr);
    const size_t mrow = (size_t)row * cap + past;
    store_row<D>(pk, cache.mem.k_sum + mrow * D, lane);
    store_row<D>(vr, cache.mem.v_sum + mrow * D, lane);
    if (lane == 0) cache.mem.vlen[mrow] = vl;
    refresh_memory_row<D>(L, pk, vr, vl, cache.mem.k_attn + mrow * D, cache.mem.v_attn + mrow * D, lane);
  }
  return piece;
}

constexpr int kDecConsumers = 8;                           // math warps (16 keys of every chunk each)
constexpr int kDecThreads = (kDecConsumers + 1) * 32;      // + one producer warp
constexpr int kDecChunk = kDecConsumers * 16;              // rows per pipeline stage
constexpr int kDecBoxRows = 16;                            // rows per TMA box: the fetch granularity of a run's tail
constexpr int kDecMaxBatch = 1024;                         // sequences per launch (their chunk table lives in shared memory)
constexpr int kDecMaxSmem = 227 * 1024;   // dynamic shared memory one CTA may use (one CTA per SM)

// Chunk geometry of one sequence's kv rows: up to three contiguous runs (memory rows, window part up to
// the end of the ring, wrapped window part), each cut into chunks of kDecChunk rows.
struct DecGeo {
  int S_act, slot0, len_a, len_b, c_mem, c_a, c_b;
  __device__ __forceinline__ int chunks() const { return c_mem + c_a + c_b; }
};
__device__ __forceinline__ DecGeo dec_geometry(int S, int total, int C, int W) {
  DecGeo g;
  const int WC = W * C;
  const int new_begin = bswa_begin_dev(total, C, W);
  g.S_act = new_begin > 0 ? S : 0;
  const int n_win = total - new_begin;
  g.slot0 = new_begin % WC;
  g.len_a = min(n_win, WC - g.slot0);
  g.len_b = n_win - g.len_a;
  g.c_mem = (g.S_act + kDecChunk - 1) / kDecChunk;
  g.c_a = (g.len_a + kDecChunk - 1) / kDecChunk;
  g.c_b = (g.len_b + kDecChunk - 1) / kDecChunk;
  return g;
}

// The four row arrays of the decode cache as 2-D tensors [all rows][D] with boxes of kDecBoxRows rows.
struct DecMaps {
  CUtensorMap mem_k, mem_v, ring_k, ring_v;
};

// byte offset of the 16-byte piece j of row r inside the K (or V) part of a stage
template <int D>
__device__ __forceinline__ uint32_t dec_piece(int r, int j) {
  if constexpr (D >= 64) return (uint32_t)((j >> 3) * (kDecChunk * 128) + r * 128 + (((j & 7) ^ (r & 7)) << 4));
  else return (uint32_t)(r * (D * 2) + j * 16);
}

// Bounded wait that also gives up when another warp of the CTA has given up.
__device__ __forceinline__ bool dec_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t i = 0; i < tc::kSpinLimit; ++i) {
    if (tc::mbar_try_wait(bar, parity)) return true;
    if (i >= 8) {
      if (*abort_flag) return false;
      __nanosleep(i < 64 ? 32 : 200);
    }
  }
  return false;
}

// ------------------------------------------------------------------------------------- host side
constexpr int kMaxDevices = 64;  // device ordinals the per-device caches below cover

int device_sm_count();
// The tensor maps of a decode cache (kept between calls, keyed by the arrays' addresses and sizes).
bool decode_maps(const DecodeCacheDev& c, uint64_t kv_rows, int cap, int WC, int D, DecMaps* out);

// The boundary updates of the listed sequences (nothing else runs on the GPU meanwhile).
cudaError_t decode_update(int D, const LayerDev& L, int batch, const DecodeCacheDev& cache, const UpdateSet& upd, bf16* pk_scr,
                          cudaStream_t stream);

}  // namespace kvm
