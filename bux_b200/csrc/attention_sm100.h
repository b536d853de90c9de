// Host-visible types of the tcgen05 attention kernels (attention_sm100.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace bux {

struct Status;

// q, o, d_o, dq: [B, T, H, D] bf16.  k, v, dk, dv: [B, S, G, D] bf16 (H % G == 0).
// lse, delta: [B, H, T] fp32.  sinks / dsinks: [H] fp32 or null.  D is 64 or 128.
// Causal alignment is bottom-right (query t sees keys <= t + S - T); window > 0 keeps
// keys in (t + S - T - window, t + S - T].
// Documents packed into a row (self-attention, T == S): row_lo[b, t] is the first key that
// query t may see (the start of its document) and key_hi[b, s] the last query that may see
// key s (the end of its document); both int32, both non-decreasing along a row, or null.
// The forward and the mask use row_lo; key_hi only bounds the backward's walk over query tiles.
struct AttnArgs {
  const void* q = nullptr; const void* k = nullptr; const void* v = nullptr;
  void* o = nullptr; float* lse = nullptr;
  const void* d_o = nullptr; void* dq = nullptr; void* dk = nullptr; void* dv = nullptr;
  float* delta = nullptr;
  const float* sinks = nullptr; float* dsinks = nullptr;
  const int* row_lo = nullptr; const int* key_hi = nullptr;
  int B = 0, T = 0, S = 0, H = 0, G = 0, D = 0;
  float scale = 1.f; bool causal = true; int window = 0;
  Status* status = nullptr;
  // backward only, optional: 32 counters that the CTA of the first key tile adds the cycles of
  // its phases to (softmax warp 0: slots 0-13, MMA issuer: 16-23), for reading the schedule
  unsigned int* phase_cycles = nullptr;
};

#ifdef __CUDACC__
// Which (tile, head) a block of a one-dimensional grid works on. Blocks start in order, so the grid
// walks the tiles of all heads with the longest walks first (tile 0 of every head, then tile 1, ...):
// the short ones fill the gaps at the end. With the tiles of one head after another, long
// walks of the last heads started late: the SMs had work 61 % of the backward's time (2 x 4096
// tokens, 4 key heads, 256 blocks, forward + backward: 1796 us, then 1409) and 86 % of the forward's.
// Heads go 64 at a time, so that the keys in use stay within L2 however large the batch is. Where all
// walks have about one length (no causal mask, or a window under half the row) the tiles of a head
// stay together, since neighbours read the same keys.
struct AttnSlot { int tile, pair; };
__device__ __forceinline__ AttnSlot attn_slot(unsigned id, int tiles, int pairs, bool by_length) {
  if (!by_length) return {(int)(id % (unsigned)tiles), (int)(id / (unsigned)tiles)};
  constexpr unsigned CHUNK = 64;
  const unsigned per_chunk = CHUNK * (unsigned)tiles, chunk = id / per_chunk, local = id % per_chunk;
  const unsigned here = min(CHUNK, (unsigned)pairs - chunk * CHUNK);
  return {(int)(local / here), (int)(chunk * CHUNK + local % here)};
}
inline bool attn_by_length(const AttnArgs& a) { return a.causal && (a.window <= 0 || a.window >= a.S / 2); }
#endif

const char* attn_fwd_launch(const AttnArgs& a, cudaStream_t stream);
const char* attn_bwd_launch(const AttnArgs& a, cudaStream_t stream);

}  // namespace bux
