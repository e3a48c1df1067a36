// hj_launch.h -- thread layouts of the fused particle pass and its grid rule
// (host only, no CUDA: the rules are checked on the CPU as well).
#pragma once

#include <cstdint>

namespace hj {

// Particles one block of the fused pass may deposit per turn (its counters and
// trip counts are 32-bit; the bound leaves them far from wrapping).
constexpr int64_t kMaxBlockParticles = (1 << 20) - 8;

// Thread layouts of the fused pass (particles/thread x threads/block; the next
// group prefetched into registers except in 3): 0 = 4 x 512, 1 = 2 x 1024,
// 2 = 2 x 768, 3 = 2 x 512 without prefetch, 4 = 2 x 512 at 64 registers (two
// blocks per SM where shared memory allows), 5 = 4 x 256 at 128 registers
// (two blocks per SM: one block's set-up and write-out overlap the other's
// particles).
constexpr int kNumPassCfgs = 6;       // thread layouts of the fused pass
constexpr int kPassLayoutMask = 7;    // layout bits of a pass configuration
constexpr int kPassN32 = 8;           // + 32-bit counters of a cell's halves (else 16-bit ones)
constexpr int kPassFastNormals = 16;  // + single-precision quantum-excitation normals
// Launch-only bit (never in a caller's configuration): the pass's hot window
// holds fewer than all B + 1 cells, so its deposits are range-checked.
constexpr int kPassWindowed = 32;
// Bit of a bunch's configuration (never in a caller's): its grid's cells do not halve its
// bins, which one layout serves (0 with 32-bit counters).
constexpr int kPassSplit = 64;
inline int split_pass_cfg(int cfg) { return kPassSplit | kPassN32 | (cfg & kPassFastNormals); }

inline int pass_cfg_threads(int cfg) {
  const int l = cfg & kPassLayoutMask;
  return l == 1 ? 1024 : (l == 2 ? 768 : (l == 5 ? 256 : 512));
}
inline int pass_cfg_ppt(int cfg) {
  const int l = cfg & kPassLayoutMask;
  return (l == 0 || l == 5) ? 4 : 2;
}
// Layouts that keep two blocks on an SM (each takes at most half of it).
inline bool pass_cfg_two_blocks(int cfg) {
  const int l = cfg & kPassLayoutMask;
  return l == 4 || l == 5;
}
// Entries of a warp's staging queue of particles whose Float64 normal takes
// the ziggurat's slow path (the fused pass finishes them 32 at a time).
constexpr int kDeferStage = 64;
inline bool pass_cfg_valid(int cfg) {
  return cfg >= 0 && (cfg & ~(kPassLayoutMask | kPassN32 | kPassFastNormals)) == 0 &&
         (cfg & kPassLayoutMask) < kNumPassCfgs;
}

// A caller's layout request: -1 = automatic; kPassAutoFast = the automatic
// layout with single-precision normals; otherwise a valid configuration.
constexpr int kPassAutoFast = kPassFastNormals | kPassLayoutMask;
inline bool pass_request_valid(int r) { return r == -1 || r == kPassAutoFast || pass_cfg_valid(r); }
// The configuration a request gives for bins B, `automatic` being the
// library's choice for them.
inline int resolve_pass_request(int r, int automatic) {
  if (r == -1) return automatic;
  if (r == kPassAutoFast) return automatic | kPassFastNormals;
  return r;
}

// Particles per block of a batch member of n particles, in a batch of `slots`
// bunches created with `chunk` particles per block.  A chunk of the caller's own is
// taken as it is.  The default one leaves the size to this rule: member_blocks(slots)
// blocks of kMinChunk to 2 kDefaultChunk particles.  A block costs about 8 us beside its
// particles (1 us a thousand), so large bunches take large blocks, while a batch of few or
// small bunches must not wait for one block each: eight, or what fills the SMs
// twice when every slot is taken.  Measured, us a turn, against 65532 for
// all: 256 bunches of 1e4 to 2e6 870 -> 862, 32 bunches of 1e6 303 -> 262, 64 of 1e4
// to 5e4 58 -> 32, 16 served ones (1.6e6 particles) 81 -> 45; but 256 of 1e5 272 -> 319,
// 148 of 1e5 144 -> 185, where a caller does better with blocks of their own.
// A function of n and of how the batch was created: a bunch's sums do not depend
// on the bunches that share it.
constexpr int64_t kDefaultChunk = 65536;
constexpr int64_t kMinChunk = 16384;
inline int64_t member_blocks(int64_t slots, int64_t sms = 148) {
  const int64_t b = 2 * sms / (slots > 0 ? slots : 1);
  return b > 8 ? b : 8;
}
inline int64_t member_chunk(int64_t n, int64_t chunk, int64_t slots, int64_t sms = 148) {
  constexpr int64_t kMost = kMaxBlockParticles & ~int64_t(127);
  if (chunk != kDefaultChunk) return chunk < kMost - 128 ? chunk : kMost;
  const int64_t blocks = member_blocks(slots, sms);
  int64_t c = (n + blocks - 1) / blocks;
  c = (c + 127) / 128 * 128;                       // whole warps of four-particle groups
  if (c < kMinChunk) c = kMinChunk;
  return c < 2 * kDefaultChunk ? c : 2 * kDefaultChunk;
}
// First particle of block i of a member split into blocks of `chunk`: on a whole warp of
// four-particle groups, so that only the bunch's last block has particles left over by
// its warps, while the blocks keep `chunk` particles on average (a chunk that fills the
// GPU's waves still does).
inline int64_t member_first(int64_t i, int64_t chunk) {
  return chunk >= 128 ? i * chunk & ~int64_t(127) : i * chunk;
}
inline int64_t member_chunks(int64_t n, int64_t chunk) { return (n + chunk - 1) / chunk; }
inline int64_t member_end(int64_t i, int64_t n, int64_t chunk) {
  return i + 1 < member_chunks(n, chunk) ? member_first(i + 1, chunk) : n;
}

// Blocks of the particle pass: enough to fill the GPU, but each block should
// move at least B/2 particles, since it clears and adds up a window of up to
// B + 1 counters.
inline int track_grid_size(int64_t n, int B, int num_sms, int blocks_per_sm, int cfg) {
  int64_t per_block = (int64_t)pass_cfg_ppt(cfg) * pass_cfg_threads(cfg);
  if (per_block < (int64_t)B / 2) per_block = (int64_t)B / 2;
  int64_t g = (n + per_block - 1) / per_block;
  int64_t cap = (int64_t)num_sms * blocks_per_sm;
  if (g > cap) g = cap;
  // At most kMaxBlockParticles per block and turn.  Block b takes the groups of PPT
  // particles b·T + t + k·g·T: at most ceil((n / PPT) / (g·T)) steps of T·PPT particles,
  // and block 0 also the tail that whole warps leave over.  So g is raised until no block
  // takes more steps than fit.
  const int64_t threads = pass_cfg_threads(cfg);
  const int64_t steps = kMaxBlockParticles / ((int64_t)pass_cfg_ppt(cfg) * threads);
  const int64_t groups = n / pass_cfg_ppt(cfg);
  const int64_t need = (groups + steps * threads - 1) / (steps * threads);
  if (g < need) g = need;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace hj
