// Uniform walk on the smallest array that serves a step (StepReader), 32-bit ids.
//
// A step is one dependent access (packed records) or two (row descriptor, then the edge), and nothing in a walk can
// shorten that chain; what is left is how many walks an SM keeps in flight and how large the arrays are that they hit.
// An SM's misses in flight are tracked in L1 lines, so shared memory is what must be small: a warp owns 32 walks and one
// tile of S steps x 32 walks of 4-byte slots, which holds the chunk's draws and, as they are consumed, the nodes reached.
// Draws come in as row segments by cp.async (no registers, no second buffer: their latency is exposed once in S steps and
// covered by the SM's other warps), nodes leave as row segments of S int64. With the carve-out for the tiles held at
// 100 KB a launch of 200,000 walks on a 21 MB graph takes 62 us, with 132 KB 69, and 5.5 times as long at 32 KB, where one
// block fits; the 8-byte tiles of uniform_walk_staged_kernel: 120 us.
//
// SRC: where the draws come from. DRAW_GIVEN: the caller's rand array. DRAW_UNIFORM: the uniform walk's Philox stream
// (four steps per block). DRAW_NODE2VEC: the node2vec stream; a node2vec walk with prob_2 >= prob_0, prob_1 (q <= 1,
// q <= p; (1, 1) among them) accepts by prob_2 alone, so its steps are uniform steps on that stream. prob_2 is then 1
// and only the draw 2^31 - 1, which stands for r = 1, is rejected.
#pragma once
#include "walk_kernels.cuh"

namespace walk_b200 {

enum : int { DRAW_GIVEN = 0, DRAW_UNIFORM = 1, DRAW_NODE2VEC = 2 };
__device__ __forceinline__ void cp_async4(uint32_t* smem, const void* gmem) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int SRC, int GATHER, bool HAS_EOUT, int S, int BLOCK, int BLOCKS_PER_SM, bool SECTORS>
__global__ void __launch_bounds__(BLOCK, BLOCKS_PER_SM) uniform_steps_kernel(const UniformParams P) {
  static_assert(!SECTORS || (S == 16 && !HAS_EOUT), "whole-sector flushes are built for 16-step chunks of the node matrix");
  constexpr int kSlots = SECTORS ? S + 4 : S;
  static_assert(S == 8 || S == 16, "a chunk is a whole number of Philox blocks and fits the lanes");
  constexpr int kWarps = BLOCK / 32, kPitch = 33, kRows = 32 / S;  // kRows: walks served by one segment instruction
  __shared__ uint32_t tiles[kWarps][kSlots][kPitch];
  __shared__ uint32_t etiles[HAS_EOUT ? kWarps : 1][S][kPitch];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  uint32_t (*tile)[kPitch] = tiles[wib];
  uint32_t (*etile)[kPitch] = etiles[HAS_EOUT ? wib : 0];
  const int64_t w0 = ((int64_t)blockIdx.x * kWarps + wib) * 32;
  if (w0 >= P.num_walks) return;  // whole warp leaves together
  const L2Policy pol = make_policies(P.hints);
  const StepReader<GATHER> reader(P.col, P.steps, P.step_bits);
  const int32_t L = P.walk_length;
  const int nw = (int)min((int64_t)32, P.num_walks - w0);
  const int seg = lane & (S - 1), row0 = lane / S;  // this lane's place in the row segments
  const float* rand = SRC == DRAW_GIVEN ? P.rand + w0 * L + seg : nullptr;
  int64_t* out = P.n_out + w0 * ((int64_t)L + 1) + 1 + seg;

  // Tile slot of the chunk's step j. SECTORS: a ring, in which the last steps of the chunk before stay unwritten until
  // their row's next 32-byte boundary is reached.
  int first_slot = 0;
  auto slot_of = [&](int j) -> int {
    if (!SECTORS) return j;
    const int k = first_slot + j;
    return k >= kSlots ? k - kSlots : k;
  };
  // Row r of this warp starts this many elements behind a 32-byte boundary.
  auto row_phase = [&](int r) -> int {
    return (int)(((reinterpret_cast<uintptr_t>(P.n_out) >> 3) + (uint64_t)(w0 + r) * (uint64_t)(L + 1)) & 3);
  };

  auto load_draws = [&](int32_t l0) {
    if (l0 + seg < L) {
#pragma unroll
      for (int k = 0; k < S; k++) {
        const int wi = k * kRows + row0;
        if (wi < nw) cp_async4(&tile[slot_of(seg)][wi], rand + (int64_t)wi * L + l0);
      }
    }
  };

  if (SRC == DRAW_GIVEN) load_draws(0);
  bool parked = lane >= nw;
  uint32_t cur = 0, rs = 0, deg = kNoRow;
  int64_t bad = 0;  // a start that is no node: written as it is
  bool bad_start = false;
  if (!parked) {
    const int64_t first = ld8(P.start + w0 + lane, pol.stream);
    st8(P.n_out + (w0 + lane) * ((int64_t)L + 1), first, pol.stream);
    cur = (uint32_t)first;
    if ((uint64_t)first >= (uint64_t)P.num_nodes) {
      raise_flag(P.flags, WALK_B200_FLAG_BAD_NODE);
      parked = bad_start = true;
      bad = first;
    }
  }
  const uint64_t gw = P.walk_index_base + (uint64_t)(w0 + lane) * P.walk_index_stride;

  for (int32_t l0 = 0; l0 < L; l0 += S) {
    const int sc = min(S, L - l0);
    if (SRC == DRAW_GIVEN) {
      cp_async_wait();
      __syncwarp();
    }
    Philox4 blk = {0, 0, 0, 0};
    for (int j = 0; j < sc; j++) {
      uint32_t edge = 0;  // edge + 1, 0: none
      uint32_t word = 0;
      if (SRC == DRAW_UNIFORM) {
        if (!parked && (j & 3) == 0) blk = uniform_block(P.key0, P.key1, gw, (uint32_t)(l0 + j) >> 2);
        word = (j & 3) == 0 ? blk.x : (j & 3) == 1 ? blk.y : (j & 3) == 2 ? blk.z : blk.w;
      }
      if (!parked) {
        if (GATHER != GATHER_PACKED || deg == kNoRow) {
          const uint64_t d = (uint64_t)ld8(P.desc + cur, pol.keep);
          rs = (uint32_t)(d & kDescStartMask);
          deg = (uint32_t)(d >> kDescStartBits);
        }
        uint32_t e = rs;
        bool move = true;
        if (SRC == DRAW_NODE2VEC) {
          uint32_t cand, acc, a = 0;
          node2vec_draw(P.key0, P.key1, gw, (uint32_t)(l0 + j), 0, cand, acc);
          while (acc >= P.cut2 && l0 + j > 0 && deg > 1) {  // one draw in 2^31
            if (++a >= P.max_attempts) { raise_flag(P.flags, WALK_B200_FLAG_ATTEMPT_CAP); move = false; break; }
            node2vec_draw(P.key0, P.key1, gw, (uint32_t)(l0 + j), a, cand, acc);
          }
          if (deg > 1) e += cand % deg;
          if ((uint64_t)rs + deg > (uint64_t)P.num_edges) { raise_flag(P.flags, WALK_B200_FLAG_BAD_ROWPTR); deg = 0; }
        } else {
          const float r = SRC == DRAW_GIVEN ? __uint_as_float(tile[slot_of(j)][lane]) : uniform_from_word(word);
          const float prod = __fmul_rn(r, __uint2float_rn(deg));
          const int64_t wide = (int64_t)rs + __float2ll_rz(prod);
          e = (uint32_t)wide;
          if (deg && (uint64_t)wide >= (uint64_t)P.num_edges) {  // rand >= 1, NaN, negative, or corrupt rowptr
            raise_flag(P.flags, WALK_B200_FLAG_BAD_EDGE);
            e = wide < 0 || P.num_edges == 0 ? 0u : (uint32_t)(P.num_edges - 1);
            if (P.num_edges == 0) deg = 0;
          }
        }
        if (deg == 0) {  // no way out of this node: the walk stays for good
          parked = true;
        } else if (move) {
          edge = e + 1;
          uint32_t to, to_rs, to_deg;
          if (reader.read(e, pol, (uint64_t)P.num_nodes, to, to_rs, to_deg)) {
            cur = to;
            if (GATHER == GATHER_PACKED) { rs = to_rs; deg = to_deg; }
          } else {  // an id that is no node: keep cur
            raise_flag(P.flags, WALK_B200_FLAG_BAD_NODE);
            if (SRC != DRAW_NODE2VEC) parked = true;
          }
        }
      }
      tile[slot_of(j)][lane] = cur;
      if (HAS_EOUT) etile[j][lane] = edge;
    }
    __syncwarp();
    if (SECTORS) {
      // Positions p = 0 .. l0 + S of each row are known (p = 0 the start, written above); those from l0 - phase up to
      // l0 - phase + S are written now, whole sectors in the middle of a row. The last chunk writes the rest too.
#pragma unroll 4
      for (int k = 0; k < S; k++) {
        const int wi = k * kRows + row0;
        if (wi >= nw) continue;
        int64_t* row = P.n_out + (w0 + wi) * ((int64_t)L + 1);
        for (int32_t p = l0 - row_phase(wi) + seg; p <= l0 + sc; p += S) {
          if (p >= 1 && (p < l0 - row_phase(wi) + S || l0 + S >= L)) {
            int at = first_slot + (p - 1 - l0);
            if (at < 0) at += kSlots;
            if (at >= kSlots) at -= kSlots;
            st8(row + p, (int64_t)tile[at][wi], pol.stream);
          }
        }
      }
      first_slot = first_slot + S >= kSlots ? first_slot + S - kSlots : first_slot + S;
    } else if (seg < sc) {
#pragma unroll 4
      for (int k = 0; k < S; k++) {
        const int wi = k * kRows + row0;
        if (wi < nw) {
          st8(out + (int64_t)wi * ((int64_t)L + 1) + l0, (int64_t)tile[seg][wi], pol.stream);
          if (HAS_EOUT) st8(P.e_out + (w0 + wi) * (int64_t)L + l0 + seg, (int64_t)etile[seg][wi] - 1, pol.stream);
        }
      }
    }
    __syncwarp();
    if (SRC == DRAW_GIVEN && l0 + S < L) load_draws(l0 + S);
  }
  if (bad_start) {  // overwrite what the 32-bit tile could not hold
    for (int32_t l = 0; l < L; l++) st8(P.n_out + (w0 + lane) * ((int64_t)L + 1) + 1 + l, bad, pol.stream);
  }
}

}  // namespace walk_b200
