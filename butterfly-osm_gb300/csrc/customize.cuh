// customize.cuh — what the two relaxation forms of the customization share
// (customize.cu: a level of apexes; cchpanel.cu: a level of panels).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "engine.cuh"

namespace bf {

// Target of a pair candidate: the pair's slot index with the directions
// present in the topology; neither bit set = nothing to relax.
constexpr uint32_t T_UP = 1u << 31;
constexpr uint32_t T_DOWN = 1u << 30;
constexpr uint32_t T_PAIR = T_DOWN - 1;
// per-pair flag byte
constexpr uint8_t P_UP = 1, P_DOWN = 2, P_UP_SHORT = 4, P_DOWN_SHORT = 8;

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Candidate value of a triangle from its two packed legs; false when a leg
// has weight (time) u32::MAX, which the reference skips.
template <bool LEX>
__device__ __forceinline__ bool candidate(uint64_t leg1, uint64_t leg2, uint32_t m,
                                          uint64_t* out) {
  const uint32_t a = (uint32_t)(leg1 >> 32), b = (uint32_t)(leg2 >> 32);
  if (a == INF || b == INF) return false;
  const uint32_t lo = LEX ? sat_add((uint32_t)leg1, (uint32_t)leg2) : m;
  *out = ((uint64_t)sat_add(a, b) << 32) | lo;
  return true;
}

// Panels of apexes (cchpanel.cu): up to 16 consecutive ranks, each the lowest
// upper neighbour of the one before. A panel's columns are the upper neighbours
// of its rows outside it.
struct CchPanels {
  uint32_t first_level = 0xFFFFFFFFu;  // apexes of this level and above are relaxed by panels
  std::vector<uint64_t> lvl_solve, lvl_push;  // level of panels -> first work unit
  uint4* d_pan = nullptr;     // {lowest rank, rows, columns, first column}
  uint64_t* d_e0 = nullptr;   // first entry
  uint32_t* d_col = nullptr;  // column ranks, ascending in a panel
  uint32_t* d_ent = nullptr;  // pairs [row][row], then [column][row, padded]: T_* words
  uint2* d_solve = nullptr;   // {panel, block of 32 columns}
  uint2* d_push = nullptr;    // {panel, block of 16 columns | the other << 16}
  uint32_t* d_tgt = nullptr;  // per push unit: T_* words of its 16 x 16 column pairs
};

// Builds the panels of the rows at or above the level the rule picks (none, or no
// memory for them: P stays empty). qo, qt, pf: pair rows; lev: levels; d_qo .. d_pf: their device
// copies; room: bytes the panels may take. Synchronises `s`.
bf_status build_cch_panels(CchPanels& P, uint32_t n, const std::vector<uint64_t>& qo,
                           const std::vector<uint32_t>& qt, const std::vector<uint8_t>& pf,
                           const std::vector<uint32_t>& lev, uint32_t n_levels,
                           const uint64_t* d_qo, const uint32_t* d_qt, const uint8_t* d_pf,
                           uint64_t room, cudaStream_t s);
void free_cch_panels(CchPanels& P);
// The relaxation of all panels on `s`, after the levels below them; `pdl`
// whether the first launch may start while what is before it drains.
cudaError_t relax_cch_panels(const CchPanels& P, bool lex, bool pdl, ulonglong2* sl,
                             cudaStream_t s);

}  // namespace bf
