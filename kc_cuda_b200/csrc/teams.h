// Teams of blocks for the graphs of a union: each takes a stretch of the graphs
// in a cooperative launch of its own pace.
#pragma once
#include <algorithm>
#include <vector>

#include "kt_internal.h"

namespace kt {

// off[at[i]] for every i.
std::vector<uint64_t> gather_offsets(Ctx* c, const uint64_t* off, const std::vector<uint64_t>& at);

// Graphs [first, last) and blocks [block0, block0 + blocks) of a team.
struct TeamSpan {
  uint64_t first, last;
  unsigned block0, blocks;
};

// Up to `most` teams over graphs of weights before[g + 1] - before[g]: stretches
// of about the same weight, a graph beyond that by itself, with blocks of `grid`
// by their weights.  Empty where there would be one.
inline std::vector<TeamSpan> split_teams(const std::vector<uint64_t>& before, unsigned most, unsigned grid) {
  std::vector<TeamSpan> teams;
  const uint64_t G = before.size() - 1, total = before[G] - before[0];
  most = (unsigned)std::min<uint64_t>({most, G, grid});
  if (most < 2) return teams;
  const uint64_t share = total / most + 1;
  uint64_t first = 0;
  for (uint64_t i = 1; i <= G; ++i) {
    // A team is closed before a graph that would take it past its share, and at
    // the end.
    if (i < G && (before[i + 1] - before[first] <= share || teams.size() + 1 == most)) continue;
    teams.push_back(TeamSpan{first, i, 0, 0});
    first = i;
  }
  if (teams.size() < 2) return {};
  unsigned block = 0;
  const unsigned spare = grid - (unsigned)teams.size();
  for (TeamSpan& t : teams) {
    t.block0 = block;
    t.blocks = 1 + (unsigned)((double)(before[t.last] - before[t.first]) / (double)std::max<uint64_t>(total, 1) * spare);
    block += t.blocks;
  }
  return teams;
}

// Blocks that the teams use.
inline unsigned team_blocks(const std::vector<TeamSpan>& teams) { return teams.back().block0 + teams.back().blocks; }

// Adds the errors that the teams flagged to the context's.
void merge_team_errors(Ctx* c, const void* team_words, uint32_t nteams);

}  // namespace kt
