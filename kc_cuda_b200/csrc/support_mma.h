// Supports of dense working graphs on the tensor cores (support_mma.cu).
#pragma once
#include <vector>

#include "subgraph.h"

namespace kt {

// Exact supports from the product of the rows' bitsets, where that takes less
// time than popcounts (capped ones, where those would do) and has room; returns whether anything was counted.  Of a
// grouped union, counted[g] tells for which graphs; otherwise it stays empty and
// every edge is.  words: the words of expanded rows that the tiles read.
bool support_products(Ctx* c, const Sub& s, uint32_t* sup, bool capped, std::vector<uint8_t>& counted,
                      uint64_t* words);

}  // namespace kt
