// Counted loops whose body holds work that is not part of the chain of iterations (loops.cc).
#pragma once
#include "ir.h"

namespace b200 {
void split_counted_loops(Module& m, Block* b);
}  // namespace b200
