// Counted loops whose body holds work that is not part of the chain of iterations (loops.cc).
#pragma once
#include <functional>

#include "ir.h"

namespace b200 {
// Modelled times of fp32 products, us.
struct LoopProductModel {
  std::function<double(Op*)> in_loop;                                   // an iteration's, on whatever pipe is best; negative: it has to stay
  std::function<double(Op*, int64_t)> in_front;                         // so many iterations' as one, on the FMA pipe
  std::function<double(int64_t, int64_t, int64_t, int64_t)> behind;     // G products M x K x N of k-major operands, on the FMA pipe
};

void split_counted_loops(Module& m, Block* b, const LoopProductModel& model);
}  // namespace b200
