// CUDA source generation for fused kernels.
//
// A fused kernel evaluates a DAG of StableHLO operations per output element.
// Every value is computed "in a context": an index tuple into its own shape.
// Elementwise operations pass the context through; broadcast, transpose,
// reshape, reverse, slice, pad, concatenate, dynamic_slice and
// dynamic_update_slice rewrite it for their operand(s); values that are not
// part of the fusion are loaded from memory at the context's position.
// The reference gets the same effect from mlx::core::compile
// (src/pjrt_plugin/mlx_executable.cc:882); here the composition is printed
// as straight-line CUDA over the device functions of the prelude.
#pragma once
#include <functional>
#include <map>
#include <set>
#include <sstream>
#include <string>
#include <vector>

#include "ir.h"

namespace b200 {

const char* c_type(DT d);        // register type
const char* s_type(DT d);        // storage type
std::string literal(DT d, const uint8_t* bytes);

// A context in which a thread evaluates `Emitter::run` consecutive positions one after the other (e = 0, 1, ...) keeps track
// of how they lie: either along one dimension, starting on a multiple of `run` (run_dim, run_base), or along the linear index
// (lin_base), or they are all the same position. Where that is lost (a transposed or unaligned run) nothing is assumed.
struct Ctx {
  static constexpr int kUnknown = -2, kSame = -1;
  std::vector<std::string> idx;   // one index expression per dimension (may be empty until needed)
  std::string lin;                // row-major linear index expression, when known
  std::vector<int64_t> shape;
  int run_dim = kUnknown;         // >= 0: idx[run_dim] is run_base + e, run_base a multiple of run, the other indices do not change with e
  std::string run_base;
  std::string lin_base;           // not empty: lin is lin_base + e, lin_base a multiple of run
  static Ctx scalar() { Ctx c; c.lin = "0"; c.run_dim = kSame; return c; }
};

class Emitter {
 public:
  std::function<bool(Op*)> is_internal;        // op evaluated inline (fusion member or duplicable)
  std::string idx_t = "int";
  std::vector<Value*> inputs;                  // external values, in parameter order
  std::map<Value*, std::string> bound;         // values bound to a fixed expression (region arguments)
  bool round_small_floats = true;              // round bf16/f16 results after every op
  std::string name_prefix;                     // keeps variable names of cooperating emitters apart
  int run = 0;                                 // consecutive positions per thread (0: one), numbered by run_var
  std::string run_var = "e";

  std::string emit(Value* v, Ctx c);
  std::string input_name(Value* v);
  // The value `e` of type `d` as it is stored. A value that was just rounded to 16 bits, or loaded, is stored as those bits.
  std::string stored(DT d, const std::string& e) const;
  void seed_inputs(const std::vector<Value*>& vs) { for (Value* v : vs) input_name(v); }   // fix the first parameters
  void line(const std::string& s);
  std::string fresh(const char* prefix);
  void ensure_idx(Ctx& c);
  std::string lin_of(Ctx& c);
  void push_scope() { memo_.emplace_back(); indent_ += 2; }
  void pop_scope() { memo_.pop_back(); indent_ -= 2; }
  std::string str() const { return os_.str(); }
  std::string run_arrays(int indent) const;    // declarations in front of the loop over run_var
  std::string run_array(DT d);                 // one of them, `run` elements of storage type `d`: its name
  // Evaluates a region whose operations are all scalar elementwise ops.
  std::vector<std::string> emit_scalar_region(Block* b, const std::vector<std::string>& args);
  int indent_ = 4;

 private:
  std::string shifted(const std::string& base, int64_t by);
  std::string elementwise(Op* op, const std::vector<std::string>& a);
  std::string load(Value* v, Ctx& c);
  bool expensive(Value* v);
  std::string key(Value* v, Ctx& c);
  std::ostringstream os_;
  std::vector<std::map<std::string, std::string>> memo_{1};
  std::map<Value*, int> in_index_;
  std::vector<std::string> arrays_;
  std::map<std::string, std::string> bits_;    // variable of a 16-bit float type -> its bits
  int nvar_ = 0;
};

// moves W elements of `es` bytes between a thread's array `arr` and `ptr + at` in the widest aligned pieces
std::string wide_move(const std::string& arr, const std::string& ptr, int W, int es, bool is_load, int indent = 2, const std::string& at = "base");
// ... which is possible for these sizes
inline bool wide_size(int W, int es) { return W > 0 && (es == 1 || es == 2 || es == 4) && (W * es) % 4 == 0; }

bool is_elementwise_op(const std::string& short_name);

}  // namespace b200
