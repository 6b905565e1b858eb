// Loop fission of counted `while` loops (what lax.scan becomes), for fp32 products.
//
// An iteration of a recurrent network's reverse scan is a chain of small dependent kernels, but much of what it computes is
// not on the chain:
//   * products whose operands are known before the loop (the pre-activations of a step recomputed from the stacked carries of
//     the forward scan): all iterations' are made by one product in front of the loop, and an iteration reads its slice;
//   * accumulators that only ever receive a term (weight and bias gradients): the iterations stack what the terms are made
//     of, and one product (or reduction) behind the loop makes their sum.
// The chain of an LSTM training step of two layers (64 x 256, 100 steps) shrinks from 15 kernels per reverse iteration to
// 6, and 400 products of 64 rows become 2 of 6400 rows and 2 of 25 groups.
//
// Nothing is computed with less precision: these products go to the FMA pipe ("b200.fma"), whatever pipe an iteration's would
// take, and a sum over iterations is made of partial products over at most 256 rows each, all with the k of a tile shared by at
// least four warps, which are then added up: chains of 64 additions, where an iteration's product and the additions over iterations
// made chains of 16 and one per iteration. Against 64 bits, the gradients of four LSTM steps (100 x 64 x 32 x 256 and smaller),
// norm of the difference over the norm: 2.0e-7 to 2.9e-7 before, 1.8e-7 to 2.6e-7 now; over 512 rows in one chain the largest was
// 5.3e-7.
//
// Taken when the loop's trip count is known and at least 8, for each product that the time models (compiler.cc) give no more
// time so than all iterations' own products, and as long as all that is written in front of a loop, by its iterations and behind it
// for the sake of the split is below 512 MB: stacks, the operands they are made of, partial sums. A sum over an operand that is the same in all
// iterations stays in the loop: its stack would be as many copies of one tensor. Sums of rows leave only where what they read is
// stacked for a product. Training steps of two recurrent layers and 50 iterations, batch x hidden, us, products in the
// loop / split: 16 x 256 2610 / 1615, 64 x 256 3030 / 2305, 128 x 256 3820 / 2925, 256 x 256 5220 / 4670, 64 x 512 4980 / 4160,
// 256 x 512 8170 - 8760 / 8050, 512 x 512 (20 iterations) 4565 / 4560, 16 x 1024 8000 / 5200, 64 x 1024 11270 / 10505, 256 x 1024 15520 / 15515.
// (All products below 2^30 multiply-adds split and all sums of rows: 4910 at 512 x 512, 15660 at 256 x 1024.)
#include "loops.h"

#include <algorithm>
#include <cstring>
#include <functional>
#include <map>
#include <set>

#include "codegen.h"

namespace b200 {
namespace {

constexpr int64_t kMinTrips = 8, kMaxStackBytes = 512LL << 20, kSumRows = 256;

std::string i64s(const std::vector<int64_t>& v) {
  std::string s = "array<i64: ";
  for (size_t k = 0; k < v.size(); k++) s += (k ? ", " : "") + std::to_string(v[k]);
  return s + ">";
}
std::string dot_numbers(const std::vector<int64_t>& lb, const std::vector<int64_t>& rb, const std::vector<int64_t>& lc, const std::vector<int64_t>& rc) {
  auto list = [](const std::vector<int64_t>& v) {
    std::string s = "[";
    for (size_t k = 0; k < v.size(); k++) s += (k ? ", " : "") + std::to_string(v[k]);
    return s + "]";
  };
  return "#stablehlo.dot<lhs_batching_dimensions = " + list(lb) + ", rhs_batching_dimensions = " + list(rb) +
         ", lhs_contracting_dimensions = " + list(lc) + ", rhs_contracting_dimensions = " + list(rc) + ">";
}
bool const_int(Value* v, long long& out) {
  if (!v->def || v->def->short_name() != "constant") return false;
  DenseValue d = attr_dense(v->def->attr("value"));
  if (d.type.numel() != 1 || !d.type.dims.empty()) return false;
  if (d.type.dt == DT::I32) { int32_t t; memcpy(&t, d.data.data(), 4); out = t; return true; }
  if (d.type.dt == DT::I64) { int64_t t; memcpy(&t, d.data.data(), 8); out = t; return true; }
  return false;
}
bool inside(Value* v, Block* b) {
  for (Block* p = v->def ? v->def->parent : v->owner; p; p = p->parent_op ? p->parent_op->parent : nullptr)
    if (p == b) return true;
  return false;
}
int count_uses(Block* b, Value* v) {
  int n = 0;
  for (auto& o : b->ops) {
    n += (int)std::count(o->operands.begin(), o->operands.end(), v);
    for (auto& r : o->regions) n += count_uses(r.get(), v);
  }
  return n;
}
void replace_uses(Block* b, Value* from, Value* to) {
  for (auto& o : b->ops) {
    std::replace(o->operands.begin(), o->operands.end(), from, to);
    for (auto& r : o->regions) replace_uses(r.get(), from, to);
  }
}
TensorType stacked_type(const TensorType& t, int64_t T) {
  TensorType s = t;
  s.dims.insert(s.dims.begin(), T);
  return s;
}

struct Splitter {
  Module& m;
  Block* outer;
  Op* w;
  Block *cond, *body;
  Op* next;                                          // the body's return
  const LoopProductModel& model;
  int counter = -1;
  long long first = 0, trips = 0;
  std::vector<std::unique_ptr<Op>> front, back;      // in front of the loop, behind it
  bool changed = false;
  std::map<Value*, bool> known_;                     // can be stacked in front of the loop
  std::map<Op*, bool> quicker_;
  std::map<Value*, Value*> stack_, outside_;
  std::map<Value*, Value*> carried_;                 // stacked by the loop itself: the loop's result

  Value* add(std::vector<std::unique_ptr<Op>>& where, Block* parent, const std::string& name, std::vector<Value*> ins, const TensorType& t,
             std::map<std::string, std::string> attrs = {}) {
    auto op = std::make_unique<Op>();
    op->name = "stablehlo." + name;
    op->operands = std::move(ins);
    op->attrs = std::move(attrs);
    op->parent = parent;
    Value* v = m.new_value(t, "");
    v->def = op.get();
    v->def_index = 0;
    op->results.push_back(v);
    where.push_back(std::move(op));
    return v;
  }
  Value* zero(std::vector<std::unique_ptr<Op>>& where, Block* parent, const TensorType& t) {
    return add(where, parent, "constant", {}, t, {{"value", std::string(dt_is_float(t.dt) ? "dense<0.000000e+00> : " : "dense<0> : ") + t.str()}});
  }

  bool find_counter() {
    if (w->regions.size() != 2 || w->operands.size() != w->results.size()) return false;
    Op* cret = cond->ops.empty() ? nullptr : cond->ops.back().get();
    if (!cret || cret->operands.size() != 1 || !cret->operands[0]->def) return false;
    Op* cmp = cret->operands[0]->def;
    if (cmp->short_name() != "compare" || attr_enum(cmp->attr("comparison_direction")) != "LT") return false;
    Value* c = cmp->operands[0];
    long long limit, step;
    if (c->def || c->owner != cond || !const_int(cmp->operands[1], limit)) return false;
    counter = c->arg_index;
    Value *arg = body->args[counter], *nv = next->operands[counter];
    if (!const_int(w->operands[counter], first) || !nv->def || nv->def->short_name() != "add") return false;
    Value *a = nv->def->operands[0], *b = nv->def->operands[1];
    if (!((a == arg && const_int(b, step)) || (b == arg && const_int(a, step))) || step != 1) return false;
    trips = limit - first;
    return trips >= kMinTrips && trips <= 65536;
  }

  // Scalar integers of the body as base + slope * (iteration number).
  bool affine(Value* v, long long& base, long long& slope, int depth = 0) {
    if (depth > 8 || !v->type.dims.empty()) return false;
    if (const_int(v, base)) { slope = 0; return true; }
    if (v == body->args[counter]) { base = first; slope = 1; return true; }
    Op* d = v->def;
    if (!d || d->parent != body || (d->short_name() != "add" && d->short_name() != "subtract")) return false;
    long long b0, s0, b1, s1;
    if (!affine(d->operands[0], b0, s0, depth + 1) || !affine(d->operands[1], b1, s1, depth + 1)) return false;
    const int sign = d->short_name() == "add" ? 1 : -1;
    base = b0 + sign * b1;
    slope = s0 + sign * s1;
    return true;
  }

  // The value outside the loop of something that is the same in all iterations; null when it is not.
  Value* fixed(Value* v) {
    if (!inside(v, body)) return v;
    auto it = outside_.find(v);
    if (it != outside_.end()) return it->second;
    Value* r = nullptr;
    if (!v->def) {
      if (v->owner == body && next->operands[v->arg_index] == v) r = w->operands[v->arg_index];
    } else if (v->def->parent == body && v->def->results.size() == 1 && v->def->regions.empty()) {
      const std::string sh = v->def->short_name();
      if (sh == "constant" || sh == "iota") r = add(front, outer, sh, {}, v->type, v->def->attrs);
      else if (sh == "broadcast_in_dim" || sh == "reshape") {
        if (Value* o = fixed(v->def->operands[0])) r = add(front, outer, sh, {o}, v->type, v->def->attrs);
      }
    }
    return outside_[v] = r;
  }

  // Products of all iterations stay on the FMA pipe, whatever pipe an iteration's would take: they leave where that is no slower.
  double in_loop_us(Op* d) {
    if (d->operands[0]->type.dt != DT::F32 || d->operands[1]->type.dt != DT::F32 || d->results[0]->type.dt != DT::F32) return -1.0;
    return (double)trips * model.in_loop(d);
  }
  bool quicker_in_front(Op* d) {
    auto it = quicker_.find(d);
    if (it != quicker_.end()) return it->second;
    const double us = in_loop_us(d);
    return quicker_[d] = us > 0 && model.in_front(d, trips) <= us;
  }
  // The sum of A^T B: partial products, what remains of them, and their sum, against a product and an addition an iteration.
  bool quicker_behind(Op* d, int64_t per) {
    const int64_t M = d->operands[0]->type.dims[1], N = d->operands[1]->type.dims[1], rows = d->operands[0]->type.dims[0], groups = trips / per, left = trips % per;
    const double us = in_loop_us(d), mb = (double)M * N * 4e-6;
    if (us <= 0) return false;
    return model.behind(M, N, per * rows, groups) + (left ? model.behind(M, N, left * rows, 1) : 0.0) + (groups > 1 ? 2.0 + 2.0 * groups * mb / 6.0 : 0.0) <=
           us + (double)trips * std::max(2.0, 3.0 * mb / 6.0);
  }

  // Can all iterations' values of `v` be made in front of the loop?
  bool known(Value* v) {
    if (fixed(v)) return true;
    auto it = known_.find(v);
    if (it != known_.end()) return it->second;
    bool& ok = known_[v];
    ok = false;
    Op* d = v->def;
    if (!d || d->parent != body || !d->regions.empty() || d->results.size() != 1 || d->name.rfind("stablehlo.", 0) != 0 || v->type.dims.empty()) return false;
    const std::string sh = d->short_name();
    if (sh == "dynamic_slice") {
      Value* o = d->operands[0];
      long long base, slope;
      if (o->type.rank() != v->type.rank() || v->type.dims[0] != 1 || !fixed(o) || !affine(d->operands[1], base, slope) || (slope != 1 && slope != -1)) return false;
      if (std::min(base, base + slope * (trips - 1)) < 0 || std::max(base, base + slope * (trips - 1)) >= o->type.dims[0]) return false;
      for (int i = 1; i < o->type.rank(); i++)
        if (o->type.dims[i] != v->type.dims[i]) return false;
      return known_[v] = true;
    }
    if (is_elementwise_op(sh)) {
      for (Value* o : d->operands)
        if (o->type.dims != v->type.dims || !known(o)) return false;
      return known_[v] = true;
    }
    if (sh == "reshape" || sh == "slice" || sh == "transpose" || sh == "broadcast_in_dim" || sh == "concatenate") {
      for (Value* o : d->operands)
        if (!known(o)) return false;
      return known_[v] = true;
    }
    if (sh == "dot_general") {
      auto f = attr_struct(d->attr("dot_dimension_numbers"));
      return known_[v] = f["lhs_batching_dimensions"].empty() && f["rhs_batching_dimensions"].empty() && known(d->operands[0]) && !fixed(d->operands[0]) &&
                         fixed(d->operands[1]) && quicker_in_front(d);
    }
    return false;
  }

  // All iterations' values of a known `v`, iteration number outermost.
  Value* stacked(Value* v) {
    auto it = stack_.find(v);
    if (it != stack_.end()) return it->second;
    const TensorType t = stacked_type(v->type, trips);
    Value* r = nullptr;
    if (Value* o = fixed(v)) {
      std::vector<int64_t> dims;
      for (int i = 0; i < v->type.rank(); i++) dims.push_back(i + 1);
      r = add(front, outer, "broadcast_in_dim", {o}, t, {{"broadcast_dimensions", i64s(dims)}});
      return stack_[v] = r;
    }
    Op* d = v->def;
    const std::string sh = d->short_name();
    auto shifted = [&](const char* attr) {
      std::vector<int64_t> out{0};
      for (int64_t x : attr_i64s(d->attr(attr))) out.push_back(x + 1);
      return out;
    };
    if (sh == "dynamic_slice") {
      Value* o = fixed(d->operands[0]);
      long long base, slope;
      affine(d->operands[1], base, slope);
      std::vector<int64_t> lo(o->type.rank(), 0), hi = o->type.dims, one(o->type.rank(), 1);
      lo[0] = slope > 0 ? base : base - (trips - 1);
      hi[0] = lo[0] + trips;
      TensorType rt = o->type;
      rt.dims[0] = trips;
      Value* rows = rt.dims == o->type.dims ? o : add(front, outer, "slice", {o}, rt, {{"start_indices", i64s(lo)}, {"limit_indices", i64s(hi)}, {"strides", i64s(one)}});
      if (slope < 0) rows = add(front, outer, "reverse", {rows}, rt, {{"dimensions", i64s({0})}});
      r = add(front, outer, "reshape", {rows}, t);
    } else if (is_elementwise_op(sh)) {
      std::vector<Value*> ins;
      for (Value* o : d->operands) ins.push_back(stacked(o));
      r = add(front, outer, sh, ins, t, d->attrs);
    } else if (sh == "reshape") {
      r = add(front, outer, "reshape", {stacked(d->operands[0])}, t);
    } else if (sh == "slice") {
      auto with = [&](const char* attr, int64_t x) {
        std::vector<int64_t> out{x};
        for (int64_t y : attr_i64s(d->attr(attr))) out.push_back(y);
        return i64s(out);
      };
      r = add(front, outer, "slice", {stacked(d->operands[0])}, t,
              {{"start_indices", with("start_indices", 0)}, {"limit_indices", with("limit_indices", trips)}, {"strides", with("strides", 1)}});
    } else if (sh == "transpose") {
      r = add(front, outer, "transpose", {stacked(d->operands[0])}, t, {{"permutation", i64s(shifted("permutation"))}});
    } else if (sh == "broadcast_in_dim") {
      r = add(front, outer, "broadcast_in_dim", {stacked(d->operands[0])}, t, {{"broadcast_dimensions", i64s(shifted("broadcast_dimensions"))}});
    } else if (sh == "concatenate") {
      std::vector<Value*> ins;
      for (Value* o : d->operands) ins.push_back(stacked(o));
      r = add(front, outer, "concatenate", ins, t, {{"dimension", std::to_string(attr_int(d->attr("dimension")) + 1) + " : i64"}});
    } else {
      auto f = attr_struct(d->attr("dot_dimension_numbers"));
      std::vector<int64_t> lc;
      for (int64_t x : f["lhs_contracting_dimensions"]) lc.push_back(x + 1);
      auto attrs = d->attrs;
      attrs["dot_dimension_numbers"] = dot_numbers({}, {}, lc, f["rhs_contracting_dimensions"]);
      attrs["b200.fma"] = "true";
      r = add(front, outer, "dot_general", {stacked(d->operands[0]), fixed(d->operands[1])}, t, attrs);
    }
    return stack_[v] = r;
  }

  // The iteration number as the type of the counter, in the body.
  std::vector<std::unique_ptr<Op>> body_ops;
  Value* zero_index = nullptr;
  Value* iteration = nullptr;
  void need_indices() {
    if (iteration) return;
    Value* c = body->args[counter];
    zero_index = zero(body_ops, body, c->type);
    iteration = c;
    if (first != 0) {
      Value* f = add(body_ops, body, "constant", {}, c->type, {{"value", "dense<" + std::to_string(first) + "> : " + c->type.str()}});
      iteration = add(body_ops, body, "subtract", {c, f}, c->type);
    }
  }

  // All iterations' values of any `v` of the body, behind the loop: known in front of it, or stacked by the loop.
  Value* history(Value* v) {
    if (known(v)) return stacked(v);
    auto it = carried_.find(v);
    if (it != carried_.end()) return it->second;
    need_indices();
    const TensorType t = stacked_type(v->type, trips);
    TensorType scalar;
    scalar.dt = t.dt;
    Value* init = add(front, outer, "broadcast_in_dim", {zero(front, outer, scalar)}, t, {{"broadcast_dimensions", i64s({})}});
    w->operands.push_back(init);
    for (Block* b : {cond, body}) {
      Value* a = m.new_value(t, "");
      a->owner = b;
      a->arg_index = (int)b->args.size();
      b->args.push_back(a);
    }
    TensorType row = v->type;
    row.dims.insert(row.dims.begin(), 1);
    std::vector<std::unique_ptr<Op>> tail;
    Value* as_row = add(tail, body, "reshape", {v}, row);
    std::vector<Value*> ins{body->args.back(), as_row, iteration};
    for (int i = 0; i < v->type.rank(); i++) ins.push_back(zero_index);
    Value* upd = add(tail, body, "dynamic_update_slice", ins, t);
    for (auto& o : tail) body->ops.insert(body->ops.end() - 1, std::move(o));
    next->operands.push_back(upd);
    Value* res = m.new_value(t, "");
    res->def = w;
    res->def_index = (int)w->results.size();
    w->results.push_back(res);
    return carried_[v] = res;
  }
  // Memory that the split asks for: stacks that live across the loop, what they are made of in front of it (each step counts as a
  // tensor, although kernels take pointwise ones in; and so does what a carried stack is to begin with), and what a sum behind it
  // needs while it is made, one after the other. `Claim` is what would come on top.
  struct Claim { std::set<Value*> stacks, steps; int64_t behind = 0; };
  Value* unshaped(Value* v) { return known(v) && !fixed(v) && v->def->short_name() == "reshape" ? unshaped(v->def->operands[0]) : v; }
  void claim_steps(Value* v, Claim& c) {
    v = unshaped(v);
    if (!c.steps.insert(v).second || fixed(v) || v->def->short_name() == "dynamic_slice") return;
    for (size_t k = 0; k < (v->def->short_name() == "dot_general" ? 1 : v->def->operands.size()); k++) claim_steps(v->def->operands[k], c);
  }
  void claim(Value* v, Claim& c) {
    c.stacks.insert(unshaped(v));
    if (known(v)) claim_steps(v, c);
  }
  int64_t step_bytes(Value* v) {
    const int64_t all = trips * (int64_t)v->type.bytes();
    if (fixed(v) || v->def->short_name() != "dynamic_slice") return all;
    long long base, slope;
    affine(v->def->operands[1], base, slope);
    return all * ((fixed(v->def->operands[0])->type.dims[0] != trips) + (slope < 0));        // a slice, reversed
  }
  Claim taken;
  bool fits(const Claim& more) {
    Claim c = taken;
    c.stacks.insert(more.stacks.begin(), more.stacks.end());
    c.steps.insert(more.steps.begin(), more.steps.end());
    c.behind = std::max(c.behind, more.behind);
    int64_t stacks = 0, front = 0;
    for (Value* v : c.stacks) {
      const int64_t all = trips * (int64_t)v->type.bytes(), written = c.steps.count(v) ? step_bytes(v) : 2 * all;       // carried: zeros, and the stack
      stacks += std::min(all, written);
      front += written - std::min(all, written);
    }
    for (Value* v : c.steps)
      if (!c.stacks.count(v)) front += step_bytes(v);
    if (stacks + std::max(front, c.behind) > kMaxStackBytes) return false;
    taken = std::move(c);
    return true;
  }

  Value* sum_over(Value* v, const std::vector<int64_t>& dims, const TensorType& t) {
    TensorType scalar;
    scalar.dt = t.dt;
    Value* r = add(back, outer, "reduce", {v, zero(back, outer, scalar)}, t, {{"dimensions", i64s(dims)}});
    Op* red = r->def;
    auto b = std::make_unique<Block>();
    b->parent_op = red;
    for (int k = 0; k < 2; k++) {
      Value* a = m.new_value(scalar, "");
      a->owner = b.get();
      a->arg_index = k;
      b->args.push_back(a);
    }
    Value* s = add(b->ops, b.get(), "add", {b->args[0], b->args[1]}, scalar);
    auto ret = std::make_unique<Op>();
    ret->name = "stablehlo.return";
    ret->operands = {s};
    ret->parent = b.get();
    b->ops.push_back(std::move(ret));
    red->regions.push_back(std::move(b));
    return r;
  }

  // Sum over iterations and rows of A^T B, from stacks [trips, rows, ..]: products over whole iterations of up to kSumRows rows
  // in all, added up; what remains of the iterations is a product of its own.
  Value* sum_of_products(Value* A, Value* B, const TensorType& t) {
    const int64_t rows = A->type.dims[1], per = std::min<int64_t>(trips, std::max<int64_t>(1, kSumRows / rows)), groups = trips / per;
    auto part = [&](Value* v, int64_t from, int64_t to, const std::vector<int64_t>& dims) {
      TensorType st = v->type;
      st.dims[0] = to - from;
      if (st.dims[0] != v->type.dims[0])
        v = add(back, outer, "slice", {v}, st, {{"start_indices", i64s({from, 0, 0})}, {"limit_indices", i64s({to, st.dims[1], st.dims[2]})}, {"strides", i64s({1, 1, 1})}});
      TensorType rt = v->type;
      rt.dims = dims;
      return add(back, outer, "reshape", {v}, rt);
    };
    const int64_t MA = A->type.dims[2], NB = B->type.dims[2];
    Value* sum = nullptr;
    if (groups > 1) {
      Value* l = part(A, 0, groups * per, {groups, per * rows, MA});
      Value* r = part(B, 0, groups * per, {groups, per * rows, NB});
      Value* each = add(back, outer, "dot_general", {l, r}, stacked_type(t, groups), {{"dot_dimension_numbers", dot_numbers({0}, {0}, {1}, {1})}, {"b200.fma", "true"}});
      sum = sum_over(each, {0}, t);
    }
    for (auto [from, to] : {std::pair<int64_t, int64_t>{0, groups == 1 ? per : 0}, {groups * per, trips}}) {
      if (from >= to) continue;
      Value* l = part(A, from, to, {(to - from) * rows, MA});
      Value* r = part(B, from, to, {(to - from) * rows, NB});
      Value* one = add(back, outer, "dot_general", {l, r}, t, {{"dot_dimension_numbers", dot_numbers({}, {}, {0}, {0})}, {"b200.fma", "true"}});
      sum = sum ? add(back, outer, "add", {sum, one}, t) : one;
    }
    return sum;
  }

  void products_in_front() {
    for (size_t i = 0; i < body->ops.size(); i++) {
      Op* d = body->ops[i].get();
      if (d->short_name() != "dot_general" || d->results.size() != 1 || !known(d->results[0])) continue;
      Claim c;
      claim(d->results[0], c);
      if (!fits(c)) continue;
      Value* all = stacked(d->results[0]);
      need_indices();
      TensorType row = d->results[0]->type;
      row.dims.insert(row.dims.begin(), 1);
      std::vector<Value*> ins{all, iteration};
      for (int q = 0; q < d->results[0]->type.rank(); q++) ins.push_back(zero_index);
      std::vector<std::unique_ptr<Op>> at;
      Value* mine = add(at, body, "dynamic_slice", ins, row, {{"slice_sizes", i64s(row.dims)}});
      // the product turns into a reshape of its slice: the same result value, so its users need no change
      d->name = "stablehlo.reshape";
      d->operands = {mine};
      d->attrs.clear();
      body->ops.insert(body->ops.begin() + i, std::move(at[0]));
      i++;
      changed = true;
    }
  }

  void sums_behind() {
    std::set<int> gone;
    const int n = (int)body->args.size();
    // products first: sums of rows leave where what they read is known in front of the loop or stacked for a product anyway
    for (int i = 0; i < 2 * n; i++) {
      const int k = i % n;
      const bool products = i < n;
      Value *a = body->args[k], *r = next->operands[k];
      Op* s = r->def;
      if (k == counter || gone.count(k) || a->type.dt != DT::F32 || !s || s->parent != body || s->short_name() != "add" || count_uses(cond, cond->args[k])) continue;
      Value* term = s->operands[0] == a ? s->operands[1] : s->operands[1] == a ? s->operands[0] : nullptr;
      if (!term || term == a || count_uses(body, a) != 1 || count_uses(body, r) != 1 || !term->def || term->def->parent != body || count_uses(body, term) != 1) continue;
      Op* d = term->def;
      Value* sum = nullptr;
      if (products && d->short_name() == "dot_general") {
        auto f = attr_struct(d->attr("dot_dimension_numbers"));
        Value *A = d->operands[0], *B = d->operands[1];
        if (A->type.rank() != 2 || B->type.rank() != 2 || A->type.dt != DT::F32 || B->type.dt != DT::F32 || A == B) continue;
        if (!f["lhs_batching_dimensions"].empty() || f["lhs_contracting_dimensions"] != std::vector<int64_t>{0} || f["rhs_contracting_dimensions"] != std::vector<int64_t>{0}) continue;
        if (fixed(A) || fixed(B) || d->results[0]->type.numel() * A->type.dims[0] == 0) continue;
        const int64_t per = std::min<int64_t>(trips, std::max<int64_t>(1, kSumRows / A->type.dims[0]));
        if (!quicker_behind(d, per)) continue;
        Claim c;
        claim(A, c);
        claim(B, c);
        c.behind = (trips / per + 3) * (int64_t)term->type.bytes();
        if (trips % per) c.behind += trips * (int64_t)(A->type.bytes() + B->type.bytes());      // the whole sums' iterations, sliced
        if (!fits(c)) continue;
        sum = sum_of_products(history(A), history(B), term->type);
      } else if (!products && d->short_name() == "reduce" && d->operands.size() == 2) {
        Op* z = d->operands[1]->def;
        Block* rb = d->regions[0].get();
        if (!z || z->short_name() != "constant" || rb->ops.size() != 2 || rb->ops[0]->short_name() != "add" || rb->ops[0]->operands[0] == rb->ops[0]->operands[1]) continue;
        DenseValue dv = attr_dense(z->attr("value"));
        float zero_value = 1.f;
        if (dv.type.dt != DT::F32 || dv.type.numel() != 1) continue;
        memcpy(&zero_value, dv.data.data(), 4);
        Claim c;
        if (zero_value != 0.f || d->operands[0]->type.dt != DT::F32 || fixed(d->operands[0])) continue;
        if (!known(d->operands[0]) && !carried_.count(d->operands[0])) continue;
        claim(d->operands[0], c);
        if (!fits(c)) continue;
        std::vector<int64_t> dims{0};
        for (int64_t x : attr_i64s(d->attr("dimensions"))) dims.push_back(x + 1);
        sum = sum_over(history(d->operands[0]), dims, term->type);
      } else continue;
      Value* total = add(back, outer, "add", {w->operands[k], sum}, term->type);
      replace_uses(outer, w->results[k], total);
      gone.insert(k);
      changed = true;
    }
    // the accumulators leave the loop
    for (auto it = gone.rbegin(); it != gone.rend(); ++it) {
      const int k = *it;
      w->operands.erase(w->operands.begin() + k);
      w->results.erase(w->results.begin() + k);
      next->operands.erase(next->operands.begin() + k);
      for (Block* b : {cond, body}) {
        replace_uses(b, b->args[k], b->args[counter]);      // only the dropped additions read it
        b->args.erase(b->args.begin() + k);
        for (size_t i = k; i < b->args.size(); i++) b->args[i]->arg_index = (int)i;
      }
      for (size_t i = k; i < w->results.size(); i++) w->results[i]->def_index = (int)i;
      if (k < counter) counter--;
    }
  }

  bool run() {
    if (!find_counter()) return false;
    products_in_front();
    sums_behind();
    body->ops.insert(body->ops.begin(), std::make_move_iterator(body_ops.begin()), std::make_move_iterator(body_ops.end()));
    return changed;
  }
};

}  // namespace

void split_counted_loops(Module& m, Block* b, const LoopProductModel& model) {
  for (size_t i = 0; i < b->ops.size(); i++) {
    Op* op = b->ops[i].get();
    if (op->short_name() != "while" || op->regions.size() != 2 || op->regions[1]->ops.empty()) continue;
    Splitter s{m, b, op, op->regions[0].get(), op->regions[1].get(), op->regions[1]->ops.back().get(), model};
    s.run();
    const size_t f = s.front.size(), k = s.back.size();
    b->ops.insert(b->ops.begin() + i + 1, std::make_move_iterator(s.back.begin()), std::make_move_iterator(s.back.end()));
    b->ops.insert(b->ops.begin() + i, std::make_move_iterator(s.front.begin()), std::make_move_iterator(s.front.end()));
    i += f + k;
  }
}

}  // namespace b200
