// A graph's walk as data: the primitive operations of a Forward or Backward walk in order, and their execution as one kernel.
#pragma once

#include <memory>
#include <vector>

#include "common.cuh"

namespace prad {

enum PrimKind : int {
  // elementwise over n values
  PRIM_ACT_FORWARD, PRIM_ACT_BACKWARD, PRIM_ADD2, PRIM_ADD3, PRIM_MUL2, PRIM_MUL_BACKWARD, PRIM_SCALE, PRIM_COPY, PRIM_SUM, PRIM_ADD_ROW,
  PRIM_LAST_ELEMENTWISE = PRIM_ADD_ROW,
  PRIM_PRODUCT, PRIM_COLUMN_SUM, PRIM_TRANSPOSE, PRIM_SOFTMAX, PRIM_SOFTMAX_BACKWARD, PRIM_SINE_SOFTMAX, PRIM_SINE_SOFTMAX_BACKWARD,
  PRIM_LAYERNORM, PRIM_LAYERNORM_BACKWARD
};

// One primitive operation.  in / out in the order of the entry point it stands for; rows x cols of a row-wise operation,
// M, N, K ... of a product (PRIM_PRODUCT: out[0] = alpha op(in[0]) op(in[1]) over `batch` slices).
struct Prim {
  PrimKind kind;
  int act = 0;
  double scalar = 0;              // activation parameter, factor, alpha of a product
  std::vector<const void*> in;
  std::vector<void*> out;
  int64_t n = 0;                  // values of an elementwise operation
  int64_t rows = 0;
  int cols = 0, depth = 1;
  bool tA = false, tB = false;
  int M = 0, N = 0, K = 0, batch = 1;
  int64_t sA = 0, sB = 0, sC = 0; // batch strides in elements (0: shared); leading dimensions are dense
};

// The start gradients of a Backward are another program's matrices every time.  Operations name the i-th one by this stand-in
// (no device address has these high bits), and a run says which matrices they are.
inline const void* start_stand_in(int i) { return (const void*)(((uint64_t)1 << 62) | ((uint64_t)i << 40)); }
inline bool is_stand_in(const void* p) { return ((uint64_t)p >> 62) == 1; }
inline int stand_in_index(const void* p) { return (int)(((uint64_t)p >> 40) & 0x3fffff); }
constexpr int MOST_STARTS = 4000;            // what a kernel's arguments have room for

struct GraphPlan;
struct GraphPlanFree { void operator()(GraphPlan* p) const; };
using GraphPlanPtr = std::unique_ptr<GraphPlan, GraphPlanFree>;

// A plan for these operations, or null when one launch per operation is the better way to run them (few of them, large ones,
// or a device that cannot run the cluster).
GraphPlanPtr graph_plan_build(prad_ctx* ctx, prad_dtype dt, const std::vector<Prim>& ops);
prad_status graph_plan_run(prad_ctx* ctx, GraphPlan* plan, const void* const* starts = nullptr, int count = 0);
// how many products its programs compute for themselves
int graph_plan_products(const GraphPlan* plan);
// whether the plan's operations write anywhere in [p, p + bytes)
bool graph_plan_writes(const GraphPlan* plan, const void* p, size_t bytes);

}  // namespace prad
