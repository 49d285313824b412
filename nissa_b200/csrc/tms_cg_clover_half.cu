// The e/o twisted-clover CG with FP16 inner spinors, in a unit of its own: it would
// double the longest compilation.
#include "tms_clov_op.cuh"

namespace tms_int
{
  template tms_status cg_half<ClovOp>(tms_ctx*, int, double, bool, tms_stats*);
}
