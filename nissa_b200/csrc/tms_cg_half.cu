// The e/o twisted-mass CG with FP16 inner spinors, in a unit of its own: it is
// compiled differently from the others (SPLIT_UNITS in build.py).
#include "tms_eo_op.cuh"

namespace tms_int
{
  template tms_status cg_half<EoOp>(tms_ctx*, int, double, bool, tms_stats*);
}
