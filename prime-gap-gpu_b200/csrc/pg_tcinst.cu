// pg_tcinst.cu -- one operand size of the tensor-core search kernel (built
// once per L with -DPG_TCL=L; see pg_tc_search.cuh).
#include "pg_tc_search.cuh"

#ifndef PG_TCL
#error "compile with -DPG_TCL=<limb count>"
#endif

namespace pg {
PG_TC_INSTANTIATE(PG_TCL)
}  // namespace pg
