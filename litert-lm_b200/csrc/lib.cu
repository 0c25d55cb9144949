// The executor, the prefill kernels and the operator-level ABI; the kernels with many instantiations are
// translation units of their own.
#include "executor.cu"
#include "ops.cu"
#include "ops_static.cu"
