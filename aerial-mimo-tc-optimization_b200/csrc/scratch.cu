// scratch.cu -- device memory of the library's own, for aerial_pusch_eq_plain_static
// alone: a cell whose outputs overlap its own inputs runs stage by stage and
// has to keep the stages' results somewhere.  The array is the only symbol of this
// file, and with it of its module, so that with lazy module loading a GPU holds
// the 16 MiB only once a call has asked for them.
#include "common.cuh"

namespace aeq {

__device__ __align__(256) unsigned char g_static_scratch[AERIAL_STATIC_SCRATCH_BYTES];

// Its address in the current context (loads the module on the first call there).
int static_scratch(char** out) {
    void* p = nullptr;
    const int s = rt_status(cudaGetSymbolAddress(&p, g_static_scratch));
    *out = static_cast<char*>(p);
    return s;
}

}  // namespace aeq
