// The PK steps of the free-space pipeline in FP32 (see op_impl.cuh).
#include "op_impl.cuh"

namespace asb {

template <>
void free_pk_eval<float, float>(const Operator& op, const PkFields<float>& f, cplx<float>* spec, cudaStream_t s,
        int B) {
    ASB_FREE_SWITCH(op.Ns, (pk_eval_apply<FreeImpl<float, NS>, float, float>(op, f, spec, s, B)));
}
template <>
void free_pk_line<float, float>(const Operator& op, const PkFields<float>& f, cplx<float>* spec, cudaStream_t s,
        int B) {
    ASB_FREE_SWITCH(op.Ns, (pk_line_apply<FreeImpl<float, NS>, float, float>(op, f, spec, s, B)));
}

}  // namespace asb
