// The PK steps of the free-space pipeline on FP64 fields with FP32 transforms (the
// defect-corrected applies; see op_impl.cuh).
#include "op_impl.cuh"

namespace asb {

template <>
void free_pk_eval<double, float>(const Operator& op, const PkFields<double>& f, cplx<float>* spec, cudaStream_t s,
        int B) {
    ASB_FREE_SWITCH(op.Ns, (pk_eval_apply<FreeImpl<float, NS>, double, float>(op, f, spec, s, B)));
}
template <>
void free_pk_line<double, float>(const Operator& op, const PkFields<double>& f, cplx<float>* spec, cudaStream_t s,
        int B) {
    ASB_FREE_SWITCH(op.Ns, (pk_line_apply<FreeImpl<float, NS>, double, float>(op, f, spec, s, B)));
}

}  // namespace asb
