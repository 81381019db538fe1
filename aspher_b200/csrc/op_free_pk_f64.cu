// The PK steps of the free-space pipeline in FP64 (see op_impl.cuh).
#include "op_impl.cuh"

namespace asb {

template <>
void free_pk_eval<double, double>(const Operator& op, const PkFields<double>& f, cplx<double>* spec, cudaStream_t s,
        int B) {
    ASB_FREE_SWITCH(op.Ns, (pk_eval_apply<FreeImpl<double, NS>, double, double>(op, f, spec, s, B)));
}
template <>
void free_pk_line<double, double>(const Operator& op, const PkFields<double>& f, cplx<double>* spec, cudaStream_t s,
        int B) {
    ASB_FREE_SWITCH(op.Ns, (pk_line_apply<FreeImpl<double, NS>, double, double>(op, f, spec, s, B)));
}

}  // namespace asb
