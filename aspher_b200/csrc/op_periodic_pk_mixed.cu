// The PK steps of the periodic pipeline on FP64 fields with FP32 transforms (the
// defect-corrected applies; see op_impl.cuh).
#include "op_impl.cuh"

namespace asb {

template <>
void periodic_pk_eval<double, float>(const Operator& op, const PkFields<double>& f, cplx<float>* spec, cudaStream_t s,
        int B) {
    ASB_SIZE_SWITCH(op.Ns, (pk_eval_apply<PeriodicImpl<float, NS>, double, float>(op, f, spec, s, B)));
}
template <>
void periodic_pk_line<double, float>(const Operator& op, const PkFields<double>& f, cplx<float>* spec, cudaStream_t s,
        int B) {
    ASB_SIZE_SWITCH(op.Ns, (pk_line_apply<PeriodicImpl<float, NS>, double, float>(op, f, spec, s, B)));
}

}  // namespace asb
