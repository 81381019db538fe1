// The PK steps of the periodic pipeline in FP64 (see op_impl.cuh).
#include "op_impl.cuh"

namespace asb {

template <>
void periodic_pk_eval<double, double>(const Operator& op, const PkFields<double>& f, cplx<double>* spec, cudaStream_t s,
        int B) {
    ASB_SIZE_SWITCH(op.Ns, (pk_eval_apply<PeriodicImpl<double, NS>, double, double>(op, f, spec, s, B)));
}
template <>
void periodic_pk_line<double, double>(const Operator& op, const PkFields<double>& f, cplx<double>* spec, cudaStream_t s,
        int B) {
    ASB_SIZE_SWITCH(op.Ns, (pk_line_apply<PeriodicImpl<double, NS>, double, double>(op, f, spec, s, B)));
}

}  // namespace asb
