// The periodic pipeline and the full-grid |k| preconditioner in FP32 (see
// op_impl.cuh).
#include "op_impl.cuh"

namespace asb {

template <>
void periodic_matvec<float>(const Operator& op, const float* x, float* y, cplx<float>* spec, cudaStream_t s,
                        const int* gate, int B) {
    ASB_SIZE_SWITCH(op.Ns, (PeriodicImpl<float, NS>::matvec(op, x, y, spec, s, gate, B)));
}

template <>
void periodic_precond<float>(Operator& op, const float* ga, const float* gb, const uint8_t* mask, PkState* st,
                        float* z,
                         double* part, cudaStream_t s, const int* gate, int B, void* spec) {
    ASB_SIZE_SWITCH(op.Ns, (FourierImpl<float, NS>::run(op, ga, gb, mask, st, z, part, s, gate, B, spec)));
}

template <>
void periodic_pk_eval<float, float>(const Operator& op, const PkFields<float>& f, cplx<float>* spec, cudaStream_t s,
        int B) {
    ASB_SIZE_SWITCH(op.Ns, (pk_eval_apply<PeriodicImpl<float, NS>, float, float>(op, f, spec, s, B)));
}
template <>
void periodic_pk_line<float, float>(const Operator& op, const PkFields<float>& f, cplx<float>* spec, cudaStream_t s,
        int B) {
    ASB_SIZE_SWITCH(op.Ns, (pk_line_apply<PeriodicImpl<float, NS>, float, float>(op, f, spec, s, B)));
}
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
