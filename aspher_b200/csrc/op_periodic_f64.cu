// The periodic pipeline and the full-grid |k| preconditioner in FP64 (see
// op_impl.cuh).
#include "op_impl.cuh"

namespace asb {

template <>
void periodic_matvec<double>(const Operator& op, const double* x, double* y, cplx<double>* spec, cudaStream_t s,
                        const int* gate, int B) {
    ASB_SIZE_SWITCH(op.Ns, (PeriodicImpl<double, NS>::matvec(op, x, y, spec, s, gate, B)));
}

template <>
void periodic_precond<double>(Operator& op, const double* ga, const double* gb, const uint8_t* mask, PkState* st,
                        double* z,
                         double* part, cudaStream_t s, const int* gate, int B, void* spec) {
    ASB_SIZE_SWITCH(op.Ns, (FourierImpl<double, NS>::run(op, ga, gb, mask, st, z, part, s, gate, B, spec)));
}

}  // namespace asb
