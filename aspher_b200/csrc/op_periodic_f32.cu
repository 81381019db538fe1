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

}  // namespace asb
