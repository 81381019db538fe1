// The free-space pipeline in FP32 (see op_impl.cuh).
#include "op_impl.cuh"

namespace asb {

template <>
void free_matvec<float>(const Operator& op, const float* x, float* y, cplx<float>* spec, cudaStream_t s,
                    const int* gate, int B) {
    ASB_FREE_SWITCH(op.Ns, (FreeImpl<float, NS>::matvec(op, x, y, spec, s, gate, B)));
}

template <>
void free_apply_block<float>(const Operator& op, const float* x, float* y, cplx<float>* spec, cudaStream_t s) {
    const long nl = (long)op.Nl * op.Nl;
    ASB_FREE_SWITCH(op.Ns, (FreeImpl<float, NS>::apply_block(op, x, y, nl, spec, s)));
}

template <>
void embedded_precond<float>(Operator& op, const float* ga, const float* gb, const uint8_t* mask, PkState* st,
                        float* z,
                         double* part, cudaStream_t s, const int* gate, int B, void* spec) {
    ASB_FREE_SWITCH(op.Ns, (EmbeddedFourierImpl<float, NS>::run(op, ga, gb, mask, st, z, part, s, gate, B,
                                                            spec)));
}

}  // namespace asb
