// The free-space pipeline in FP64 (see op_impl.cuh).
#include "op_impl.cuh"

namespace asb {

template <>
void free_matvec<double>(const Operator& op, const double* x, double* y, cplx<double>* spec, cudaStream_t s,
                    const int* gate, int B) {
    ASB_FREE_SWITCH(op.Ns, (FreeImpl<double, NS>::matvec(op, x, y, spec, s, gate, B)));
}

template <>
void free_apply_block<double>(const Operator& op, const double* x, double* y, cplx<double>* spec, cudaStream_t s) {
    const long nl = (long)op.Nl * op.Nl;
    ASB_FREE_SWITCH(op.Ns, (FreeImpl<double, NS>::apply_block(op, x, y, nl, spec, s)));
}

template <>
void embedded_precond<double>(Operator& op, const double* ga, const double* gb, const uint8_t* mask, PkState* st,
                        double* z,
                         double* part, cudaStream_t s, const int* gate, int B, void* spec) {
    ASB_FREE_SWITCH(op.Ns, (EmbeddedFourierImpl<double, NS>::run(op, ga, gb, mask, st, z, part, s, gate, B,
                                                            spec)));
}

}  // namespace asb
