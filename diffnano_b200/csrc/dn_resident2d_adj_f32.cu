#include "dn_resident2d_adj.cuh"

template int dn::res::run_resident_adjoint<float>(const AdjJob<float>&, const SampleSet<float>&,
                                                const Split&, uint64_t*, int*, cudaStream_t);
