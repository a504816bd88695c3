#include "dn_resident2d_adj.cuh"

template int dn::res::run_resident_adjoint<double>(const AdjJob<double>&, const SampleSet<double>&,
                                                const Split&, uint64_t*, int*, cudaStream_t);
