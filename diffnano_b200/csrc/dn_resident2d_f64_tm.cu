#include "dn_resident2d_fwd.cuh"

template int dn::res::run_resident<double, DN_TM>(const Job<double>&, const SampleSet<double>&, const Split&,
                                              uint64_t*, int*, cudaStream_t);
