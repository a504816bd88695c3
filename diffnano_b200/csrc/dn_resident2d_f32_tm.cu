#include "dn_resident2d_fwd.cuh"

template int dn::res::run_resident<float, DN_TM>(const Job<float>&, const SampleSet<float>&, const Split&,
                                              uint64_t*, int*, cudaStream_t);
