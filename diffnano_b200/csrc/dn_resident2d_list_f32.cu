#include "dn_resident2d_list.cuh"

template int dn::res::run_resident_list<float>(const List&, bool, bool, int, int, int*, cudaStream_t);
