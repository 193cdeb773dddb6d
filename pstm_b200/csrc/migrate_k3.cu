// Instantiations of the gather kernel for traveltime kind 3.
#include "migrate_dispatch.cuh"
namespace pstm {
template cudaError_t launch_gather<3>(const KParams &, int, const Launch &);
}
