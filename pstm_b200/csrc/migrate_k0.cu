// Instantiations of the gather kernel for traveltime kind 0.
#include "migrate_dispatch.cuh"
namespace pstm {
template cudaError_t launch_gather<0>(const KParams &, int, const Launch &);
}
