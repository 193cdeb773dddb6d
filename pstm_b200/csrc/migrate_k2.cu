// Instantiations of the gather kernel for traveltime kind 2.
#include "migrate_dispatch.cuh"
namespace pstm {
template cudaError_t launch_gather<2>(const KParams &, int, const Launch &);
}
