// Resident runs of the classes with 2 reference primes.
#include "resident.cuh"

namespace ab
{

cudaError_t launch_resident2(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits)
{
	return resident_k<2, 1>(J, c, s, ncand, fits);
}

} // namespace ab
