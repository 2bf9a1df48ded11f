// Resident runs of the classes with 3 reference primes.
#include "resident.cuh"

namespace ab
{

cudaError_t launch_resident3(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits)
{
	return resident_k<3, 2>(J, c, s, ncand, fits);
}

} // namespace ab
