// Resident runs of the classes with 5 reference primes.
#include "resident.cuh"

namespace ab
{

cudaError_t launch_resident5(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits)
{
	return resident_k<5, 4>(J, c, s, ncand, fits);
}

} // namespace ab
