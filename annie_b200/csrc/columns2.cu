// The column pass of the classes with 2 reference primes.
#include "columns.cuh"

namespace ab
{

cudaError_t launch_colpass2(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	return colpass_k<2, 1>(g, c, jobs, njobs, s, ncand);
}

} // namespace ab
