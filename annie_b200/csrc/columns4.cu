// The column pass of the classes with 4 reference primes.
#include "columns.cuh"

namespace ab
{

cudaError_t launch_colpass4(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	return colpass_k<4, 2>(g, c, jobs, njobs, s, ncand);
}

} // namespace ab
