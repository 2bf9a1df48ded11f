// The column pass of the classes with 5 reference primes.
#include "columns.cuh"

namespace ab
{

cudaError_t launch_colpass5(const Geometry & g, const TConst & c, const ColJobs & jobs, int njobs, cudaStream_t s, int ncand)
{
	return colpass_k<5, 4>(g, c, jobs, njobs, s, ncand);
}

} // namespace ab
