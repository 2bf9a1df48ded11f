// Resident runs: the choice of the class (resident.cuh, one translation unit
// per class).
#include "kernels.h"

namespace ab
{

cudaError_t launch_resident2(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits);
cudaError_t launch_resident3(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits);
cudaError_t launch_resident4(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits);
cudaError_t launch_resident5(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits);

static cudaError_t resident_any(const ResJob & J, const TConst & c, cudaStream_t s, int ncand, bool * fits)
{
	switch (c.K)
	{
	case 2: return launch_resident2(J, c, s, ncand, fits);
	case 3: return launch_resident3(J, c, s, ncand, fits);
	case 4: return launch_resident4(J, c, s, ncand, fits);
	case 5: return launch_resident5(J, c, s, ncand, fits);
	default: if (fits) *fits = false; return (ncand == 0) ? cudaSuccess : cudaErrorNotSupported;
	}
}

bool resident_fits(const TConst & c)
{
	bool fits = false;
	const ResJob none{};
	return resident_any(none, c, nullptr, 0, &fits) == cudaSuccess && fits;
}

cudaError_t launch_resident(const ResJob & J, const TConst & c, cudaStream_t s, int ncand)
{
	if (ncand == 0) return cudaSuccess;
	return resident_any(J, c, s, ncand, nullptr);
}

} // namespace ab
