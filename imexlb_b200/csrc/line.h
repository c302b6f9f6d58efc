// Shared-memory staged step for the 8- and 4-byte storage formats (line.cu).
#pragma once

#include "lattice.h"

namespace imx {

bool line_supported(const LaunchCfg& c, int nx, int ny, int nz, int64_t pitch);
cudaError_t launch_line(const LaunchCfg& c, const StepArgs& a, cudaStream_t s);

// The staged copies of one lattice (see imexlb_debug_line_plan).
int64_t line_plan(int nx, int ny, int nz, bool wrap, int elem, int32_t* geo, int32_t* runs, int64_t max_runs);

}  // namespace imx
