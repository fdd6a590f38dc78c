// fdga_ring.h -- uses of a ring of pipeline stages, one mbarrier phase per use (host and device).
#pragma once

#ifdef __CUDACC__
#define FDGA_HD __host__ __device__
#else
#define FDGA_HD
#endif

namespace fdga {

// stage of use c in a ring of ns stages, and the parity of the stage's mbarrier phase that the use completes
FDGA_HD constexpr int ring_stage(int c, int ns) { return c % ns; }
FDGA_HD constexpr unsigned ring_parity(int c, int ns) { return (unsigned)(c / ns) & 1u; }

}  // namespace fdga
