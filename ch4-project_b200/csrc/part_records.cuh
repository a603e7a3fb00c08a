// Particle records as the caller holds them: ch4_particle of consecutive state slots, from
// the planes of the particle state.
//
// Bound by the copy to the host that follows (560 bytes per particle over PCIe), so the tile
// is simply the smallest that makes both sides whole runs: 32 slots, read as 32 consecutive
// values of a plane and written record by record.  The odd row length lets a warp's column
// in shared memory meet every bank.  What it replaces is a transposition by one
// host thread out of pageable memory: reading back 160^3 fields and 250,000 records after 600
// steps took 167 ms of 373 ms and takes 28 ms of 234 ms.
#pragma once

#include "particles.cuh"

namespace ch4 {

#ifdef __CUDACC__

constexpr int PREC_SLOTS = 32, PREC_THREADS = 256, PREC_ROW = PF_FIELDS | 1;

// out: m records of PF_FIELDS values, slots s0 .. s0 + m - 1 of np
__global__ void __launch_bounds__(PREC_THREADS) particle_records_kernel(const double* __restrict__ pf, long long np,
                                                                        int s0, int m, double* __restrict__ out) {
  __shared__ double tile[PREC_SLOTS][PREC_ROW];
  const int first = blockIdx.x * PREC_SLOTS, n = min(PREC_SLOTS, m - first);
  const int lane = threadIdx.x & 31;
  if (lane < n)
    for (int f = threadIdx.x >> 5; f < PF_FIELDS; f += PREC_THREADS / 32)
      tile[lane][f] = pf[f * np + s0 + first + lane];
  __syncthreads();
  for (int r = threadIdx.x >> 5; r < n; r += PREC_THREADS / 32)
    for (int f = lane; f < PF_FIELDS; f += 32) out[(long long)(first + r) * PF_FIELDS + f] = tile[r][f];
}

#endif  // __CUDACC__
}  // namespace ch4
