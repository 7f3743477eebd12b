// Device-side reductions shared by the fused Krylov solvers (PCG and flexible CG): exact
// dot products whose last block produces the solver's scalars without a host round trip.
#pragma once
#include "kernels.cuh"
#include "sts_internal.cuh"

// Block combine of up to two exact accumulators into s->limbs (device scalar block S with
// limbs[2][NL], flags[2] and ticket); the last block to arrive finalises the sums, resets
// the accumulators and runs `fin` on the results.
template <int NT, int NACC, typename S, typename Fin>
__device__ __forceinline__ void krylov_block_finish(xsum::Limbs* a, unsigned* fl, S* s, Fin fin)
{
  __shared__ long long sm[NACC][NT / 32][xsum::NL];
  __shared__ unsigned sflags[NACC];
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  long long v[NACC];
#pragma unroll
  for (int c = 0; c < NACC; ++c) v[c] = xsum_block_limbs<NT>(a[c], &fl[c], sm[c], &sflags[c]);
  if (tid >= 32) return;
#pragma unroll
  for (int c = 0; c < NACC; ++c)
  {
    if (tid < xsum::NL && v[c] != 0) atomicAdd(&s->limbs[c][tid], (unsigned long long)v[c]);
    if (tid == 0 && fl[c]) atomicOr(&s->flags[c], fl[c]);
  }
  __threadfence();
  __syncwarp();
  unsigned t = 0;
  if (tid == 0) t = atomicAdd(&s->ticket, 1u);
  t = __shfl_sync(0xffffffffu, t, 0);
  if (t != gridDim.x * gridDim.y - 1) return;
  __threadfence();
  unsigned f[NACC];
#pragma unroll
  for (int c = 0; c < NACC; ++c)
  {
    f[c] = 0;
    if (tid < xsum::NL) sm[c][0][tid] = (long long)atomicExch(&s->limbs[c][tid], 0ULL);
    else if (tid == xsum::NL) f[c] = atomicExch(&s->flags[c], 0u);
  }
  if (tid == xsum::NL + 1) s->ticket = 0u;
#pragma unroll
  for (int c = 0; c < NACC; ++c) f[c] = __shfl_sync(0xffffffffu, f[c], xsum::NL);
  __syncwarp(); // lane 0 reads the other lanes' limbs: a shuffle orders no memory
  if (tid == 0)
  {
    double r[NACC];
#pragma unroll
    for (int c = 0; c < NACC; ++c) r[c] = xsum::finalize(sm[c][0], f[c]);
    fin(r);
  }
}
