// Host side of the any-extent step kernels (lfts_step_any.cu).
#pragma once
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/lfts_b200.h"

namespace lfts {

struct AnyGrid;  // plan, device tables and launch limits of one grid and precision

// nullptr when a plane or a column tile does not fit in shared memory (err empty)
// or on a CUDA error (err says which).  axis extents as the context pads them.
AnyGrid *any_create(int prec, const int n[3], int nsm, int max_smem, std::string &err);
void any_destroy(AnyGrid *a);
// Radices of an n-point transform, outermost first: register radices (2 .. 13, 16) and
// primes above 13; false when a prime is too large for the kernels.
bool any_radices(int n, std::vector<int> &r);

void any_steps_continuous(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps);
void any_steps_discrete(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps, int half, int with_fac);
// zy-transforms of one real field per job into spectrum slot 0 (half the 3D transform)
void any_planes_forward(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj);
void any_xpass_forward(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj);

// stress: x-transform of both zy spectra of a job and the weighted sums over k;
// partials[(job * tiles + tile) * 3 + axis]
int any_stress_tiles(const AnyGrid *a, int nj);
void any_xstress(const AnyGrid *a, cudaStream_t st, const lfts_step_job *sj, const lfts_stress_job *jobs, int nj,
                 const double *basis, double *partials);

// CTAs per job of the cluster sweep for nj jobs; 0: the grid does not fit or the
// separate passes are faster.  force: 0 by that rule, else this cluster size where it fits.
int any_sweep_size(const AnyGrid *a, bool continuous, int nj, int force);
int any_sweep_continuous(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps, int cs);
int any_sweep_discrete(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps, int half,
                       int with_fac, int cs);

}  // namespace lfts
