// Coefficient-form (FMA) sweeps: the FP64 fast sweeps and the kernels of the
// mixed-precision defect-correction form.
//
// Mixed precision.  One iteration of the solver is an affine map x -> F(x) of
// the padded state.  Writing the iterate as x + e with x a fixed FP64 state,
// e evolves by e -> L(e) + r, where L is the linear part of F (same stencil,
// homogeneous boundary values) and r = F(x) - x.  The correction e and the
// residual r are stored in FP32 (half the bytes of a sweep); every block of
// sweeps ends with the FP64 update x += e and a fresh FP64 residual, so FP32
// rounding only ever touches the (shrinking) correction and the iterate
// converges to the FP64 fixed point.
#include <algorithm>

#include "pm_internal.h"
#include "pm_stencil.cuh"

namespace pm {

// ------------------------------------------------------------------ FP64 fast sweeps
template <int SOLVER, int PHASE>
__global__ void __launch_bounds__(256) k_sweep64_fast(Fields<double> A, Fields<double> B,
                                                      const uint8_t* codes, const int* list,
                                                      int nlist, Grid g) {
  __shared__ Tables64 tab;
  fill_tables64<SOLVER>(tab);
  __syncthreads();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nlist; q += gridDim.x * blockDim.x)
    sweep64_voxel<SOLVER, PHASE, false>(A, B, codes, g, list[q], &tab);
}

cudaError_t sweep64_exact(Fields<double> A, Fields<double> B, const uint8_t* codes,
                          const int* list, int nlist, const Grid& g, int solver, int phase,
                          cudaStream_t st);

// Persistent form: one wave of MINB CTAs per SM walks the list with a grid
// stride, each thread loading its next list entry before it computes the
// current voxel.  Launches overlap: a CTA's slot goes to the next sweep's as it
// ends, which loads its tables and first list entries and waits for this sweep
// before it touches a field.
// Bound: the FP64 pipe (31 instructions of a warp per voxel, 25 of them FMAs of
// 16 clocks per SM and 6 others of 19: 40 us for the 734k voxels of a 128^3
// pack) and, between a warp's instructions there, its loads; the half-sweeps
// of that pack also miss L2 (their two states touch 120 MB).  Two CTAs leave
// 128 registers, so that all of a voxel's loads are in flight at once; three
// leave 80, next to no spills, and keep the pipe busier where there is enough work:
// Jacobi on the 128^3 pack 44.0 us against 46.5 with two, red-black 57.6 against
// 59.8 (55.7 with the hint of update64); a 97x61x118 pack 25.7 against 21.9 (its half-sweeps are 1.2 waves of
// three).  With the whole stencil loaded and plain launches: 48.4, 63 and 26.1.
template <int SOLVER, int PHASE, int MINB>
__global__ void __launch_bounds__(256, MINB) k_sweep64_pf(Fields<double> A, Fields<double> B,
                                                      const uint8_t* codes, const int* list,
                                                      int nlist, Grid g) {
  __shared__ Tables64 tab;
  fill_tables64<SOLVER>(tab);
  __syncthreads();
  const int stride = gridDim.x * blockDim.x;
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  int lin = q < nlist ? __ldg(list + q) : 0;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (; q < nlist; q += stride) {
    const int qn = q + stride;
    if (qn >= nlist) asm volatile("griddepcontrol.launch_dependents;");
    const int next = qn < nlist ? __ldg(list + qn) : 0;
    sweep64_voxel<SOLVER, PHASE, false, kLdPlain>(A, B, codes, g, lin, &tab);
    lin = next;
  }
}

// The whole stencil per voxel, two CTAs per SM (128 registers), plain launches:
// no load waits for the code byte.  Bound as the sweep above; where its voxels'
// values come from beyond L2, or are dense, the 37 loads cost less than the wait
// (choose_fp64_shapes has both sides), and beside other problems the plain
// launches do (a CTA that waits for its predecessor takes the place of one that
// could run).
template <int SOLVER, int PHASE>
__global__ void __launch_bounds__(256, 2) k_sweep64_whole(Fields<double> A, Fields<double> B,
                                                         const uint8_t* codes, const int* list,
                                                         int nlist, Grid g) {
  __shared__ double centre[16];
  fill_centre64<SOLVER>(centre);
  __syncthreads();
  const int stride = gridDim.x * blockDim.x;
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  int lin = q < nlist ? __ldg(list + q) : 0;
  for (; q < nlist; q += stride) {
    const int qn = q + stride;
    const int next = qn < nlist ? __ldg(list + qn) : 0;
    sweep64_voxel<SOLVER, PHASE, false>(A, B, codes, g, lin, nullptr, centre);
    lin = next;
  }
}

template <int SOLVER, int MINB>
static cudaError_t sweep_pf(Fields<double> A, Fields<double> B, const uint8_t* codes,
                            const int* list, int nlist, const Grid& g, int phase,
                            cudaStream_t st) {
  const int blocks = std::min((nlist + 255) / 256, MINB * sm_count());
  auto* k = phase == 0 ? k_sweep64_pf<SOLVER, 0, MINB>
                       : phase == 1 ? k_sweep64_pf<SOLVER, 1, MINB> : k_sweep64_pf<SOLVER, 2, MINB>;
  count_launches(1);
  return launch_overlapped(k, blocks, 256, st, A, B, codes, list, nlist, g);
}

template <int SOLVER>
static cudaError_t sweep_fast_s(Fields<double> A, Fields<double> B, const uint8_t* codes,
                                const int* list, int nlist, const Grid& g, int phase,
                                int form, cudaStream_t st) {
  const int blocks = (nlist + 255) / 256;
  if (blocks < 1) return cudaSuccess;
  if (form == kForm64Two) {
    return sweep_pf<SOLVER, 2>(A, B, codes, list, nlist, g, phase, st);
  } else if (form == kForm64Three) {
    return sweep_pf<SOLVER, 3>(A, B, codes, list, nlist, g, phase, st);
  } else if (form == kForm64Whole) {
    const int wave = std::min(blocks, 2 * sm_count());
    auto* k = phase == 0 ? k_sweep64_whole<SOLVER, 0>
                         : phase == 1 ? k_sweep64_whole<SOLVER, 1> : k_sweep64_whole<SOLVER, 2>;
    k<<<wave, 256, 0, st>>>(A, B, codes, list, nlist, g);
  } else {
    if (phase == 0) k_sweep64_fast<SOLVER, 0><<<blocks, 256, 0, st>>>(A, B, codes, list, nlist, g);
    else if (phase == 1) k_sweep64_fast<SOLVER, 1><<<blocks, 256, 0, st>>>(A, B, codes, list, nlist, g);
    else k_sweep64_fast<SOLVER, 2><<<blocks, 256, 0, st>>>(A, B, codes, list, nlist, g);
  }
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_sweep64(Fields<double> A, Fields<double> B, const uint8_t* codes,
                           const int* list, int nlist, const Grid& g, int solver, int exact,
                           int phase, cudaStream_t st, int form) {
  if (exact) return sweep64_exact(A, B, codes, list, nlist, g, solver, phase, st);
  if (solver == 1) return sweep_fast_s<1>(A, B, codes, list, nlist, g, phase, form, st);
  if (solver == 2) return sweep_fast_s<2>(A, B, codes, list, nlist, g, phase, form, st);
  return sweep_fast_s<3>(A, B, codes, list, nlist, g, phase, form, st);
}

// ------------------------------------------------------------------ mixed precision
// x += e over the fluid list and the periodic halo copies its sweeps write:
// the only places where e is non-zero (residual and correction sweeps write a
// fluid voxel and its copies), so the state equals that of the dense form
// while solid regions are never touched.
__global__ void k_dc_correct_list(Fields<double> x, const float4* e, const int* list, int nlist,
                                  Grid g) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nlist; q += gridDim.x * blockDim.x)
    dc_correct_voxel(x, e, g, __ldg(list + q));
}

cudaError_t launch_dc_correct_list(Fields<double> x, const float4* e, const int* list, int nlist,
                                   const Grid& g, cudaStream_t st) {
  int blocks = (nlist + 255) / 256;
  if (blocks < 1) return cudaSuccess;
  k_dc_correct_list<<<blocks, 256, 0, st>>>(x, e, list, nlist, g);
  count_launches(1);
  return cudaGetLastError();
}


// r = F(x) - x in FP64 (stored FP32) and the first correction e1 = r.
template <int SOLVER>
__global__ void __launch_bounds__(256, 2) k_dc_residual(Fields<double> X, float4* R, float4* E,
                                                      const uint8_t* codes, const int* list,
                                                      int nlist, Grid g) {
  // persistent, next list entry prefetched (as the FP64 sweeps)
  __shared__ double centre[16];
  fill_centre64<SOLVER>(centre);
  __syncthreads();
  const int stride = gridDim.x * blockDim.x;
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  int lin = q < nlist ? __ldg(list + q) : 0;
  for (; q < nlist; q += stride) {
    const int qn = q + stride;
    const int next = qn < nlist ? __ldg(list + qn) : 0;
    dc_residual_voxel<SOLVER>(X, R, E, codes, g, lin, centre);
    lin = next;
  }
}

cudaError_t launch_dc_residual(Fields<double> x, float4* r, float4* e, const uint8_t* codes,
                               const int* list, int nlist, const Grid& g, int solver,
                               cudaStream_t st) {
  const int sms = sm_count();
  int blocks = (nlist + 255) / 256;
  if (blocks < 1) return cudaSuccess;
  if (blocks > 2 * sms) blocks = 2 * sms;
  if (solver == 1) k_dc_residual<1><<<blocks, 256, 0, st>>>(x, r, e, codes, list, nlist, g);
  else if (solver == 2) k_dc_residual<2><<<blocks, 256, 0, st>>>(x, r, e, codes, list, nlist, g);
  else k_dc_residual<3><<<blocks, 256, 0, st>>>(x, r, e, codes, list, nlist, g);
  count_launches(1);
  return cudaGetLastError();
}

// e2 = L(e) + r over the fluid list (FP32, interleaved fields).
template <int SOLVER>
__global__ void __launch_bounds__(256) k_dc_inner(const float4* E, float4* E2, const float4* R,
                                                  const uint8_t* codes, const int* list,
                                                  int nlist, Grid g) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nlist; q += gridDim.x * blockDim.x)
    dc_inner_voxel<SOLVER>(E, E2, R, codes, g, list[q]);
}

// The same sweep compiled for four resident blocks per SM (at most 64
// registers per thread): more warps in flight to hide the gather latency.
template <int SOLVER>
__global__ void __launch_bounds__(256, 4) k_dc_inner_occ(const float4* E, float4* E2,
                                                         const float4* R, const uint8_t* codes,
                                                         const int* list, int nlist, Grid g) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nlist; q += gridDim.x * blockDim.x)
    dc_inner_voxel<SOLVER>(E, E2, R, codes, g, list[q]);
}

// Persistent form of the fluid-list sweep: one wave of CTAs (MINB per SM)
// walks the list with a grid stride, and every thread loads its next list
// entry before it computes the current voxel, so the list read's latency
// overlaps the stencil instead of preceding it.  MINB 3 leaves each thread
// ~80 registers: all 13 float4 gathers of a voxel stay in flight at once
// (at 64 registers the compiler splits them and spills), which is worth more
// than the extra warps of MINB 4.
template <int SOLVER, int MINB>
__global__ void __launch_bounds__(256, MINB) k_dc_inner_pf(const float4* E, float4* E2,
                                                          const float4* R, const uint8_t* codes,
                                                          const int* list, int nlist, Grid g) {
  const int stride = gridDim.x * blockDim.x;
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  int lin = q < nlist ? __ldg(list + q) : 0;
  for (; q < nlist; q += stride) {
    const int qn = q + stride;
    const int next = qn < nlist ? __ldg(list + qn) : 0;
    dc_inner_voxel<SOLVER>(E, E2, R, codes, g, lin);
    lin = next;
  }
}

template <int MINB>
static cudaError_t launch_pf(const float4* e, float4* e2, const float4* r, const uint8_t* codes,
                             const int* list, int nlist, const Grid& g, int solver,
                             cudaStream_t st) {
  const int sms = sm_count();
  int blocks = (nlist + 255) / 256;
  if (blocks < 1) return cudaSuccess;
  if (blocks > MINB * sms) blocks = MINB * sms;
  if (solver == 1) k_dc_inner_pf<1, MINB><<<blocks, 256, 0, st>>>(e, e2, r, codes, list, nlist, g);
  else if (solver == 2) k_dc_inner_pf<2, MINB><<<blocks, 256, 0, st>>>(e, e2, r, codes, list, nlist, g);
  else k_dc_inner_pf<3, MINB><<<blocks, 256, 0, st>>>(e, e2, r, codes, list, nlist, g);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_dc_inner_pf(const float4* e, float4* e2, const float4* r,
                               const uint8_t* codes, const int* list, int nlist, const Grid& g,
                               int solver, int minb, cudaStream_t st) {
  if (minb <= 2) return launch_pf<2>(e, e2, r, codes, list, nlist, g, solver, st);
  if (minb == 3) return launch_pf<3>(e, e2, r, codes, list, nlist, g, solver, st);
  return launch_pf<4>(e, e2, r, codes, list, nlist, g, solver, st);
}

cudaError_t launch_dc_inner_occ(const float4* e, float4* e2, const float4* r,
                                const uint8_t* codes, const int* list, int nlist, const Grid& g,
                                int solver, cudaStream_t st) {
  int blocks = (nlist + 255) / 256;
  if (blocks < 1) return cudaSuccess;
  if (solver == 1) k_dc_inner_occ<1><<<blocks, 256, 0, st>>>(e, e2, r, codes, list, nlist, g);
  else if (solver == 2) k_dc_inner_occ<2><<<blocks, 256, 0, st>>>(e, e2, r, codes, list, nlist, g);
  else k_dc_inner_occ<3><<<blocks, 256, 0, st>>>(e, e2, r, codes, list, nlist, g);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_dc_inner(const float4* e, float4* e2, const float4* r, const uint8_t* codes,
                            const int* list, int nlist, const Grid& g, int solver,
                            cudaStream_t st) {
  int blocks = (nlist + 255) / 256;
  if (blocks < 1) return cudaSuccess;
  if (solver == 1) k_dc_inner<1><<<blocks, 256, 0, st>>>(e, e2, r, codes, list, nlist, g);
  else if (solver == 2) k_dc_inner<2><<<blocks, 256, 0, st>>>(e, e2, r, codes, list, nlist, g);
  else k_dc_inner<3><<<blocks, 256, 0, st>>>(e, e2, r, codes, list, nlist, g);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_zero4(float4* e, const Grid& g, cudaStream_t st) {
  return cudaMemsetAsync(e, 0, sizeof(float4) * (size_t)g.pl4 * g.NZ, st);
}

}  // namespace pm
