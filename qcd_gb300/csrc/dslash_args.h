// dslash_args.h -- launch arguments shared by the operator kernels.
#pragma once

#include "internal.h"

namespace qg {

// Partial sums that an operator launch adds up beside its own work, in a block
// of its own (block 0, before the others' blocks), and the scalars it forms from
// the total (cg_scalars_from; mode 2: the total goes to s[0]). The block sums
// that an earlier launch left: no launch counts its blocks, which held every
// block for a fence and an atomic and the last one for the sum.
struct CgReduce {
  const double *part = nullptr;
  int n = 0;
  double *s = nullptr;
  int mode = 0, hist = 0;
};

struct DArgs {
  void *out;
  float *out_norm;
  const void *in;
  const float *in_norm;
  const void *gauge;
  qgd::Geom geo;
  int x0;  // sites x0 .. V-1 (a range of a full-lattice launch; 0 otherwise)
  int V;
  int64_t stride;   // spinor block stride
  int64_t gstride;  // gauge block stride
  // scalars in double and as float pairs (hi + lo), so kernels of every
  // arithmetic type read them without converting on the FP64 pipe
  double phr[4], phi[4], mp4, tm;  // tm already negated for D^+
  float phr_h[4], phr_l[4], phi_h[4], phi_l[4], mp4_h, mp4_l, tm_h, tm_l;
  int twist_mask;
  int op_q;          // multiply the result by i g5
  double *partials;  // non-null: block b writes sum over its sites of |out|^2 to partials[b]
  // even/odd kernels (k_wilson_eo): the sites of parity eo_par only, V = half
  // volume; in, out and z are half fields indexed by (full site index) >> 1
  // (t extent even). out = ch * [A^{-1}] H in + {0 | z | A z}, with
  // A = mp4 + i tm g5 and H the hopping sum of the operator.
  int eo_par;
  const void *z;
  const float *z_norm;
  int zmode;  // 0: no addend, 1: + z, 2: + A z, 3: + A z + w (float-float kernel)
  const void *w;
  int ainv;   // 1: hopping term multiplied by A^{-1}
  double ch, ai_r, ai_i;  // A^{-1} = ai_r + i ai_i g5
  float ch_h, ch_l, ai_r_h, ai_r_l, ai_i_h, ai_i_l;
  // 1: in and out are in the host layout, [site][spin][colour] complex
  // double (12 double2 per site), instead of component blocks of `stride`
  // sites (full-lattice float-float kernel only)
  int aos = 0;
  CgReduce red;  // not with partials
};

// |v|^2 summed over the block into partials[blockIdx.x]; every thread of the
// block must call it (blockDim.x a multiple of 32, at most 1024)
__device__ __forceinline__ void block_partial(double v, double *partials)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __shared__ double sh[32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += sh[i];
    partials[blockIdx.x] = s;
  }
}

// scalar slots (S_A0, S_A1: alpha of the last even and odd iteration of a chunk)
enum { S_RR = 0, S_PAP = 1, S_RRNEW = 2, S_ALPHA = 3, S_BETA = 4, S_RES = 5, S_A0 = 6, S_A1 = 7, S_HIST = 8 };

// the CG scalars from a reduced total: mode 0 t = p^+ A p -> alpha;
// mode 1 t = |r|^2 -> beta and the residual history; mode 2 the total itself;
// mode 3 t = |r|^2 of a restarted residual: beta' = t / |r_prev|^2 with
// |r_prev|^2 = rr / beta, the residual before the last iteration
__device__ __forceinline__ void cg_scalars_from(double t, double *s, int mode, int hist)
{
  if (mode == 0) {
    s[S_PAP] = t;
    s[S_ALPHA] = s[S_A0 + (hist & 1)] = t > 0.0 ? s[S_RR] / t : nan("");  // p^+ A p <= 0: breakdown
  } else if (mode == 1) {
    s[S_RRNEW] = t;
    s[S_BETA] = t / s[S_RR];
    s[S_RR] = t;
    s[S_HIST + hist] = t;
  } else if (mode == 2) {
    s[0] = t;
  } else {
    s[S_BETA] = s[S_BETA] > 0.0 && s[S_RR] > 0.0 ? t * s[S_BETA] / s[S_RR] : 0.0;
    s[S_RR] = t;
  }
}

// every thread of a block: the sum of r.n partials in a fixed order (the same
// for one block size) and the scalars from it; 24 independent loads in flight
// per thread
__device__ __forceinline__ void cg_sum(const CgReduce &r)
{
  __shared__ double sh[32];
  double v = 0.0;
  const int nt = (int)blockDim.x;
  constexpr int kLoads = 24;
  for (int i0 = threadIdx.x; i0 < r.n; i0 += kLoads * nt) {
    double w[kLoads];
#pragma unroll
    for (int k = 0; k < kLoads; k++) w[k] = i0 + k * nt < r.n ? __ldcg(r.part + i0 + k * nt) : 0.0;
#pragma unroll
    for (int k = 0; k < kLoads; k++) v += w[k];
  }
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < nt >> 5; i++) t += sh[i];
    cg_scalars_from(t, r.s, r.mode, r.hist);
  }
}

// the sum and its scalars in a launch of its own (cg.cu)
bool cg_total(const CgReduce &r);

// this block's index among the blocks of the operator's own work; block 0 of
// a launch with partials to add adds them and returns -1
__device__ __forceinline__ int work_block(const CgReduce &r)
{
  if (r.n == 0) return (int)blockIdx.x;
  if (blockIdx.x == 0) cg_sum(r);
  return (int)blockIdx.x - 1;
}

// Called by every thread of a block after block_partial wrote the
// block's partial: the block that finishes last sums all gridDim.x partials
// in index order (the same order whichever block is last), updates the
// scalars and re-arms the counter. No block waits for another.
__device__ __forceinline__ void cg_last_block(const double *partials, unsigned *done, double *s, int mode, int hist)
{
  __shared__ unsigned last;
  if (threadIdx.x == 0) {
    __threadfence();  // this block's partial before its count
    last = atomicAdd(done, 1u) == gridDim.x - 1 ? 1u : 0u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  cg_sum(CgReduce{partials, (int)gridDim.x, s, mode, hist});
  if (threadIdx.x == 0) *done = 0u;
}

// a launch scalar in the kernel's arithmetic type R
template <typename R>
struct Scalar;
template <>
struct Scalar<double> {
  __device__ __forceinline__ static double get(double d, float, float) { return d; }
};
template <>
struct Scalar<float> {
  __device__ __forceinline__ static float get(double, float h, float) { return h; }
};

inline void split_host(double d, float *h, float *l)
{
  *h = (float)d;
  *l = (float)(d - (double)*h);
}

}  // namespace qg
