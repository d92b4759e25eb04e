// Flow-map advection and the fused FTLE kernel.
//
// flow map: one particle per seed of flow_map_generator's lattice
//   (flow_map_generator.cpp:23-43 + seed_generator.cpp:9-21, seeds generated in
//   the kernel from the voxel index), advected with particle_advector's rules
//   (particle_advector.cpp:74-139, one block: a particle stops with its current
//   position when it leaves the grid, meets a zero velocity, or has taken
//   iterations - 1 steps) and written to its voxel (flow_map_generator.cpp:44-52).
//   Frozen stages keep absolute positions and the reference's arithmetic;
//   re-sampled stages of the tableau and Adams schemes run in local cell
//   coordinates.
// FTLE: per voxel, the flow map's central-difference gradient J (FP32, one-sided
//   at the borders), the Cauchy-Green tensor C = J^T J (FP32) and its largest
//   eigenvalue (largest_eigenvalue: an error of a few FP32 ulps of ||C||, also
//   where eigenvalues nearly coincide and closed forms lose half their digits),
//   then log(sqrt(lambda_max)) / |T| =
//   0.5 log(lambda_max) / |T| — the intent of vector_field::gradient +
//   ftle_map_generator::generate (vector_field.cpp:49-93,
//   ftle_map_generator.cpp:22-60).  All FP32: a GB300 SM issues FP64 at 1/64
//   of its FP32 rate, and FP64 evaluation made this kernel FP64-pipe bound.
//   The fractional-anisotropy mode (ftle_map_generator.cpp:51-54) needs no
//   eigen-solve: it is evaluated from the invariants of C.
#include <algorithm>

#include "context.hpp"

namespace pars
{
namespace
{
struct flow_map_args
{
  field_view f;
  step_rule  rule;
  int        iterations;
  float      ox, oy, oz;          // seed lattice offset
  float      sx, sy, sz;          // seed lattice spacing (field spacing / scale)
  int        px, py, pz;          // seeds per dimension
  int        fx, fy, fz;          // flow-map shape
  float4*    flow;
  unsigned long long* steps;
  unsigned long long* next;       // pool counter (zero before the launch)
};

// The stepping scheme a flow-map kernel is compiled for.
enum flow_scheme { flow_frozen = 0, flow_classic, flow_midpoint, flow_cash_karp, flow_dormand_prince, flow_fehlberg,
                   flow_adams_bashforth, flow_adams_moulton, flow_schemes };

flow_scheme flow_scheme_of(const step_rule& r)
{
  if (r.frozen) return flow_frozen;
  switch (r.scheme)
  {
  case scheme_tableau:         return flow_scheme(flow_midpoint + r.tableau);
  case scheme_adams_bashforth: return flow_adams_bashforth;
  case scheme_adams_moulton:   return flow_adams_moulton;
  default:                     return flow_classic;
  }
}

template <int SCHEME>
__device__ __forceinline__ void flow_step(const flow_map_args& a, corner_cache& cache, local_position& q, const float3& v, frozen_history& hist)
{
  if constexpr (SCHEME == flow_classic)              local_step(a.f, cache, a.rule.rk4, a.rule.h, q, v);
  else if constexpr (SCHEME == flow_adams_bashforth) adams_step_local<false>(a.f, cache, a.rule.h, q, v, hist);
  else if constexpr (SCHEME == flow_adams_moulton)   adams_step_local<true>(a.f, cache, a.rule.h, q, v, hist);
  else                                               tableau_step_local<SCHEME - flow_midpoint>(a.f, cache, a.rule.h, q, v);
}

// Maps of many steps: one particle per lane, and lanes whose particles have ended take the next
// seeds of their warp's pool (refill_rule): particles leave the grid
// after very different step counts, and with one seed per thread a warp's lanes
// idled until its longest particle ended.  Warps take pools of 32 consecutive
// seeds from a device counter, as the batched engine does.  Bound by instruction issue and the
// corner loads' L1 wavefronts, as the batched engine.  One seed per thread
// against this: 5.51 -> 3.9 ms (frozen RK4, 150 x 128 x 141, 300 steps, with the
// reciprocal divisions), 657 -> 549 us (re-sampled RK4, 61 x 64 x 67, 120 steps,
// whole call).
// Frozen steps need few registers once the corners are cached: seven CTAs of 128
// per SM (72 registers) took 4.0 ms where 80 registers took 4.3 and 94 took 4.4
// (150 x 128 x 141 vertices, 300 steps).  The others: five (96 registers); the
// tableaux, which took what the compiler chose before (95 to 112), 3489 -> 3386 us
// (Dormand-Prince, 100^3, 200 steps) and 7858 -> 7375 us (Fehlberg 7(8)), 64^3
// within 3 %.
constexpr int flow_min_ctas(int scheme) { return scheme == flow_frozen ? 7 : 5; }

template <int SCHEME>
__global__ void __launch_bounds__(128, flow_min_ctas(SCHEME)) flow_map_kernel(const __grid_constant__ flow_map_args a, refill_rule refill)
{
  constexpr unsigned full = 0xffffffffu;
  const long long total = (long long)a.px * a.py * a.pz;
  const int lane = threadIdx.x & 31;
  const unsigned lanes_below = (1u << lane) - 1u;
  long long pool_next = 0, pool_end = 0;   // warp-uniform
  bool exhausted = false, alive = false, ended = false;   // ended: holds a particle not yet written
  unsigned int steps = 0;                  // this lane's steps, those not yet added to a.steps
  long long out = 0;                       // the particle's voxel, -1: none
  int it = 1;
  float4 pos = make_float4(0.f, 0.f, 0.f, 0.f);
  local_position q {0, 0, 0, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  corner_cache cache;
  frozen_history hist;
  for (;;)
  {
    unsigned need = __ballot_sync(full, !alive);
    if (__popc(need) >= (exhausted ? 32 : refill.lanes))
    {
      // write the ended particles, then give every idle lane a seed
      if (ended)
      {
        // With iterations <= 1 the reference never assigns the voxel; it keeps the
        // seed position here.
        if constexpr (SCHEME != flow_frozen) { if (it > 1) pos = flow_position(a.f, q); }
        if (out >= 0) a.flow[out] = pos;
        // (a lane takes particle after particle, and the warp's sum has 32 bits)
        if (steps >> 26) { atomicAdd(a.steps, (unsigned long long)steps); steps = 0; }
        ended = false;
      }
      while (need && !exhausted)
      {
        if (pool_next < pool_end)
        {
          const long long s = pool_next + __popc(need & lanes_below);
          if (!alive && s < pool_end)
          {
            int ix, iy, iz;
            lattice_index(s, a.py, a.pz, ix, iy, iz);
            out = ix < a.fx && iy < a.fy && iz < a.fz ? ((long long)ix * a.fy + iy) * a.fz + iz : -1;
            pos = make_float4(__fadd_rn(a.ox, __fmul_rn(a.sx, float(ix))), __fadd_rn(a.oy, __fmul_rn(a.sy, float(iy))),
                              __fadd_rn(a.oz, __fmul_rn(a.sz, float(iz))), 0.0f);
            hist = frozen_history();
            // Re-sampled schemes in local cell coordinates (cell + offset +
            // compensation); the position leaves them once, at the end.
            if constexpr (SCHEME != flow_frozen) q = to_local(a.f, pos);
            it = 1;
            alive = true;
          }
          pool_next = min(pool_end, pool_next + (long long)__popc(need));
          need = __ballot_sync(full, !alive);
          continue;
        }
        long long p = 0;
        if (lane == 0) p = (long long)atomicAdd(a.next, 32ULL);
        p = __shfl_sync(full, p, 0);
        if (p >= total) exhausted = true;
        else { pool_next = p; pool_end = min(p + 32, total); }
      }
      if (need == full) break;   // every lane idle, and the pools are exhausted
    }
    // every live lane's next steps, without a look at the others between them
    for (int k = 0; k < refill.steps && alive; ++k)
    {
      bool retire = it >= a.iterations;
      if constexpr (SCHEME == flow_frozen)
      {
        if (!retire)
        {
          float3 v;
          if (!sample_inside_cached(a.f, cache, pos, v) || is_zero(v)) retire = true;
          else { pos = frozen_step(a.rule, pos, v, hist); ++steps; ++it; }
        }
      }
      else
      {
        if (!retire) retire = !local_inside(a.f, q);
        if (!retire)
        {
          const float3 v = sample_local(a.f, cache, q.ix, q.iy, q.iz, q.ux, q.uy, q.uz);
          if (is_zero_local(a.f, v)) retire = true;
          else { flow_step<SCHEME>(a, cache, q, v, hist); ++steps; ++it; }
        }
      }
      if (retire) { alive = false; ended = true; }
    }
  }
  const unsigned int warp_steps = __reduce_add_sync(full, steps);
  if (lane == 0 && warp_steps) atomicAdd(a.steps, (unsigned long long)warp_steps);
}

// One seed per thread, for maps of few steps: refilled lanes are out of step, and a
// lane that ends between two looks idles until the next, which few steps do not make
// up for.  200^3 Euler frozen, 11 / 29 / 49 / 81 steps, seeds from the counter against
// this: 1028 / 2328 / 3881 / 5845 against 870 / 2082 / 3440 / 5599 us; 128^3, 129 steps:
// 2182 against 2331.
template <int SCHEME>
__global__ void __launch_bounds__(128, flow_min_ctas(SCHEME)) flow_map_once_kernel(const __grid_constant__ flow_map_args a)
{
  const long long total = (long long)a.px * a.py * a.pz, s = (long long)blockIdx.x * 128 + threadIdx.x;
  unsigned int steps = 0;
  if (s < total)
  {
    int ix, iy, iz;
    lattice_index(s, a.py, a.pz, ix, iy, iz);
    float4 pos = make_float4(__fadd_rn(a.ox, __fmul_rn(a.sx, float(ix))), __fadd_rn(a.oy, __fmul_rn(a.sy, float(iy))),
                             __fadd_rn(a.oz, __fmul_rn(a.sz, float(iz))), 0.0f);
    corner_cache cache;
    frozen_history hist = frozen_history();
    if constexpr (SCHEME == flow_frozen)
    {
      for (int it = 1; it < a.iterations; ++it, ++steps)
      {
        float3 v;
        if (!sample_inside_cached(a.f, cache, pos, v) || is_zero(v)) break;
        pos = frozen_step(a.rule, pos, v, hist);
      }
    }
    else
    {
      local_position q = to_local(a.f, pos);
      for (int it = 1; it < a.iterations; ++it, ++steps)
      {
        if (!local_inside(a.f, q)) break;
        const float3 v = sample_local(a.f, cache, q.ix, q.iy, q.iz, q.ux, q.uy, q.uz);
        if (is_zero_local(a.f, v)) break;
        flow_step<SCHEME>(a, cache, q, v, hist);
      }
      if (steps) pos = flow_position(a.f, q);   // (iterations <= 1: the seed position, as in flow_map_kernel)
    }
    if (ix < a.fx && iy < a.fy && iz < a.fz) a.flow[((long long)ix * a.fy + iy) * a.fz + iz] = pos;
  }
  const unsigned int warp_steps = __reduce_add_sync(0xffffffffu, steps);
  if ((threadIdx.x & 31) == 0 && warp_steps) atomicAdd(a.steps, (unsigned long long)warp_steps);
}

const void* flow_map_once_kernels[flow_schemes] = {
  (const void*)flow_map_once_kernel<flow_frozen>, (const void*)flow_map_once_kernel<flow_classic>,
  (const void*)flow_map_once_kernel<flow_midpoint>, (const void*)flow_map_once_kernel<flow_cash_karp>,
  (const void*)flow_map_once_kernel<flow_dormand_prince>, (const void*)flow_map_once_kernel<flow_fehlberg>,
  (const void*)flow_map_once_kernel<flow_adams_bashforth>, (const void*)flow_map_once_kernel<flow_adams_moulton>};

const void* flow_map_kernels[flow_schemes] = {
  (const void*)flow_map_kernel<flow_frozen>, (const void*)flow_map_kernel<flow_classic>, (const void*)flow_map_kernel<flow_midpoint>,
  (const void*)flow_map_kernel<flow_cash_karp>, (const void*)flow_map_kernel<flow_dormand_prince>,
  (const void*)flow_map_kernel<flow_fehlberg>, (const void*)flow_map_kernel<flow_adams_bashforth>,
  (const void*)flow_map_kernel<flow_adams_moulton>};

// Resident CTAs of the kernel on the device, all SMs together.  (Loads both kernels:
// a later launch may be inside a stream capture.)
cudaError_t flow_map_resident(flow_scheme scheme, int device, int* ctas)
{
  int per_sm = 0, sms = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, flow_map_once_kernels[scheme], 128, 0);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, flow_map_kernels[scheme], 128, 0);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  *ctas = std::max(1, per_sm) * std::max(1, sms);
  return e;
}

// The lattice's seeds (at least one) on at most `resident` CTAs that take them from the
// counter, or each on its own thread.  With refilled lanes (six seeds a lane and more)
// the two break even at about 100 steps: 128^3 Euler, midpoint and Adams-Bashforth
// frozen are 1 to 3 % slower from the counter at 81 steps and 5 to 6 % faster at 129.
// Below, warps run their seeds to the end either way, and the counter's trips show in
// short launches only: 64^3, 4 steps 42 against 32 us, 11 to 39 steps within 3 %.
constexpr int flow_once_refilled = 96, flow_once_whole = 16;
cudaError_t launch_flow_map_kernel(const flow_map_args& a, flow_scheme scheme, int resident, cudaStream_t stream)
{
  const long long total = (long long)a.px * a.py * a.pz;
  refill_rule refill = refill_for(total, resident * 128LL);
  const long long ctas = (total + 127) / 128;
  if (a.iterations <= (refill.lanes < 32 ? flow_once_refilled : flow_once_whole) && ctas < (1LL << 31))
  {
    void* args[] = {(void*)&a};
    return cudaLaunchKernel(flow_map_once_kernels[scheme], (unsigned)ctas, 128, args, 0, stream);
  }
  const unsigned grid = (unsigned)std::min<long long>(resident, ctas);
  void* args[] = {(void*)&a, (void*)&refill};
  return cudaLaunchKernel(flow_map_kernels[scheme], grid, 128, args, 0, stream);
}

// The largest eigenvalue of the symmetric 3x3 matrix with diagonal c00, c11, c22
// (non-negative trace), in FP32 without iterating over rotations: Eberly's
// construction ("A Robust Eigensolver for 3x3 Symmetric Matrices", Geometric
// Tools, 2014).  With q = tr / 3, p^2 = |C - q I|^2 / 6 and B = (C - q I) / p the
// eigenvalues of B are the roots of beta^3 - 3 beta = det B.  The root of the
// sign of det B is the well separated one (|beta| in [sqrt 3, 2], where the
// root's derivative by det B is at most 1/6), so:
//  * det B >= 0: that root is the largest eigenvalue.
//  * det B < 0: it is the smallest; the largest then comes from B on the plane
//    orthogonal to its eigenvector (the largest cross product of two rows of
//    B - beta I).  Its 2x2 eigenvalue is mean + sqrt(difference^2 + m01^2), a
//    sum of squares, so nearly equal eigenvalues lose no digits there, as they
//    would in the closed forms; the eigenvector's error enters squared.
// The root is found by two Newton steps from a quadratic fit (error below
// 4e-3, squared at each step).  Relative errors against FP64 on 200,000 matrices
// each (random, near-degenerate, near-isotropic, strongly anisotropic): rms 3.2e-8
// to 4.6e-8, largest 1.6e-7; the cyclic Jacobi sweeps that this replaces (12
// rotations with two divisions and a square root each): 3.4e-8 to 6.2e-8, largest
// 2.7e-7.  The FTLE of 320 x 300 x 311 vertices: 1.47 -> 0.46 ms, with the decoding
// and the quotients below (its 597 MB take 0.09 ms).
__device__ __forceinline__ float largest_eigenvalue(float c00, float c11, float c22, float c01, float c02, float c12)
{
  const float trace = c00 + c11 + c22;
  if (!(trace < INFINITY)) return trace;
  // a power of two brings the trace into [1, 2): exact, and no square or cube leaves the range
  const unsigned e = min(__float_as_uint(trace) & 0x7f800000u, 253u << 23);
  const float scale = __uint_as_float((254u << 23) - e), unscale = __uint_as_float(e ? e : 1u << 22);
  c00 *= scale; c11 *= scale; c22 *= scale; c01 *= scale; c02 *= scale; c12 *= scale;
  if (c02 == 0.0f && c12 == 0.0f)
  {
    // decoupled z (planar flows): one Jacobi rotation of the x-y block
    const float d = 0.5f * (c00 - c11), s = fabsf(d) + __fsqrt_rn(fmaf(d, d, c01 * c01));
    return fmaxf(c22, fmaf(c01, c01 == 0.0f ? 0.0f : __fdiv_rn(c01, s), fmaxf(c00, c11))) * unscale;
  }
  const float q = (c00 + c11 + c22) * (1.0f / 3.0f);
  const float d0 = c00 - q, d1 = c11 - q, d2 = c22 - q;
  const float off = fmaf(c01, c01, fmaf(c02, c02, c12 * c12));
  const float p2 = fmaf(2.0f, off, fmaf(d0, d0, fmaf(d1, d1, d2 * d2))) * (1.0f / 6.0f);
  // p and 1 / p from one reciprocal root, each with a Newton step
  const float y = p2 > 1e-36f ? rsqrtf(p2) : 0.0f, p0 = p2 * y;
  const float p = fmaf(0.5f * y, fmaf(-p0, p0, p2), p0);
  const float inv = fmaf(y, fmaf(-p, y, 1.0f), y);
  const float b00 = d0 * inv, b11 = d1 * inv, b22 = d2 * inv, b01 = c01 * inv, b02 = c02 * inv, b12 = c12 * inv;
  const float m0 = fmaf(b11, b22, -b12 * b12), m1 = fmaf(b01, b22, -b12 * b02), m2 = fmaf(b01, b12, -b11 * b02);
  const float det = fmaf(b00, m0, fmaf(-b01, m1, b02 * m2));
  const float r = fminf(fabsf(det), 2.0f);                    // beta^3 - 3 beta = r
  float beta = fmaf(r, fmaf(r, -0.0163373f, 0.1666667f), 1.7320508f);
  #pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    const float s = fmaf(beta, beta, -3.0f);
    beta -= __fdividef(fmaf(beta, s, -r), fmaf(3.0f, s, 6.0f));
  }
  float largest = beta;
  if (det < 0.0f)
  {
    // rows of B - beta I with beta the smallest eigenvalue, -|beta|
    const float a00 = b00 + beta, a11 = b11 + beta, a22 = b22 + beta;
    const float x0 = fmaf(b01, b12, -b02 * a11), x1 = fmaf(b02, b01, -a00 * b12), x2 = fmaf(a00, a11, -b01 * b01);   // row 0 x row 1
    const float y0 = fmaf(b01, a22, -b02 * b12), y1 = fmaf(b02, b02, -a00 * a22), y2 = fmaf(a00, b12, -b01 * b02);   // row 0 x row 2
    const float z0 = fmaf(a11, a22, -b12 * b12), z1 = fmaf(b12, b02, -b01 * a22), z2 = fmaf(b01, b12, -a11 * b02);   // row 1 x row 2
    const float nx = fmaf(x0, x0, fmaf(x1, x1, x2 * x2)), ny = fmaf(y0, y0, fmaf(y1, y1, y2 * y2)), nz = fmaf(z0, z0, fmaf(z1, z1, z2 * z2));
    float v0 = x0, v1 = x1, v2 = x2, n = nx;
    if (ny > n) { v0 = y0; v1 = y1; v2 = y2; n = ny; }
    if (nz > n) { v0 = z0; v1 = z1; v2 = z2; n = nz; }
    const float inv_n = rsqrtf(n);                            // the largest of the three is of order one
    v0 *= inv_n; v1 *= inv_n; v2 *= inv_n;
    // orthonormal u, w to v (Duff et al., "Building an Orthonormal Basis, Revisited", 2017)
    const float sign = copysignf(1.0f, v2), g = -__frcp_rn(sign + v2), h = v0 * v1 * g;
    const float u0 = fmaf(sign * v0, v0 * g, 1.0f), u1 = sign * h, u2 = -sign * v0;
    const float w0 = h, w1 = fmaf(v1, v1 * g, sign), w2 = -v1;
    const float t0 = fmaf(b00, u0, fmaf(b01, u1, b02 * u2)), t1 = fmaf(b01, u0, fmaf(b11, u1, b12 * u2)),
                t2 = fmaf(b02, u0, fmaf(b12, u1, b22 * u2));
    const float s0 = fmaf(b00, w0, fmaf(b01, w1, b02 * w2)), s1 = fmaf(b01, w0, fmaf(b11, w1, b12 * w2)),
                s2 = fmaf(b02, w0, fmaf(b12, w1, b22 * w2));
    const float m00 = fmaf(u0, t0, fmaf(u1, t1, u2 * t2)), m01 = fmaf(w0, t0, fmaf(w1, t1, w2 * t2)),
                m11 = fmaf(w0, s0, fmaf(w1, s1, w2 * s2));
    // the plane's trace is that of B (0) less the smallest eigenvalue
    const float difference = 0.5f * (m00 - m11);
    largest = fmaf(0.5f, beta, __fsqrt_rn(fmaf(difference, difference, m01 * m01)));
  }
  // the trace that the rounding of q left in C - q I belongs to every eigenvalue
  return (q + fmaf(p, largest, (d0 + d1 + d2) * (1.0f / 3.0f))) * unscale;
}

struct ftle_args
{
  const float4* flow;
  unsigned int  codes;            // ~0: the w lanes hold residual codes, 0: they do not
  int           nx, ny, nz;
  float         width[3], inverse_width[3];   // 2 h per axis and its reciprocal
  float         inverse_time;     // 1 / |T|
  int           mode;
  int           planes;           // 1: a row of CTAs per x plane; 0: one row over all vertices
  float*        out;
};

// x / d; y = RN(1 / d), 0 for a width whose reciprocal leaves the normal range.
__device__ __forceinline__ float quotient(float x, float d, float y) { return y == 0.0f ? __fdiv_rn(x, d) : quotient_rn(x, d, y); }

// A flow-map position: its stored coordinates and its residuals (code 2^e; the
// factor 2^-23 / 1022 is left out, so they are exact).
struct flow_vertex
{
  float3 x, r;
};
__device__ __forceinline__ float binade(float x) { return __uint_as_float(__float_as_uint(x) & 0x7f800000u); }
__device__ __forceinline__ flow_vertex load_vertex(const ftle_args& a, const float4* p)
{
  const float4 v = __ldg(p);
  const unsigned w = __float_as_uint(v.w) & a.codes;
  // each 10-bit code plus 512 as mantissa bits of a power of two: bits 0-9 of
  // 2^23, bits 10-19 of 2^13, bits 20-29 (shifted down) of 2^23
  return {make_float3(v.x, v.y, v.z), make_float3((__uint_as_float((w & 0x3ffu) ^ 0x4b000200u) - 8389120.0f) * binade(v.x),
                                                  (__uint_as_float((w & 0xffc00u) ^ 0x46080000u) - 8704.0f) * binade(v.y),
                                                  (__uint_as_float(((w >> 20) & 0x3ffu) ^ 0x4b000200u) - 8389120.0f) * binade(v.z))};
}

// b - a: the FP32 difference of neighbouring coordinates is exact where they lie
// within a factor of two of each other (Sterbenz); the residuals' difference, exact
// for neighbours of the same binade, is added to it.
__device__ __forceinline__ float difference(float b, float rb, float a, float ra)
{
  return fmaf(__fsub_rn(rb, ra), 0x1p-23f / 1022.0f, __fsub_rn(b, a));
}

// Column j of J: (phi(+e_j) - phi(-e_j)) / (2 h_j); a one-sided difference divides
// by h_j (half the width, exactly).
__device__ __forceinline__ float3 jacobian_column(const ftle_args& a, int j, const flow_vertex& hi, const flow_vertex& lo, bool one_sided)
{
  const float width = one_sided ? 0.5f * a.width[j] : a.width[j], inverse = one_sided ? 2.0f * a.inverse_width[j] : a.inverse_width[j];
  return make_float3(quotient(difference(hi.x.x, hi.r.x, lo.x.x, lo.r.x), width, inverse),
                     quotient(difference(hi.x.y, hi.r.y, lo.x.y, lo.r.y), width, inverse),
                     quotient(difference(hi.x.z, hi.r.z, lo.x.z, lo.r.z), width, inverse));
}

// One vertex per thread.  Bound by instruction issue (88 % of the cycles), so the
// place in the lattice costs one 32-bit division (CTAs by x plane), the codes are
// decoded by masks, and a column's borders by selects: 320 x 300 x 311 vertices 491
// -> 460 us with the reciprocal root above, 256^3 278 -> 261, 150 x 128 x 141 51 ->
// 49.  (16 planes per thread, the vertices at x - 1 and x kept decoded: 446, 253, 49,
// but 64^3 12 instead of 11: not worth a second kernel.)
template <int MODE>
__global__ void __launch_bounds__(256) ftle_kernel(const __grid_constant__ ftle_args a)
{
  const long long plane = (long long)a.ny * a.nz, p = (long long)blockIdx.x * 256 + threadIdx.x;
  int x, y, z;
  if (a.planes)
  {
    if (p >= plane) return;
    x = int(blockIdx.y);
    y = int(unsigned(p) / unsigned(a.nz));
    z = int(p) - y * a.nz;
  }
  else
  {
    if (p >= plane * a.nx) return;
    lattice_index(p, a.ny, a.nz, x, y, z);
  }
  const long long i = ((long long)x * a.ny + y) * a.nz + z;
  const float4* v = a.flow + i;
  const float4 *x_lo = x == 0 ? v : v - plane, *x_hi = x == a.nx - 1 ? v : v + plane;
  const int y_lo = y == 0 ? 0 : a.nz, y_hi = y == a.ny - 1 ? 0 : a.nz, z_lo = z == 0 ? 0 : 1, z_hi = z == a.nz - 1 ? 0 : 1;
  const float3 none = make_float3(0.f, 0.f, 0.f);   // the column of an axis of one vertex
  const float3 J0 = a.nx > 1 ? jacobian_column(a, 0, load_vertex(a, x_hi), load_vertex(a, x_lo), x_lo == v || x_hi == v) : none;
  const float3 J1 = a.ny > 1 ? jacobian_column(a, 1, load_vertex(a, v + y_hi), load_vertex(a, v - y_lo), y_lo == 0 || y_hi == 0) : none;
  const float3 J2 = a.nz > 1 ? jacobian_column(a, 2, load_vertex(a, v + z_hi), load_vertex(a, v - z_lo), z_lo == 0 || z_hi == 0) : none;
  const float J[3][3] = {{J0.x, J1.x, J2.x}, {J0.y, J1.y, J2.y}, {J0.z, J1.z, J2.z}};
  // Cauchy-Green tensor C = J^T J (FP32) and its eigenvalues.
  float C[3][3];
  #pragma unroll
  for (int r = 0; r < 3; ++r)
    #pragma unroll
    for (int c = r; c < 3; ++c)
      C[r][c] = fmaf(J[2][r], J[2][c], fmaf(J[1][r], J[1][c], J[0][r] * J[0][c]));
  float value;
  if constexpr (MODE == PARS_FTLE_REGULAR)
  {
    // log(sqrt(lambda_max)) / |T|
    const float lambda = largest_eigenvalue(C[0][0], C[1][1], C[2][2], C[0][1], C[0][2], C[1][2]);
    value = 0.5f * logf(lambda) * a.inverse_time;
  }
  else
  {
    // Fractional anisotropy of the eigenvalues (ftle_map_generator.cpp:51-54),
    // sqrt(1/2) sqrt(sum_{i<j} (l_i - l_j)^2) / sqrt(sum_i l_i^2), from the
    // invariants: sum_{i<j} (l_i - l_j)^2 = 3 |C - (tr C / 3) I|_F^2 and
    // sum_i l_i^2 = |C|_F^2, so FA = sqrt(3/2) |dev C|_F / |C|_F — no
    // eigen-solve, and the deviator's diagonal is formed before squaring, so
    // nearly isotropic tensors keep their small anisotropy.
    const float m = (C[0][0] + C[1][1] + C[2][2]) * (1.0f / 3.0f);
    const float d0 = C[0][0] - m, d1 = C[1][1] - m, d2 = C[2][2] - m;
    const float off = fmaf(C[0][1], C[0][1], fmaf(C[0][2], C[0][2], C[1][2] * C[1][2]));
    const float dev = fmaf(2.0f, off, fmaf(d0, d0, fmaf(d1, d1, d2 * d2)));
    const float all = fmaf(2.0f, off, fmaf(C[0][0], C[0][0], fmaf(C[1][1], C[1][1], C[2][2] * C[2][2])));
    value = 1.22474487f * __fsqrt_rn(__fdiv_rn(dev, all));
  }
  a.out[i] = value;
}

void set_widths(ftle_args& a, float hx, float hy, float hz)
{
  const float h[3] = {hx, hy, hz};
  for (int j = 0; j < 3; ++j) { a.width[j] = 2.0f * h[j]; a.inverse_width[j] = h[j] > 1e-30f && h[j] < 1e30f ? 1.0f / a.width[j] : 0.0f; }
}

void launch_ftle_kernel(ftle_args& a, cudaStream_t stream)
{
  // by plane where its last CTA is a small part of it
  const long long plane = (long long)a.ny * a.nz;
  a.planes = plane >= 4096 && plane < (1LL << 31) && a.nx <= 65535 ? 1 : 0;
  const dim3 grid((unsigned)(((a.planes ? plane : plane * a.nx) + 255) / 256), a.planes ? (unsigned)a.nx : 1u);
  if (a.mode == PARS_FTLE_REGULAR) ftle_kernel<PARS_FTLE_REGULAR><<<grid, 256, 0, stream>>>(a);
  else                             ftle_kernel<PARS_FTLE_FRACTIONAL_ANISOTROPY><<<grid, 256, 0, stream>>>(a);
}
}

const unsigned long long* launch_flow_map(pars_gpu_context& ctx, const field_view& f, const step_rule& rule, int iterations,
                                          const float offset[3], const float fm_spacing[3], const int seeds_per_dimension[3],
                                          const int fm_shape[3], float4* flow)
{
  ctx.counters.reserve(sizeof(unsigned long long) * 2);   // steps taken, seeds handed out
  auto* counters = ctx.counters.as<unsigned long long>();
  PARS_CUDA(cudaMemsetAsync(counters, 0, sizeof(unsigned long long) * 2, ctx.stream));
  flow_map_args a;
  a.f = f; a.rule = rule; a.iterations = iterations;
  a.ox = offset[0]; a.oy = offset[1]; a.oz = offset[2];
  a.sx = fm_spacing[0]; a.sy = fm_spacing[1]; a.sz = fm_spacing[2];
  a.px = seeds_per_dimension[0]; a.py = seeds_per_dimension[1]; a.pz = seeds_per_dimension[2];
  a.fx = fm_shape[0]; a.fy = fm_shape[1]; a.fz = fm_shape[2];
  a.flow = flow; a.steps = counters; a.next = counters + 1;
  const long long total = (long long)a.px * a.py * a.pz;
  if (total <= 0) return counters;
  const flow_scheme scheme = flow_scheme_of(rule);
  int& resident = ctx.flow_map_ctas[scheme];
  if (resident < 0) PARS_CUDA(flow_map_resident(scheme, ctx.device, &resident));
  launch_scope scope(ctx, "advect_flow_map");
  PARS_CUDA(launch_flow_map_kernel(a, scheme, resident, ctx.stream));
  return counters;
}

void launch_ftle(pars_gpu_context& ctx, const field_view& flow, double time, int mode, float* out)
{
  ftle_args a;
  a.flow = flow.data; a.codes = flow.z_pairs ? 0u : ~0u; a.nx = flow.nx; a.ny = flow.ny; a.nz = flow.nz;
  set_widths(a, flow.hx, flow.hy, flow.hz);
  a.inverse_time = float(1.0 / fabs(time));
  a.mode = mode;
  a.out = out;
  const long long total = (long long)a.nx * a.ny * a.nz;
  if (total <= 0) return;
  launch_scope scope(ctx, "ftle_fused");
  launch_ftle_kernel(a, ctx.stream);
}

// ---- Allocation-free FTLE ------------------------------------------------------
// pars_gpu_ftle_no_alloc (declared in pars_gpu.h) runs the pack kernel, the
// per-seed flow-map kernel (flow_map_kernel, frozen or re-sampled stages) and
// the FTLE kernel, and keeps its scratch — the float4 copy of the field, the
// flow map, and the step counter — in the one file-scope device array below
// instead of allocating it.  The context path runs re-sampled RK4 / Euler
// flow maps through the batched engine instead, so for those the two paths
// agree to rounding (the engine's per-step arithmetic differs), not bit for
// bit; frozen stages and the other schemes use the same kernel in both.
// Every GPU that loads this library holds the array (no_alloc_max_voxels * 32
// bytes + 256, 8 MiB) until the process exits.
namespace
{
constexpr long long no_alloc_max_voxels = 1LL << 18;   // 64^3
constexpr long long no_alloc_entries = 2 * no_alloc_max_voxels + 16;   // field | flow map | counter
static __device__ __align__(256) float4 no_alloc_scratch[no_alloc_entries];

__global__ void pack_into_scratch_kernel(const float* __restrict__ xyz, float4* __restrict__ out, long long count, long long plane)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count)   // field_view::z_pairs
    out[i] = make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], i + plane < count ? xyz[3 * (i + plane) + 2] : 0.0f);
}

__global__ void steps_to_int64_kernel(const unsigned long long* __restrict__ counter, int64_t* __restrict__ out)
{
  *out = (int64_t)*counter;
}

// Host code must not use the array's name as a device address: it is a host
// stand-in.  The device address, and how many CTAs of the flow-map kernel fit
// on the device, are looked up once per device, with that device current, and
// cached; later calls on the device reuse them.
constexpr int no_alloc_max_devices = 64;
std::mutex no_alloc_mutex;
float4* no_alloc_address[no_alloc_max_devices] = {};
int no_alloc_resident[no_alloc_max_devices][flow_schemes] = {};

int32_t no_alloc_device(int device, flow_scheme scheme, float4** out, int* resident)
{
  if (device < 0 || device >= no_alloc_max_devices) return PARS_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(no_alloc_mutex);
  if (!no_alloc_address[device])
  {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, no_alloc_scratch) != cudaSuccess) { (void)cudaGetLastError(); return PARS_ERR_CUDA; }
    // every scheme's at once: a later call may be the first of its scheme inside a stream capture
    for (int k = 0; k < flow_schemes; ++k)
      if (flow_map_resident(flow_scheme(k), device, &no_alloc_resident[device][k]) != cudaSuccess)
      {
        (void)cudaGetLastError();
        return PARS_ERR_CUDA;
      }
    no_alloc_address[device] = static_cast<float4*>(p);
  }
  *out = no_alloc_address[device];
  *resident = no_alloc_resident[device][scheme];
  return PARS_OK;
}
}

// Checks the geometry of an allocation-free call before anything is
// multiplied or launched: every shape entry within the static scratch on its
// own (so the voxel product cannot overflow), the product within it, and the
// seed lattice int(size / spacing) per axis between shape and shape + 1 (the
// lattice flow_map_generator builds over a block: one seed per vertex), so
// the seed count and the launch's grid stay small.  Host-only; no CUDA call.
static int32_t no_alloc_geometry(const int32_t shape[3], const float size[3], const float spacing[3], long long* voxels,
                          int seeds[3])
{
  for (int i = 0; i < 3; ++i)
  {
    if (shape[i] < 2 || !(spacing[i] > 0.0f)) return PARS_ERR_INVALID_ARGUMENT;
    if (shape[i] > no_alloc_max_voxels) return PARS_ERR_BUDGET;
  }
  const long long v = (long long)shape[0] * shape[1] * shape[2];   // each factor <= 2^18: no overflow
  if (v > no_alloc_max_voxels) return PARS_ERR_BUDGET;
  for (int i = 0; i < 3; ++i)
  {
    const float q = size[i] / spacing[i];
    seeds[i] = (q > 0.0f && q < 2147483647.0f) ? int(q) : 0;
    if (seeds[i] < shape[i] || seeds[i] > shape[i] + 1) return PARS_ERR_INVALID_ARGUMENT;
  }
  *voxels = v;
  return PARS_OK;
}
}

#pragma GCC visibility push(default)
extern "C" int32_t pars_gpu_ftle_no_alloc(const float* device_xyz, const int32_t shape[3], const float offset[3], const float size[3],
                                          const float spacing[3], int32_t iterations, int32_t integrator, int32_t stage_mode,
                                          float step_size, float time, int32_t mode, float* device_ftle, int64_t* device_steps,
                                          void* stream)
{
  using namespace pars;
  if (!device_xyz || !shape || !offset || !size || !spacing || !device_ftle) return PARS_ERR_INVALID_ARGUMENT;
  if (mode != PARS_FTLE_REGULAR && mode != PARS_FTLE_FRACTIONAL_ANISOTROPY) return PARS_ERR_INVALID_ARGUMENT;
  if (time == 0.0f) return PARS_ERR_INVALID_ARGUMENT;
  // Flow map at the field's own resolution (resolution scale 1): one seed per
  // vertex (seed_generator.cpp:11), so every flow-map voxel is written and the
  // flow-map part of the scratch needs no clearing.
  long long voxels = 0;
  int seeds[3];
  const int32_t geometry = no_alloc_geometry(shape, size, spacing, &voxels, seeds);
  if (geometry != PARS_OK) return geometry;   // PARS_ERR_BUDGET: larger than the static scratch
  step_rule rule;
  try { rule = make_step_rule(integrator, stage_mode, step_size); }
  catch (const error& e) { return e.status; }

  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) { (void)cudaGetLastError(); return PARS_ERR_CUDA; }
  float4* scratch = nullptr;
  const flow_scheme scheme = flow_scheme_of(rule);
  int resident = 0;
  const int32_t status = no_alloc_device(device, scheme, &scratch, &resident);
  if (status != PARS_OK) return status;
  float4* field_data = scratch;
  float4* flow = scratch + no_alloc_max_voxels;
  auto* counter = reinterpret_cast<unsigned long long*>(scratch + 2 * no_alloc_max_voxels);
  cudaStream_t s = static_cast<cudaStream_t>(stream);

  field_view f;
  f.data = field_data;
  f.nx = shape[0]; f.ny = shape[1]; f.nz = shape[2];
  f.ox = offset[0]; f.oy = offset[1]; f.oz = offset[2];
  f.hx = spacing[0]; f.hy = spacing[1]; f.hz = spacing[2];
  f.maxx = offset[0] + size[0]; f.maxy = offset[1] + size[1]; f.maxz = offset[2] + size[2];
  set_derived(f);
  f.z_pairs = 1;

  // The counters (steps, seeds handed out) keep the previous call's values: clear them first.
  if (cudaMemsetAsync(counter, 0, 2 * sizeof(unsigned long long), s) != cudaSuccess) { (void)cudaGetLastError(); return PARS_ERR_CUDA; }
  pack_into_scratch_kernel<<<(unsigned)((voxels + 255) / 256), 256, 0, s>>>(device_xyz, field_data, voxels, (long long)shape[1] * shape[2]);
  if (cudaGetLastError() != cudaSuccess) return PARS_ERR_CUDA;

  flow_map_args a;
  a.f = f; a.rule = rule; a.iterations = iterations;
  a.ox = offset[0]; a.oy = offset[1]; a.oz = offset[2];
  a.sx = spacing[0]; a.sy = spacing[1]; a.sz = spacing[2];
  a.px = seeds[0]; a.py = seeds[1]; a.pz = seeds[2];
  a.fx = shape[0]; a.fy = shape[1]; a.fz = shape[2];
  a.flow = flow; a.steps = counter; a.next = counter + 1;
  if (launch_flow_map_kernel(a, scheme, resident, s) != cudaSuccess) { (void)cudaGetLastError(); return PARS_ERR_CUDA; }

  ftle_args t;
  t.flow = flow; t.codes = ~0u; t.nx = shape[0]; t.ny = shape[1]; t.nz = shape[2];
  set_widths(t, spacing[0], spacing[1], spacing[2]);
  t.inverse_time = float(1.0 / fabs(double(time)));
  t.mode = mode;
  t.out = device_ftle;
  launch_ftle_kernel(t, s);
  if (cudaGetLastError() != cudaSuccess) return PARS_ERR_CUDA;
  if (device_steps) steps_to_int64_kernel<<<1, 1, 0, s>>>(counter, device_steps);
  if (cudaGetLastError() != cudaSuccess) return PARS_ERR_CUDA;
  return PARS_OK;
}
#pragma GCC visibility pop
