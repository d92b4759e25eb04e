// Index and colour generation on device-resident curve batches.
//
// index_generator::generate (pa/source/stages/index_generator.cpp:10-24):
//   indices = [ i for i in 0..n-2 if v[i] != termination and v[i+1] != termination ]
//   in increasing order — a stream compaction, done here by a pass over the
//   vertices (one flag bit each, tile counts), a scan of the tile counts and a
//   pass over the flags that writes the indices.
// color_generator::generate (pa/source/stages/color_generator.cpp:16-98): one
//   thread per index; the FP32 operations follow the reference one by one with
//   explicit round-to-nearest intrinsics (no FMA contraction).  The tangent's
//   squared norm is reduced in the order of Eigen's SSE packet reduction,
//   (d0^2 + d2^2) + (d1^2 + d3^2).  atan2 and acos are FP32 functions on both
//   sides (the host libm's there, CUDA's here), so hue / saturation colours
//   agree to a few FP32 ulps rather than bit for bit.
#include "context.hpp"

namespace pars
{
namespace
{
constexpr unsigned full_mask = 0xffffffffu;
constexpr int index_threads = 256;
constexpr int warp_words    = 8;                            // words of 32 flags per warp
constexpr int warp_vertices = 32 * warp_words;
constexpr int tile_words    = index_threads / 32 * warp_words;
constexpr int index_tile    = 32 * tile_words;              // vertices per CTA

// ---- colours ----------------------------------------------------------------
__device__ __forceinline__ float clamp01(float x) { return x < 0.0f ? 0.0f : (1.0f < x ? 1.0f : x); }

__device__ __forceinline__ float4 hue_to_rgba(float hue)
{
  const float six_h = __fmul_rn(6.0f, hue);
  return make_float4(clamp01(__fsub_rn(fabsf(__fsub_rn(six_h, 3.0f)), 1.0f)),
                     clamp01(__fsub_rn(2.0f, fabsf(__fsub_rn(six_h, 2.0f)))),
                     clamp01(__fsub_rn(2.0f, fabsf(__fsub_rn(six_h, 4.0f)))),
                     1.0f);
}

// Error-free sum (Knuth's TwoSum): s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
  s = __fadd_rn(a, b);
  const float bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

// float(sqrt(double(x)^2 + double(y)^2 + double(z)^2)) — the reference's
// radius (coordinates.hpp:8-16: std::pow(float, int) promotes to double) — in
// FP32 arithmetic: each square as an exact pair (product + FMA remainder), the
// six terms summed error-free into hi + lo, then the correctly rounded square
// root of hi + lo, decided against the rounding midpoints of sqrtf(hi) with the
// exact remainder hi - r0^2.  It can differ from the double evaluation only
// where the root lies within about 2^-46 of a float midpoint (no case in
// 300,000 random and axis-aligned tangents).
__device__ __forceinline__ float reference_radius(float x, float y, float z)
{
  const float px = __fmul_rn(x, x), py = __fmul_rn(y, y), pz = __fmul_rn(z, z);
  const float ex = __fmaf_rn(x, x, -px), ey = __fmaf_rn(y, y, -py), ez = __fmaf_rn(z, z, -pz);
  float s1, t1, s2, t2;
  two_sum(px, py, s1, t1);
  two_sum(s1, pz, s2, t2);
  float lo = __fadd_rn(__fadd_rn(__fadd_rn(t1, t2), __fadd_rn(ex, ey)), ez);
  const float hi = __fadd_rn(s2, lo);
  lo = __fsub_rn(lo, __fsub_rn(hi, s2));
  const float r0 = __fsqrt_rn(hi);
  const float rho = __fadd_rn(__fmaf_rn(-r0, r0, hi), lo);          // (hi + lo) - r0^2
  const float up = __int_as_float(__float_as_int(r0) + 1), dn = __int_as_float(__float_as_int(r0) - 1);
  const float u = __fsub_rn(up, r0), ud = __fsub_rn(r0, dn);       // ulps above and below r0
  // (r0 + u/2)^2 - r0^2 = r0 u + u^2/4, (r0 - ud/2)^2 - r0^2 = -r0 ud + ud^2/4
  if (rho > __fadd_rn(__fmul_rn(r0, u), __fmul_rn(__fmul_rn(u, u), 0.25f))) return up;
  if (rho < __fadd_rn(__fmul_rn(-r0, ud), __fmul_rn(__fmul_rn(ud, ud), 0.25f))) return dn;
  return r0;
}

__device__ float4 color_of(const float4& a, const float4& b, int mode, float parameter)
{
  // (b - a).normalized() as Eigen evaluates it for Vector4f.
  float4 d = make_float4(__fsub_rn(b.x, a.x), __fsub_rn(b.y, a.y), __fsub_rn(b.z, a.z), __fsub_rn(b.w, a.w));
  const float z = __fadd_rn(__fadd_rn(__fmul_rn(d.x, d.x), __fmul_rn(d.z, d.z)), __fadd_rn(__fmul_rn(d.y, d.y), __fmul_rn(d.w, d.w)));
  if (z > 0.0f)
  {
    const float r = __fsqrt_rn(z);
    d = make_float4(__fdiv_rn(d.x, r), __fdiv_rn(d.y, r), __fdiv_rn(d.z, r), __fdiv_rn(d.w, r));
  }
  if (mode == PARS_COLOR_RGB) return make_float4(fabsf(d.x), fabsf(d.z), fabsf(d.y), 1.0f);

  // to_spherical (coordinates.hpp:8-16): the radius as the reference rounds
  // it (acos near +-1 would magnify any difference in it); atan2 and acos are
  // the FP32 functions, as the reference calls them (the host libm's atan2f /
  // acosf there, CUDA's here: within 3 and 2 ulp).
  const float radius = reference_radius(d.x, d.y, d.z);
  float s1 = atan2f(d.y, d.x);
  float s2 = acosf(__fdiv_rn(d.z, radius));
  // correct_range (color_generator.cpp:41-54).
  const float pi = float(3.14159265358979323846);
  if (s1 <  0.0f) s1 = __fadd_rn(s1, pi);
  if (s1 >= pi)   s1 = __fsub_rn(s1, pi);
  s1 = __fsub_rn(pi, s1);
  if (s2 <  0.0f) s2 = fabsf(s2);
  if (s2 >= float(3.14159265358979323846 / 2.0)) s2 = __fsub_rn(pi, s2);
  // s / M_PI and s / (M_PI / 2): the reference divides in double and rounds to
  // float; an FP32 multiply by the rounded reciprocal is within one ulp of
  // that (hue and saturation are already a few ulps apart from the reference
  // through atan2f / acosf).
  const float hue    = __fmul_rn(s1, float(1.0 / 3.14159265358979323846));
  const float second = __fmul_rn(s2, float(2.0 / 3.14159265358979323846));

  const bool constant_first = (mode == PARS_COLOR_HSL_CONSTANT_S || mode == PARS_COLOR_HSV_CONSTANT_S);
  const float sat   = constant_first ? parameter : second;
  const float third = constant_first ? second : parameter;
  float4 c = hue_to_rgba(hue);
  if (mode == PARS_COLOR_HSL_CONSTANT_S || mode == PARS_COLOR_HSL_CONSTANT_L)
  {
    // hsl_to_rgba (color_generator.cpp:65-72)
    const float pre = __fmul_rn(__fsub_rn(1.0f, fabsf(__fsub_rn(__fmul_rn(2.0f, third), 1.0f))), sat);
    c.x = __fadd_rn(__fmul_rn(__fsub_rn(c.x, 0.5f), pre), third);
    c.y = __fadd_rn(__fmul_rn(__fsub_rn(c.y, 0.5f), pre), third);
    c.z = __fadd_rn(__fmul_rn(__fsub_rn(c.z, 0.5f), pre), third);
  }
  else
  {
    // hsv_to_rgba (color_generator.cpp:73-79)
    c.x = __fmul_rn(__fadd_rn(__fmul_rn(__fsub_rn(c.x, 1.0f), sat), 1.0f), third);
    c.y = __fmul_rn(__fadd_rn(__fmul_rn(__fsub_rn(c.y, 1.0f), sat), 1.0f), third);
    c.z = __fmul_rn(__fadd_rn(__fmul_rn(__fsub_rn(c.z, 1.0f), sat), 1.0f), third);
  }
  c.w = 1.0f;
  return c;
}

__global__ void __launch_bounds__(256) color_kernel(const float4* __restrict__ v, const int* __restrict__ indices, long long m,
                                                    int mode, float parameter, float4* __restrict__ colors)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int index = indices[i];
  const float4 c = color_of(v[index], v[index + 1], mode, parameter);
  colors[index] = c;
  // The last vertex of a run copies its colour (color_generator.cpp:36-37).
  if (i != m - 1 && indices[i + 1] != index + 1) colors[index + 1] = c;
}

// ---- every batch of a curves store at once ------------------------------------
// The batches are consecutive ranges of one vertex buffer (bounds[b] ..
// bounds[b + 1]).  Index generation runs over the whole buffer with each
// vertex's flag confined to its batch; one scan gives every flagged vertex its
// position in the packed index buffer, which holds the batches' indices one
// after the other (each index relative to its batch, as the reference's).
//
// The index passes are bound by memory: a warp takes 256 consecutive vertices, 32
// at a time, looks its first batch up once and then steps over the bounds it meets,
// and the write pass reads the flags' bits instead of the vertices.  Colours (bound
// by memory as rgb, by atan2 and acos as hsl / hsv) go vertex by vertex in one
// write.  26.5 M vertices in 300 batches, count / write / colours: 83 / 42 / 177 us;
// eight consecutive vertices per thread, the vertices read again by the write pass,
// a search per index and zeroed colours took 120 / 182 / 203 us and 60 us to zero.

// The first s in [0, batches) with bounds[s] >= x, else batches.
__device__ __forceinline__ int bound_from(const long long* __restrict__ bounds, int batches, long long x)
{
  int lo = 0, hi = batches;
  while (lo < hi)
  {
    const int mid = (lo + hi) >> 1;
    if (bounds[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Flags of every vertex (a word per 32) and the flagged vertices of every tile.
// One batch: vbounds is not read.
__global__ void __launch_bounds__(index_threads) index_count_kernel(const float4* __restrict__ v, long long n,
                                                                    const long long* __restrict__ vbounds, int batches,
                                                                    unsigned int* __restrict__ flags, int* __restrict__ tile_counts)
{
  __shared__ int counts[index_threads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long first = (long long)blockIdx.x * index_tile + warp * warp_vertices;
  int count = 0;
  if (first < n)
  {
    unsigned term[warp_words + 1];
    #pragma unroll
    for (int k = 0; k < warp_words; ++k)
    {
      const long long i = first + 32 * k + lane;
      const float4 vertex = v[min(i, n - 1)];   // (no branch: the loads go out together)
      term[k] = __ballot_sync(full_mask, i >= n || is_termination_vertex(vertex));
    }
    const long long beyond = first + warp_vertices;
    term[warp_words] = beyond < n ? (is_termination_vertex(v[beyond]) ? 1u : 0u) : 1u;
    int s = batches == 1 ? 1 : bound_from(vbounds, batches, first + 1);   // the next batch
    long long bound = s < batches ? vbounds[s] : n;
    unsigned word = 0;
    #pragma unroll
    for (int k = 0; k < warp_words; ++k)
    {
      const long long c = first + 32 * k;
      unsigned f = ~term[k] & ~((term[k] >> 1) | (term[k + 1] << 31));
      // the vertex before a batch has no next one
      while (s < batches && bound <= c + 32)
      {
        f &= ~(1u << int(bound - 1 - c));
        ++s;
        bound = s < batches ? vbounds[s] : n;
        // (bounds of empty batches repeat: the same bit again)
      }
      count += __popc(f);
      if (lane == k) word = f;
    }
    if (lane < warp_words && first + 32 * lane < n) flags[(first >> 5) + lane] = word;
  }
  if (lane == 0) counts[warp] = count;
  __syncthreads();
  if (threadIdx.x == 0)
  {
    int total = 0;
    #pragma unroll
    for (int w = 0; w < index_threads / 32; ++w) total += counts[w];
    tile_counts[blockIdx.x] = total;
  }
}

// Writes the packed indices and, for every batch that starts in the warp's range,
// the batch's first position in the packed buffer (ibounds, if given).
__global__ void __launch_bounds__(index_threads) index_write_kernel(const unsigned int* __restrict__ flags, long long n,
                                                                    const long long* __restrict__ vbounds, int batches,
                                                                    const long long* __restrict__ tile_offsets, int* __restrict__ indices,
                                                                    long long* __restrict__ ibounds)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lanes_below = (1u << lane) - 1u;
  const long long first = (long long)blockIdx.x * index_tile + warp * warp_vertices;
  if (first >= n) return;
  // the tile's flags before this warp's
  const long long tile_word = (long long)blockIdx.x * tile_words, words = (n + 31) >> 5;
  int before = 0;
  for (int w = lane; w < warp * warp_words; w += 32) before += __popc(flags[tile_word + w]);
  long long out = tile_offsets[blockIdx.x] + __reduce_add_sync(full_mask, before);
  const long long own = tile_word + warp * warp_words + lane;
  const unsigned word = lane < warp_words && own < words ? flags[own] : 0u;

  int s = batches == 1 ? 1 : bound_from(vbounds, batches, first);   // the first batch that starts at or after `first`
  if (batches == 1 && ibounds && first == 0 && lane == 0) ibounds[0] = 0;
  long long bound = s < batches ? vbounds[s] : n;
  long long begin = batches > 1 && s > 0 ? vbounds[s - 1] : 0;      // the batch of the lane's vertex
  #pragma unroll
  for (int k = 0; k < warp_words; ++k)
  {
    const long long c = first + 32 * k, i = c + lane;
    const unsigned f = __shfl_sync(full_mask, word, k);
    while (s < batches && bound < c + 32)
    {
      if (lane == 0 && ibounds) ibounds[s] = out + __popc(f & ((1u << int(bound - c)) - 1u));
      if (i >= bound) begin = bound;
      ++s;
      bound = s < batches ? vbounds[s] : n;
    }
    if (f >> lane & 1u) indices[out + __popc(f & lanes_below)] = int(i - begin);
    out += __popc(f);
    begin = __shfl_sync(full_mask, begin, 31);   // the next vertices' batch
  }
}

// Colours of every vertex: an indexed vertex takes its segment's; the last vertex
// of a run copies its colour, but for the batch's last run (color_generator.cpp:
// 36-37); others stay 0.
__global__ void __launch_bounds__(256) batch_color_kernel(const float4* __restrict__ v, const int* __restrict__ indices, long long n,
                                                          const long long* __restrict__ vbounds, const long long* __restrict__ ibounds,
                                                          int batches, const color_spec* __restrict__ specs, float4* __restrict__ colors, int words)
{
  const int lane = threadIdx.x & 31;
  const long long first = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 * words);
  if (first >= n) return;
  int s = bound_from(vbounds, batches, first + 1);   // the batch after the lane's vertex's
  for (int k = 0; k < words; ++k)
  {
    const long long i = first + 32 * k + lane;
    if (i >= n) return;
    while (s < batches && vbounds[s] <= i) ++s;
    const int b = s - 1;
    const long long begin = vbounds[b], end = vbounds[b + 1], last_index = ibounds[b + 1];
    const float4 here = v[i];
    float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
    if (last_index > ibounds[b] && !is_termination_vertex(here))
    {
      const color_spec spec = specs[b];
      float4 from = here, to = here;
      bool colored = false;
      if (i + 1 < end) { to = v[i + 1]; colored = !is_termination_vertex(to); }
      if (!colored && i > begin && i - 1 - begin != indices[last_index - 1])
      {
        from = v[i - 1];
        to = here;
        colored = !is_termination_vertex(from);
      }
      if (colored) out = color_of(from, to, spec.mode, spec.parameter);
    }
    colors[i] = out;
  }
}
}

void index_batches(pars_gpu_context& ctx, curves_store& c)
{
  const int batches = int(c.batches.size());
  std::vector<long long> vbounds(batches + 1), ibounds(batches + 1, 0);
  for (int b = 0; b < batches; ++b) vbounds[b] = c.batches[b].vertex_offset;
  vbounds[batches] = c.vertex_total;
  for (int b = 0; b < batches; ++b)
    PARS_REQUIRE(c.batches[b].vertex_offset + c.batches[b].vertex_count == vbounds[b + 1], "curve batches are not consecutive");
  c.indices.reserve(sizeof(int) * (std::size_t)std::max<long long>(c.vertex_total, 1));
  ctx.curve_bounds.reserve(sizeof(long long) * 2 * (batches + 1));
  long long* d_vbounds = ctx.curve_bounds.as<long long>();
  long long* d_ibounds = d_vbounds + batches + 1;
  const long long n = c.vertex_total;
  if (batches > 0 && n > 0)
  {
    PARS_CUDA(cudaMemcpyAsync(d_vbounds, vbounds.data(), sizeof(long long) * (batches + 1), cudaMemcpyHostToDevice, ctx.stream));
    const long long tiles = (n + index_tile - 1) / index_tile;
    ctx.tile_counts.reserve(sizeof(int) * tiles);
    ctx.tile_offsets.reserve(sizeof(long long) * (tiles + 1));
    ctx.index_flags.reserve(sizeof(unsigned int) * tiles * tile_words);
    {
      launch_scope scope(ctx, "index_count");
      index_count_kernel<<<(unsigned)tiles, index_threads, 0, ctx.stream>>>(c.vertices.as<const float4>(), n, d_vbounds, batches,
                                                                            ctx.index_flags.as<unsigned int>(), ctx.tile_counts.as<int>());
    }
    exclusive_sum(ctx, ctx.tile_counts.as<int>(), ctx.tile_offsets.as<long long>(), tiles);
    {
      launch_scope scope(ctx, "index_write");
      index_write_kernel<<<(unsigned)tiles, index_threads, 0, ctx.stream>>>(ctx.index_flags.as<const unsigned int>(), n, d_vbounds, batches,
                                                                            ctx.tile_offsets.as<const long long>(), c.indices.as<int>(),
                                                                            d_ibounds);
    }
    long long total = 0;
    PARS_CUDA(cudaMemcpyAsync(ibounds.data(), d_ibounds, sizeof(long long) * batches, cudaMemcpyDeviceToHost, ctx.stream));
    PARS_CUDA(cudaMemcpyAsync(&total, ctx.tile_offsets.as<long long>() + tiles, sizeof(long long), cudaMemcpyDeviceToHost, ctx.stream));
    PARS_CUDA(cudaStreamSynchronize(ctx.stream));
    ibounds[batches] = total;
    // batches starting at the very end (empty) were not seen by any thread
    for (int b = batches - 1; b >= 0; --b) if (vbounds[b] == n) ibounds[b] = total;
    PARS_CUDA(cudaMemcpyAsync(d_ibounds, ibounds.data(), sizeof(long long) * (batches + 1), cudaMemcpyHostToDevice, ctx.stream));
  }
  else if (batches > 0)
  {
    PARS_CUDA(cudaMemcpyAsync(d_vbounds, vbounds.data(), sizeof(long long) * (batches + 1), cudaMemcpyHostToDevice, ctx.stream));
    PARS_CUDA(cudaMemcpyAsync(d_ibounds, ibounds.data(), sizeof(long long) * (batches + 1), cudaMemcpyHostToDevice, ctx.stream));
  }
  for (int b = 0; b < batches; ++b)
  {
    c.batches[b].index_offset = ibounds[b];
    c.batches[b].index_count = ibounds[b + 1] - ibounds[b];
  }
  c.index_total = ibounds[batches];
}

void color_batches(pars_gpu_context& ctx, curves_store& c, const std::vector<color_spec>& specs)
{
  const int batches = int(c.batches.size());
  PARS_REQUIRE(specs.size() == std::size_t(batches), "one colour spec per batch");
  c.colors.reserve(sizeof(float4) * (std::size_t)std::max<long long>(c.vertex_total, 1));
  if (batches == 0 || c.index_total == 0)
  {
    if (c.vertex_total > 0) PARS_CUDA(cudaMemsetAsync(c.colors.get(), 0, sizeof(float4) * c.vertex_total, ctx.stream));
    return;
  }
  ctx.color_specs.reserve(sizeof(color_spec) * batches);
  PARS_CUDA(cudaMemcpyAsync(ctx.color_specs.get(), specs.data(), sizeof(color_spec) * batches, cudaMemcpyHostToDevice, ctx.stream));
  const long long* d_vbounds = ctx.curve_bounds.as<const long long>();
  const long long* d_ibounds = d_vbounds + batches + 1;
  launch_scope scope(ctx, "color_generate");
  // 32 vertices a warp while there are few (4096 curves of 1000 vertices: 9 us, 12
  // with 256), 256 a warp from 8 M on (26.5 M: 177 us, 207 with 32: fewer searches)
  const int words = c.vertex_total < (8LL << 20) ? 1 : warp_words;
  batch_color_kernel<<<(unsigned)((c.vertex_total + 256 * words - 1) / (256 * words)), 256, 0, ctx.stream>>>(
    c.vertices.as<const float4>(), c.indices.as<const int>(), c.vertex_total, d_vbounds, d_ibounds, batches, ctx.color_specs.as<const color_spec>(),
    c.colors.as<float4>(), words);
}

long long launch_index_generate(pars_gpu_context& ctx, const float4* vertices, long long n, int* indices)
{
  if (n < 2) return 0;
  const long long tiles = (n + index_tile - 1) / index_tile;
  ctx.tile_counts.reserve(sizeof(int) * tiles);
  ctx.tile_offsets.reserve(sizeof(long long) * (tiles + 1));
  ctx.index_flags.reserve(sizeof(unsigned int) * tiles * tile_words);
  {
    launch_scope scope(ctx, "index_count");
    index_count_kernel<<<(unsigned)tiles, index_threads, 0, ctx.stream>>>(vertices, n, nullptr, 1, ctx.index_flags.as<unsigned int>(),
                                                                          ctx.tile_counts.as<int>());
  }
  exclusive_sum(ctx, ctx.tile_counts.as<int>(), ctx.tile_offsets.as<long long>(), tiles);
  {
    launch_scope scope(ctx, "index_write");
    index_write_kernel<<<(unsigned)tiles, index_threads, 0, ctx.stream>>>(ctx.index_flags.as<const unsigned int>(), n, nullptr, 1,
                                                                          ctx.tile_offsets.as<const long long>(), indices, nullptr);
  }
  long long total = 0;
  PARS_CUDA(cudaMemcpyAsync(&total, ctx.tile_offsets.as<long long>() + tiles, sizeof(long long), cudaMemcpyDeviceToHost, ctx.stream));
  PARS_CUDA(cudaStreamSynchronize(ctx.stream));
  return total;
}

void launch_color_generate(pars_gpu_context& ctx, const float4* vertices, const int* indices, long long index_count,
                           int mode, float parameter, float4* colors)
{
  if (index_count <= 0) return;
  launch_scope scope(ctx, "color_generate");
  color_kernel<<<(unsigned)((index_count + 255) / 256), 256, 0, ctx.stream>>>(vertices, indices, index_count, mode, parameter, colors);
}
}
