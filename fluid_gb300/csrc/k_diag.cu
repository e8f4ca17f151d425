// Diagnostics and field views (pkg/fluid/fluid.go:529-557, 798-891;
// pressure.go, smoke.go): reductions accumulate in FP64 through fixed-slot
// block partials, so repeated runs give identical numbers.
#include <algorithm>
#include <cfloat>
#include <cstddef>

#include "fg_internal.cuh"
#include "fg_reduce.cuh"

namespace fg {
namespace {

constexpr int BX = 32, BY = 8;
inline dim3 cell_grid(const fg_fluid* f) {
  return dim3((f->NY + BX - 1) / BX, (f->NX + BY - 1) / BY);
}
__device__ __forceinline__ bool fluid_interior(uint8_t fl) {
  return (fl & (F_FLUID | F_INTERIOR)) == (F_FLUID | F_INTERIOR);
}

// Where the reductions' total rows go.
struct StoreDiv {
  DevStats* st;
  __device__ void operator()(const float* r) const {
    st->div_l2_sq = row_sum(r, 0);
    st->div_max = (double)r[2];
    st->div_count = row_sum(r, 2);
  }
};

// (max v, max -v) -> float (min, max), with the reference's initial values
// (MaxFloat32, -MaxFloat32) when no cell was seen. To device or pinned host
// memory.
struct StoreMinMax {
  float* out;
  __device__ void operator()(const float* r) const {
    float hi = r[0], nlo = r[2];
    out[0] = nlo == -INFINITY ? FLT_MAX : -nlo;
    out[1] = hi == -INFINITY ? -FLT_MAX : hi;
  }
};

// A max slot of a final row -> float, 0 when no cell was seen.
struct StoreMax0 {
  float* out;
  __device__ void operator()(const float* r) const { out[0] = r[0] < 0.0f ? 0.0f : r[0]; }
};

// body(c) for the cells of a block's tiles.
template <typename Body>
__device__ __forceinline__ void each_cell(const Grid& g, Body body) {
  const int tx = (g.NY + BX - 1) / BX, tiles = tx * ((g.NX + BY - 1) / BY);
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int y = t / tx, j = (t - y * tx) * BX + threadIdx.x, i = y * BY + threadIdx.y;
    if (i < g.NX && j < g.NY) body(i * g.P + j);
  }
}

// Post-projection divergence statistics: rows {sum div^2, max |div|, count}
// over fluid interior cells.
__global__ void __launch_bounds__(256)
    k_div_stats(const float* __restrict__ U, const float* __restrict__ V,
                const uint8_t* __restrict__ flags, float* __restrict__ part, Grid g, int* ticket,
                StoreDiv store) {
  __shared__ float sh[64 * 3];
  pdl_enter();
  FF v[3] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
  each_cell(g, [&](int c) {
    if (!fluid_interior(flags[c])) return;
    float div = U[c + g.P] - U[c] + V[c + 1] - V[c];
    ff_acc(v[0], ff_sq(div));
    v[1].hi = fmaxf(v[1].hi, fabsf(div));
    v[2].hi += 1.0f;
  });
  grid_row<3>(v, 2u, sh, part, blockIdx.x, gridDim.x, ticket, store);
}

// MaxDivergence (fluid.go:876-891): float32 |div|, NaN ignored (fmaxf).
__global__ void __launch_bounds__(256)
    k_max_divergence(const float* __restrict__ U, const float* __restrict__ V,
                     const uint8_t* __restrict__ flags, float* __restrict__ part, Grid g,
                     int* ticket, StoreMax0 store) {
  __shared__ float sh[64];
  FF v[1] = {{0.0f, 0.0f}};
  each_cell(g, [&](int c) {
    if (fluid_interior(flags[c]))
      v[0].hi = fmaxf(v[0].hi, fabsf(U[c + g.P] - U[c] + V[c + 1] - V[c]));
  });
  grid_row<1>(v, 1u, sh, part, blockIdx.x, gridDim.x, ticket, store);
}

// |U| + |V| on fluid interior cells (GetAdaptiveTimeStep fluid.go:534-543).
__global__ void __launch_bounds__(256)
    k_max_speed(const float* __restrict__ U, const float* __restrict__ V,
                const uint8_t* __restrict__ flags, float* __restrict__ part, Grid g, int* ticket,
                StoreMax0 store) {
  __shared__ float sh[64];
  FF v[1] = {{0.0f, 0.0f}};
  each_cell(g, [&](int c) {
    if (fluid_interior(flags[c])) v[0].hi = fmaxf(v[0].hi, fabsf(U[c]) + fabsf(V[c]));
  });
  grid_row<1>(v, 1u, sh, part, blockIdx.x, gridDim.x, ticket, store);
}

// A value's part in a range {max v, max -v}: NaN is left out.
__device__ __forceinline__ void range_of(FF (&v)[2], float x) {
  if (isnan(x)) return;
  v[0].hi = fmaxf(v[0].hi, x);
  v[1].hi = fmaxf(v[1].hi, -x);
}

// Vorticity (fluid.go:806-838, kind 0) and VelocityMagnitude (fluid.go:841-873,
// kind 1) on fluid interior cells, 0 elsewhere; rows {max v, max -v} over
// the computed cells (-inf when a block saw none).
__global__ void __launch_bounds__(256)
    k_view(const float* __restrict__ U, const float* __restrict__ V,
           const uint8_t* __restrict__ flags, float* __restrict__ out, int kind,
           float* __restrict__ part, Grid g, int* ticket, StoreMinMax store) {
  __shared__ float sh[128];
  FF v[2] = {{-INFINITY, 0.0f}, {-INFINITY, 0.0f}};
  each_cell(g, [&](int c) {
    float x = 0.0f;
    if (fluid_interior(flags[c])) {
      if (kind == 0) {
        float dvdx = (V[c + g.P] - V[c - g.P]) * 0.5f / g.h;
        float dudy = (U[c + 1] - U[c - 1]) * 0.5f / g.h;
        x = dvdx - dudy;
      } else {
        float u = (U[c] + U[c + g.P]) * 0.5f;
        float w = (V[c] + V[c + 1]) * 0.5f;
        x = sqrtf(u * u + w * w);
      }
      range_of(v, x);
    }
    out[c] = x;
  });
  grid_row<2>(v, 3u, sh, part, blockIdx.x, gridDim.x, ticket, store);
}

// min / max over all cells of a field (Pressure(), Smoke()).
__global__ void __launch_bounds__(256)
    k_field_minmax(const float* __restrict__ F, float* __restrict__ part, Grid g, int* ticket,
                   StoreMinMax store) {
  __shared__ float sh[128];
  FF v[2] = {{-INFINITY, 0.0f}, {-INFINITY, 0.0f}};
  each_cell(g, [&](int c) { range_of(v, F[c]); });
  grid_row<2>(v, 3u, sh, part, blockIdx.x, gridDim.x, ticket, store);
}

__global__ void k_sample_velocity(const float* __restrict__ U, const float* __restrict__ V,
                                  float x, float y, float* __restrict__ out, Grid g) {
  out[0] = sample_field(U, x, y, 0.0f, g.hh, g);
  out[1] = sample_field(V, x, y, g.hh, 0.0f, g);
}

}  // namespace

cudaError_t launch_clear_stats(fg_fluid* f, bool keep_timeout) {
  // (A batch's and a recorded rollout's mark of a wait that gave up outlives
  // the step: it is read once for many steps.  The ticket is 0 at rest.)
  return cudaMemsetAsync(f->dstats, 0, keep_timeout ? offsetof(DevStats, timeout) : sizeof(DevStats),
                         f->stream);
}

// Blocks of a reduction over the cells' tiles, 0 when their rows do not fit.
static int stat_blocks(const fg_fluid* f, int ns) {
  const dim3 gr = cell_grid(f);
  const int nb = (int)std::min<long long>((long long)gr.x * gr.y, kStatBlocks);
  return partials_fit(f, ns, nb) ? nb : 0;
}

cudaError_t launch_div_stats(fg_fluid* f) {
  const int nb = stat_blocks(f, 3);
  if (!nb) return cudaErrorInvalidValue;
  count(f);
  return launch_pdl(k_div_stats, dim3(nb), dim3(BX, BY), 0, f->stream, f->d[FG_U], f->d[FG_V],
                    f->flags, f->partials, f->g, &f->dstats->ticket, StoreDiv{f->dstats});
}

cudaError_t launch_max_divergence(fg_fluid* f, float* out) {
  const int nb = stat_blocks(f, 1);
  if (!nb) return cudaErrorInvalidValue;
  count(f);
  k_max_divergence<<<nb, dim3(BX, BY), 0, f->stream>>>(f->d[FG_U], f->d[FG_V], f->flags,
                                                       f->partials, f->g, &f->dstats->ticket,
                                                       StoreMax0{out});
  return cudaGetLastError();
}

cudaError_t launch_max_speed(fg_fluid* f, float* out) {
  const int nb = stat_blocks(f, 1);
  if (!nb) return cudaErrorInvalidValue;
  count(f);
  k_max_speed<<<nb, dim3(BX, BY), 0, f->stream>>>(f->d[FG_U], f->d[FG_V], f->flags, f->partials,
                                                  f->g, &f->dstats->ticket, StoreMax0{out});
  return cudaGetLastError();
}

cudaError_t launch_view(fg_fluid* f, int kind, float* minmax) {
  const int nb = stat_blocks(f, 2);
  if (!nb) return cudaErrorInvalidValue;
  count(f);
  k_view<<<nb, dim3(BX, BY), 0, f->stream>>>(f->d[FG_U], f->d[FG_V], f->flags, f->view, kind,
                                             f->partials, f->g, &f->dstats->ticket,
                                             StoreMinMax{minmax});
  return cudaGetLastError();
}

cudaError_t launch_field_minmax(fg_fluid* f, int field, float* minmax) {
  const int nb = stat_blocks(f, 2);
  if (!nb) return cudaErrorInvalidValue;
  count(f);
  k_field_minmax<<<nb, dim3(BX, BY), 0, f->stream>>>(f->d[field], f->partials, f->g,
                                                     &f->dstats->ticket, StoreMinMax{minmax});
  return cudaGetLastError();
}

cudaError_t launch_sample_velocity(fg_fluid* f, float x, float y, float* dev_uv) {
  count(f);
  k_sample_velocity<<<1, 1, 0, f->stream>>>(f->d[FG_U], f->d[FG_V], x, y, dev_uv, f->g);
  return cudaGetLastError();
}

// Copies between the mirrors' layout (rows of NY floats) and the device
// pitch, on the device (faster than a strided DMA copy for device sources).
__global__ void k_repitch(float* __restrict__ dst, const float* __restrict__ src, int rows,
                          int cols, int dpitch, int spitch) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= rows || j >= cols) return;
  dst[(size_t)i * dpitch + j] = src[(size_t)i * spitch + j];
}

cudaError_t launch_repitch(fg_fluid* f, float* dst, const float* src, int dpitch, int spitch) {
  count(f);
  dim3 gr((f->NY + 31) / 32, (f->NX + 7) / 8);
  k_repitch<<<gr, dim3(32, 8), 0, f->stream>>>(dst, src, f->NX, f->NY, dpitch, spitch);
  return cudaGetLastError();
}

}  // namespace fg
