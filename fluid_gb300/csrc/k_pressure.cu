// Pressure projection (pkg/fluid/fluid.go:144-234).
//
// The parallel schemes (the reference's serial ones: k_lexsor.cu):
//  * JACOBI relaxes the same masked Poisson system for the cell potential
//    phi (the accumulated per-cell correction of the SOR loop):
//        s_c phi_c - sum_n phi_n = -div_c,   phi = 0 off the active cells,
//    then applies U_face += S_R phi_L - S_L phi_R (and likewise V) and
//    p = cp * phi.  Sweeps run temporally blocked: a block relaxes a tile
//    with a halo as wide as its sweep count (8) in registers, so memory sees
//    one read and one write of phi per block of sweeps (k_jacobi_rb; fed by
//    TMA copies in k_jacobi_tma; a whole fixed-count solve as one cooperative
//    dataflow launch in k_jacobi_flow).  Optional outer correction: an
//    FP64-class residual of the FP32 iterate, a correction solve on it,
//    phi += e.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <mutex>

#include "fg_batch.cuh"
#include "fg_internal.cuh"
#include "fg_reduce.cuh"

namespace fg {

// Device control block of the parallel schemes.
struct PCtl {
  int stop;         // early-exit latch
  int sel;          // buffer holding the latest phi (0: phi, 1: phi2)
  int sweeps;       // sweeps executed
  int last_launch;  // index of the last executed launch
  int esel;         // buffer holding the latest correction (0: err, 1: err2)
  int pad[3];
  unsigned slots[1];  // per-launch max |r| of its last sweep (float bits)
};

namespace {

constexpr unsigned long long MBAR_WAIT_NS = 1000000000ull;  // 1 s
constexpr int MBAR_MAX_TRIES = 1 << 24;
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

constexpr int BX = 32, BY = 8;
inline dim3 cell_grid(const fg_fluid* f) {
  return dim3((f->NY + BX - 1) / BX, (f->NX + BY - 1) / BY);
}

// ------------------------------------------------------------------ parallel scheme
struct WTab {
  float w[5];  // w[s] = (omega * damping) / s
};

// U + Fu at face u (the force field of a recorded step, null otherwise).
__device__ __forceinline__ float with_force(const float* __restrict__ U,
                                            const float* __restrict__ F, int u) {
  return F ? U[u] + F[u] : U[u];
}

// Per cell: b = -div, w = om / s and bw = w * b on active cells, all 0
// elsewhere (ring included); phi = 0 when `zero_phi` (a solve with no sweeps
// reads it directly).
// U, V use the grid pitch g.P, the solver arrays the pitch Ps.
__device__ __forceinline__ void setup_cell_p(int i, int j, const float* __restrict__ U,
                                             const float* __restrict__ V, float* __restrict__ phi,
                                             float* __restrict__ rhs, float* __restrict__ W,
                                             float* __restrict__ BW,
                                             const uint8_t* __restrict__ flags, float om,
                                             int zero_phi, const Grid& g, int Ps,
                                             const float* __restrict__ Fu = nullptr,
                                             const float* __restrict__ Fv = nullptr) {
  int u = i * g.P + j;
  int c = i * Ps + j;
  float b = 0.0f, w = 0.0f, bw = 0.0f;
  uint8_t fl = flags[c];
  // Active cells are interior.  Below the last row and column the four face
  // loads are in range whatever the flags say, so they issue beside the flag
  // load and the flags only select the result.
  if (i <= g.NX - 2 && j <= g.NY - 2) {
    float div = with_force(U, Fu, u + g.P) - with_force(U, Fu, u) + with_force(V, Fv, u + 1) -
                with_force(V, Fv, u);
    bool act = flag_active(fl);
    b = act ? -div : 0.0f;
    w = act ? om / (float)flag_count(fl) : 0.0f;
    bw = w * b;
  }
  rhs[c] = b;
  W[c] = w;
  BW[c] = bw;
  if (zero_phi) phi[c] = 0.0f;
}
__device__ __forceinline__ void setup_cell(int i, int j, const float* __restrict__ U,
                                           const float* __restrict__ V, float* __restrict__ phi,
                                           float* __restrict__ rhs, float* __restrict__ W,
                                           float* __restrict__ BW,
                                           const uint8_t* __restrict__ flags, float om,
                                           int zero_phi, const Grid& g) {
  setup_cell_p(i, j, U, V, phi, rhs, W, BW, flags, om, zero_phi, g, g.P);
}
// The flags of an interior fluid cell with four fluid neighbours.
constexpr uint8_t kPlain = F_W | F_E | F_S | F_N | F_FLUID | F_INTERIOR;
__global__ void k_setup_system(const float* __restrict__ U, const float* __restrict__ V,
                               float* __restrict__ phi, float* __restrict__ rhs,
                               float* __restrict__ W, float* __restrict__ BW,
                               const uint8_t* __restrict__ flags, float om, int zero_phi, Grid g,
                               int Ps, const float* __restrict__ Fu, const float* __restrict__ Fv) {
  pdl_enter();
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.NX || j >= g.NY) return;
  setup_cell_p(i, j, U, V, phi, rhs, W, BW, flags, om, zero_phi, g, Ps, Fu, Fv);
}

// The same for a handle's own fields (g.P the pitch of all of them), 4 columns
// a thread in 16-byte pieces; a piece of plain cells has one weight.  Bound by
// memory traffic from 1500 x 1100 on; one cell a thread, with a division each,
// was bound by its instructions (2048 x 2048: 20.1 us, 14.1 this way; the
// traffic takes 12).
__global__ void __launch_bounds__(256)
    k_setup_pieces(const float* __restrict__ U, const float* __restrict__ V,
                   float* __restrict__ phi, float* __restrict__ rhs, float* __restrict__ W,
                   float* __restrict__ BW, const uint8_t* __restrict__ flags, float om,
                   int zero_phi, Grid g, const float* __restrict__ Fu,
                   const float* __restrict__ Fv) {
  pdl_enter();
  const int nq = (g.NY + 3) / 4, idx = blockIdx.x * 256 + threadIdx.x;
  const int i = idx / nq, j = 4 * (idx - i * nq);
  if (i >= g.NX) return;
  const int c = i * g.P + j, cn = i <= g.NX - 2 ? c + g.P : c;
  auto sum4 = [](const float* x, const float* y, int k, float (&o)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(x + k);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
    if (y) {
      const float4 b = *reinterpret_cast<const float4*>(y + k);
      o[0] = o[0] + b.x; o[1] = o[1] + b.y; o[2] = o[2] + b.z; o[3] = o[3] + b.w;
    }
  };
  const bool more = j + 4 < g.NY;  // the column right of the piece is a cell
  const uint32_t f = *reinterpret_cast<const uint32_t*>(flags + c);
  float u[4], un[4], v[4];
  sum4(U, Fu, c, u);
  sum4(U, Fu, cn, un);
  sum4(V, Fv, c, v);
  const float vr = more ? with_force(V, Fv, c + 4) : 0.0f;
  const bool plain = more && f == kPlain * 0x01010101u;
  float b[4], w[4], bw[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    b[k] = w[k] = bw[k] = 0.0f;
    const uint8_t fl = (uint8_t)(f >> 8 * k);
    if (plain) {
      b[k] = -(un[k] - u[k] + (k < 3 ? v[k + 1] : vr) - v[k]);
      w[k] = om * 0.25f;
      bw[k] = w[k] * b[k];
    } else if (i <= g.NX - 2 && j + k <= g.NY - 2) {
      const bool act = flag_active(fl);
      const float div = un[k] - u[k] + (k < 3 ? v[k + 1] : vr) - v[k];
      b[k] = act ? -div : 0.0f;
      w[k] = act ? om / (float)flag_count(fl) : 0.0f;
      bw[k] = w[k] * b[k];
    }
  }
  auto put = [&](float* d, const float (&x)[4]) {
    if (j + 4 <= g.NY) {
      *reinterpret_cast<float4*>(d + c) = make_float4(x[0], x[1], x[2], x[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (j + k < g.NY) d[c + k] = x[k];
    }
  };
  put(rhs, b);
  put(W, w);
  put(BW, bw);
  if (zero_phi) {
    const float z[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    put(phi, z);
  }
}

// Register-blocked, temporally blocked Jacobi.  A CTA of 8 warps holds a
// 64 x 128 region (rows i x columns j) in registers: each thread a block of
// RT = 8 rows by JT = 4 consecutive columns.  Vertical neighbours come from
// the thread's own rows, or through shared memory from the warp above/below
// at its first/last row; horizontal neighbours from the thread's own columns
// or a warp shuffle.  `ns` <= H sweeps run per launch; inside the grid the
// region carries a halo of H = 8 cells, so the CTA owns the inner 48 x 112
// cells, and at the grid's edges it owns up to the edge (span_count and
// span_own, fg_internal.cuh); it writes only what it owns.  Cells outside
// the grid or inactive have w = bw = 0 and stay 0.  The TMA-fed kernels
// below keep regions at t S - H with the inner 48 x 112 owned.  Launch k
// first decides whether the solve already stopped
// (thread 0 of every CTA reads the same control words, so all CTAs agree);
// a running launch records the max |r| of its last sweep over the active
// cells it owns, r = fma(-s, phi, b + nb), in slots[k].
constexpr int JT = 4, RT = 8, NWARP = 8, TMAX = 8;
constexpr int RJ = 32 * JT;        // 128 region columns
constexpr int RI = NWARP * RT;     // 64 region rows
constexpr int OJ = RJ - 2 * TMAX;  // 112 owned columns
constexpr int OI = RI - 2 * TMAX;  // 48 owned rows
constexpr int TB_THREADS = 32 * NWARP;
static_assert(RI == kJacRegionRows && RJ == kJacRegionCols && TMAX == kJacHalo && RT == kJacWarpRows,
              "Jacobi region geometry");

// RINIT (first launch of the outer correction): instead of loading bw, the
// kernel loads the main potential phi (from the buffer the main solve's
// control block names), b and the flags, forms the correction right-hand
// side b_e = r(phi) = resid_ff(...) rounded to float on every region cell
// (garbage only on the region's outermost ring, which the halo absorbs),
// sets bw = w * b_e, starts the correction from 0 and, when more launches
// follow, writes b_e and bw_e of the owned cells to rhs_e / bwe.
template <bool OMEGA1, bool FULL, bool CHECK, bool RINIT, int NW = NWARP>
__device__ __forceinline__ void jacobi_tile(
    int ri0, int rj0, uint32_t own, bool lead, const float* __restrict__ src, float* __restrict__ dst,
    const float* __restrict__ W, const float* __restrict__ BW, const float* __restrict__ rhs,
    const uint8_t* __restrict__ flags, float om1, PCtl* ctl, int k, int t0, int ns, float tol,
    int out_sel, int zero_init, Grid g, const float* __restrict__ mphi0,
    const float* __restrict__ mphi1, const PCtl* __restrict__ mctl, float* __restrict__ rhs_e,
    float* __restrict__ bwe) {
  __shared__ float4 xch[2][2][NW][32];
  __shared__ float red[NW];
  __shared__ int skip;
  pdl_enter();
  if (threadIdx.x == 0) {
    int sk = ctl->stop;
    if (!sk && CHECK && k > 0 && __uint_as_float(ctl->slots[k - 1]) < tol) {
      sk = 1;
      ctl->stop = 1;
    }
    skip = sk;
  }
  __syncthreads();
  if (skip) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gi0 = ri0 + warp * RT;
  const int gj = rj0 + lane * JT;
  const int oi0 = own & 255, oi1 = own >> 8 & 255, oj0 = own >> 16 & 255, oj1 = own >> 24;
  // gj is a multiple of 4 (rj0 is) and the pitch a multiple of 4: a 4-column
  // group is either wholly left of the grid or a 16-byte aligned read inside
  // the row.
  const bool colok = gj >= 0 && gj < g.P;
  float x[RT][JT], w[RT][JT], bw[RT][JT];
  uint32_t fr[RINIT ? RT : 1];
  const float* ph = RINIT ? (mctl->sel ? mphi1 : mphi0) : src;
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    int gi = gi0 + r;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), ww = a, bb = a;
    uint32_t f4 = 0;
    if (colok && gi >= 0 && gi < g.NX) {
      size_t c = (size_t)gi * g.P + gj;
      if (RINIT || !zero_init) a = *reinterpret_cast<const float4*>(ph + c);
      ww = *reinterpret_cast<const float4*>(W + c);
      bb = *reinterpret_cast<const float4*>((RINIT ? rhs : BW) + c);
      if (RINIT) f4 = *reinterpret_cast<const uint32_t*>(flags + c);
    }
    x[r][0] = a.x; x[r][1] = a.y; x[r][2] = a.z; x[r][3] = a.w;
    w[r][0] = ww.x; w[r][1] = ww.y; w[r][2] = ww.z; w[r][3] = ww.w;
    bw[r][0] = bb.x; bw[r][1] = bb.y; bw[r][2] = bb.z; bw[r][3] = bb.w;
    if (RINIT) fr[r] = f4;
#pragma unroll
    for (int q = 0; q < JT; ++q)
      if (gj + q >= g.NY) {
        x[r][q] = 0.0f;
        w[r][q] = 0.0f;
        bw[r][q] = 0.0f;
        if (RINIT) fr[r] &= ~(0xffu << (8 * q));
      }
  }
  const bool own_col = lane * JT >= oj0 && lane * JT < oj1;
  if (RINIT) {
    // Residual of the main potential held in x, with b in bw.
    xch[1][0][warp][lane] = make_float4(x[0][0], x[0][1], x[0][2], x[0][3]);
    xch[1][1][warp][lane] = make_float4(x[RT - 1][0], x[RT - 1][1], x[RT - 1][2], x[RT - 1][3]);
    __syncthreads();
    float4 u4 = warp > 0 ? xch[1][1][warp - 1][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 d4 = warp < NW - 1 ? xch[1][0][warp + 1][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    float prev[JT] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      float lf = __shfl_up_sync(0xffffffffu, x[r][JT - 1], 1);
      float rt = __shfl_down_sync(0xffffffffu, x[r][0], 1);
      float nxt[JT];
      if (r < RT - 1) {
#pragma unroll
        for (int q = 0; q < JT; ++q) nxt[q] = x[r + 1][q];
      } else {
        nxt[0] = d4.x; nxt[1] = d4.y; nxt[2] = d4.z; nxt[3] = d4.w;
      }
      float be[JT];
#pragma unroll
      for (int q = 0; q < JT; ++q) {
        uint8_t fl = (uint8_t)(fr[r] >> (8 * q));
        float left = q == 0 ? lf : x[r][q - 1];
        float right = q == JT - 1 ? rt : x[r][q + 1];
        be[q] = 0.0f;
        if (flag_active(fl))
          be[q] = resid_ff(bw[r][q], prev[q], nxt[q], left, right, (float)flag_count(fl), x[r][q]).hi;
      }
#pragma unroll
      for (int q = 0; q < JT; ++q) {
        prev[q] = x[r][q];
        bw[r][q] = w[r][q] * be[q];
      }
      if (rhs_e && own_col && warp * RT + r >= oi0 && warp * RT + r < oi1) {
        int gi = gi0 + r;
        if (gi < g.NX && gj < g.NY) {
          size_t c = (size_t)gi * g.P + gj;
          if (gj + JT <= g.NY) {
            *reinterpret_cast<float4*>(rhs_e + c) = make_float4(be[0], be[1], be[2], be[3]);
            *reinterpret_cast<float4*>(bwe + c) =
                make_float4(bw[r][0], bw[r][1], bw[r][2], bw[r][3]);
          } else {
#pragma unroll
            for (int q = 0; q < JT; ++q)
              if (gj + q < g.NY) {
                rhs_e[c + q] = be[q];
                bwe[c + q] = bw[r][q];
              }
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int q = 0; q < JT; ++q) x[r][q] = 0.0f;
    __syncthreads();  // xch[1] is read above and written again by the second sweep
  }
  float mx = 0.0f;
  auto sweep = [&](int sw, bool last) {
    const int buf = sw & 1;
    xch[buf][0][warp][lane] = make_float4(x[0][0], x[0][1], x[0][2], x[0][3]);
    xch[buf][1][warp][lane] = make_float4(x[RT - 1][0], x[RT - 1][1], x[RT - 1][2], x[RT - 1][3]);
    __syncthreads();
    float4 u4 = warp > 0 ? xch[buf][1][warp - 1][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 d4 = warp < NW - 1 ? xch[buf][0][warp + 1][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    float prev[JT] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      float lf = __shfl_up_sync(0xffffffffu, x[r][JT - 1], 1);
      float rt = __shfl_down_sync(0xffffffffu, x[r][0], 1);
      float nxt[JT];
      if (r < RT - 1) {
#pragma unroll
        for (int q = 0; q < JT; ++q) nxt[q] = x[r + 1][q];
      } else {
        nxt[0] = d4.x; nxt[1] = d4.y; nxt[2] = d4.z; nxt[3] = d4.w;
      }
      float nw[JT];
      float nbv[JT];
#pragma unroll
      for (int q = 0; q < JT; ++q) {
        float left = q == 0 ? lf : x[r][q - 1];
        float right = q == JT - 1 ? rt : x[r][q + 1];
        float nb = prev[q] + nxt[q] + left + right;  // (i-1) + (i+1) + (j-1) + (j+1)
        nbv[q] = nb;
        float y = __fmaf_rn(w[r][q], nb, bw[r][q]);
        if (!OMEGA1) y = __fmaf_rn(om1, x[r][q], y);
        nw[q] = y;
      }
      if (CHECK && last) {
        const int ri = warp * RT + r;
        const int gi = gi0 + r;
        if (own_col && ri >= oi0 && ri < oi1 && gi < g.NX && gj < g.NY) {
          size_t c = (size_t)gi * g.P + gj;
          float4 b4 = *reinterpret_cast<const float4*>(rhs + c);
          uint32_t f4 = *reinterpret_cast<const uint32_t*>(flags + c);
          float bq[JT] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
          for (int q = 0; q < JT; ++q) {
            uint8_t fl = (uint8_t)(f4 >> (8 * q));
            if (gj + q < g.NY && flag_active(fl)) {
              float rr = __fmaf_rn(-(float)flag_count(fl), x[r][q], bq[q] + nbv[q]);
              float ar = fabsf(rr);
              if (ar > mx) mx = ar;
            }
          }
        }
      }
#pragma unroll
      for (int q = 0; q < JT; ++q) {
        prev[q] = x[r][q];
        x[r][q] = nw[q];
      }
    }
  };
  if (FULL) {
#pragma unroll
    for (int sw = 0; sw < TMAX; ++sw) sweep(sw, sw == TMAX - 1);
  } else {
    for (int sw = 0; sw < ns; ++sw) sweep(sw, sw == ns - 1);
  }
  // Owned cells: rows [oi0, oi1), columns [oj0, oj1) of the region.
  if (own_col) {
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      int gi = gi0 + r;
      if (warp * RT + r < oi0 || warp * RT + r >= oi1 || gi >= g.NX || gj >= g.NY) continue;
      size_t c = (size_t)gi * g.P + gj;
      if (gj + JT <= g.NY) {
        *reinterpret_cast<float4*>(dst + c) = make_float4(x[r][0], x[r][1], x[r][2], x[r][3]);
      } else {
#pragma unroll
        for (int q = 0; q < JT; ++q)
          if (gj + q < g.NY) dst[c + q] = x[r][q];
      }
    }
  }
  if (CHECK) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    if (lane == 0) red[warp] = mx;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (CHECK) {
      float m = 0.0f;
#pragma unroll
      for (int q = 0; q < NW; ++q) m = fmaxf(m, red[q]);
      if (m > 0.0f) atomicMax(&ctl->slots[k], __float_as_uint(m));
    }
    if (lead) {
      ctl->sweeps = t0 + ns;
      ctl->last_launch = k;
      ctl->sel = out_sel;
    }
  }
}

// NW warps (8, or 4 on grids with fewer 8-warp regions than SMs): a region
// of 8 NW rows x 128 columns, so a small grid spreads over more SMs.
template <bool OMEGA1, bool FULL, bool CHECK, bool RINIT, int NW = NWARP>
__global__ void __launch_bounds__(32 * NW, 2 * NWARP / NW)
    k_jacobi_rb(const float* __restrict__ src, float* __restrict__ dst,
                const float* __restrict__ W, const float* __restrict__ BW,
                const float* __restrict__ rhs, const uint8_t* __restrict__ flags, float om1,
                PCtl* ctl, int k, int t0, int ns, float tol, int out_sel, int zero_init, Grid g,
                const float* __restrict__ mphi0, const float* __restrict__ mphi1,
                const PCtl* __restrict__ mctl, float* __restrict__ rhs_e,
                float* __restrict__ bwe) {
  constexpr int R = NW * RT;  // region rows
  jacobi_tile<OMEGA1, FULL, CHECK, RINIT, NW>((int)blockIdx.y * (R - 2 * TMAX), (int)blockIdx.x * OJ,
                                              span_own(blockIdx.y, g.NX, R) |
                                                  span_own(blockIdx.x, g.NY, RJ) << 16,
                                              blockIdx.x == 0 && blockIdx.y == 0, src, dst, W,
                                              BW, rhs, flags, om1, ctl, k, t0, ns, tol, out_sel,
                                              zero_init, g, mphi0, mphi1, mctl, rhs_e, bwe);
}

// A batch's Jacobi launch k of L: scene s runs its nl_s = ceil(iters_s / T)
// launches as the last nl_s of the L, the first of them with the remainder
// sweeps, so every scene ends in the same buffer.  The table lists the
// scenes with more sweeps first and launch k runs only the prefix of
// scenes that have started (a block of another would return at once).
// Each block's table entry gives its region's origin and owned window
// (fg_internal.cuh): regions at a scene's edges start or end there and own
// up to it, so a scene is cut into fewer regions than whole 48 x 112 tiles
// with halos on every side.  The tables are constant and read before
// jacobi_tile waits on the previous launch (programmatic dependent launch).
template <bool OMEGA1>
__global__ void __launch_bounds__(TB_THREADS, 2)
    kb_jacobi(const BTile* __restrict__ tiles, const BScene* __restrict__ sc,
              const float* __restrict__ src, float* __restrict__ dst, const float* __restrict__ W,
              const float* __restrict__ BW, const uint8_t* __restrict__ flags, float om1,
              PCtl* ctl, int k, int L, int T, int out_sel) {
  const BTile t = tiles[blockIdx.x];
  const BScene& s = sc[t.s];
  const int nl = (s.iters + T - 1) / T;
  const int first = L - nl;
  if (k < first) return;
  const int ns = k == first ? s.iters - (nl - 1) * T : T;
  const long long o = s.off;
  if (ns == TMAX)
    jacobi_tile<OMEGA1, true, false, false>(t.y, t.x, (uint32_t)t.pad, blockIdx.x == 0, src + o, dst + o, W + o,
                                            BW + o, nullptr, flags + o, om1, ctl, k, 0, ns, 0.0f,
                                            out_sel, k == first, s.g, nullptr, nullptr, nullptr,
                                            nullptr, nullptr);
  else
    jacobi_tile<OMEGA1, false, false, false>(t.y, t.x, (uint32_t)t.pad, blockIdx.x == 0, src + o, dst + o, W + o,
                                             BW + o, nullptr, flags + o, om1, ctl, k, 0, ns, 0.0f,
                                             out_sel, k == first, s.g, nullptr, nullptr, nullptr,
                                             nullptr, nullptr);
}


// ------------------------------------------------------------------ TMA-fed Jacobi
// The full 8-sweep launches without residual check, as a persistent kernel:
// each block (two per SM) walks tiles t = blockIdx.x, + gridDim.x, ...; the
// tensor memory accelerator copies the next tile's phi, w and w*b boxes (64 x
// 128, zero outside the arrays) into shared memory while the block sweeps the
// current tile in registers, so the loads no longer sit in front of the
// sweeps.  Same per-cell arithmetic as k_jacobi_rb, same results.
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
// The same without the arrival: the phase stays open.
__device__ __forceinline__ void mbar_expect_more(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void tma_load_2d(float* dst, const CUtensorMap* tm, int x, int y,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

constexpr int TILE_FLOATS = RI * RJ;  // one 64 x 128 box


// Waits for phase `parity` of the barrier for at most about a second (and a
// bounded number of polls); false when it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (int it = 0; it < MBAR_MAX_TRIES; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > MBAR_WAIT_NS) return false;
  }
  return false;
}

// After a wait gave up, before the block leaves: waits for its copy in
// flight for up to about eight more seconds, so a copy that is only slow
// lands before the block's shared memory passes to another block.  A copy
// still outstanding after nine seconds means the device is not progressing;
// the wait stays bounded all the same.
constexpr int MBAR_DRAIN_SLICES = 8;
__device__ __forceinline__ void mbar_drain(uint64_t* bar, unsigned parity) {
  for (int s = 0; s < MBAR_DRAIN_SLICES; ++s)
    if (mbar_wait_bounded(bar, parity)) return;
}

// The barrier of a tile's NW warps: the block's, or (OWN) a named one of
// theirs alone in a block with other warps.
template <int NW, bool OWN>
__device__ __forceinline__ void tile_barrier() {
  if (OWN)
    asm volatile("barrier.cta.sync 1, %0;" ::"n"(32 * NW) : "memory");
  else
    __syncthreads();
}
// One sweep of a tile in registers, with the arithmetic of jacobi_tile;
// buf alternates between consecutive sweeps (the row exchange is double
// buffered, one barrier per sweep).
template <bool OMEGA1, int NW = NWARP, bool OWN = false>
__device__ __forceinline__ void tile_sweep(float (&x)[RT][JT], const float (&w)[RT][JT],
                                           const float (&bw)[RT][JT], float om1,
                                           float4 (&xch)[2][2][NW][32], int warp, int lane,
                                           int buf) {
  xch[buf][0][warp][lane] = make_float4(x[0][0], x[0][1], x[0][2], x[0][3]);
  xch[buf][1][warp][lane] = make_float4(x[RT - 1][0], x[RT - 1][1], x[RT - 1][2], x[RT - 1][3]);
  tile_barrier<NW, OWN>();
  float4 u4 = warp > 0 ? xch[buf][1][warp - 1][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  float4 d4 = warp < NW - 1 ? xch[buf][0][warp + 1][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  float prev[JT] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    float lf = __shfl_up_sync(0xffffffffu, x[r][JT - 1], 1);
    float rt = __shfl_down_sync(0xffffffffu, x[r][0], 1);
    float nxt[JT];
    if (r < RT - 1) {
#pragma unroll
      for (int q = 0; q < JT; ++q) nxt[q] = x[r + 1][q];
    } else {
      nxt[0] = d4.x; nxt[1] = d4.y; nxt[2] = d4.z; nxt[3] = d4.w;
    }
    float nw[JT];
#pragma unroll
    for (int q = 0; q < JT; ++q) {
      float left = q == 0 ? lf : x[r][q - 1];
      float right = q == JT - 1 ? rt : x[r][q + 1];
      float nb = prev[q] + nxt[q] + left + right;  // (i-1) + (i+1) + (j-1) + (j+1)
      float y = __fmaf_rn(w[r][q], nb, bw[r][q]);
      if (!OMEGA1) y = __fmaf_rn(om1, x[r][q], y);
      nw[q] = y;
    }
#pragma unroll
    for (int q = 0; q < JT; ++q) {
      prev[q] = x[r][q];
      x[r][q] = nw[q];
    }
  }
}

// The TMAX sweeps of one tile.  hook(sw) runs before sweep sw (sw a
// constant after unrolling), so callers can spread latency-bound side work
// over the sweeps.
struct NoHook {
  __device__ __forceinline__ void operator()(int) const {}
};
template <bool OMEGA1, typename Hook = NoHook, int NW = NWARP, bool OWN = false>
__device__ __forceinline__ void tile_sweeps(float (&x)[RT][JT], const float (&w)[RT][JT],
                                            const float (&bw)[RT][JT], float om1,
                                            float4 (&xch)[2][2][NW][32], int warp, int lane,
                                            Hook hook = Hook()) {
#pragma unroll
  for (int sw = 0; sw < TMAX; ++sw) {
    hook(sw);
    tile_sweep<OMEGA1, NW, OWN>(x, w, bw, om1, xch, warp, lane, sw & 1);
  }
}

// 16 bytes from global to shared memory without passing through registers;
// the bytes past src_bytes (0 or 16) are zero-filled.
__device__ __forceinline__ void cp_async16(float* smem, const float* gmem, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem)), "l"(gmem),
               "r"(src_bytes)
               : "memory");
}

// A batch's Jacobi launch k (as kb_jacobi, same regions, same per-cell
// arithmetic, same results) as a persistent kernel: block b runs the
// started scenes' regions b, b + G, ... in turn, and while it sweeps one,
// its threads' asynchronous copies bring the next region's boxes (phi, w,
// w*b; zero outside the scene's rows and pitch) into shared memory, so the
// loads no longer sit in front of the sweeps.  The tables are constant;
// the copies read the previous launch's result, after the programmatic
// wait.
template <bool OMEGA1>
__global__ void __launch_bounds__(TB_THREADS, 2)
    kb_jacobi_pf(const BTile* __restrict__ tiles, const BScene* __restrict__ sc, int n,
                 const float* __restrict__ src, float* __restrict__ dst,
                 const float* __restrict__ W, const float* __restrict__ BW, float om1, PCtl* ctl,
                 int k, int L, int T, int out_sel) {
  extern __shared__ __align__(128) float4 pbuf4[];  // [3][RI][RJ] floats: phi, w, w*b
  float* pbuf = reinterpret_cast<float*>(pbuf4);
  __shared__ float4 xch[2][2][NWARP][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // Thread tid copies float4 q = tid + 256 m (m < 8) of each box: region
  // row q / 32, columns 4 (q % 32) .. + 3, for a region starting at (ri0,
  // rj0) of a scene of NX rows of pitch P at element offset off.
  auto issue_at = [&](int ri0, int rj0, int NX, int P, long long off, bool zi) {
    const float* xs = src + off;
    const float* ws = W + off;
    const float* bs = BW + off;
#pragma unroll
    for (int m = 0; m < TILE_FLOATS / 4 / TB_THREADS; ++m) {
      const int q = tid + TB_THREADS * m;
      const int row = q / (RJ / JT), col = JT * (q % (RJ / JT));
      const int gi = ri0 + row, gj = rj0 + col;
      const bool ok = gi >= 0 && gi < NX && gj >= 0 && gj < P;
      const size_t c = ok ? (size_t)gi * P + gj : 0;
      float* d = pbuf + row * RJ + col;
      cp_async16(d, xs + c, ok && !zi ? 16 : 0);
      cp_async16(d + TILE_FLOATS, ws + c, ok ? 16 : 0);
      cp_async16(d + 2 * TILE_FLOATS, bs + c, ok ? 16 : 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // (A scene's first launch starts from 0: its phi box is not copied.)
  auto issue = [&](int i) {
    const BTile t = tiles[i];
    const BScene& s = sc[t.s];
    issue_at(t.y, t.x, s.g.NX, s.g.P, s.off, k == L - (s.iters + T - 1) / T);
  };
  int i = blockIdx.x;
  pdl_enter();
  if (i < n) issue(i);
  while (i < n) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // every thread's copies of region i landed
    const BTile t = tiles[i];
    const BScene& s = sc[t.s];
    const Grid g = s.g;
    const int nl = (s.iters + T - 1) / T;
    const int ns = k == L - nl ? s.iters - (nl - 1) * T : T;
    const int gi0 = t.y + warp * RT, gj = t.x + lane * JT;
    float x[RT][JT], w[RT][JT], bw[RT][JT];
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const int o = (warp * RT + r) * RJ + lane * JT;
      const float4 a = *reinterpret_cast<const float4*>(pbuf + o);
      const float4 ww = *reinterpret_cast<const float4*>(pbuf + TILE_FLOATS + o);
      const float4 bb = *reinterpret_cast<const float4*>(pbuf + 2 * TILE_FLOATS + o);
      x[r][0] = a.x; x[r][1] = a.y; x[r][2] = a.z; x[r][3] = a.w;
      w[r][0] = ww.x; w[r][1] = ww.y; w[r][2] = ww.z; w[r][3] = ww.w;
      bw[r][0] = bb.x; bw[r][1] = bb.y; bw[r][2] = bb.z; bw[r][3] = bb.w;
#pragma unroll
      for (int q = 0; q < JT; ++q)
        if (gj + q >= g.NY) {  // the pitch padding: outside the grid
          x[r][q] = 0.0f;
          w[r][q] = 0.0f;
          bw[r][q] = 0.0f;
        }
    }
    const int nx = i + gridDim.x;
    if (i == 0 && tid == 0) ctl->sweeps = ns;
    // (The host launches the started scenes' regions only; a region of a
    // scene that has not started would be left alone.)
    const bool run = k >= L - nl;
    if (run && ns == TMAX) {
      // The next region's table entry is read before sweep 0, its scene's
      // before sweep 1, and its copies start before sweep 2 (sweep 0's
      // barrier has ordered every thread's register fill before them), so
      // neither the dependent table reads nor the copies sit in front of a
      // sweep.
      BTile tn{};
      int nNX = 0, nP = 0, nit = 0;
      long long noff = 0;
      auto hook = [&](int sw) {
        if (nx >= n) return;
        if (sw == 0) {
          tn = tiles[nx];
        } else if (sw == 1) {
          const BScene& sn = sc[tn.s];
          nNX = sn.g.NX;
          nP = sn.g.P;
          noff = sn.off;
          nit = sn.iters;
        } else if (sw == 2) {
          issue_at(tn.y, tn.x, nNX, nP, noff, k == L - (nit + T - 1) / T);
        }
      };
      tile_sweeps<OMEGA1>(x, w, bw, om1, xch, warp, lane, hook);
    } else {
      __syncthreads();  // the boxes are in registers: the buffer takes the next region
      if (nx < n) issue(nx);
      if (run)
        for (int sw = 0; sw < ns; ++sw) tile_sweep<OMEGA1>(x, w, bw, om1, xch, warp, lane, sw & 1);
    }
    const uint32_t own = (uint32_t)t.pad;
    const int oi0 = own & 255, oi1 = own >> 8 & 255, oj0 = own >> 16 & 255, oj1 = own >> 24;
    if (run && lane * JT >= oj0 && lane * JT < oj1) {
      float* xd = dst + s.off;
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const int gi = gi0 + r;
        if (warp * RT + r < oi0 || warp * RT + r >= oi1 || gi >= g.NX || gj >= g.NY) continue;
        const size_t c = (size_t)gi * g.P + gj;
        if (gj + JT <= g.NY) {
          *reinterpret_cast<float4*>(xd + c) = make_float4(x[r][0], x[r][1], x[r][2], x[r][3]);
        } else {
#pragma unroll
          for (int q = 0; q < JT; ++q)
            if (gj + q < g.NY) xd[c + q] = x[r][q];
        }
      }
    }
    i = nx;
  }
  if (blockIdx.x == 0 && tid == 0) {
    ctl->last_launch = k;
    ctl->sel = out_sel;
  }
}

template <bool OMEGA1>
__global__ void __launch_bounds__(TB_THREADS, 2)
    k_jacobi_tma(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw,
                 const __grid_constant__ CUtensorMap tmb, float* __restrict__ dst, float om1,
                 PCtl* ctl, int k, int t0, int out_sel, int zero_init, Grid g, int ntx,
                 int ntiles, int* err, int stall_tile) {
  extern __shared__ __align__(128) float4 tbuf4[];  // [3][RI][RJ] floats: phi, w, w*b
  float* tbuf = reinterpret_cast<float*>(tbuf4);
  __shared__ float4 xch[2][2][NWARP][32];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_skip;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    s_skip = ctl->stop;
    if (!s_skip) mbar_init(&bar, 1);
  }
  __syncthreads();
  if (s_skip) return;
  const unsigned bytes = (zero_init ? 2u : 3u) * TILE_FLOATS * 4u;
  auto issue = [&](int t) {
    const int ty = t / ntx, tx = t - ty * ntx;
    const int x = tx * OJ - TMAX, y = ty * OI - TMAX;  // x: a multiple of 4 floats (16 bytes)
    // Order this block's earlier shared-memory reads before the copy's writes.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // Fault injection: tile `stall_tile` expects 16 bytes more than its
    // copies bring, so its barrier phase never completes and the bounded
    // wait below gives up (every copy issued still lands).
    mbar_expect_tx(&bar, bytes + (t == stall_tile ? 16u : 0u));
    if (!zero_init) tma_load_2d(tbuf, &tmx, x, y, &bar);
    tma_load_2d(tbuf + TILE_FLOATS, &tmw, x, y, &bar);
    tma_load_2d(tbuf + 2 * TILE_FLOATS, &tmb, x, y, &bar);
  };
  if (tid == 0 && (int)blockIdx.x < ntiles) issue(blockIdx.x);
  unsigned parity = 0;
  const bool own_col = lane * JT >= TMAX && lane * JT < RJ - TMAX;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const bool landed = mbar_wait_bounded(&bar, parity);
    if (__syncthreads_or(!landed)) {
      // A copy did not land in time (the whole block agrees): flag it, let
      // it land (bounded), stop.  The next tile's copy is issued only after
      // this one landed, so nothing else is in flight.
      if (tid == 0) {
        atomicExch(&ctl->pad[0], 1);
        if (err) atomicExch(err, 1);
      }
      if (!landed) mbar_drain(&bar, parity);
      return;
    }
    parity ^= 1u;
    const int ty = t / ntx, tx = t - ty * ntx;
    const int gi0 = ty * OI - TMAX + warp * RT;
    const int gj = tx * OJ - TMAX + lane * JT;
    float x[RT][JT], w[RT][JT], bw[RT][JT];
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const int o = (warp * RT + r) * RJ + lane * JT;
      float4 a = zero_init ? make_float4(0.f, 0.f, 0.f, 0.f)
                           : *reinterpret_cast<const float4*>(tbuf + o);
      float4 ww = *reinterpret_cast<const float4*>(tbuf + TILE_FLOATS + o);
      float4 bb = *reinterpret_cast<const float4*>(tbuf + 2 * TILE_FLOATS + o);
      x[r][0] = a.x; x[r][1] = a.y; x[r][2] = a.z; x[r][3] = a.w;
      w[r][0] = ww.x; w[r][1] = ww.y; w[r][2] = ww.z; w[r][3] = ww.w;
      bw[r][0] = bb.x; bw[r][1] = bb.y; bw[r][2] = bb.z; bw[r][3] = bb.w;
#pragma unroll
      for (int q = 0; q < JT; ++q)
        if (gj + q >= g.NY) {  // the pitch padding (outside the grid: zero-filled)
          x[r][q] = 0.0f;
          w[r][q] = 0.0f;
          bw[r][q] = 0.0f;
        }
    }
    __syncthreads();  // the boxes are in registers: the buffer takes the next tile
    if (tid == 0 && t + (int)gridDim.x < ntiles) issue(t + gridDim.x);
    tile_sweeps<OMEGA1>(x, w, bw, om1, xch, warp, lane);
    if (own_col && warp >= TMAX / RT && warp < NWARP - TMAX / RT) {
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        int gi = gi0 + r;
        if (gi >= g.NX || gj >= g.NY) continue;
        size_t c = (size_t)gi * g.P + gj;
        if (gj + JT <= g.NY) {
          *reinterpret_cast<float4*>(dst + c) = make_float4(x[r][0], x[r][1], x[r][2], x[r][3]);
        } else {
#pragma unroll
          for (int q = 0; q < JT; ++q)
            if (gj + q < g.NY) dst[c + q] = x[r][q];
        }
      }
    }
  }
  if (tid == 0 && blockIdx.x == 0) {
    ctl->sweeps = t0 + TMAX;
    ctl->last_launch = k;
    ctl->sel = out_sel;
  }
}

// ------------------------------------------------------------------ dataflow Jacobi
// A whole fixed-count solve (nphase launches of TMAX sweeps) as one
// cooperative persistent kernel.  Items (phase, tile) are numbered phase
// by phase and handed out by an atomic counter (done[ntiles]): a block
// claims its next item while it sweeps the current one, so the tensor
// memory accelerator copies the next boxes meanwhile.  Item (ph, t) starts
// once the up to nine tiles whose owned cells its region reads have
// finished phase ph - 1 (done[n] >= ph; done[t] = ph + 1 is published after
// a fence that follows the tile's stores).  That one wait covers both
// hazards of the ping-pong buffers: the neighbours' phase ph - 1 results
// are in src(ph), and they no longer read src(ph - 1), which this item
// overwrites.  Items are claimed in increasing order and depend only on
// smaller ones, so the smallest unfinished item can always proceed (all
// blocks are resident: cooperative launch).  No block idles at a launch
// boundary or in a partial last wave.  Same per-cell arithmetic, same
// results.

// Whether the tiles around t (3 x 3, clipped to the tile grid) finished
// phase ph - 1.  All 32 lanes of a warp call it: lane l < 9 reads the flag
// of neighbour (l / 3 - 1, l % 3 - 1) with a relaxed load; an acquire fence
// follows once all are set (one in every poll cost more than the poll).
__device__ __forceinline__ bool flow_ready_warp(const int* done, int ph, int t, int ntx, int nty,
                                                int lane) {
  bool ok = true;
  if (ph > 0 && lane < 9) {
    const int ty = t / ntx, tx = t - ty * ntx;
    const int y = ty + lane / 3 - 1, x = tx + lane % 3 - 1;
    if (y >= 0 && y < nty && x >= 0 && x < ntx) {
      int v;
      asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(done + y * ntx + x)
                   : "memory");
      ok = v >= ph;
    }
  }
  if (!__all_sync(0xffffffffu, ok)) return false;
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  __syncwarp();  // (a vote orders no memory: the lanes' flags before lane 0's copy)
  return true;
}

// Tiles of 12 warps, one block an SM: 96 x 128 regions owning 80 x 112 cells
// (73% of the swept cells; 66% with 8 warps and 48 x 112).  A thirteenth warp
// does everything that waits: it claims the next item, starts its w and w*b
// copies as soon as the sweeping warps have taken the present item into
// registers, its phi copy once its neighbours' flags are set, and publishes
// each tile once the warps have stored it; the sweeping warps meet only on a
// barrier of their own.  (It belongs to a warpgroup whose registers go to the
// other three: 12 x 32 x 152 + 4 x 32 x 40 = 63,488 of the 512 x 128 = 65,536
// the block is launched with.)  Bound by the sweeps' instructions: of an item's
// 8,000 cycles 5,430 are sweeps, 1,250 the fill from shared memory and 1,000
// the stores; 48 MB of boxes a phase at 2048 x 2048 stay in L2.  Each further 8
// sweeps (us), against two 8-warp blocks an SM whose own threads waited for
// boxes and flags: 2048 x 2048 13.6 (16.9), 1300 x 1300 8.5 (10.7), 1500 x 1100
// 8.2 (10.5), 1700 x 1700 9.7 (12.5), 3000 x 2500 26.9 (32.2); with the
// launch's ends a phase of 25 at 2048 x 2048 takes 14.0.  A fence in every
// poll of the flags and the timer read on every turn held the phi copy back
// 5,000 cycles an item (15.0 at 2048 x 2048).
constexpr int FW = 12, FI = FW * RT, FO = FI - 2 * TMAX, FLOW_FLOATS = FI * RJ;
constexpr int FLOW_THREADS = 32 * (FW + 4);

// Whether phase `parity` has completed, without waiting (try_wait suspends).
__device__ __forceinline__ bool mbar_test(uint64_t* bar, unsigned parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same for a whole warp: its lanes test one by one and may not see the same,
// but what follows (a claim's shuffle, the next vote) needs all of them.
__device__ __forceinline__ bool warp_test(uint64_t* bar, unsigned parity) {
  return __all_sync(0xffffffffu, mbar_test(bar, parity)) != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <bool OMEGA1>
__global__ void __launch_bounds__(FLOW_THREADS, 1)
    k_jacobi_flow(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1,
                  const __grid_constant__ CUtensorMap tmw, const __grid_constant__ CUtensorMap tmb,
                  float* __restrict__ x0, float* __restrict__ x1, float om1, PCtl* ctl,
                  int* __restrict__ done, int nphase, int zero_first, Grid g, int ntx, int nty,
                  int* err, int stall_tile) {
  extern __shared__ __align__(128) float4 tbuf4[];  // [3][FI][RJ] floats: phi, w, w*b
  float* tbuf = reinterpret_cast<float*>(tbuf4);
  __shared__ float4 xch[2][2][FW][32];
  // full: an item's boxes have landed (and s_item names it); empty: the
  // sweeping warps hold it in registers; stored: they have stored it.
  __shared__ __align__(8) uint64_t full, empty, stored;
  __shared__ int s_item;
  __shared__ unsigned s_lost;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ntiles = ntx * nty, total = ntiles * nphase;
  int* counter = done + ntiles;
  if (tid == 0) {
    mbar_init(&full, 1);
    mbar_init(&empty, FW);
    mbar_init(&stored, FW);
    s_item = 0;
    s_lost = UINT_MAX;
  }
  __syncthreads();
  bool fail = false;
  if (warp >= FW) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp > FW) return;
    auto claim = [&] {
      int i = 0;
      if (lane == 0) i = atomicAdd(counter, 1);
      return __shfl_sync(0xffffffffu, i, 0);
    };
    // With two tiles or more for each block a neighbour's flag is set well
    // before it is needed, and the next claim goes before the publication of
    // the tile just stored (2048 x 2048, 494 tiles on 152 blocks: 13.5 us per
    // phase against 14.4); with fewer the neighbours wait for that publication,
    // and it goes first (1300 x 1300, 204 tiles: 8.5 us against 9.3).
    const bool deep = ntiles >= 2 * (int)gridDim.x;
    int cur_ph = 0, cur_t = -1, next = claim();
    // The item whose boxes may be landing (its phase of `full`), and whether
    // its last box has been sent for.
    bool flight = false, whole = true;
    unsigned flight_n = 0;
    for (unsigned n = 0;; ++n) {
      // Item `next` goes into the buffer when it is free; the item before it
      // is swept meanwhile.  Everything about it that needs no buffer (its
      // place, the neighbours' flags) is known by then.
      const bool have = next < total;
      const int ph = next / ntiles, t = next - ph * ntiles, ty = t / ntx, tx = t - ty * ntx;
      const int x = tx * OJ - TMAX, y = ty * FO - TMAX;  // x: a multiple of 4 floats (16 bytes)
      const bool zi = zero_first && ph == 0;  // phi starts from 0: not copied
      int after = 0;
      bool unused = n == 0, ready = !have, copied = !have, told = cur_t < 0;
      bool taken = false;
      unsigned long long t0 = 0;
      for (int it = 0;; ++it) {
        if (!taken && (unused || warp_test(&empty, (n - 1) & 1))) {
          taken = true;
          flight = have;
          flight_n = n;
          whole = !have;
          if (lane == 0) {
            s_item = next;
            if (have) {
              // The warps' earlier shared-memory reads before the copies' writes.
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
              mbar_expect_more(&full, 2u * FLOW_FLOATS * 4u);
              tma_load_2d(tbuf + 2 * FLOW_FLOATS, &tmb, x, y, &full);
              tma_load_2d(tbuf + FLOW_FLOATS, &tmw, x, y, &full);
            } else {
              mbar_arrive(&full);
            }
          }
        }
        if (!ready) ready = flow_ready_warp(done, ph, t, ntx, nty, lane);
        if (!copied && ready && taken) {
          if (lane == 0) {
            if (zi) {
              mbar_arrive(&full);
            } else {
              // The neighbours' (generic) stores, acquired above, before the copy's reads.
              asm volatile("fence.proxy.async.global;" ::: "memory");
              mbar_expect_tx(&full, FLOW_FLOATS * 4u);
              tma_load_2d(tbuf, (ph & 1) ? &tm1 : &tm0, x, y, &full);
            }
          }
          copied = whole = true;
        }
        if (taken && !told && warp_test(&stored, (n - 1) & 1)) {
          if (deep) after = claim();
          if (lane == 0 && cur_t != stall_tile) {  // (a stalled tile: fault injection)
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(done + cur_t), "r"(cur_ph + 1)
                         : "memory");
          }
          told = true;
        }
        if (taken && copied && told) break;
        if ((it & 63) == 63) {  // (the timer is slow to read)
          const unsigned long long now = global_ns();
          if (t0 == 0) t0 = now;
          if (__any_sync(0xffffffffu, it >= MBAR_MAX_TRIES || now - t0 > MBAR_WAIT_NS)) {
            fail = true;
            break;
          }
        }
      }
      if (fail || !have) break;
      next = n == 0 || !deep ? claim() : after;
      cur_ph = ph;
      cur_t = t;
    }
    if (fail && flight && lane == 0) {
      // A wait gave up.  An item without its phi is ended here, marked lost, so
      // that the warps that wait for it leave too; then the copies still
      // landing.  (Left incomplete, the phase held the block for 9 s more.)
      if (!whole) {
        atomicMin(&s_lost, flight_n);
        mbar_arrive(&full);
      }
      mbar_drain(&full, flight_n & 1);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
    const bool own_col = lane * JT >= TMAX && lane * JT < RJ - TMAX;
    for (unsigned n = 0;; ++n) {
      const bool landed = __all_sync(0xffffffffu, mbar_wait_bounded(&full, n & 1));
      // A warp whose wait gave up sweeps whatever the buffer holds, as item 0,
      // and a warp that has seen the end meets the same barriers before it
      // leaves: whatever each warp saw, all of them pass TMAX barriers here, so
      // none is left waiting in one.  s_lost names the first item given up:
      // set before the first barrier, it is seen by all after the last, and a
      // faster warp (or the thirteenth) that gives up the next item neither
      // makes a slower one leave before that item's barriers nor hides that
      // this one is lost.
      const int item = landed ? s_item : 0;
      if (!landed) atomicMin(&s_lost, n);
      if (item >= total) {
#pragma unroll 1
        for (int sw = 0; sw < TMAX; ++sw) tile_barrier<FW, true>();
        break;
      }
      const int ph = item / ntiles, t = item - ph * ntiles;
      const int ty = t / ntx, tx = t - ty * ntx;
      const int gi0 = ty * FO - TMAX + warp * RT;
      const int gj = tx * OJ - TMAX + lane * JT;
      const bool zi = zero_first && ph == 0;
      float x[RT][JT], w[RT][JT], bw[RT][JT];
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const int o = (warp * RT + r) * RJ + lane * JT;
        float4 a = zi ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(tbuf + o);
        float4 ww = *reinterpret_cast<const float4*>(tbuf + FLOW_FLOATS + o);
        float4 bb = *reinterpret_cast<const float4*>(tbuf + 2 * FLOW_FLOATS + o);
        x[r][0] = a.x; x[r][1] = a.y; x[r][2] = a.z; x[r][3] = a.w;
        w[r][0] = ww.x; w[r][1] = ww.y; w[r][2] = ww.z; w[r][3] = ww.w;
        bw[r][0] = bb.x; bw[r][1] = bb.y; bw[r][2] = bb.z; bw[r][3] = bb.w;
#pragma unroll
        for (int q = 0; q < JT; ++q)
          if (gj + q >= g.NY) {  // the pitch padding (outside the grid: zero-filled)
            x[r][q] = 0.0f;
            w[r][q] = 0.0f;
            bw[r][q] = 0.0f;
          }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty);
      tile_sweeps<OMEGA1, NoHook, FW, true>(x, w, bw, om1, xch, warp, lane);
      if (*(volatile unsigned*)&s_lost <= n) {
        fail = true;
        break;
      }
      float* dst = (ph & 1) ? x0 : x1;
      if (own_col && warp >= TMAX / RT && warp < FW - TMAX / RT) {
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          int gi = gi0 + r;
          if (gi >= g.NX || gj >= g.NY) continue;
          size_t c = (size_t)gi * g.P + gj;
          if (gj + JT <= g.NY) {
            *reinterpret_cast<float4*>(dst + c) = make_float4(x[r][0], x[r][1], x[r][2], x[r][3]);
          } else {
#pragma unroll
            for (int q = 0; q < JT; ++q)
              if (gj + q < g.NY) dst[c + q] = x[r][q];
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&stored);
    }
  }
  if (fail && lane == 0) {
    atomicExch(&ctl->pad[0], 1);
    if (err) atomicExch(err, 1);
  }
  if (tid == 0 && blockIdx.x == 0 && nphase > 0) {
    ctl->sweeps = nphase * TMAX;
    ctl->last_launch = nphase - 1;
    ctl->sel = ((nphase - 1) & 1) ? 0 : 1;
  }
}

// ------------------------------------------------------------------ resident Jacobi
// A whole fixed-count solve with every region in registers from the first
// sweep to the last: one block per region (the placement of k_jacobi_rb:
// span_count, span_own), all resident at once (a cooperative launch), 8
// sweeps between exchanges.  Only the values that a neighbour's halo holds
// leave a block: the 8 rows of its first and last owned warps and the 8
// columns of lanes 2, 3 and 28, 29, written as 16-byte packets of three
// values and a tag.  A packet is stored and read whole (one 128-bit access
// each way) and its tag names the solve and the phase, so the receiver polls
// the data itself: no fence, flag or grid barrier.  Two slots by phase
// parity suffice: a neighbour writes phase p + 2 only after it has this
// block's p + 1, sent after its p was read.  Same per-cell arithmetic as the
// other kernels, the same bits.
//
// For grids whose regions fit the GPU at once.  Bound by the sweeps' own
// latency (1.35 us per 8 sweeps for 4 warps, each alone on its scheduler) and
// the packets' flight (0.7 us): 196 warp instructions a warp and sweep, the
// exchange included, in 30 % of the issue slots of the SMs that hold a region
// of 4 warps (128^2, 40 sweeps), 189 in 46 % with 8 warps (512x256, 100
// sweeps); per issue 0.8-0.9 warps wait on the packets, 0.2-0.4 on the sweeps'
// barrier.  With 8-warp regions the registers decide: 128 a thread
// (two blocks an SM) spill and take 3.9 us, 190 take 3.0.  Barriers split
// into arrive and wait around the inner rows measured slower (2.2 against
// 1.35 us without exchange), as did the boundary rows computed first (1.41).
constexpr int JP = (RT * JT + 2) / 3;        // packets of a thread's 8 x 4 cells
constexpr int JROWS = 2 * JP * 32;           // a slot's row packets: first, last owned warp
template <int NW>
struct JSlot {
  static constexpr int N = JROWS + 2 * NW * JP * 2;  // + the column packets: left, right lanes
  static constexpr int PER = (N + 32 * NW - 1) / (32 * NW);  // a thread's share of the items
};

struct JResArgs {
  float* x;                    // the solution
  const float *W, *BW;
  float om1;
  int iters;
  unsigned* epoch;             // per block: the tag its last solve ended on (all alike)
  unsigned inc;                // the launch's phases (a batch: of its longest solve)
  int cap;                     // a batch: the regions of its largest group
  uint4* pkt;                  // [region][parity][JSlot::N]
  PCtl* ctl;
  const JRegion* regions;      // batch: the launch's regions (nullptr: one grid)
  Grid g;
  int ntx, nty;
  int last_launch;             // what ctl->last_launch reports
  int* err;
  int stall;                   // fault injection: a region that sends nothing
};

__device__ __forceinline__ void jst_pkt(uint4* p, float x, float y, float z, unsigned tag) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
      "mov.b128 t, {a, b};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "f"(x), "f"(y), "f"(z), "r"(tag)
      : "memory");
}
__device__ __forceinline__ uint4 jld_pkt(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .b128 t;\n\t.reg .b64 a, b;\n\tld.relaxed.gpu.global.b128 t, [%4];\n\t"
      "mov.b128 {a, b}, t;\n\tmov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}

// MB: blocks per SM the registers are limited for.
template <bool OMEGA1, int NW, bool BATCH, int MB>
__global__ void __launch_bounds__(32 * NW, MB) k_jacobi_res(JResArgs a) {
  using S = JSlot<NW>;
  constexpr int NT = 32 * NW, R = NW * RT;
  __shared__ float4 xch[2][2][NW][32];
  __shared__ float stage[3 * S::N];
  __shared__ int from[S::N];
  __shared__ JRegion rg;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, id = blockIdx.x;
  const unsigned epoch = a.epoch[id];
  if (BATCH) {
    if (tid == 0) rg = a.regions[id];
  } else if (tid == 0) {
    const int ty = id / a.ntx, tx = id - ty * a.ntx;
    rg.NX = a.g.NX;
    rg.NY = a.g.NY;
    rg.P = a.g.P;
    rg.iters = a.iters;
    rg.off = 0;
    rg.r0 = ty * (R - 2 * TMAX);
    rg.c0 = tx * OJ;
    rg.own = span_own(ty, a.g.NX, R) | span_own(tx, a.g.NY, RJ) << 16;
    rg.ntx = a.ntx;
    rg.up = ty > 0;
    rg.down = ty < a.nty - 1;
    rg.left = tx > 0;
    rg.right = tx < a.ntx - 1;
  }
  __syncthreads();
  const int gi0 = rg.r0 + warp * RT, gj = rg.c0 + lane * JT;
  float x[RT][JT], w[RT][JT], bw[RT][JT];
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    float4 ww = make_float4(0.f, 0.f, 0.f, 0.f), bb = ww;
    if (gi0 + r < rg.NX && gj < rg.P) {
      const size_t c = (size_t)rg.off + (size_t)(gi0 + r) * rg.P + gj;
      ww = *reinterpret_cast<const float4*>(a.W + c);
      bb = *reinterpret_cast<const float4*>(a.BW + c);
    }
    w[r][0] = ww.x; w[r][1] = ww.y; w[r][2] = ww.z; w[r][3] = ww.w;
    bw[r][0] = bb.x; bw[r][1] = bb.y; bw[r][2] = bb.z; bw[r][3] = bb.w;
#pragma unroll
    for (int q = 0; q < JT; ++q) {
      x[r][q] = 0.0f;
      if (gj + q >= rg.NY) {  // the pitch padding: outside the grid
        w[r][q] = 0.0f;
        bw[r][q] = 0.0f;
      }
    }
  }
  // Where each item the block receives lies, relative to its own slots
  // (INT_MIN: not needed).  Items are numbered as a slot's packets: the rows
  // above and below (all 32 lanes; the corners from the diagonal regions),
  // then the columns left and right of the rows no halo covers.
  for (int k = tid; k < S::N; k += NT) {
    int at = INT_MIN;
    if (k < JROWS) {
      const int side = k / (JP * 32), rest = k - side * (JP * 32), l = rest & 31;
      const int dx = l < 2 && rg.left ? -1 : l >= 30 && rg.right ? 1 : 0;
      if (side ? rg.down : rg.up)
        at = ((side ? rg.ntx : -rg.ntx) + dx) * 2 * S::N + (1 - side) * JP * 32 + rest - 28 * dx;
    } else {
      const int c = k - JROWS, side = c / (NW * JP * 2), wr = (c / (JP * 2)) % NW;
      const bool covered = (wr == 0 && rg.up) || (wr == NW - 1 && rg.down);
      if ((side ? rg.right : rg.left) && !covered)
        at = (side ? 2 * S::N : -2 * S::N) + JROWS + (1 - side) * NW * JP * 2 +
             (c - side * NW * JP * 2);
    }
    from[k] = at;
  }
  const bool up = rg.up, down = rg.down, left = rg.left, right = rg.right;
  const int iters = rg.iters;
  uint4* own_slot = a.pkt + (size_t)id * 2 * S::N;
  const int nph = (iters + TMAX - 1) / TMAX;
  bool fail = false;
  for (int ph = 0; ph < nph; ++ph) {
    const int ns = iters - ph * TMAX;
    if (ns >= TMAX) {
      tile_sweeps<OMEGA1, NoHook, NW>(x, w, bw, a.om1, xch, warp, lane);
    } else {
      for (int sw = 0; sw < ns; ++sw)
        tile_sweep<OMEGA1, NW>(x, w, bw, a.om1, xch, warp, lane, sw & 1);
    }
    if (ph + 1 == nph) break;
    const unsigned tag = epoch + 1u + (unsigned)ph;
    uint4* slot = own_slot + (ph & 1) * S::N;
    auto val = [&](int k) { return k < RT * JT ? x[k / JT][k % JT] : 0.0f; };
    if (id != a.stall) {
      // The rows of the first and last owned warps, for the regions above
      // and below; the columns for those left and right.
      if (warp == 1 && up) {
#pragma unroll
        for (int m = 0; m < JP; ++m)
          jst_pkt(slot + m * 32 + lane, val(3 * m), val(3 * m + 1), val(3 * m + 2), tag);
      }
      if (warp == NW - 2 && down) {
#pragma unroll
        for (int m = 0; m < JP; ++m)
          jst_pkt(slot + (JP + m) * 32 + lane, val(3 * m), val(3 * m + 1), val(3 * m + 2), tag);
      }
      const int cl = lane - 2, cr = lane - 28;  // 0, 1: a lane whose columns go left / right
      const bool goes_l = (unsigned)cl < 2u && left, goes_r = (unsigned)cr < 2u && right;
      if (goes_l || goes_r) {
        uint4* d = slot + JROWS + ((goes_r ? NW : 0) + warp) * JP * 2 + (goes_r ? cr : cl);
#pragma unroll
        for (int m = 0; m < JP; ++m)
          jst_pkt(d + m * 2, val(3 * m), val(3 * m + 1), val(3 * m + 2), tag);
      }
    }
    // Receive: each thread polls its items into the staging area.
    uint4 v[S::PER];
    auto source = [&](int m) {
      const int k = tid + NT * m;
      return k < S::N ? from[k] : INT_MIN;
    };
    bool miss = false;
#pragma unroll
    for (int m = 0; m < S::PER; ++m) {
      const int at = source(m);
      v[m].w = tag;
      if (at != INT_MIN) v[m] = jld_pkt(slot + at);
    }
#pragma unroll
    for (int m = 0; m < S::PER; ++m) miss = miss || v[m].w != tag;
    if (miss) {
      unsigned long long t0 = 0;
      for (int it = 1; miss; ++it) {
        miss = false;
#pragma unroll
        for (int m = 0; m < S::PER; ++m) {
          if (v[m].w != tag) v[m] = jld_pkt(slot + source(m));
          miss = miss || v[m].w != tag;
        }
        if ((it & 63) == 0) {  // (the timer is slow to read)
          const unsigned long long now = global_ns();
          if (t0 == 0) t0 = now;
          if (it >= MBAR_MAX_TRIES || now - t0 > MBAR_WAIT_NS) break;
        }
      }
      fail = miss;
    }
#pragma unroll
    for (int m = 0; m < S::PER; ++m)
      if (source(m) != INT_MIN) {
        float* d = stage + 3 * (tid + NT * m);
        d[0] = __uint_as_float(v[m].x);
        d[1] = __uint_as_float(v[m].y);
        d[2] = __uint_as_float(v[m].z);
      }
    if (__syncthreads_or(fail)) {
      fail = true;
      break;
    }
    const bool above = warp == 0 && up, below = warp == NW - 1 && down;
    const bool lcol = lane < 2 && left, rcol = lane >= 30 && right;
    if (above || below || lcol || rcol) {
      const bool row = above || below;
      const float* d =
          stage + 3 * (row ? (below ? JP * 32 : 0) + lane
                           : JROWS + ((rcol ? NW : 0) + warp) * JP * 2 + (rcol ? lane - 30 : lane));
      const int step = 3 * (row ? 32 : 2);
#pragma unroll
      for (int k = 0; k < RT * JT; ++k) x[k / JT][k % JT] = d[(k / 3) * step + k % 3];
    }
  }
  if (tid == 0) {
    a.epoch[id] = epoch + a.inc;
    // (A batch's groups share the slots: those this one does not use keep step.)
    if (BATCH)
      for (int k = id + gridDim.x; k < a.cap; k += gridDim.x) a.epoch[k] = epoch + a.inc;
    if (fail) atomicExch(a.err, 1);
    if (id == 0) {
      a.ctl->sweeps = iters;
      a.ctl->last_launch = a.last_launch;
      a.ctl->sel = 0;
    }
  }
  const int oi0 = rg.own & 255, oi1 = rg.own >> 8 & 255, oj0 = rg.own >> 16 & 255,
            oj1 = rg.own >> 24;
  if (lane * JT < oj0 || lane * JT >= oj1) return;
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    const int gi = gi0 + r;
    if (warp * RT + r < oi0 || warp * RT + r >= oi1 || gi >= rg.NX || gj >= rg.NY) continue;
    float* d = a.x + rg.off + (size_t)gi * rg.P + gj;
    if (gj + JT <= rg.NY) {
      *reinterpret_cast<float4*>(d) = make_float4(x[r][0], x[r][1], x[r][2], x[r][3]);
    } else {
#pragma unroll
      for (int q = 0; q < JT; ++q)
        if (gj + q < rg.NY) d[q] = x[r][q];
    }
  }
}

// Final potential at cell c: the main iterate, plus the outer correction on
// active cells when one ran (phi = phi + e, fluid.go's p accumulation aside).
__device__ __forceinline__ float phi_final(const float* __restrict__ phi,
                                           const float* __restrict__ e, int c, bool act) {
  float x = phi[c];
  if (e && act) x = x + e[c];
  return x;
}

// Gradient subtract and pressure: U_face += S_R phi_L - S_L phi_R on faces
// with an active neighbour, V likewise, p = cp * phi on active cells, 0
// elsewhere (fill(f.p, 0) fluid.go:83 plus p += cp * delta fluid.go:224).
// U, V, p use the grid pitch g.P; phi, e and the flags the pitch Ps.
__global__ void k_grad(float* __restrict__ U, float* __restrict__ V, float* __restrict__ p,
                       const float* __restrict__ phi0, const float* __restrict__ phi1,
                       const PCtl* __restrict__ ctl, const float* __restrict__ e0,
                       const float* __restrict__ e1, const PCtl* __restrict__ ectl,
                       const uint8_t* __restrict__ flags, float cp, Grid g, int Ps) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.NX || j >= g.NY) return;
  const float* phi = ctl->sel ? phi1 : phi0;
  const float* e = ectl ? (ectl->sel ? e1 : e0) : nullptr;
  int c = i * Ps + j;
  int u = i * g.P + j;
  uint8_t fl = flags[c];
  bool act = flag_active(fl);
  float pc = phi_final(phi, e, c, act);
  if (i >= 1 && j >= 1 && j <= g.NY - 2) {
    uint8_t fL = flags[c - Ps];
    bool actL = flag_active(fL);
    if (act || actL) {
      float d = fbit(fl, F_FLUID) * phi_final(phi, e, c - Ps, actL) - fbit(fl, F_W) * pc;
      U[u] = U[u] + d;
    }
  }
  if (j >= 1 && i >= 1 && i <= g.NX - 2) {
    uint8_t fB = flags[c - 1];
    bool actB = flag_active(fB);
    if (act || actB) {
      float d = fbit(fl, F_FLUID) * phi_final(phi, e, c - 1, actB) - fbit(fl, F_S) * pc;
      V[u] = V[u] + d;
    }
  }
  p[u] = act ? cp * pc : 0.0f;
}

// Gradient subtract for the parallel scheme, fused with what follows it in
// the step: the post-projection divergence statistics (sum div^2 in float
// pairs, max |div|, fluid cell count), the residual statistics of the final
// potential (resid_ff per cell, sum r^2 and max |r|) and, when confinement
// is off, addTurbulence (fluid.go:496-526), which only touches a cell's own
// U, V.  Reads U, V and writes the rotated buffers Uo, Vo, so the divergence
// can recompute a neighbour's projected face from its original value.
struct GradAcc {
  FF d2, r2;
  float dmax, rmax, n;
};

// A cell's inputs: its flags and its four neighbours', the final potential
// (phi + e) there (0 past the domain edge), U and V at its faces (plus the
// recorded step's forces) and at the faces (i+1, j), (i, j+1), b and the
// turbulence noise.
struct GradIn {
  uint8_t fl, fL, fR, fB, fT;
  float pc, pL, pR, pB, pT;
  float u, v, uR0, vT0, bc;
  float2 nz;
};

// Its results: the faces, p, and the faces before turbulence (which a recorded
// step keeps).
struct GradOut {
  float u, v, p, u2, v2;
};

// addTurbulence (fluid.go:496-526) on a fluid cell's own faces.
__device__ __forceinline__ void turbulence(float& u, float& v, float2 nz, float turbStrength) {
  float noiseU = nz.x * turbStrength;
  float noiseV = nz.y * turbStrength;
  float localVel = sqrtf(u * u + v * v);
  if (localVel > 0.1f) {
    float turbulenceFactor = go_min(localVel * 0.5f, 1.0f);
    u += noiseU * turbulenceFactor;
    v += noiseV * turbulenceFactor;
  }
}

// The cell's update from its inputs: the projected faces, p, the residual
// and divergence statistics, turbulence.
__device__ __forceinline__ GradOut grad_apply(bool hasL, bool hasR, bool hasB, bool hasT,
                                              const GradIn& in, float cp, float turbStrength,
                                              int do_turb, GradAcc& acc) {
  const uint8_t fl = in.fl, fR = in.fR, fT = in.fT;
  const bool act = flag_active(fl), aL = flag_active(in.fL), aR = flag_active(fR);
  const bool aB = flag_active(in.fB), aT = flag_active(fT);
  const float pc = in.pc, pL = in.pL, pR = in.pR, pB = in.pB, pT = in.pT;
  float u = in.u, v = in.v;
  if (hasL && hasB && hasT && (act || aL)) u = u + (fbit(fl, F_FLUID) * pL - fbit(fl, F_W) * pc);
  if (hasB && hasL && hasR && (act || aB)) v = v + (fbit(fl, F_FLUID) * pB - fbit(fl, F_S) * pc);
  GradOut out;
  out.p = act ? cp * pc : 0.0f;
  out.u2 = u;
  out.v2 = v;
  if (act) {
    FF r = resid_ff(in.bc, pL, pR, pB, pT, (float)flag_count(fl), pc);
    FF q = ff_sq(r.hi);
    q.lo = q.lo + 2.0f * r.hi * r.lo;
    ff_acc(acc.r2, q);
    acc.rmax = fmaxf(acc.rmax, fabsf(r.hi));
  }
  if ((fl & (F_FLUID | F_INTERIOR)) == (F_FLUID | F_INTERIOR)) {
    // Projected faces (i+1, j) and (i, j+1), as their own threads compute them.
    float uR = in.uR0;
    if (act || aR) uR = uR + (fbit(fR, F_FLUID) * pc - fbit(fR, F_W) * pR);
    float vT = in.vT0;
    if (act || aT) vT = vT + (fbit(fT, F_FLUID) * pc - fbit(fT, F_S) * pT);
    float div = uR - u + vT - v;
    ff_acc(acc.d2, ff_sq(div));
    acc.dmax = fmaxf(acc.dmax, fabsf(div));
    acc.n = acc.n + 1.0f;
    if (do_turb) turbulence(u, v, in.nz, turbStrength);
  }
  out.u = u;
  out.v = v;
  return out;
}

// grad_apply of a plain cell: an interior fluid cell with four fluid
// neighbours (flags kPlain), whose bits are all 1 and whose neighbours' flags
// say nothing more.  The same operations without the factors of 1.
__device__ __forceinline__ GradOut grad_plain(const GradIn& in, float cp, float turbStrength,
                                              int do_turb, GradAcc& acc) {
  GradOut out;
  float u = in.u + (in.pL - in.pc), v = in.v + (in.pB - in.pc);
  out.p = cp * in.pc;
  const FF r = resid_ff(in.bc, in.pL, in.pR, in.pB, in.pT, 4.0f, in.pc);
  FF q = ff_sq(r.hi);
  q.lo = q.lo + 2.0f * r.hi * r.lo;
  ff_acc(acc.r2, q);
  acc.rmax = fmaxf(acc.rmax, fabsf(r.hi));
  const float uR = in.uR0 + (in.pc - in.pR), vT = in.vT0 + (in.pc - in.pT);
  const float div = uR - u + vT - v;
  ff_acc(acc.d2, ff_sq(div));
  acc.dmax = fmaxf(acc.dmax, fabsf(div));
  acc.n = acc.n + 1.0f;
  out.u2 = u;
  out.v2 = v;
  if (do_turb) turbulence(u, v, in.nz, turbStrength);
  out.u = u;
  out.v = v;
  return out;
}

__device__ __forceinline__ void grad_cell(int i, int j, const float* __restrict__ U,
                                          const float* __restrict__ V, float* __restrict__ Uo,
                                          float* __restrict__ Vo, float* __restrict__ p,
                                          const float* __restrict__ phi,
                                          const float* __restrict__ e,
                                          const float* __restrict__ rhs,
                                          const uint8_t* __restrict__ flags, float cp,
                                          const float2* __restrict__ noise, float turbStrength,
                                          int do_turb, const Grid& g, GradAcc& acc,
                                          const float* __restrict__ Fu = nullptr,
                                          const float* __restrict__ Fv = nullptr,
                                          float* __restrict__ U2o = nullptr,
                                          float* __restrict__ V2o = nullptr) {
  const int P = g.P;
  const int c = i * P + j;
  const bool hasL = i >= 1, hasR = i <= g.NX - 2, hasB = j >= 1, hasT = j <= g.NY - 2;
  // Neighbour indices clamped to the cell at the domain edge, so every load
  // below is issued at once and valid; the edge values are masked after.
  const int cL = hasL ? c - P : c, cR = hasR ? c + P : c;
  const int cB = hasB ? c - 1 : c, cT = hasT ? c + 1 : c;
  GradIn in;
  in.fl = flags[c];
  in.fL = hasL ? flags[cL] : 0;
  in.fR = hasR ? flags[cR] : 0;
  in.fB = hasB ? flags[cB] : 0;
  in.fT = hasT ? flags[cT] : 0;
  // phi and the correction are both exactly 0 off the active cells, so the
  // final potential phi + e needs no activity test.
  float pc = phi[c], pL = phi[cL], pR = phi[cR], pB = phi[cB], pT = phi[cT];
  if (e) {
    pc = pc + e[c];
    pL = pL + e[cL];
    pR = pR + e[cR];
    pB = pB + e[cB];
    pT = pT + e[cT];
  }
  if (!hasL) pL = 0.0f;
  if (!hasR) pR = 0.0f;
  if (!hasB) pB = 0.0f;
  if (!hasT) pT = 0.0f;
  in.pc = pc;
  in.pL = pL;
  in.pR = pR;
  in.pB = pB;
  in.pT = pT;
  // U1 = U + the recorded step's forces (when given).
  in.u = with_force(U, Fu, c);
  in.v = with_force(V, Fv, c);
  in.uR0 = with_force(U, Fu, cR);
  in.vT0 = with_force(V, Fv, cT);
  in.bc = rhs[c];
  in.nz = do_turb ? noise[c] : make_float2(0.0f, 0.0f);
  const GradOut o = grad_apply(hasL, hasR, hasB, hasT, in, cp, turbStrength, do_turb, acc);
  Uo[c] = o.u;
  Vo[c] = o.v;
  p[c] = o.p;
  if (U2o) {
    U2o[c] = o.u2;
    V2o[c] = o.v2;
  }
}

// The step's statistics from the combined row of k_grad_fused's partials
// (sum div^2, max |div|, fluid cells, sum r^2, max |r|) and, after a solve,
// its sweep count and last checked max |r| from the control block.
struct StoreDivP {
  DevStats* st;
  const PCtl* ctl;
  __device__ void operator()(const float* r) const {
    st->div_l2_sq = row_sum(r, 0);
    st->div_max = (double)r[2];
    st->div_count = row_sum(r, 2);
    st->resid_l2_sq = row_sum(r, 3);
    st->resid_max = (double)r[8];
    if (ctl) {
      st->sweeps = ctl->sweeps;
      st->last_maxdiv = (double)__uint_as_float(ctl->slots[ctl->last_launch]);
    }
  }
};

// The gradient subtract and its fused statistics, 4 columns of a row a thread
// at a time: fields move in 16-byte pieces (rows start on 128 bytes; a piece
// past the last column reads pitch padding, which nothing uses).  At most
// kGradBlocks blocks walk the grid, three an SM (held to 80 registers a thread,
// which spills 36 bytes, 104 when a step is recorded), so the reduction at the
// end of a block is paid once per block and its rows are few enough to combine
// in the same launch.  Plain cells take 150 operations of the 240 the
// flag-by-flag form takes.  With the combining (us; before: one column of 8
// rows a thread and a second launch): 128 x 128 9.1 (11.7 + 4.9), 512 x 256 9.3
// (11.4 + 5.3), 1500 x 1100 24 (27.7 + 5.9), 2048 x 2048 42 (56 + 7.1).  One
// piece a thread in 4109 blocks: 66; two rows a piece 82.
constexpr int kGradBlocks = 3 * 152;
// REC: a recorded step (force fields, the faces before turbulence kept).
template <bool REC>
__global__ void __launch_bounds__(256, 3)
    k_grad_fused(const float* __restrict__ U, const float* __restrict__ V,
                 float* __restrict__ Uo, float* __restrict__ Vo, float* __restrict__ p,
                 const float* __restrict__ phi0, const float* __restrict__ phi1,
                 const PCtl* __restrict__ ctl, const float* __restrict__ e0,
                 const float* __restrict__ e1, const PCtl* __restrict__ ectl,
                 const float* __restrict__ rhs, const uint8_t* __restrict__ flags, float cp,
                 const float2* __restrict__ noise, float turbStrength, int do_turb,
                 float* __restrict__ part, Grid g, const float* __restrict__ Fu,
                 const float* __restrict__ Fv, float* __restrict__ U2o,
                 float* __restrict__ V2o, int* ticket, StoreDivP store) {
  __shared__ float shr[64 * 5];
  pdl_enter();
  const float *fu = REC ? Fu : nullptr, *fv = REC ? Fv : nullptr;
  const float* phi = ctl->sel ? phi1 : phi0;
  const float* e = ectl ? (ectl->sel ? e1 : e0) : nullptr;
  const int nq = (g.NY + 3) / 4, total = nq * g.NX, P = g.P;
  GradAcc acc{{0.0f, 0.0f}, {0.0f, 0.0f}, 0.0f, 0.0f, 0.0f};
  for (int idx = blockIdx.x * 256 + threadIdx.x; idx < total; idx += gridDim.x * 256) {
    const int i = idx / nq, j = 4 * (idx - i * nq);
    auto ld4 = [](const float* x, int c) { return *reinterpret_cast<const float4*>(x + c); };
    auto sum4 = [&](const float* x, const float* y, int c) {
      float4 a = ld4(x, c);
      if (y) {
        const float4 b = ld4(y, c);
        a = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
      }
      return a;
    };
    auto sum1 = [](const float* x, const float* y, int c) { return y ? x[c] + y[c] : x[c]; };
    auto fl4 = [&](int c) { return *reinterpret_cast<const uint32_t*>(flags + c); };
    auto at = [](const float4& x, int k) { return k == 0 ? x.x : k == 1 ? x.y : k == 2 ? x.z : x.w; };
    auto fat = [](uint32_t x, int k) { return (uint8_t)(x >> 8 * k); };
    const bool more = j + 4 < g.NY;  // the column right of the piece is a cell
    const int c = i * P + j;
    const bool hasL = i >= 1, hasR = i <= g.NX - 2;
    // (Off the grid: the row itself, masked below.)
    const int cl = hasL ? c - P : c, cn = hasR ? c + P : c;
    const float4 pprev = sum4(phi, e, cl), pcur = sum4(phi, e, c), pnext = sum4(phi, e, cn);
    const float4 ucur = sum4(U, fu, c), unext = sum4(U, fu, cn);
    const uint32_t f = fl4(c);
    const float4 v = sum4(V, fv, c), b = ld4(rhs, c);
    const float pl = j >= 1 ? sum1(phi, e, c - 1) : 0.0f;
    const float pr = more ? sum1(phi, e, c + 4) : 0.0f;
    const float vr = more ? sum1(V, fv, c + 4) : 0.0f;
    float4 n0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), n1 = n0;
    if (do_turb) {
      n0 = ld4(reinterpret_cast<const float*>(noise + c), 0);
      n1 = ld4(reinterpret_cast<const float*>(noise + c), 4);
    }
    GradIn in[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool hasT = j + k <= g.NY - 2;
      in[k].pc = at(pcur, k);
      in[k].pL = hasL ? at(pprev, k) : 0.0f;
      in[k].pR = hasR ? at(pnext, k) : 0.0f;
      in[k].pB = k ? at(pcur, k - 1) : pl;
      in[k].pT = !hasT ? 0.0f : k < 3 ? at(pcur, k + 1) : pr;
      in[k].u = at(ucur, k);
      in[k].v = at(v, k);
      in[k].uR0 = at(unext, k);
      in[k].vT0 = k < 3 ? at(v, k + 1) : vr;
      in[k].bc = at(b, k);
      in[k].nz = k == 0 ? make_float2(n0.x, n0.y) : k == 1 ? make_float2(n0.z, n0.w)
                 : k == 2 ? make_float2(n1.x, n1.y) : make_float2(n1.z, n1.w);
    }
    float o[5][4];
    auto out = [&](int k, const GradOut& x) {
      o[0][k] = x.u; o[1][k] = x.v; o[2][k] = x.p; o[3][k] = x.u2; o[4][k] = x.v2;
    };
    if (more && f == kPlain * 0x01010101u) {
#pragma unroll
      for (int k = 0; k < 4; ++k) out(k, grad_plain(in[k], cp, turbStrength, do_turb, acc));
    } else {
      const uint32_t fp = hasL ? fl4(c - P) : 0, fn = hasR ? fl4(cn) : 0;
      const uint8_t fb = j >= 1 ? flags[c - 1] : 0, ft = more ? flags[c + 4] : 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool hasB = j + k >= 1, hasT = j + k <= g.NY - 2;
        if (j + k >= g.NY) continue;
        in[k].fl = fat(f, k);
        in[k].fL = fat(fp, k);
        in[k].fR = fat(fn, k);
        in[k].fB = k ? fat(f, k - 1) : fb;
        in[k].fT = !hasT ? 0 : k < 3 ? fat(f, k + 1) : ft;
        out(k, grad_apply(hasL, hasR, hasB, hasT, in[k], cp, turbStrength, do_turb, acc));
      }
    }
    float* dst[5] = {Uo, Vo, p, U2o, V2o};
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      if (q >= 3 && !(REC && U2o)) break;
      if (j + 4 <= g.NY) {
        *reinterpret_cast<float4*>(dst[q] + c) = make_float4(o[q][0], o[q][1], o[q][2], o[q][3]);
      } else {
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (j + k < g.NY) dst[q][c + k] = o[q][k];
      }
    }
  }
  // Row slots: sum div^2, max |div|, fluid cells (exact), sum r^2, max |r|.
  FF row[5] = {acc.d2, {acc.dmax, 0.0f}, {acc.n, 0.0f}, acc.r2, {acc.rmax, 0.0f}};
  grid_row<5, 0x4u>(row, 0x12u, shr, part, blockIdx.x, gridDim.x, ticket, store);
}

// Copies the solve's final potential (the buffer the control block names),
// plus the outer correction when one ran (both exactly 0 off the active
// cells, as k_grad_fused adds them).
__global__ void k_store_phi(const float* __restrict__ phi0, const float* __restrict__ phi1,
                            const PCtl* __restrict__ ctl, const float* __restrict__ e0,
                            const float* __restrict__ e1, const PCtl* __restrict__ ectl,
                            float* __restrict__ dst, int n) {
  const float* src = ctl->sel ? phi1 : phi0;
  const float* e = ectl ? (ectl->sel ? e1 : e0) : nullptr;
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) dst[k] = e ? src[k] + e[k] : src[k];
}

// A batch's gradient subtract: grad_cell without the statistics.
__device__ __forceinline__ void grad_batch_cell(int i, int j, const float* __restrict__ U,
                                                const float* __restrict__ V,
                                                float* __restrict__ Uo, float* __restrict__ Vo,
                                                float* __restrict__ p,
                                                const float* __restrict__ phi0,
                                                const float* __restrict__ phi1,
                                                const PCtl* __restrict__ ctl,
                                                const float* __restrict__ rhs,
                                                const uint8_t* __restrict__ flags, float cp,
                                                const float2* __restrict__ noise,
                                                float turbStrength, int do_turb,
                                                float* __restrict__ U2o, float* __restrict__ V2o,
                                                const Grid& g) {
  GradAcc acc{{0.0f, 0.0f}, {0.0f, 0.0f}, 0.0f, 0.0f, 0.0f};
  grad_cell(i, j, U, V, Uo, Vo, p, ctl->sel ? phi1 : phi0, nullptr, rhs, flags, cp, noise,
            turbStrength, do_turb, g, acc, nullptr, nullptr, U2o, V2o);
}

}  // namespace

size_t pctl_bytes(int n_slots) { return sizeof(PCtl) + sizeof(unsigned) * (size_t)n_slots; }

// Tensor maps of the TMA-fed Jacobi kernel: a 2D float array of rows x
// pitch, boxes of 64 rows x 128 columns, zero outside.  false when the
// driver entry point or the encoding is unavailable (the plain kernel runs).
// Per CUDA context: the SM count, the dataflow kernel's blocks per SM,
// whether the set-up ran (the kernels' shared-memory limit is state of the
// context the module is loaded in).
constexpr int kMaxContexts = 64;
struct TmaDevice {
  std::once_flag once;
  std::atomic<bool> ready{false};
  int sms = 0;
  int flow_per_sm = 0;
  int batch_pf_per_sm = 0;  // blocks of kb_jacobi_pf per SM (0: the plain batch kernel runs)
  int res_blocks[4] = {};   // blocks of k_jacobi_res's forms the device holds (0: none)
};
static TmaDevice g_tma_dev[kMaxContexts];
static unsigned long long g_tma_key[kMaxContexts];
static int g_tma_used = 0;
static std::mutex g_tma_mu;
static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
static std::once_flag g_encode_once;

// Identity of the CUDA context current on the calling thread: its
// cuCtxGetId value (unique for the life of the process) with the top bit
// clear, or, when the driver entry points are missing, the device ordinal
// with the top bit set; 0 when neither is known (no context yet).  Module
// state -- a __device__ array's address, a kernel's shared-memory limit --
// belongs to a context, and a caller may make its own context current
// (cuCtxCreate, cuCtxSetCurrent) or replace the primary one
// (cudaDeviceReset), so caches of that state are keyed by this value.
typedef CUresult (*PfnCtxGetCurrent)(CUcontext*);
typedef CUresult (*PfnCtxGetId)(CUcontext, unsigned long long*);
static PfnCtxGetCurrent g_ctx_current = nullptr;
static PfnCtxGetId g_ctx_id = nullptr;
static std::once_flag g_ctx_once;

unsigned long long context_key() {
  std::call_once(g_ctx_once, [] {
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_ctx_current = reinterpret_cast<PfnCtxGetCurrent>(fn);
    fn = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_ctx_id = reinterpret_cast<PfnCtxGetId>(fn);
    cudaGetLastError();
  });
  if (g_ctx_current && g_ctx_id) {
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (g_ctx_current(&c) != CUDA_SUCCESS || !c) return 0;
    if (g_ctx_id(c, &id) != CUDA_SUCCESS) return 0;
    return (id & ~(1ull << 63)) + 1;  // nonzero, top bit clear
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return (1ull << 63) | (unsigned long long)dev;
}

static bool encode_box_map(CUtensorMap* tm, const float* base, int rows, int pitch,
                           int box_rows = RI) {
  if (!g_encode || (reinterpret_cast<uintptr_t>(base) & 15) || (pitch % 4) != 0) return false;
  cuuint64_t dims[2] = {(cuuint64_t)pitch, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)pitch * sizeof(float)};
  cuuint32_t box[2] = {(cuuint32_t)RJ, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Forms of the resident solve: regions of 4, 8 and 12 warps, one to an SM (all
// the registers they want), and of 8 warps two to an SM.
enum { JRES_4 = 0, JRES_8 = 1, JRES_12 = 2, JRES_8X2 = 3 };
static int res_warps(int form) { return form == JRES_4 ? 4 : form == JRES_12 ? 12 : 8; }
typedef void (*ResKernel)(JResArgs);
static ResKernel res_kernel(bool o1, bool batch, int form) {
#define FG_RES1(NW, MB, B) (o1 ? k_jacobi_res<true, NW, B, MB> : k_jacobi_res<false, NW, B, MB>)
#define FG_RES(NW, MB) (batch ? FG_RES1(NW, MB, true) : FG_RES1(NW, MB, false))
  return form == JRES_4    ? FG_RES1(4, 2, false)  // (a batch has no use for it)
         : form == JRES_8  ? FG_RES(8, 1)
         : form == JRES_12 ? FG_RES(12, 1)
                           : FG_RES(8, 2);
#undef FG_RES
#undef FG_RES1
}

// The current context's entry, or nullptr (no context identity, or more
// contexts than entries: the plain kernels run).
static TmaDevice* tma_device() {
  const unsigned long long key = context_key();
  if (!key) return nullptr;
  std::lock_guard<std::mutex> lk(g_tma_mu);
  for (int k = 0; k < g_tma_used; ++k)
    if (g_tma_key[k] == key) return &g_tma_dev[k];
  if (g_tma_used == kMaxContexts) return nullptr;
  g_tma_key[g_tma_used] = key;
  return &g_tma_dev[g_tma_used++];
}

// Resolves the tensor-map encoder (once per process) and, once per device,
// the SM count and the TMA kernels' shared-memory limit (outside any stream
// capture).
void init_jacobi_tma() {
  std::call_once(g_encode_once, [] {
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    cudaGetLastError();
  });
  TmaDevice* d = tma_device();
  if (!d) return;
  std::call_once(d->once, [d] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
      d->sms = n;
    const int smem = 3 * TILE_FLOATS * (int)sizeof(float);
    if (cudaFuncSetAttribute(k_jacobi_tma<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem) != cudaSuccess ||
        cudaFuncSetAttribute(k_jacobi_tma<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem) != cudaSuccess)
      d->sms = 0;
    // Blocks of the dataflow kernel that fit on one SM (co-residency bound).
    int b1 = 0, b2 = 0;
    const int fsmem = 3 * FLOW_FLOATS * (int)sizeof(float);
    if (cudaFuncSetAttribute(k_jacobi_flow<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             fsmem) == cudaSuccess &&
        cudaFuncSetAttribute(k_jacobi_flow<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             fsmem) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_jacobi_flow<true>, FLOW_THREADS, fsmem) ==
            cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, k_jacobi_flow<false>, FLOW_THREADS, fsmem) ==
            cudaSuccess)
      d->flow_per_sm = b1 < b2 ? b1 : b2;
    int coop = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
      d->flow_per_sm = 0;
    int p1 = 0, p2 = 0;
    if (cudaFuncSetAttribute(kb_jacobi_pf<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem) == cudaSuccess &&
        cudaFuncSetAttribute(kb_jacobi_pf<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p1, kb_jacobi_pf<true>, TB_THREADS,
                                                      smem) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p2, kb_jacobi_pf<false>, TB_THREADS,
                                                      smem) == cudaSuccess)
      d->batch_pf_per_sm = p1 < p2 ? p1 : p2;
    if (coop)
      for (int form = 0; form < 4; ++form) {
        int least = INT_MAX;
        for (int v = 0; v < 4; ++v) {
          int per = 0;
          if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                  &per, res_kernel(v & 1, (v & 2) != 0, form), 32 * res_warps(form), 0) !=
              cudaSuccess)
            per = 0;
          least = std::min(least, per);
        }
        d->res_blocks[form] = std::min(least, 2) * d->sms;
      }
    cudaGetLastError();
    d->ready.store(true);
  });
}

// The current device's set-up, done here unless the stream is capturing
// (then nullptr: the plain kernels run).
static const TmaDevice* tma_ready(cudaStream_t st) {
  TmaDevice* d = tma_device();
  if (!d) return nullptr;
  if (!d->ready.load()) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusActive;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
      cudaGetLastError();
      return nullptr;
    }
    init_jacobi_tma();
  }
  return d->ready.load() ? d : nullptr;
}

// Launches one full, unchecked Jacobi launch through the TMA-fed kernel;
// false (nothing launched) when the tensor maps cannot be made.
static bool launch_jacobi_tma(cudaStream_t st, const Grid& g, PCtl* ctl, const float* src,
                              float* dst, const float* W, const float* BW, float om1, bool o1,
                              int k, int t0, int sel, int zero_init, int* err, int stall_tile) {
  const TmaDevice* dv = tma_ready(st);
  if (!dv) return false;
  CUtensorMap tmx, tmw, tmb;
  if (!encode_box_map(&tmx, src, g.NX, g.P) || !encode_box_map(&tmw, W, g.NX, g.P) ||
      !encode_box_map(&tmb, BW, g.NX, g.P))
    return false;
  const int nsm = dv->sms;
  if (nsm <= 0) return false;
  const int ntx = (g.NY + OJ - 1) / OJ, nty = (g.NX + OI - 1) / OI;
  const int ntiles = ntx * nty;
  const int grid = ntiles < 2 * nsm ? ntiles : 2 * nsm;
  const size_t smem = 3 * (size_t)TILE_FLOATS * sizeof(float);
  if (o1)
    k_jacobi_tma<true><<<grid, TB_THREADS, smem, st>>>(tmx, tmw, tmb, dst, om1, ctl, k, t0, sel,
                                                       zero_init, g, ntx, ntiles, err, stall_tile);
  else
    k_jacobi_tma<false><<<grid, TB_THREADS, smem, st>>>(tmx, tmw, tmb, dst, om1, ctl, k, t0, sel,
                                                        zero_init, g, ntx, ntiles, err, stall_tile);
  return true;
}

inline int clamp_tb(int t) { return t < 1 ? 1 : (t > TMAX ? TMAX : t); }

int jacobi_launches(const fg_fluid* f, int iters) {
  // In 64 bits: iters near INT_MAX must not wrap (at most INT_MAX launches).
  const long long T = clamp_tb(f->prm.tb_depth);
  return (int)(((long long)iters + T - 1) / T);
}

int jacobi_tile_count(int NX, int NY) {
  return ((NY + OJ - 1) / OJ) * ((NX + OI - 1) / OI);
}

// Launches the first `nphase` full phases of a fixed-count solve as one
// cooperative dataflow kernel (x0 -> x1 -> x0 ...); `done` holds one flag
// per tile and the item counter.  false (nothing launched) when the grid is
// below one tile per SM, the flags are missing, or the tensor maps or the
// cooperative launch are unavailable.
static bool launch_jacobi_flow(cudaStream_t st, const Grid& g, PCtl* ctl, float* x0, float* x1,
                               const float* W, const float* BW, float om1, bool o1, int nphase,
                               int* done, int* err, int stall_tile) {
  if (!done || nphase < 2) return false;
  const TmaDevice* dv = tma_ready(st);
  if (!dv || dv->flow_per_sm <= 0 || dv->sms <= 0) return false;
  // Grids of fewer 48 x 112 tiles than SMs stay with the per-launch kernels
  // (which run there only without the resident solve's buffers).
  if (jacobi_tile_count(g.NX, g.NY) < dv->sms) return false;
  const int ntx = (g.NY + OJ - 1) / OJ, nty = (g.NX + FO - 1) / FO;
  const int ntiles = ntx * nty;
  CUtensorMap tm0, tm1, tmw, tmb;
  if (!encode_box_map(&tm0, x0, g.NX, g.P, FI) || !encode_box_map(&tm1, x1, g.NX, g.P, FI) ||
      !encode_box_map(&tmw, W, g.NX, g.P, FI) || !encode_box_map(&tmb, BW, g.NX, g.P, FI))
    return false;
  // The tile flags and the item counter.
  if (cudaMemsetAsync(done, 0, sizeof(int) * ((size_t)ntiles + 1), st) != cudaSuccess) return false;
  const int cap = dv->flow_per_sm * dv->sms;
  const int grid = ntiles < cap ? ntiles : cap;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(FLOW_THREADS);
  cfg.dynamicSmemBytes = 3 * (size_t)FLOW_FLOATS * sizeof(float);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int zero_first = 1;
  cudaError_t e = o1 ? cudaLaunchKernelEx(&cfg, k_jacobi_flow<true>, tm0, tm1, tmw, tmb, x0, x1,
                                          om1, ctl, done, nphase, zero_first, g, ntx, nty, err,
                                          stall_tile)
                     : cudaLaunchKernelEx(&cfg, k_jacobi_flow<false>, tm0, tm1, tmw, tmb, x0, x1,
                                          om1, ctl, done, nphase, zero_first, g, ntx, nty, err,
                                          stall_tile);
  return e == cudaSuccess;
}

// Enqueues `iters` Jacobi sweeps of A x = b from x = 0 in launches of T
// sweeps; x ping-pongs between x0 and x1 and ctl->sel names the buffer that
// holds the result.  The grid g's pitch is the solver arrays' pitch.
// With `mphi0` set, the first launch forms the right-hand side from the main
// potential (RINIT): b is then the main right-hand side, and b_e / bw_e are
// written to rhs_e / bwe when more launches follow (which then read them).
static cudaError_t enqueue_jacobi(cudaStream_t st, const Grid& g, PCtl* ctl, const float* b,
                                  const float* bw, const float* W, const uint8_t* flags, float* x0,
                                  float* x1, int iters, int T, float om, int check, float tol,
                                  int* n_launched, const float* mphi0 = nullptr,
                                  const float* mphi1 = nullptr, const PCtl* mctl = nullptr,
                                  float* rhs_e = nullptr, float* bwe = nullptr,
                                  int* err = nullptr, int* done = nullptr,
                                  int stall_tile = -1, int tma_stall_tile = -1,
                                  int* kind = nullptr) {
  float om1 = 1.0f - om;
  int used = FG_JACOBI_KERNEL_SWEEP;
  bool o1 = om1 == 0.0f;
  dim3 gr(span_count(g.NY, RJ), span_count(g.NX, RI));
  // Grids with fewer 8-warp regions than SMs run every launch on 4-warp
  // regions (half the rows), spread over twice the SMs.
  const TmaDevice* dv = tma_ready(st);
  const bool narrow = dv && dv->sms > 0 && (long long)gr.x * gr.y < dv->sms;
  const dim3 gr4(span_count(g.NY, RJ), span_count(g.NX, RI / 2));
  int nlaunch = (int)(((long long)iters + T - 1) / T);
  int k0 = 0, kernels = 0;
  // Fixed sweep counts in full launches: the leading full phases as one
  // dataflow kernel where the grid is large enough.
  if (!check && !mphi0 && T == TMAX && iters / TMAX >= 2 &&
      launch_jacobi_flow(st, g, ctl, x0, x1, W, bw, om1, o1, iters / TMAX, done, err,
                         stall_tile)) {
    k0 = iters / TMAX;
    kernels = 1;
    used = FG_JACOBI_KERNEL_DATAFLOW;
  }
  for (int k = k0; k < nlaunch; ++k) {
    ++kernels;
    int t0 = k * T;
    int ns = iters - t0 < T ? iters - t0 : T;
    const float* src = (k & 1) ? x1 : x0;
    float* dst = (k & 1) ? x0 : x1;
    int sel = (k & 1) ? 0 : 1;
    int zi = k == 0 ? 1 : 0;
    bool full = ns == TMAX;
    bool rinit = k == 0 && mphi0 != nullptr;
    const float* bk = rinit ? b : (mphi0 ? rhs_e : b);
    const float* bwk = mphi0 && k > 0 ? bwe : bw;
    float* re = rinit && nlaunch > 1 ? rhs_e : nullptr;
    if (full && !check && !rinit && !mphi0 && !narrow &&
        launch_jacobi_tma(st, g, ctl, src, dst, W, bwk, om1, o1, k, t0, sel, zi, err,
                          tma_stall_tile)) {
      if (used == FG_JACOBI_KERNEL_SWEEP) used = FG_JACOBI_KERNEL_TMA;
      continue;
    }
#define FG_JAC(O, F, C, R)                                                                      \
  (narrow ? launch_pdl(k_jacobi_rb<O, F, C, R, NWARP / 2>, gr4, dim3(TB_THREADS / 2), 0, st, src, \
                       dst, W, bwk, bk, flags, om1, ctl, k, t0, ns, tol, sel, zi, g, mphi0,     \
                       mphi1, mctl, re, bwe)                                                    \
          : launch_pdl(k_jacobi_rb<O, F, C, R>, gr, dim3(TB_THREADS), 0, st, src, dst, W, bwk, \
                       bk, flags, om1, ctl, k, t0, ns, tol, sel, zi, g, mphi0, mphi1, mctl, re, \
                       bwe))
    if (rinit) {
      if (o1) { if (full) FG_JAC(true, true, false, true); else FG_JAC(true, false, false, true); }
      else { if (full) FG_JAC(false, true, false, true); else FG_JAC(false, false, false, true); }
    } else if (o1) {
      if (full) { if (check) FG_JAC(true, true, true, false); else FG_JAC(true, true, false, false); }
      else { if (check) FG_JAC(true, false, true, false); else FG_JAC(true, false, false, false); }
    } else {
      if (full) { if (check) FG_JAC(false, true, true, false); else FG_JAC(false, true, false, false); }
      else { if (check) FG_JAC(false, false, true, false); else FG_JAC(false, false, false, false); }
    }
#undef FG_JAC
  }
  *n_launched = kernels;
  if (kind) *kind = used;
  return cudaGetLastError();
}

// ---------------------------------------------------------------- resident solves
// Regions of NW warps that cover a grid; 0 above the buffers' limit.
static int res_regions(int NX, int NY, int NW) {
  const long long n = (long long)span_count(NX, NW * RT) * span_count(NY, RJ);
  return n > JRES_MAX_REGIONS ? 0 : (int)n;
}
// Regions the current device holds at once in a form.
static int res_capacity(const TmaDevice* dv, int form) {
  return form == JRES_8X2 ? dv->res_blocks[form] : std::min(dv->sms, dv->res_blocks[form]);
}
size_t jres_bytes(int regions, int warps) {
  const size_t n = warps == 4 ? JSlot<4>::N : warps == 8 ? JSlot<8>::N : JSlot<12>::N;
  return JRES_MAX_REGIONS * sizeof(unsigned) + 2 * n * (size_t)regions * sizeof(uint4);
}

// The smallest regions that get an SM each, but 4 warps only for up to 16
// regions; else two 8-warp regions an SM.  Measured per 8 sweeps (us), against
// the launches or the dataflow kernel they replace: 4 warps 128^2 2.2 (3.5);
// 8 warps 512x256 3.1 (3.5), 512^2 2.9 (4.4), 800^2 3.0 (6.6); 12 warps
// 1024x768 4.2 (7.4), 1200x800 4.1 (9.4); 8 warps twice 1200^2 6.0 (11.0).  A
// larger form where a smaller one fits is slower.  4 warps take a solve alone
// on the GPU further (512x256: 2.4), but own half of the cells they sweep and
// hold more SMs while they wait, at the cost of every other stream's work:
// a step of many handles in turn (us; 4 warps, 8 warps, the launches) 64 of
// 256^2 673, 585, 648; 32 of 360^2 695, 570, 567; 32 of 512x256 836, 659, 694;
// 64 of 192^2 439, 397, 432.  Up to 128^2 (16 regions) they cost nothing there:
// 64 of 128^2 386, 403, 406; alone 58 us a step against 60 and 68.
// (Outside any capture.)
constexpr int kRes4Regions = 16;
int jres_grid_form(int NX, int NY) {
  init_jacobi_tma();
  const TmaDevice* dv = tma_device();
  if (!dv || !dv->ready.load()) return -1;
  for (int form = JRES_4; form <= JRES_8X2; ++form) {
    const int n = res_regions(NX, NY, res_warps(form));
    const int most = form == JRES_4 ? kRes4Regions : JRES_MAX_REGIONS;
    if (n > 0 && n <= std::min(most, res_capacity(dv, form))) return form;
  }
  return -1;
}
size_t jres_bytes_grid(int NX, int NY, int form) {
  return form < 0 ? 0 : jres_bytes(res_regions(NX, NY, res_warps(form)), res_warps(form));
}

// The forms a batch may be solved in: rows of a region, regions at once, and
// the measured time of 8 sweeps (us); 0 regions: unavailable.  (Outside any
// capture.)
void jres_batch_forms(JresForm (&out)[3]) {
  init_jacobi_tma();
  const TmaDevice* d = tma_device();
  const bool ok = d && d->ready.load();
  const int form[3] = {JRES_8, JRES_12, JRES_8X2};
  const float us[3] = {3.0f, 4.1f, 6.0f};
  for (int k = 0; k < 3; ++k) {
    const int cap = ok ? res_capacity(d, form[k]) : 0;
    out[k] = JresForm{form[k], res_warps(form[k]) * RT, std::min(cap, JRES_MAX_REGIONS), us[k]};
  }
}

static cudaError_t launch_res(cudaStream_t st, const JResArgs& a, bool o1, bool batch, int form,
                              int blocks) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(32 * res_warps(form));
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, res_kernel(o1, batch, form), a);
}

// A fixed-count solve of one grid from x = 0 into x as one resident launch.
// What fg_stats.jacobi_resident reports of it, or 0 (nothing launched) where
// the grid has no form or its buffers could not be had.
static int launch_jacobi_res(fg_fluid* f, PCtl* ctl, float* x, const float* W, const float* BW,
                             float om1, int iters, int T, int stall) {
  if (!f->jres) return 0;
  const TmaDevice* dv = tma_ready(f->stream);
  if (!dv) return 0;
  const int form = f->jres_form, nw = res_warps(form), n = res_regions(f->NX, f->NY, nw);
  if (n > res_capacity(dv, form)) return 0;  // (another context than the handle's first)
  JResArgs a = {};
  a.x = x;
  a.W = W;
  a.BW = BW;
  a.om1 = om1;
  a.iters = iters;
  a.inc = (unsigned)((iters + TMAX - 1) / TMAX);
  a.epoch = static_cast<unsigned*>(f->jres);
  a.pkt = reinterpret_cast<uint4*>(a.epoch + JRES_MAX_REGIONS);
  a.ctl = ctl;
  a.g = f->g;
  a.ntx = span_count(f->NY, RJ);
  a.nty = span_count(f->NX, nw * RT);
  a.last_launch = (iters + T - 1) / T - 1;
  a.err = &f->dstats->timeout;
  a.stall = stall;
  if (launch_res(f->stream, a, om1 == 0.0f, false, form, n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return form == JRES_8X2 ? 16 : nw;
}

// A batch's solves: every scene runs its own sweep count, no early exit.
static cudaError_t jacobi_solve_batch(fg_fluid* f, PCtl* ctl, const float* bw, float* x0,
                                      float* x1) {
  const BatchGeom* bt = f->batch;
  int T = clamp_tb(f->prm.tb_depth);
  int L = (bt->max_iters + T - 1) / T;
  cudaError_t e = cudaMemsetAsync(ctl, 0, sizeof(PCtl), f->stream);
  if (e != cudaSuccess) return e;
  float om = f->prm.jacobi_omega * f->prm.pressure_damping;
  float om1 = 1.0f - om;
  const TmaDevice* dv = tma_ready(f->stream);
  const int pf_blocks = dv && dv->sms > 0 ? dv->batch_pf_per_sm * dv->sms : 0;
  // Groups of scenes whose regions fit the GPU at once, each group's whole
  // solve one resident launch.
  if (f->jres && dv && bt->res_regions && bt->res_cap > 0) {
    JResArgs a = {};
    a.x = x0;
    a.W = f->wgt;
    a.BW = bw;
    a.om1 = om1;
    a.ctl = ctl;
    a.last_launch = L - 1;
    a.err = &f->dstats->timeout;
    a.stall = f->stall_tile;  // (that region of every group)
    unsigned* epochs = static_cast<unsigned*>(f->jres);
    uint4* pkts = reinterpret_cast<uint4*>(epochs + JRES_MAX_REGIONS);
    bool ok = true;
    for (const ResGroup& gp : bt->res_groups) {  // (groups run in turn: they share the buffers)
      a.regions = bt->res_regions + gp.first;
      a.cap = bt->res_cap;
      a.inc = (unsigned)((bt->max_iters + TMAX - 1) / TMAX);
      a.epoch = epochs;
      a.pkt = pkts;
      ok = dv->res_blocks[gp.form] >= gp.count &&
           launch_res(f->stream, a, om1 == 0.0f, true, gp.form, gp.count) == cudaSuccess;
      if (!ok) break;
      count(f);
    }
    if (ok) return cudaGetLastError();
    cudaGetLastError();
  }
  size_t sc = 0;  // scenes (in the table's order) started by launch k
  int n_act = 0;  // their regions: the prefix of the table launch k runs
  for (int k = 0; k < L; ++k) {
    while (sc < bt->jac_iters.size() && L - (bt->jac_iters[sc] + T - 1) / T <= k)
      n_act += bt->jac_regions[sc++];
    const float* src = (k & 1) ? x1 : x0;
    float* dst = (k & 1) ? x0 : x1;
    int sel = (k & 1) ? 0 : 1;
    if (n_act == 0) continue;
    if (pf_blocks > 0)
      launch_pdl(om1 == 0.0f ? kb_jacobi_pf<true> : kb_jacobi_pf<false>,
                 dim3(n_act < pf_blocks ? n_act : pf_blocks), dim3(TB_THREADS),
                 3 * (size_t)TILE_FLOATS * sizeof(float), f->stream, bt->jac_tiles,
                 bt->scenes_dev, n_act, src, dst, f->wgt, bw, om1, ctl, k, L, T, sel);
    else
      launch_pdl(om1 == 0.0f ? kb_jacobi<true> : kb_jacobi<false>, dim3(n_act),
                 dim3(TB_THREADS), 0, f->stream, bt->jac_tiles, bt->scenes_dev, src, dst, f->wgt,
                 bw, f->flags, om1, ctl, k, L, T, sel);
  }
  count(f, L);
  return cudaGetLastError();
}

// kind: where to record the kernel that ran the sweeps (the main solve's).
static cudaError_t jacobi_solve(fg_fluid* f, PCtl* ctl, const float* b, const float* bw, float* x0,
                                float* x1, int iters, bool allow_exit, bool rinit = false,
                                int* kind = nullptr) {
  if (f->batch) return jacobi_solve_batch(f, ctl, bw, x0, x1);
  int T = clamp_tb(f->prm.tb_depth);
  const long long nlaunch = ((long long)iters + T - 1) / T;
  if (nlaunch > f->n_slots) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(ctl, 0, pctl_bytes((int)nlaunch), f->stream);
  if (e != cudaSuccess) return e;
  int check = allow_exit && f->prm.early_exit ? 1 : 0;
  const bool prof = f->profile && allow_exit;
  if (prof && (e = cudaEventRecord(f->prof_ev[0], f->stream)) != cudaSuccess) return e;
  int n = 0;
  const TmaDevice* dv = tma_ready(f->stream);
  const int resident = rinit || check || iters <= 0
                           ? 0
                           : launch_jacobi_res(f, ctl, x0, f->wgt, bw,
                                               1.0f - f->prm.jacobi_omega * f->prm.pressure_damping,
                                               iters, T, f->stall_tile);
  if (kind) f->jacobi_resident = resident;
  if (resident) {
    // (kind: the kernel that such a solve takes without the resident launch.)
    n = 1;
    if (kind)
      *kind = T < TMAX || iters < TMAX ? FG_JACOBI_KERNEL_SWEEP
              : iters >= 2 * TMAX && jacobi_tile_count(f->NX, f->NY) >= dv->sms
                  ? FG_JACOBI_KERNEL_DATAFLOW
              : res_regions(f->NX, f->NY, 8) >= dv->sms ? FG_JACOBI_KERNEL_TMA
                                                        : FG_JACOBI_KERNEL_SWEEP;
  } else if (rinit)
    e = enqueue_jacobi(f->stream, f->g, ctl, b, bw, f->wgt, f->flags, x0, x1, iters, T,
                       f->prm.jacobi_omega * f->prm.pressure_damping, 0, f->prm.tolerance, &n,
                       f->phi, f->phi2, (const PCtl*)f->pctl, f->rhs_e, f->bwe);
  else
    e = enqueue_jacobi(f->stream, f->g, ctl, b, bw, f->wgt, f->flags, x0, x1, iters, T,
                       f->prm.jacobi_omega * f->prm.pressure_damping, check, f->prm.tolerance, &n,
                       nullptr, nullptr, nullptr, nullptr, nullptr, &f->dstats->timeout,
                       f->tile_done, f->stall_tile, -1, kind);
  count(f, n);
  if (e != cudaSuccess) return e;
  if (prof) {
    if ((e = cudaEventRecord(f->prof_ev[1], f->stream)) != cudaSuccess) return e;
    f->prof_launches = (int)nlaunch;
  }
  return cudaGetLastError();
}

cudaError_t launch_jacobi_solve(fg_fluid* f, void* ctl, const float* b, const float* bw, float* x0,
                                float* x1, int iters) {
  return jacobi_solve(f, (PCtl*)ctl, b, bw, x0, x1, iters, false);
}

// ------------------------------------------------------------------ multigrid Jacobi
// The MULTIGRID scheme: V(2,2) cycles on the masked Poisson system of the
// Jacobi scheme.  A coarse cell covers up to 2 x 2 fine cells (the ghost
// ring coarsens along its own row or column) and is fluid if any of them is;
// its flag bytes come from that mask as the fine ones come from S.  The
// smoother is the Jacobi scheme's sweep kernel with weight kMgOmega *
// PressureDamping (undamped Jacobi leaves the high frequencies a coarse grid
// cannot see); the coarse right-hand side is the sum of the children's
// residuals (the coarse operator has the fine one's form at twice the
// spacing, so the sum is the scaled average); the correction returns by
// bilinear interpolation (weights 9, 3, 3, 1) over the active coarse cells
// around each fine cell.  Every operation has a fixed order, restated by
// the oracle, so the result is bitwise reproducible.
constexpr int kMgPre = 2, kMgPost = 2, kMgCoarse = 32;

namespace {

// Rows of the fine grid (NXf rows) under coarse row I of NXc: the ring row
// under the ring, else rows 2I-1 and 2I of the interior.
__host__ __device__ __forceinline__ void mg_children(int I, int NXc, int NXf, int& a, int& b) {
  if (I == 0) {
    a = b = 0;
  } else if (I == NXc - 1) {
    a = b = NXf - 1;
  } else {
    a = 2 * I - 1;
    b = min(2 * I, NXf - 2);
  }
}

__global__ void k_mg_mask(const float* __restrict__ Sf, Grid gf, float* __restrict__ Sc, Grid gc) {
  int J = blockIdx.x * blockDim.x + threadIdx.x;
  int I = blockIdx.y * blockDim.y + threadIdx.y;
  if (I >= gc.NX || J >= gc.NY) return;
  int a0, a1, b0, b1;
  mg_children(I, gc.NX, gf.NX, a0, a1);
  mg_children(J, gc.NY, gf.NY, b0, b1);
  float v = 0.0f;
  for (int a = a0; a <= a1; ++a)
    for (int b = b0; b <= b1; ++b) v = fmaxf(v, Sf[a * gf.P + b]);
  Sc[I * gc.P + J] = v;
}

__global__ void k_mg_weights(const uint8_t* __restrict__ flags, float* __restrict__ w, float om,
                             Grid g) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.NX || j >= g.NY) return;
  const uint8_t fl = flags[i * g.P + j];
  w[i * g.P + j] = flag_active(fl) ? om / (float)flag_count(fl) : 0.0f;
}

// Coarse right-hand side at coarse cell (I, J): the sum of the active
// children's residuals b - (s x - (x_w + x_e + x_s + x_n)), and w * b.
__device__ __forceinline__ void mg_restrict_cell(int I, int J, const float* __restrict__ xf,
                                                 const float* __restrict__ bf,
                                                 const uint8_t* __restrict__ flf, const Grid& gf,
                                                 const uint8_t* __restrict__ flc,
                                                 const float* __restrict__ wc,
                                                 float* __restrict__ bc, float* __restrict__ bwc,
                                                 const Grid& gc) {
  // (Interior cells: the children are rows 2I-1, 2I and columns 2J-1, 2J, the
  // last without its pair on odd sides.  Every load is issued before the flags
  // select.)
  const int cc = I * gc.P + J;
  float rs = 0.0f;
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int i = 2 * I - 1 + a, j = 2 * J - 1 + b;
      const int cf = min(i, gf.NX - 2) * gf.P + min(j, gf.NY - 2);
      const uint8_t fl = flf[cf];
      float nb = xf[cf - gf.P] + xf[cf + gf.P] + xf[cf - 1] + xf[cf + 1];
      float ax = (float)flag_count(fl) * xf[cf] - nb;
      const float sum = rs + (bf[cf] - ax);
      rs = flag_active(fl) && i <= gf.NX - 2 && j <= gf.NY - 2 ? sum : rs;
    }
  rs = flag_active(flc[cc]) ? rs : 0.0f;
  bc[cc] = rs;
  bwc[cc] = wc[cc] * rs;
}
__global__ void k_mg_restrict(const float* __restrict__ xf, const float* __restrict__ bf,
                              const uint8_t* __restrict__ flf, Grid gf,
                              const uint8_t* __restrict__ flc, const float* __restrict__ wc,
                              float* __restrict__ bc, float* __restrict__ bwc, Grid gc) {
  pdl_enter();
  int J = blockIdx.x * blockDim.x + threadIdx.x;
  int I = blockIdx.y * blockDim.y + threadIdx.y;
  if (I < 1 || J < 1 || I > gc.NX - 2 || J > gc.NY - 2) return;
  mg_restrict_cell(I, J, xf, bf, flf, gf, flc, wc, bc, bwc, gc);
}

// x_f += the bilinear interpolation of x_c over the active coarse cells
// around the active fine cell (i, j).
__device__ __forceinline__ void mg_prolong_cell(int i, int j, const float* __restrict__ xc,
                                                const uint8_t* __restrict__ flc, const Grid& gc,
                                                float* __restrict__ xf,
                                                const uint8_t* __restrict__ flf, const Grid& gf) {
  const int cf = i * gf.P + j;
  const int I = (i - 1) / 2 + 1, J = (j - 1) / 2 + 1;
  const int di = ((i - 1) & 1) ? 1 : -1, dj = ((j - 1) & 1) ? 1 : -1;
  const int ci[4] = {I, I + di, I, I + di}, cj[4] = {J, J, J + dj, J + dj};
  const float wt[4] = {9.0f, 3.0f, 3.0f, 1.0f};
  const float x = xf[cf];
  const bool act = flag_active(flf[cf]);
  float num = 0.0f, den = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int cc = ci[k] * gc.P + cj[k];
    const bool on = flag_active(flc[cc]);
    const float sum = num + wt[k] * xc[cc];
    num = on ? sum : num;
    den = on ? den + wt[k] : den;
  }
  // (All four: den = 16, whose quotient the product with 1/16 is.)
  float e = num * 0.0625f;
  if (den != 16.0f) e = den > 0.0f ? num / den : 0.0f;
  if (act) xf[cf] = x + e;
}
__global__ void k_mg_prolong(const float* __restrict__ xc, const uint8_t* __restrict__ flc, Grid gc,
                             float* __restrict__ xf, const uint8_t* __restrict__ flf, Grid gf) {
  pdl_enter();
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i < 1 || j < 1 || i > gf.NX - 2 || j > gf.NY - 2) return;
  mg_prolong_cell(i, j, xc, flc, gc, xf, flf, gf);
}

// The bottom of the V-cycle in one block, in shared memory: levels l0 ..
// n-1 (a launch per operation would cost more than their work, and their
// arrays fit on one SM).  The block copies the levels' weights and flags
// and level l0's right-hand side into shared memory (rows of mg_pitch
// cells), zeroes the iterates, runs the same per-cell operations as the
// launches above and the Jacobi sweep kernel -- zero-started pre-smoothing
// and restriction down to the coarsest level, its sweeps, then
// prolongation and post-smoothing back up -- and writes level l0's iterate
// back to its buffer 0.  Every level starts in buffer 0 and makes an even
// number of sweeps, so its iterate ends in buffer 0; only interior cells
// are written and the ghost rings stay 0 as the sweep kernel leaves them.
// Latency bound (one block): 33 us for levels of 94 x 69 down to 6 x 5 cells
// against 41 with synchronous loads (7.6 us of it), rows of warps at every
// level and a block barrier in each of the 32 coarsest sweeps (7.5 us).
constexpr int kMgFuseLevels = 12, kMgFuseThreads = 1024;
constexpr int kMgSmemBytes = 200 * 1024;  // dynamic shared memory of k_mg_bottom
struct MgFused {
  Grid gg[kMgFuseLevels];               // the levels in global memory (pitched)
  Grid gs[kMgFuseLevels];               // the same in shared memory (pitch mg_pitch)
  const uint8_t* flags[kMgFuseLevels];  // global
  const float* w[kMgFuseLevels];        // global
  const float* b0;                      // level l0's right-hand side and w * b (global)
  const float* bw0;
  float* x0;                            // level l0's buffer 0 (global): the result
  int foff[kMgFuseLevels];              // first float of each level's arrays in shared memory
  int boff[kMgFuseLevels];              // first byte of each level's flags in shared memory
  int n;                                // levels held (the first is l0)
};
// A level's arrays in shared memory: five float arrays of NX * pitch, then flags.
struct MgSm {
  float *x0, *x1, *b, *bw, *w;
  uint8_t* fl;
};
__device__ __forceinline__ MgSm mg_sm(const MgFused& m, int l, float* fs, uint8_t* bs) {
  const int n = m.gs[l].NX * m.gs[l].P;
  float* p = fs + m.foff[l];
  return MgSm{p, p + n, p + 2 * n, p + 3 * n, p + 4 * n, bs + m.boff[l]};
}

__device__ __forceinline__ void mg_fused_sweeps(const MgSm& a, const Grid& g, int ns, bool zero,
                                                float om1) {
  const int tid = threadIdx.x, cols = g.NY - 2, n = (g.NX - 2) * cols;
  auto cell = [&](const float* xs, int c, float w, float bw, float xc, bool z) {
    float nb = z ? 0.0f : xs[c - g.P] + xs[c + g.P] + xs[c - 1] + xs[c + 1];
    float y = __fmaf_rn(w, nb, bw);
    return __fmaf_rn(om1, xc, y);
  };
  if (n <= kMgFuseThreads) {
    // One cell a thread, its weights and value in registers; a level of one
    // warp's cells needs no barrier between its sweeps.
    const int i = tid / cols, c = (1 + i) * g.P + 1 + tid - i * cols;
    const bool mine = tid < n, one = n <= 32;
    const float w = mine ? a.w[c] : 0.0f, bw = mine ? a.bw[c] : 0.0f;
    float xc = mine && !zero ? a.x0[c] : 0.0f;
    if (!one || tid < 32)
      for (int s = 0; s < ns; ++s) {
        if (mine) {
          xc = cell((s & 1) ? a.x1 : a.x0, c, w, bw, xc, zero && s == 0);
          ((s & 1) ? a.x0 : a.x1)[c] = xc;
        }
        if (one) __syncwarp();
        else __syncthreads();
      }
    if (one) __syncthreads();
    return;
  }
  const int lane = tid & 31, warp = tid >> 5, nw = kMgFuseThreads / 32;
  for (int s = 0; s < ns; ++s) {
    const float* __restrict__ xs = (s & 1) ? a.x1 : a.x0;
    float* __restrict__ xd = (s & 1) ? a.x0 : a.x1;
    const bool z = zero && s == 0;
    for (int i = 1 + warp; i < g.NX - 1; i += nw)
#pragma unroll 3
      for (int j = 1 + lane; j < g.NY - 1; j += 32) {
        const int c = i * g.P + j;
        xd[c] = cell(xs, c, a.w[c], a.bw[c], z ? 0.0f : xs[c], z);
      }
    __syncthreads();
  }
}

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem)), "l"(gmem)
               : "memory");
}

__global__ void __launch_bounds__(kMgFuseThreads, 1)
    k_mg_bottom(const __grid_constant__ MgFused m, float om1) {
  extern __shared__ __align__(16) float mg_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = kMgFuseThreads / 32;
  uint8_t* bsm = reinterpret_cast<uint8_t*>(mg_smem);
  const int last = m.n - 1;
  pdl_enter();
  // Every level's arrays in pieces of four cells, all copies in flight
  // together (pitches are multiples of 4; the pieces' last cells may be pitch
  // padding, which nothing reads).
  for (int l = 0; l <= last; ++l) {
    const MgSm a = mg_sm(m, l, mg_smem, bsm);
    const int q4 = m.gs[l].P / 4;
    for (int k = threadIdx.x; k < m.gs[l].NX * q4; k += kMgFuseThreads) {
      const int i = k / q4, cs = 4 * k, cg = i * m.gg[l].P + 4 * (k - i * q4);
      cp_async16(a.w + cs, m.w[l] + cg, 16);
      cp_async4(a.fl + cs, m.flags[l] + cg);
      if (l == 0) {
        cp_async16(a.b + cs, m.b0 + cg, 16);
        cp_async16(a.bw + cs, m.bw0 + cg, 16);
      }
      *reinterpret_cast<float4*>(a.x0 + cs) = make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(a.x1 + cs) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (int l = 0; l < last; ++l) {
    const MgSm f = mg_sm(m, l, mg_smem, bsm), c = mg_sm(m, l + 1, mg_smem, bsm);
    mg_fused_sweeps(f, m.gs[l], kMgPre, true, om1);
    const Grid& gf = m.gs[l];
    const Grid& gc = m.gs[l + 1];
    for (int k = threadIdx.x; k < (gc.NX - 2) * (gc.NY - 2); k += kMgFuseThreads) {
      const int I = k / (gc.NY - 2);
      mg_restrict_cell(1 + I, 1 + k - I * (gc.NY - 2), f.x0, f.b, f.fl, gf, c.fl, c.w, c.b, c.bw,
                       gc);
    }
    __syncthreads();
  }
  mg_fused_sweeps(mg_sm(m, last, mg_smem, bsm), m.gs[last], kMgCoarse, true, om1);
  for (int l = last - 1; l >= 0; --l) {
    const MgSm f = mg_sm(m, l, mg_smem, bsm), c = mg_sm(m, l + 1, mg_smem, bsm);
    const Grid& gf = m.gs[l];
    const Grid& gc = m.gs[l + 1];
    for (int i = 1 + warp; i < gf.NX - 1; i += nw)
      for (int j = 1 + lane; j < gf.NY - 1; j += 32)
        mg_prolong_cell(i, j, c.x0, c.fl, gc, f.x0, f.fl, gf);
    __syncthreads();
    mg_fused_sweeps(f, gf, kMgPost, false, om1);
  }
  const MgSm a = mg_sm(m, 0, mg_smem, bsm);
  for (int i = warp; i < m.gs[0].NX; i += nw)
    for (int j = lane; j < m.gs[0].NY; j += 32) m.x0[i * m.gg[0].P + j] = a.x0[i * m.gs[0].P + j];
}

inline dim3 level_grid(const Grid& g) { return dim3((g.NY + BX - 1) / BX, (g.NX + BY - 1) / BY); }

// ns (<= TMAX) damped Jacobi sweeps src -> dst on one level (4-warp
// regions on levels with fewer 8-warp regions than SMs, as enqueue_jacobi).
void mg_sweeps(cudaStream_t st, const MgLevelDev& v, const float* src, float* dst, float om1,
               PCtl* ctl, int t0, int ns, int sel, int zero) {
  dim3 gr(span_count(v.g.NY, RJ), span_count(v.g.NX, RI));
  const TmaDevice* dv = tma_ready(st);
  const bool narrow = dv && dv->sms > 0 && (long long)gr.x * gr.y < dv->sms;
#define FG_MGJ(F, NW)                                                                           \
  launch_pdl(k_jacobi_rb<false, F, false, false, NW>, dim3(gr.x, span_count(v.g.NX, RT * NW)),  \
             dim3(32 * NW), 0, st, src, dst, v.w, v.bw, nullptr, v.flags, om1, ctl, 0, t0, ns,  \
             0.0f, sel, zero, v.g, nullptr, nullptr, nullptr, nullptr, nullptr)
  if (narrow) {
    if (ns == TMAX) FG_MGJ(true, NWARP / 2); else FG_MGJ(false, NWARP / 2);
  } else {
    if (ns == TMAX) FG_MGJ(true, NWARP); else FG_MGJ(false, NWARP);
  }
#undef FG_MGJ
}

// The V-cycles of one solve.  cur[l] names the buffer of level l holding
// its iterate; the last smoothing of level 0 reports to the main control
// block (sweeps = cycles, sel = the buffer of the result).
// A level's pitch in shared memory: whole pieces of four cells.
inline int mg_pitch(int NY) { return (NY + 3) / 4 * 4; }

// The first coarse level from which all levels down fit k_mg_bottom's
// shared memory (at most kMgFuseLevels of them); the level count when none
// does.
int mg_bottom_level(const MgHier* h) {
  const int L = (int)h->lv.size();
  long long bytes = 0;
  int bottom = L;
  for (int l = L - 1; l >= 1 && L - l <= kMgFuseLevels; --l) {
    bytes += (5 * (long long)sizeof(float) + 1) * h->lv[l].g.NX * mg_pitch(h->lv[l].g.NY);
    if (bytes > kMgSmemBytes - 64) break;
    bottom = l;
  }
  return bottom;
}

struct MgRun {
  fg_fluid* f;
  MgHier* h;
  float om1;
  int cycles;
  std::vector<int> cur;
  int bottom;  // the first level run by k_mg_bottom (levels below it included)
  int launches = 0;
  void smooth(int l, int ns, bool zero, bool last) {
    MgLevelDev& v = h->lv[l];
    const int to = 1 - cur[l];
    PCtl* ctl = last ? (PCtl*)f->pctl : (PCtl*)h->ctl;
    mg_sweeps(f->stream, v, v.x[cur[l]], v.x[to], om1, ctl, last ? cycles - ns : 0, ns, to,
              zero ? 1 : 0);
    cur[l] = to;
    ++launches;
  }
  void cycle(int l, bool zero, bool last) {
    const int L = (int)h->lv.size();
    if (l == bottom) {
      MgFused m{};
      m.n = L - l;
      int fo = 0;
      for (int k = 0; k < m.n; ++k) {
        const MgLevelDev& v = h->lv[l + k];
        m.gg[k] = v.g;
        m.gs[k] = make_grid(v.g.NX, v.g.NY, mg_pitch(v.g.NY), v.g.h);
        m.flags[k] = v.flags;
        m.w[k] = v.w;
        m.foff[k] = fo;
        fo += 5 * v.g.NX * mg_pitch(v.g.NY);
      }
      int bo = fo * (int)sizeof(float);
      for (int k = 0; k < m.n; ++k) {
        m.boff[k] = bo;
        bo += h->lv[l + k].g.NX * mg_pitch(h->lv[l + k].g.NY);
      }
      m.b0 = h->lv[l].b;
      m.bw0 = h->lv[l].bw;
      m.x0 = h->lv[l].x[0];
      launch_pdl(k_mg_bottom, dim3(1), dim3(kMgFuseThreads), bo, f->stream, m, om1);
      cur[l] = 0;
      ++launches;
      return;
    }
    if (l == L - 1) {
      for (int k = 0; k < kMgCoarse / TMAX; ++k) smooth(l, TMAX, zero && k == 0, false);
      return;
    }
    MgLevelDev& v = h->lv[l];
    MgLevelDev& c = h->lv[l + 1];
    smooth(l, kMgPre, zero, false);
    launch_pdl(k_mg_restrict, level_grid(c.g), dim3(BX, BY), 0, f->stream, v.x[cur[l]], v.b,
               v.flags, v.g, c.flags, c.w, c.b, c.bw, c.g);
    ++launches;
    cycle(l + 1, true, false);
    launch_pdl(k_mg_prolong, level_grid(v.g), dim3(BX, BY), 0, f->stream, c.x[cur[l + 1]], c.flags,
               c.g, v.x[cur[l]], v.flags, v.g);
    ++launches;
    smooth(l, kMgPost, false, last && l == 0);
  }
};

cudaError_t mg_solve(fg_fluid* f, int cycles, float om) {
  MgHier* h = f->mg;
  if (!h || h->lv.size() < 2) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(h->ctl, 0, sizeof(PCtl), f->stream);
  if (e != cudaSuccess) return e;
  const int L = (int)h->lv.size();
  const int bottom = mg_bottom_level(h);
  MgRun run{f, h, 1.0f - om, cycles, std::vector<int>(h->lv.size(), 0), bottom};
  for (int k = 0; k < cycles; ++k) run.cycle(0, k == 0, k == cycles - 1);
  count(f, run.launches);
  return cudaGetLastError();
}

}  // namespace

cudaError_t mg_kernel_setup() {
  return cudaFuncSetAttribute(k_mg_bottom, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              kMgSmemBytes);
}

void mg_free(fg_fluid* f) {
  if (!f->mg) return;
  cudaFree(f->mg->block);
  cudaFree(f->mg->ctl);
  delete f->mg;
  f->mg = nullptr;
}

cudaError_t launch_mg_rebuild(fg_fluid* f) {
  MgHier* h = f->mg;
  if (!h) return cudaSuccess;
  const float om = kMgOmega * f->prm.pressure_damping;
  for (size_t l = 1; l < h->lv.size(); ++l) {
    const MgLevelDev& p = h->lv[l - 1];
    const MgLevelDev& c = h->lv[l];
    k_mg_mask<<<level_grid(c.g), dim3(BX, BY), 0, f->stream>>>(p.S, p.g, c.S, c.g);
    cudaError_t e = launch_build_flags_on(f->stream, c.S, c.flags, c.g);
    if (e != cudaSuccess) return e;
    k_mg_weights<<<level_grid(c.g), dim3(BX, BY), 0, f->stream>>>(c.flags, c.w, om, c.g);
  }
  h->omega = om;
  return cudaGetLastError();
}

// The gradient subtract; swaps in the projected U, V.  `ticket`: where the
// statistics are combined (null: they are not).
static cudaError_t launch_grad_fused(fg_fluid* f, PCtl* ctl, PCtl* ectl, const float* phi0,
                                     const float* phi1, float cp, float dt, bool fuse_turb,
                                     int* ticket, StoreDivP store) {
  const long long pieces = (long long)((f->NY + 3) / 4) * f->NX;
  const int nb = (int)std::min<long long>((pieces + 255) / 256, kGradBlocks);
  if (!partials_fit(f, 5, nb)) return cudaErrorInvalidValue;
  count(f);
  cudaError_t e = launch_pdl(
      f->step_fu || f->step_u2 ? k_grad_fused<true> : k_grad_fused<false>, dim3(nb), dim3(256), 0, f->stream, f->d[FG_U], f->d[FG_V], f->partner[FG_U],
      f->partner[FG_V], f->d[FG_P], phi0, phi1, ctl, f->err, f->err2, ectl, f->rhs, f->flags, cp,
      f->noise, f->prm.turbulence_strength * dt, fuse_turb ? 1 : 0, f->partials, f->g, f->step_fu,
      f->step_fv, f->step_u2, f->step_v2, ticket, store);
  swap_state(f, FG_U);
  swap_state(f, FG_V);
  return e;
}

cudaError_t launch_pressure(fg_fluid* f, int num_iters, float dt, bool fuse_turb) {
  float cp = f->density * f->h / dt;  // fluid.go:158
  cudaError_t e;
  f->jacobi_kernel = FG_JACOBI_KERNEL_NONE;
  f->jacobi_resident = 0;
  if (f->prm.scheme == FG_SCHEME_LEXSOR) return launch_lexsor(f, num_iters, dt);
  PCtl* ctl = (PCtl*)f->pctl;
  PCtl* ectl = (PCtl*)f->ectl;
  dim3 gr = cell_grid(f), bl(BX, BY);
  const bool mgs = f->prm.scheme == FG_SCHEME_MULTIGRID && !f->batch;
  float om = mgs ? kMgOmega * f->prm.pressure_damping
                 : f->prm.jacobi_omega * f->prm.pressure_damping;
  if (f->batch) {
    // Every scene solves (the batch forbids early exit and refinement);
    // no statistics.
    count(f);
    FG_CELLS_BATCH(f, setup_cell, (const float*)f->d[FG_U], (const float*)f->d[FG_V], f->phi,
                   f->rhs, f->wgt, f->bw, (const uint8_t*)f->flags, om, 1);
    if ((e = jacobi_solve_batch(f, ctl, f->bw, f->phi, f->phi2)) != cudaSuccess) return e;
    count(f);
    FG_CELLS_BATCH(f, grad_batch_cell, (const float*)f->d[FG_U], (const float*)f->d[FG_V],
                   f->partner[FG_U], f->partner[FG_V], f->d[FG_P], (const float*)f->phi,
                   (const float*)f->phi2, (const PCtl*)ctl, (const float*)f->rhs,
                   (const uint8_t*)f->flags, cp, (const float2*)f->noise,
                   f->prm.turbulence_strength * dt, fuse_turb ? 1 : 0, f->step_u2, f->step_v2);
    swap_state(f, FG_U);
    swap_state(f, FG_V);
    return cudaGetLastError();
  }
  // sel = 0 (phi) until a launch runs.
  if ((e = cudaMemsetAsync(ctl, 0, sizeof(PCtl), f->stream)) != cudaSuccess) return e;
  count(f);
  // Pieces of four cells leave too few threads to hide the loads on small
  // grids (us, cells against pieces: 128 x 128 2.3, 3.5; 512 x 256 2.6, 3.5;
  // 1500 x 1100 9.1, 7.2; 2048 x 2048 20.1, 14.1).
  if ((long long)f->NX * f->NY < (1 << 20)) {
    launch_pdl(k_setup_system, gr, bl, 0, f->stream, f->d[FG_U], f->d[FG_V], f->phi, f->rhs,
               f->wgt, f->bw, f->flags, om, num_iters == 0 ? 1 : 0, f->g, f->P, f->step_fu,
               f->step_fv);
  } else {
    const long long pieces = (long long)((f->NY + 3) / 4) * f->NX;
    launch_pdl(k_setup_pieces, dim3((unsigned)((pieces + 255) / 256)), dim3(256), 0, f->stream,
               f->d[FG_U], f->d[FG_V], f->phi, f->rhs, f->wgt, f->bw, f->flags, om,
               num_iters == 0 ? 1 : 0, f->g, f->step_fu, f->step_fv);
  }
  mark(f, "pressure setup");
  if (num_iters > 0) {
    e = mgs ? mg_solve(f, num_iters, om)
            : jacobi_solve(f, ctl, f->rhs, f->bw, f->phi, f->phi2, num_iters, true, false,
                           &f->jacobi_kernel);
    if (e != cudaSuccess) return e;
  }
  mark(f, "jacobi sweeps");
  bool refine = f->prm.refine_sweeps > 0;
  if (refine) {
    if ((e = jacobi_solve(f, ectl, f->rhs, f->bw, f->err, f->err2, f->prm.refine_sweeps, false,
                          true)) != cudaSuccess)
      return e;
    mark(f, "outer correction");
  }
  return launch_grad_fused(f, ctl, refine ? ectl : nullptr, f->phi, f->phi2, cp, dt, fuse_turb,
                           &f->dstats->ticket, StoreDivP{f->dstats, num_iters > 0 ? ctl : nullptr});
}

cudaError_t launch_store_phi(fg_fluid* f, float* dst) {
  int n = f->NX * f->P;
  count(f);
  const bool refine = f->prm.refine_sweeps > 0;
  k_store_phi<<<(n + 255) / 256, 256, 0, f->stream>>>(f->phi, f->phi2, (const PCtl*)f->pctl,
                                                      f->err, f->err2,
                                                      refine ? (const PCtl*)f->ectl : nullptr,
                                                      dst, n);
  return cudaGetLastError();
}

cudaError_t launch_grad_replay(fg_fluid* f, float dt, const float* phi, bool fuse_turb) {
  float cp = f->density * f->h / dt;  // fluid.go:158
  if (f->batch) {
    count(f);
    FG_CELLS_BATCH(f, grad_batch_cell, (const float*)f->d[FG_U], (const float*)f->d[FG_V],
                   f->partner[FG_U], f->partner[FG_V], f->d[FG_P], phi, phi,
                   (const PCtl*)f->pctl, (const float*)f->rhs, (const uint8_t*)f->flags, cp,
                   (const float2*)f->noise, f->prm.turbulence_strength * dt, fuse_turb ? 1 : 0,
                   f->step_u2, f->step_v2);
    swap_state(f, FG_U);
    swap_state(f, FG_V);
    return cudaGetLastError();
  }
  // The potential is the same buffer whichever one the control block names;
  // the statistics partials it writes are not combined.
  return launch_grad_fused(f, (PCtl*)f->pctl, nullptr, phi, phi, cp, dt, fuse_turb, nullptr,
                           StoreDivP{});
}

}  // namespace fg

// ===========================================================================
// Projection without allocation.
//
// Some callers cannot allocate device memory at the moment they need a
// projection: an embedding engine whose allocator owns all of the device
// memory, a real-time loop that forbids cudaMalloc (it may synchronise the
// device), or code running where allocation is not allowed at all.  For them
// fg_project_noalloc runs the Jacobi projection on caller-owned fields using
// the scratch array below instead of the handle's buffers.  The array is a
// fixed part of the library image, so every GPU that loads the library holds
// it (about 21 MiB) until the process exits.
// ===========================================================================
namespace fg {
namespace {

constexpr size_t kNoAllocMaxCells = (size_t)FG_NOALLOC_MAX_CELLS;  // num_x * padded num_y
constexpr int kNoAllocSlots = 4096;                                  // Jacobi launches per call
constexpr size_t kNoAllocCtlBytes = 256 + sizeof(unsigned) * kNoAllocSlots;
// The status word: nonzero when a bounded wait of the last call gave up.
constexpr size_t kNoAllocStatusOff = 21 * kNoAllocMaxCells + kNoAllocCtlBytes;
constexpr size_t kNoAllocBytes = kNoAllocStatusOff + 256;

// Scratch shared by every call on a device: phi, phi2, rhs, w, bw (floats),
// the flag bytes, the control block and the status word, carved at fixed
// offsets with the solver's own pitch (num_y rounded up to 32).  It keeps
// the previous call's contents; each call rewrites or clears what it reads.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// Flag bytes from a caller-owned S (nonzero = fluid).
__global__ void k_noalloc_flags(const float* __restrict__ S, uint8_t* __restrict__ flags, Grid g,
                                int Ps) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.NX || j >= g.NY) return;
  int c = i * g.P + j;
  uint8_t fl = 0;
  if (S[c] != 0.0f) fl |= F_FLUID;
  if (i > 0 && S[c - g.P] != 0.0f) fl |= F_W;
  if (i < g.NX - 1 && S[c + g.P] != 0.0f) fl |= F_E;
  if (j > 0 && S[c - 1] != 0.0f) fl |= F_S;
  if (j < g.NY - 1 && S[c + 1] != 0.0f) fl |= F_N;
  if (i >= 1 && i <= g.NX - 2 && j >= 1 && j <= g.NY - 2) fl |= F_INTERIOR;
  flags[i * Ps + j] = fl;
}

// The scratch array's address per CUDA context (context_key), looked up by
// the first call made in each context.  A full table is not an error: the
// address is then looked up on every call.
constexpr int kNoAllocCtx = 64;
std::mutex g_noalloc_mu;
unsigned long long g_noalloc_key[kNoAllocCtx] = {};
void* g_noalloc_ptr[kNoAllocCtx] = {};
int g_noalloc_used = 0;
std::atomic<int> g_noalloc_stall{-1};

cudaError_t noalloc_scratch(void** out) {
  unsigned long long key = context_key();
  if (key) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    for (int k = 0; k < g_noalloc_used; ++k)
      if (g_noalloc_key[k] == key) {
        *out = g_noalloc_ptr[k];
        return cudaSuccess;
      }
  }
  void* ptr = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
  if (e != cudaSuccess) return e;
  if (!key) key = context_key();  // the lookup made the primary context current
  if (key) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (g_noalloc_used < kNoAllocCtx) {
      g_noalloc_key[g_noalloc_used] = key;
      g_noalloc_ptr[g_noalloc_used++] = ptr;
    }
  }
  *out = ptr;
  return cudaSuccess;
}

}  // namespace

void set_noalloc_stall(int tile) { g_noalloc_stall.store(tile < 0 ? -1 : tile); }

}  // namespace fg

extern "C" int fg_project_noalloc(float* u, float* v, float* p, const float* s, int num_x,
                                  int num_y, int pitch, float density, float h, float dt,
                                  int num_iters, float jacobi_omega, float pressure_damping,
                                  int tb_depth, int early_exit, float tolerance, void* stream) {
  using namespace fg;
  if (!u || !v || !p || !s || num_x < 3 || num_y < 3 || pitch < num_y || num_iters < 0 ||
      !(h > 0.0f) || dt == 0.0f)
    return FG_ERR_INVALID;
  const int Ps = (num_y + 31) / 32 * 32;  // solver pitch inside the scratch
  if ((size_t)num_x * (size_t)Ps > kNoAllocMaxCells) return FG_ERR_TOO_LARGE;
  // The caller's fields are indexed with 32-bit integers too.
  if ((size_t)num_x * (size_t)pitch > (size_t)INT_MAX) return FG_ERR_TOO_LARGE;
  const int T = clamp_tb(tb_depth);
  // In 64 bits: a num_iters near INT_MAX must not wrap below the limit.
  const long long nlaunch = ((long long)num_iters + T - 1) / T;
  if (nlaunch > kNoAllocSlots) return FG_ERR_TOO_LARGE;
  void* base = nullptr;
  if (noalloc_scratch(&base) != cudaSuccess) return FG_ERR_CUDA;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* b = (unsigned char*)base;
  float* phi = (float*)b;
  float* phi2 = (float*)(b + 4 * kNoAllocMaxCells);
  float* rhs = (float*)(b + 8 * kNoAllocMaxCells);
  float* W = (float*)(b + 12 * kNoAllocMaxCells);
  float* BW = (float*)(b + 16 * kNoAllocMaxCells);
  uint8_t* flags = b + 20 * kNoAllocMaxCells;
  PCtl* ctl = (PCtl*)(b + 21 * kNoAllocMaxCells);
  int* status = (int*)(b + kNoAllocStatusOff);
  Grid g = make_grid(num_x, num_y, pitch, h);   // caller fields
  Grid gs = make_grid(num_x, num_y, Ps, h);     // solver arrays
  float om = jacobi_omega * pressure_damping;
  float cp = density * h / dt;
  dim3 gr((num_y + BX - 1) / BX, (num_x + BY - 1) / BY), bl(BX, BY);
  // The control words and the status word start at zero (sel = 0 until a
  // launch runs).
  if (cudaMemsetAsync(ctl, 0, pctl_bytes((int)nlaunch), st) != cudaSuccess ||
      cudaMemsetAsync(status, 0, sizeof(int), st) != cudaSuccess)
    return FG_ERR_CUDA;
  k_noalloc_flags<<<gr, bl, 0, st>>>(s, flags, g, Ps);
  k_setup_system<<<gr, bl, 0, st>>>(u, v, phi, rhs, W, BW, flags, om, num_iters == 0 ? 1 : 0, g,
                                    Ps, nullptr, nullptr);
  int n = 0;
  if (num_iters > 0 &&
      enqueue_jacobi(st, gs, ctl, rhs, BW, W, flags, phi, phi2, num_iters, T, om,
                     early_exit ? 1 : 0, tolerance, &n, nullptr, nullptr, nullptr, nullptr,
                     nullptr, status, nullptr, -1, g_noalloc_stall.load()) != cudaSuccess)
    return FG_ERR_CUDA;
  k_grad<<<gr, bl, 0, st>>>(u, v, p, phi, phi2, ctl, nullptr, nullptr, nullptr, flags, cp, g, Ps);
  return cudaGetLastError() == cudaSuccess ? FG_OK : FG_ERR_CUDA;
}

extern "C" int fg_project_noalloc_status(void* stream) {
  using namespace fg;
  int v = 0;
  cudaStream_t st = (cudaStream_t)stream;
  // The symbol is resolved in the current context, like the scratch itself.
  if (cudaMemcpyFromSymbolAsync(&v, g_noalloc_scratch, sizeof(int), kNoAllocStatusOff,
                                cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return FG_ERR_CUDA;
  return v ? FG_ERR_TIMEOUT : FG_OK;
}
