// The reference's serial pressure schemes, bit for bit
// (pkg/fluid/fluid.go:157-234, 559-758, 1122-1149).
//
// LEXSOR is solveSingleGrid / pressureJacobiIteration: the lexicographic SOR
// sweep in velocity form with the relaxation schedule 1.9 -> 1.2 and the
// early exit on max|div| < tolerance.  Cell (i, j) of a sweep needs (i-1, j)
// and (i, j-1) of that sweep and (i+1, j), (i, j+1) of the previous one.
// The V-cycle's coarse Gauss-Seidel has the same dependencies.
// k_wave runs either as a pipeline of warps in which every value sees the
// serial loop's sequence of operations, so the results are bit-identical.
#include <algorithm>
#include <climits>

#include "fg_internal.cuh"

namespace fg {

namespace {

constexpr int BX = 32, BY = 8;
inline dim3 cell_grid(const fg_fluid* f) {
  return dim3((f->NY + BX - 1) / BX, (f->NX + BY - 1) / BY);
}

// ------------------------------------------------------------------ pipeline
// One warp runs one sweep over a strip of 32 rows: lane l on row i0 - w + l
// marches along j one column behind lane l - 1, so at step s it is on column
// s - l and its west neighbour's result arrives by a warp shuffle.  The G <=
// 8 warps w of a block are consecutive sweeps of the same strip, each a chunk
// of WV_C columns behind the previous one; sweep w's rows are shifted down by
// w, which makes every dependency point to an earlier sweep or to the strip
// below (smaller i), never back: a strip needs nothing of the strip above
// within a group of G sweeps.  The strip's fields live in shared memory, a
// ring of WV_W columns that a loader warp fills and a storer warp drains, so
// the serial chain of a step is the shuffle and the arithmetic (about 50
// cycles), where a wavefront through L2 with a barrier per anti-diagonal paid
// a memory round trip and the barrier (2.4 us on one block, 2.4 us on eight).
// Between strips the topmost lane hands each column's new values on as one
// 16-byte packet {u, v, p, tag} in global memory, written and read whole, so
// the receiving warp polls the data itself and no fence or flag stands
// between the two.  Tasks (strip b, group g of sweeps) are claimed by ticket
// in the order of b + 2 g: a task needs (b-1, g), (b, g-1) and (b+1, g-1),
// all of earlier tickets, so whatever number of blocks is resident the oldest
// unfinished task can always proceed.
//
// Measured on a GB300 against the wavefront through L2 that it replaced (one
// block, an 8-block cluster or a grid barrier per anti-diagonal), whole
// passes from the host: the app's 300x251 jet with 8 sweeps and the early
// exit 1383 -> 329 us, two steps of a 128x128 jet with 40 sweeps 2891 -> 867
// us, a 1024x768 box with BFECC 4471 -> 903 us, a 512x512 box with 8
// reference V-cycles 45.7 -> 9.7 ms.
constexpr int WV_G = 8;            // sweeps per group (compute warps of a block)
constexpr int WV_C = 8;            // columns per chunk
constexpr int WV_W = 256;          // ring columns
constexpr int WV_M = WV_W - 1;
constexpr int WV_FP = WV_W + 16;   // row pitch of the ring's flag bytes
constexpr int WV_GROUPS = 256;     // groups per launch (slots of `fin` per strip)
constexpr int WV_SWEEPS = WV_G * WV_GROUPS;
constexpr int WV_A0 = 33 + WV_G, WV_A1 = 32 + WV_G;  // ring rows of the fields
constexpr unsigned long long WV_WAIT_NS = 1000000000ull;  // a wait gives up after 1 s
constexpr int WV_MAX_TRIES = 1 << 26;

// Control words of a handle's solves (zeroed once; every launch leaves them
// ready for the next).
struct WaveCtl {
  unsigned epoch;      // tag of the next launch's first group, minus 1
  unsigned ticket;     // next task
  unsigned exited;     // blocks that have left
  int fail;            // a bounded wait gave up
  int exit_sweep;      // speculative pass: first sweep below the tolerance + 1 (0: none)
  int pad[3];
  unsigned gmax[WV_SWEEPS];  // max |div| of each sweep of the launch (float bits)
};

// What the launch does with the early exit (fluid.go:177-179): PLAIN runs all
// sweeps in place; SPECULATE runs them from the state into scratch copies and
// records the first sweep whose max |div| is below the tolerance; FINISH
// copies the scratch fields into the state, or, when the serial loop would
// have stopped before the last sweep, runs exactly its sweeps on the state
// (sweeps up to that one are the same in both passes, so the result and the
// count are the serial loop's).
enum { WV_PLAIN = 0, WV_SPECULATE = 1, WV_FINISH = 2 };

struct WaveArgs {
  // SOR: U, V, p.  Coarse Gauss-Seidel: the solution (zero before group 0)
  // and the right-hand side in f0 / src[1].
  const float* src[3];  // group 0 reads these
  float* dst[3];        // every group writes these; later groups read them
  float* scratch[3];    // FINISH copies from these
  const uint8_t* flags;
  WaveCtl* ctl;
  unsigned long long* fin;  // [strip][group slot]: tag << 32 | final columns
  void* pkt;                // [strip][group parity][sweep][column]
  int NX, NY, P;
  int B;          // strips
  int G;          // sweeps per group
  int t0;         // first sweep of this launch
  int nsweeps;    // sweeps of this launch
  int iters;      // sweeps of the solve
  int last;       // the solve's last launch
  int mode;
  float relax0, relax1, damping, cp, tol;
  const int* stop;  // a multigrid solve that already converged does nothing
  DevStats* st;
  int* err;         // set when a bounded wait gave up
  int stall;        // fault injection: a strip that sends nothing (-1: none)
};

struct WaveShared {
  int prog[WV_G];  // chunks each sweep has finished
  int loaded;      // ring columns the loader has delivered
  int stored;      // columns the storer has drained
  int abort;
  int b, g;        // the task
  int last_block;
  int exit_at;
};

__device__ __forceinline__ unsigned long long wv_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ uint32_t wv_smem(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ int ld_cta(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(wv_smem(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_cta(int* p, int v) {
  asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(wv_smem(p)), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_gpu(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_gpu(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Packets: one 128-bit (SOR) or 64-bit (coarse) access each way, so a reader
// sees a packet whole or not at all.
__device__ __forceinline__ void st_pkt(uint4* p, uint4 v) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
      "mov.b128 t, {a, b};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
      : "memory");
}
__device__ __forceinline__ uint4 ld_pkt(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .b128 t;\n\t.reg .b64 a, b;\n\tld.relaxed.gpu.global.b128 t, [%4];\n\t"
      "mov.b128 {a, b}, t;\n\tmov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}
__device__ __forceinline__ void st_pkt2(uint2* p, uint2 v) {
  asm volatile("{\n\t.reg .b64 a;\n\tmov.b64 a, {%1, %2};\n\tst.relaxed.gpu.global.b64 [%0], a;\n\t}" ::"l"(p),
               "r"(v.x), "r"(v.y)
               : "memory");
}
__device__ __forceinline__ uint2 ld_pkt2(const uint2* p) {
  uint2 v;
  asm volatile(
      "{\n\t.reg .b64 a;\n\tld.relaxed.gpu.global.b64 a, [%2];\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "=r"(v.x), "=r"(v.y)
      : "l"(p)
      : "memory");
  return v;
}
// 16 bytes into shared memory, read past L1; zeros when !in.
__device__ __forceinline__ void wv_copy16(void* smem, const void* gmem, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(wv_smem(smem)), "l"(gmem),
               "r"(in ? 16 : 0)
               : "memory");
}

// Waits until *p >= need (a block's progress word); false when the wait gave
// up or the block is leaving.  The same in every lane.
__device__ __forceinline__ bool wv_wait(const int* p, int need, WaveShared* sh) {
  if (__all_sync(0xffffffffu, ld_cta(p) >= need)) return true;
  const unsigned long long t0 = wv_ns();
  for (int it = 1; it < WV_MAX_TRIES; ++it) {
    if (__all_sync(0xffffffffu, ld_cta(p) >= need)) return true;
    if ((it & 255) == 0 &&
        __any_sync(0xffffffffu, ld_cta(&sh->abort) != 0 || wv_ns() - t0 > WV_WAIT_NS))
      break;
  }
  st_cta(&sh->abort, 1);
  return false;
}

// x / n for the neighbour counts n = 1..4, correctly rounded: an exact
// scaling for the powers of two, and for 3 the quotient by the rounded
// reciprocal with Markstein's correction (IBM J. Res. Dev. 34, 1990), which
// is correctly rounded where the remainder is exact -- |x| >= 2^-100 here;
// compared with the division over every such float.  Smaller |x| divides.
__device__ __forceinline__ float div_count(float x, int n) {
  const float r = n == 4 ? 0.25f : n == 3 ? 1.0f / 3.0f : n == 2 ? 0.5f : 1.0f;
  float q = x * r;
  if (n == 3) {
    const float t = fabsf(x);
    const float q3 = __fmaf_rn(__fmaf_rn(-3.0f, q, x), r, q);
    if (t >= 0x1p-100f && t <= 3.402823466e38f)
      q = q3;
    else if (t > 0.0f && t < 0x1p-100f)
      q = x / 3.0f;
  }
  return q;
}
__device__ __forceinline__ float wv_bit(unsigned f, unsigned b) { return (f & b) ? 1.0f : 0.0f; }
__device__ __forceinline__ bool wv_active(unsigned f) {
  return (f & (F_FLUID | F_INTERIOR)) == (F_FLUID | F_INTERIOR) && (f & 15u) != 0;
}
constexpr unsigned WV_FULL = F_W | F_E | F_S | F_N | F_FLUID | F_INTERIOR;

// One sweep (warp w of the block, sweep t of the solve) of task (b, g).
// A0: U (SOR) or the solution; A1: V or the right-hand side; A2: p.  Ring row
// q of a field holds grid row i0 + q - WV_G.
template <bool GS>
__device__ void wv_sweep(const WaveArgs& a, WaveShared* sh, float* A0, float* A1, float* A2,
                         const uint8_t* F, int b, int g, int w, int Gt, int nchunks, unsigned tag) {
  const int lane = threadIdx.x & 31;
  const int q = WV_G - w + lane;
  float* r0 = A0 + q * WV_W;       // own row
  float* r0n = r0 + WV_W;          // row i + 1
  float* r0s = r0 - WV_W;          // row i - 1 (GS, lane 0)
  float* r1 = A1 + q * WV_W;
  float* r2 = GS ? nullptr : A2 + q * WV_W;
  const uint8_t* rf = F + q * WV_FP;
  const int t = a.t0 + g * a.G + w;
  const float prog_t = (float)t / (float)a.iters;
  const float rel = GS ? a.relax0 : a.relax0 - (a.relax0 - a.relax1) * prog_t;  // fluid.go:169-170
  const float damping = a.damping, cp = a.cp;
  const int NY = a.NY;
  const size_t slot = (size_t)(g & 1) * a.G + w;
  const size_t in_at = ((size_t)(b - 1) * 2 * a.G + slot) * a.P;
  const size_t out_at = ((size_t)b * 2 * a.G + slot) * a.P;
  const uint4* in4 = (const uint4*)a.pkt + in_at;
  uint4* out4 = (uint4*)a.pkt + out_at;
  const uint2* in2 = (const uint2*)a.pkt + in_at;
  uint2* out2 = (uint2*)a.pkt + out_at;
  const bool recv = b > 0, send = b + 1 < a.B && b != a.stall && lane == 31;
  float mx = 0.0f;
  // v0: V[i][j], updated by (i, j-1) (SOR); the old P[i][j] (GS).  ue: the
  // east face after the last step (SOR); the last step's new P (GS).
  float v0 = 0.0f, ue = 0.0f;
  float n1 = 0.0f, n2 = 0.0f, n3 = 0.0f, west = 0.0f;  // the next step's inputs
  unsigned nf = 0;
  int s = -2 * (w + 1);  // the chunk's first step
  uint4 pk = make_uint4(0, 0, 0, tag - 1);
  auto poll = [&](int c) {
    if (GS) {
      const uint2 x = ld_pkt2(in2 + c);
      pk.x = x.x;
      pk.w = x.y;
    } else {
      pk = ld_pkt(in4 + c);
    }
  };
  auto fetch = [&](int j) {  // inputs of column j
    const int c = j & WV_M, cn = (j + 1) & WV_M;
    n1 = r0n[c];                       // U[i+1][j]; the old P[i+1][j]
    n2 = GS ? r0[cn] : r1[cn];         // V[i][j+1]; the old P[i][j+1]
    n3 = GS ? r1[c] : r2[c];           // p; the right-hand side
    nf = rf[c];
  };
  if (recv && lane < WV_C && (unsigned)(s + lane) < (unsigned)NY) poll(s + lane);
  for (int n = 0; n < nchunks; ++n, s += WV_C) {
    if (w == 0) {
      if (!wv_wait(&sh->loaded, min(s + WV_C + 2, a.P), sh)) return;
    } else {
      if (!wv_wait(&sh->prog[w - 1], n + 1, sh)) return;
    }
    if (recv) {
      // The chunk's packets from the strip below: the west values of this
      // sweep's lowest row, and that neighbour row's other values, which
      // the next sweep's lowest row starts from.
      const int c = s + lane;
      const bool mine = lane < WV_C && (unsigned)c < (unsigned)NY;
      if (__any_sync(0xffffffffu, mine && pk.w != tag)) {
        const unsigned long long w0 = wv_ns();
        bool ok = false;
        for (int it = 1; it < WV_MAX_TRIES; ++it) {
          if (mine && pk.w != tag) poll(c);
          if (!__any_sync(0xffffffffu, mine && pk.w != tag)) {
            ok = true;
            break;
          }
          if ((it & 255) == 0 &&
              __any_sync(0xffffffffu, ld_cta(&sh->abort) != 0 || wv_ns() - w0 > WV_WAIT_NS))
            break;
        }
        if (!ok) {
          st_cta(&sh->abort, 1);
          return;
        }
      }
      if (mine) {
        const int ql = (WV_G - w) * WV_W + (c & WV_M);
        if (GS) {
          A0[ql - WV_W] = __uint_as_float(pk.x);
        } else {
          A0[ql] = __uint_as_float(pk.x);
          if (w + 1 < Gt) {
            A1[ql - WV_W] = __uint_as_float(pk.y);
            A2[ql - WV_W] = __uint_as_float(pk.z);
          }
        }
      }
      __syncwarp();
      if (lane < WV_C && (unsigned)(c + WV_C) < (unsigned)NY) poll(c + WV_C);
    }
    if (n == 0) fetch(s - lane);
    if (lane == 0) west = GS ? r0s[s & WV_M] : r0[s & WV_M];
    auto step = [&](int k, bool edge) {
      const int j = s + k - lane;
      const bool in = !edge || (unsigned)j < (unsigned)NY;
      float wv = __shfl_up_sync(0xffffffffu, ue, 1);
      if (lane == 0) wv = west;
      const float x1 = n1, x2 = n2, x3 = n3;
      const unsigned fl = in ? nf : 0u;
      fetch(j + 1);
      if (lane == 0 && k + 1 < WV_C) west = (GS ? r0s : r0)[(j + 1) & WV_M];
      const bool full = __all_sync(0xffffffffu, fl == WV_FULL);
      const int c = j & WV_M;
      if (GS) {
        float out = v0;
        if (full) {
          const float lap = (wv - v0) + (x1 - v0) + (ue - v0) + (x2 - v0);
          out = v0 + -(x3 - lap) * 0.25f * rel;
        } else if (wv_active(fl)) {
          const float lap = wv_bit(fl, F_W) * (wv - v0) + wv_bit(fl, F_E) * (x1 - v0) +
                            wv_bit(fl, F_S) * (ue - v0) + wv_bit(fl, F_N) * (x2 - v0);
          out = v0 + div_count(-(x3 - lap), __popc(fl & 15u)) * rel;
        }
        if (in) r0[c] = out;
        if (send && in) st_pkt2(out2 + j, make_uint2(__float_as_uint(out), tag));
        ue = out;
        v0 = x2;
      } else {
        const float div = x1 - wv + x2 - v0;
        float un = wv, en = x1, vn = v0, tn = x2, pn = x3;
        if (full) {
          mx = fmaxf(mx, fabsf(div));
          float pp = -div * 0.25f;
          pp *= rel;
          pp *= damping;
          pn = x3 + cp * pp;
          un = wv - pp;
          en = x1 + pp;
          vn = v0 - pp;
          tn = x2 + pp;
        } else if (wv_active(fl)) {
          mx = fmaxf(mx, fabsf(div));
          float pp = div_count(-div, __popc(fl & 15u));
          pp *= rel;
          pp *= damping;
          pn = x3 + cp * pp;
          un = wv - wv_bit(fl, F_W) * pp;
          en = x1 + wv_bit(fl, F_E) * pp;
          vn = v0 - wv_bit(fl, F_S) * pp;
          tn = x2 + wv_bit(fl, F_N) * pp;
        }
        if (in) {
          r0[c] = un;
          r1[c] = vn;
          r2[c] = pn;
        }
        if (send && in)
          st_pkt(out4 + j, make_uint4(__float_as_uint(en), __float_as_uint(vn), __float_as_uint(pn), tag));
        ue = en;
        v0 = tn;
      }
    };
    if (s - 31 >= 0 && s + WV_C <= NY) {
#pragma unroll
      for (int k = 0; k < WV_C; ++k) step(k, false);
    } else {
#pragma unroll 1
      for (int k = 0; k < WV_C; ++k) step(k, true);
    }
    __syncwarp();
    if (lane == 0) st_cta(&sh->prog[w], n + 1);
  }
  if (!GS) {
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
    if (lane == 0 && m) atomicMax(&a.ctl->gmax[g * a.G + w], m);
  }
}

// Copies 32 ring columns (from column c) of the rows [q0, q1) of a field
// whose ring row q is grid row i0 + q - WV_G; rows outside the grid, and
// everything when !data, become zeros.
template <typename T>
__device__ __forceinline__ void wv_load_rows(T* ring, int pitch, const T* src, int q0, int q1, int i0,
                                             int c, int NX, int P, bool data) {
  constexpr int PER = 16 / sizeof(T), SEG = 32 / PER;
  const int lane = threadIdx.x & 31;
  for (int it = lane; it < (q1 - q0) * SEG; it += 32) {
    const int q = q0 + it / SEG, e = (it % SEG) * PER;
    const int i = i0 + q - WV_G;
    const bool in = data && i >= 0 && i < NX;
    wv_copy16(ring + q * pitch + (c & WV_M) + e, in ? src + (size_t)i * P + c + e : src, in);
  }
}

// The loader warp: 32 columns at a time, as far ahead as the ring has room.
template <bool GS>
__device__ void wv_loader(const WaveArgs& a, WaveShared* sh, float* A0, float* A1, float* A2,
                          uint8_t* F, int b, int g, unsigned tag) {
  const int lane = threadIdx.x & 31;
  const int i0 = 1 + 32 * b, lo = WV_G - (a.G - 1), hi = WV_G + 32;
  const float* s0 = g ? a.dst[0] : a.src[0];
  const float* s1 = GS ? a.src[1] : g ? a.dst[1] : a.src[1];
  const float* s2 = GS ? nullptr : g ? a.dst[2] : a.src[2];
  // The groups below this one that it reads the results of: lane 0 watches
  // this strip's, lane 1 the strip above's.
  const bool dep = g > 0 && lane < 2 && b + lane < a.B;
  const unsigned long long* fin =
      a.fin + (size_t)(dep ? b + lane : 0) * WV_GROUPS + (dep ? (g - 1) % WV_GROUPS : 0);
  auto ready = [&](int c) {
    bool r = true;
    if (dep) {
      const unsigned long long v = ld_gpu(fin);
      r = (unsigned)(v >> 32) == tag - 1 && (int)(v & 0xffffffffu) >= min(c + 32, a.NY);
    }
    return __all_sync(0xffffffffu, r) != 0;
  };
  auto publish = [&](int cols) {
    __syncwarp();
    if (lane == 0) st_cta(&sh->loaded, cols);
  };
  bool ok = true;
  int pending = 0;  // columns copied but not yet published (0: none)
  for (int c = 0; c < a.P && ok; c += 32) {
    const int room = c + 32 - WV_W;
    bool now = (room <= 0 || __all_sync(0xffffffffu, ld_cta(&sh->stored) >= room)) && ready(c);
    if (!now) {
      if (pending) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        publish(pending);
        pending = 0;
      }
      if (room > 0) ok = wv_wait(&sh->stored, room, sh);
      const unsigned long long t0 = wv_ns();
      for (int it = 1; ok && !ready(c); ++it)
        if ((it & 63) == 0 &&
            (it >= WV_MAX_TRIES ||
             __any_sync(0xffffffffu, ld_cta(&sh->abort) != 0 || wv_ns() - t0 > WV_WAIT_NS))) {
          st_cta(&sh->abort, 1);
          ok = false;
        }
      if (!ok) break;
    }
    if (GS) {
      // Row 0 and the rows below it hold zeros (strip 0); the right-hand side
      // and the flags reach down to the last sweep's rows.
      wv_load_rows(A0, WV_W, s0, b ? WV_G : 0, hi + 1, i0, c, a.NX, a.P, g > 0);
      wv_load_rows(A1, WV_W, s1, lo, hi, i0, c, a.NX, a.P, true);
    } else {
      wv_load_rows(A0, WV_W, s0, WV_G, hi + 1, i0, c, a.NX, a.P, true);
      wv_load_rows(A1, WV_W, s1, WV_G, hi, i0, c, a.NX, a.P, true);
      wv_load_rows(A2, WV_W, s2, WV_G, hi, i0, c, a.NX, a.P, true);
    }
    wv_load_rows(F, WV_FP, a.flags, lo, hi, i0, c, a.NX, a.P, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (pending) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      publish(pending);
    }
    pending = c + 32;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (pending) publish(pending);
}

// The storer warp: the group's final values, 32 columns at a time, once its
// last sweep's topmost lane has passed them.
template <bool GS>
__device__ void wv_storer(const WaveArgs& a, WaveShared* sh, const float* A0, const float* A1,
                          const float* A2, int b, int g, int Gt, int nchunks, unsigned tag,
                          bool more) {
  const int lane = threadIdx.x & 31;
  const int i0 = 1 + 32 * b;
  constexpr int NF = GS ? 1 : 3;
  const int first = GS ? 0 : 1;  // (GS: strip 0 also writes row 0's zeros)
  for (int c = 0; c < a.P; c += 32) {
    // Lane 31 passes column c + 31 in step c + 62.
    const int need = min((c + 63 + 2 * Gt + WV_C - 1) / WV_C, nchunks);
    if (!wv_wait(&sh->prog[Gt - 1], need, sh)) return;
#pragma unroll
    for (int fd = 0; fd < NF; ++fd) {
      const float* ring = fd == 0 ? A0 : fd == 1 ? A1 : A2;
      float* dst = a.dst[fd];
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const int r = m * 4 + (lane >> 3), e = (lane & 7) * 4;
        const int q = WV_G - (Gt - 1) + r, i = i0 - (Gt - 1) + r, j = c + e;
        const float4 v = *reinterpret_cast<const float4*>(ring + q * WV_W + (c & WV_M) + e);
        if (i < first || i >= a.NX || j >= a.NY) continue;
        float* d = dst + (size_t)i * a.P + j;
        if (j + 4 <= a.NY) {
          *reinterpret_cast<float4*>(d) = v;
        } else {
          d[0] = v.x;
          if (j + 1 < a.NY) d[1] = v.y;
          if (j + 2 < a.NY) d[2] = v.z;
        }
      }
    }
    if (more) __threadfence();
    __syncwarp();
    if (lane == 0) {
      if (more)
        st_gpu(a.fin + (size_t)b * WV_GROUPS + g % WV_GROUPS,
               (unsigned long long)tag << 32 | (unsigned)(c + 32));
      st_cta(&sh->stored, c + 32);
    }
  }
}

template <bool GS>
__global__ void __launch_bounds__((WV_G + 2) * 32) k_wave(WaveArgs a) {
  extern __shared__ __align__(16) unsigned char wv_dyn[];
  __shared__ WaveShared sh;
  if (a.stop && *a.stop) return;  // (the same in every block)
  float* A0 = reinterpret_cast<float*>(wv_dyn);
  float* A1 = A0 + WV_A0 * WV_W;
  float* A2 = A1 + WV_A1 * WV_W;
  uint8_t* F = reinterpret_cast<uint8_t*>(GS ? A2 : A2 + WV_A1 * WV_W);
  WaveCtl* ctl = a.ctl;
  const int warp = threadIdx.x >> 5;
  const unsigned epoch = ctl->epoch;
  int nsw = a.nsweeps;
  bool copy = false;
  const int found = ctl->exit_sweep;  // (changed only after every block has left)
  if (a.mode == WV_SPECULATE && a.t0 > 0 && found) nsw = 0;
  if (a.mode == WV_FINISH) {
    const bool rerun = found && found < a.iters;
    nsw = rerun ? max(0, min(a.nsweeps, found - a.t0)) : 0;
    copy = !rerun && a.last;
  }
  const int ng = (nsw + a.G - 1) / a.G, ntasks = a.B * ng;
  if (threadIdx.x == 0) sh.abort = 0;
  int key = 0, before = 0;  // ticket decoding (thread 0): tasks with b + 2 g < key
  for (;;) {
    if (threadIdx.x == 0) {
      sh.b = -1;
      const int tk = ntasks ? (int)atomicAdd(&ctl->ticket, 1u) : 0;
      if (tk < ntasks && !sh.abort && !*(volatile int*)&ctl->fail) {
        for (;;) {
          const int g0 = max(0, (key - a.B + 2) / 2), g1 = min(ng - 1, key / 2);
          const int cnt = g1 - g0 + 1;
          if (tk < before + cnt) {
            sh.g = g0 + (tk - before);
            sh.b = key - 2 * sh.g;
            break;
          }
          before += max(cnt, 0);
          ++key;
        }
      }
      for (int w = 0; w < WV_G; ++w) sh.prog[w] = 0;
      sh.loaded = 0;
      sh.stored = 0;
    }
    __syncthreads();
    const int b = sh.b, g = sh.g;
    if (b < 0) break;
    const int Gt = min(a.G, nsw - g * a.G);
    const int nchunks = (a.NY + 31 + 2 * Gt + WV_C - 1) / WV_C;
    const unsigned tag = epoch + 1u + (unsigned)g;
    if (warp == a.G)
      wv_loader<GS>(a, &sh, A0, A1, A2, F, b, g, tag);
    else if (warp == a.G + 1)
      wv_storer<GS>(a, &sh, A0, A1, A2, b, g, Gt, nchunks, tag, g + 1 < ng);
    else if (warp < Gt)
      wv_sweep<GS>(a, &sh, A0, A1, A2, F, b, g, warp, Gt, nchunks, tag);
    __syncthreads();
  }
  if (copy) {
    // The speculative result: rows 1 .. NX - 1 of U, V and p.
    const int per = a.P / 4, n = (a.NX - 1) * per;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
      const size_t at = (size_t)(k / per + 1) * a.P + (size_t)(k % per) * 4;
      if ((k % per) * 4 >= a.NY) continue;
#pragma unroll
      for (int fd = 0; fd < 3; ++fd) {
        const float4 v = *reinterpret_cast<const float4*>(a.scratch[fd] + at);
        float* d = a.dst[fd] + at;
        const int left = a.NY - (k % per) * 4;
        if (left >= 4) {
          *reinterpret_cast<float4*>(d) = v;
        } else {
          d[0] = v.x;
          if (left > 1) d[1] = v.y;
          if (left > 2) d[2] = v.z;
        }
      }
    }
  }
  // The last block to leave reports the sweeps and readies the control words
  // for the next launch.
  __syncthreads();
  if (threadIdx.x == 0) {
    if (sh.abort) atomicExch(&ctl->fail, 1);
    __threadfence();
    sh.last_block = atomicAdd(&ctl->exited, 1u) == gridDim.x - 1;
    sh.exit_at = INT_MAX;
  }
  __syncthreads();
  if (!sh.last_block) return;
  __threadfence();
  if (!GS) {
    for (int t = threadIdx.x; t < nsw; t += blockDim.x) {
      const unsigned m = __ldcg(&ctl->gmax[t]);
      ctl->gmax[t] = 0u;
      if (a.mode == WV_SPECULATE && __uint_as_float(m) < a.tol) atomicMin(&sh.exit_at, t);
      if (t == nsw - 1) {
        a.st->sweeps = a.t0 + nsw;
        a.st->last_maxdiv = (double)__uint_as_float(m);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (a.mode == WV_SPECULATE && sh.exit_at != INT_MAX) ctl->exit_sweep = a.t0 + sh.exit_at + 1;
    if (a.mode == WV_FINISH && a.last) ctl->exit_sweep = 0;
    ctl->epoch = epoch + (unsigned)WV_GROUPS;
    ctl->ticket = 0;
    ctl->exited = 0;
    if (*(volatile int*)&ctl->fail) {
      ctl->fail = 0;
      atomicExch(a.err, 1);
    }
  }
}

// ------------------------------------------------------------------ without the pipeline's buffers
// The same sweeps as an anti-diagonal wavefront on one block, straight on the
// row-major fields: what runs when the pipeline's buffers cannot be allocated.
// Cell (i, j) of a sweep needs (i-1, j), (i, j-1) of that sweep and (i+1, j),
// (i, j+1) of the previous one, so consecutive sweeps run two diagonals apart.
// q / n and q % n for 0 <= q < 2^24, n > 0, from a float reciprocal and one
// correction step (exact: q and the candidate products are exact in float
// range, and the float quotient is off by at most one).
__device__ __forceinline__ int div_small(int q, int n, float inv_n, int& rem) {
  int t = __float2int_rz((float)q * inv_n);
  int r = q - t * n;
  if (r < 0) {
    --t;
    r += n;
  } else if (r >= n) {
    ++t;
    r -= n;
  }
  rem = r;
  return t;
}
constexpr int LEX_THREADS = 1024;
constexpr int LEX_RING = 4096;  // sweeps in flight (a new sweep waits while the ring is full)
constexpr int LEX_CHUNK = 4;    // cells whose loads a thread issues together

__global__ void __launch_bounds__(LEX_THREADS)
    k_lexsor(float* U, float* V, float* p, const uint8_t* __restrict__ flags, Grid g,
             int numIters, float relax0, float damping, float cp, float tol, int early_exit,
             DevStats* st, float minRelax, const int* __restrict__ stop) {
  __shared__ int s_start[LEX_RING];
  __shared__ unsigned s_max[LEX_RING];
  __shared__ uint8_t s_cont[LEX_RING];
  __shared__ int s_lo, s_hi, s_done, s_exit, s_last;
  const int P = g.P;
  const int ni = g.NX - 2, nj = g.NY - 2;  // interior extent
  const int D = ni + nj - 1;               // anti-diagonals d = i + j in [2, NX+NY-4]
  const int offE = P, offN = 1;
  const int L = ni < nj ? ni : nj;         // longest diagonal
  if (threadIdx.x == 0) {
    s_lo = 0;
    s_hi = 0;
    s_done = 0;
    s_exit = 0;
    s_last = -1;
  }
  __syncthreads();
  if (numIters <= 0 || ni <= 0 || nj <= 0) return;
  if (stop && *stop) return;  // a multigrid solve that already converged
  // The cells of the W sweeps lo .. lo+W-1 that step tau reaches; sweep t is
  // on diagonal 2 + delta_of(t) (out of range: not running) and its max
  // |div| goes to s_max[r] (r = t mod LEX_RING).
  auto step = [&](long long tau, int lo, int W, auto delta_of) {
      // Each warp takes 32 cells of one sweep's diagonal (the diagonal length
      // padded to a multiple of 32), so the sweep's max |div| and its
      // "cannot exit" mark are reduced in the warp and stored once per warp.
      // The cells a step updates share no face or pressure value (cells of one
      // diagonal are not neighbours; sweeps in flight are two diagonals
      // apart), so a thread loads the inputs of LEX_CHUNK cells at once and
      // then updates them: one memory round trip per chunk instead of one per
      // cell.
      const int Lp = (L + 31) & ~31;
      const float invLp = 1.0f / (float)Lp;
      const int items = W * Lp;
      for (int base = 0; base < items; base += LEX_CHUNK * LEX_THREADS) {
        int cc[LEX_CHUNK], rr[LEX_CHUNK], tt[LEX_CHUNK];
        bool act[LEX_CHUNK] = {};
        uint8_t fl[LEX_CHUNK];
        float u0[LEX_CHUNK], u1[LEX_CHUNK], v0[LEX_CHUNK], v1[LEX_CHUNK], p0[LEX_CHUNK];
#pragma unroll
        for (int m = 0; m < LEX_CHUNK; ++m) {
          if (base + m * LEX_THREADS >= items) break;  // (block-uniform)
          const int q = base + m * LEX_THREADS + (int)threadIdx.x;
          int k;
          const int t = lo + (items < (1 << 24) ? div_small(q, Lp, invLp, k) : (k = q % Lp, q / Lp));
          const int r = t & (LEX_RING - 1);
          const int delta = q < items ? delta_of(t) : -1;
          const int d = 2 + delta;
          const int i_lo = max(1, d - nj), i_hi = min(ni, d - 1);
          const int i = i_lo + k;
          const bool in = delta >= 0 && delta < D && k < L && i <= i_hi;
          const int c = in ? i * P + (d - i) : 0;
          cc[m] = c;
          rr[m] = r;
          tt[m] = t;
          act[m] = in;
          fl[m] = in ? flags[c] : 0;
          u0[m] = in ? U[c] : 0.0f;
          u1[m] = in ? U[c + offE] : 0.0f;
          v0[m] = in ? V[c] : 0.0f;
          v1[m] = in ? V[c + offN] : 0.0f;
          p0[m] = in ? p[c] : 0.0f;
        }
#pragma unroll
        for (int m = 0; m < LEX_CHUNK; ++m) {
          if (base + m * LEX_THREADS >= items) break;  // (whole warps: items is a multiple of 32)
          const uint8_t f = fl[m];
          bool a = act[m] && (f & F_FLUID);
          const float sx0 = fbit(f, F_W), sx1 = fbit(f, F_E), sy0 = fbit(f, F_S),
                      sy1 = fbit(f, F_N);
          const float s = sx0 + sx1 + sy0 + sy1;
          a = a && s != 0.0f;
          const float div = a ? u1[m] - u0[m] + v1[m] - v0[m] : 0.0f;
          const float absDiv = fabsf(div);
          const bool counted = a && !isnan(absDiv);
          const unsigned mx = __reduce_max_sync(0xffffffffu, counted ? __float_as_uint(absDiv) : 0u);
          const bool cont = __any_sync(0xffffffffu, counted && absDiv >= tol);
          // (Without the early exit only the last sweep's max is reported,
          // and more sweeps than ring slots may be in flight.)
          if ((threadIdx.x & 31) == 0 && (early_exit || tt[m] == numIters - 1)) {
            if (mx) atomicMax(&s_max[rr[m]], mx);
            if (cont) s_cont[rr[m]] = 1;
          }
          if (!a) continue;
          const int c = cc[m];
          // Relaxation of sweep t (fluid.go:169-170).
          float iterProgress = (float)tt[m] / (float)numIters;
          float rel = relax0 - (relax0 - minRelax) * iterProgress;
          float pp = -div / s;
          pp *= rel;
          pp *= damping;
          p[c] = p0[m] + cp * pp;
          U[c] = u0[m] - sx0 * pp;
          U[c + offE] = u1[m] + sx1 * pp;
          V[c] = v0[m] - sy0 * pp;
          V[c + offN] = v1[m] + sy1 * pp;
        }
      }
  };
  if (!early_exit) {
    // Without the early exit sweep t always starts at step 2t (two steps
    // after the previous one, as the bookkeeping below would start it):
    // sweep t covers steps 2t .. 2t + D - 1 and the steps need no
    // bookkeeping between them, one barrier each.
    for (int r = threadIdx.x; r < LEX_RING; r += LEX_THREADS) s_max[r] = 0u;
    __shared__ unsigned s_lastmax;
    if (threadIdx.x == 0) s_lastmax = 0u;
    __syncthreads();
    const long long steps = (long long)D + 2LL * (numIters - 1);
    for (long long tau = 0; tau < steps; ++tau) {
      int t_lo = (int)((tau - D + 2) / 2);
      if (t_lo < 0) t_lo = 0;
      while (tau - 2LL * t_lo >= D) ++t_lo;
      int t_hi = (int)(tau / 2);
      if (t_hi > numIters - 1) t_hi = numIters - 1;
      step(tau, t_lo, t_hi - t_lo + 1, [&](int t) { return (int)(tau - 2LL * t); });
      __syncthreads();
      // The sweep whose last diagonal ran in this step retires.
      const long long rt = tau - (D - 1);
      if (threadIdx.x == 0 && rt >= 0 && (rt & 1) == 0 && rt / 2 < numIters) {
        const int t = (int)(rt / 2), r = t & (LEX_RING - 1);
        const unsigned m = s_max[r];
        if (t == numIters - 1) s_lastmax = m;
        s_max[r] = 0u;  // (slot reused by sweep t + LEX_RING, not yet started)
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      st->sweeps = numIters;
      st->last_maxdiv = (double)__uint_as_float(s_lastmax);
    }
    return;
  }
  // Start sweep 0 at step 0.
  if (threadIdx.x == 0) {
    s_start[0] = 0;
    s_max[0] = 0u;
    s_cont[0] = 0;
    s_hi = 1;
  }
  __syncthreads();
  // Bounded: each sweep takes D steps and starts at most D + 2 steps after
  // the previous one.
  const long long max_steps = (long long)numIters * (D + 2) + D + 4;
  for (long long tau = 0; tau < max_steps; ++tau) {
    const int lo = s_lo, hi = s_hi;
    step(tau, lo, hi - lo, [&](int t) { return (int)(tau - s_start[t & (LEX_RING - 1)]); });
    __syncthreads();
    if (threadIdx.x == 0) {
      // Retire sweeps whose last diagonal ran in this step.
      while (s_lo < s_hi && tau - s_start[s_lo & (LEX_RING - 1)] >= D - 1) {
        int r = s_lo & (LEX_RING - 1);
        s_last = s_lo;
        if (early_exit && __uint_as_float(s_max[r]) < tol) s_exit = 1;
        ++s_lo;
      }
      // Start the next sweep if allowed.
      int nxt = s_hi;
      if (!s_exit && nxt < numIters) {
        int pr = (nxt - 1) & (LEX_RING - 1);
        bool prev_done = s_lo > nxt - 1;
        bool gap_ok = prev_done || (tau + 1 - s_start[pr] >= 2);
        bool safe = !early_exit || prev_done || s_cont[pr];
        if (gap_ok && safe && nxt - s_lo < LEX_RING) {
          int r = nxt & (LEX_RING - 1);
          s_start[r] = (int)(tau + 1);
          s_max[r] = 0u;
          s_cont[r] = 0;
          s_hi = nxt + 1;
        }
      }
      if (s_lo == s_hi && (s_exit || s_hi >= numIters)) s_done = 1;
    }
    __syncthreads();
    if (s_done) break;
  }
  if (threadIdx.x == 0) {
    st->sweeps = s_hi;
    st->last_maxdiv = s_last >= 0 ? (double)__uint_as_float(s_max[s_last & (LEX_RING - 1)]) : 0.0;
  }
}

// ------------------------------------------------------------------ multigrid
// solveMultigridVCycle (fluid.go:559-594) with its helpers (fluid.go:596-758,
// 1122-1149): per iteration three SOR sweeps at relaxation 1.5,
// the early exit on the last sweep's max |div|, the residual restricted by
// full weighting to the (NX+1)/2 x (NY+1)/2 grid, 40 lexicographic
// Gauss-Seidel sweeps there at relaxation 1.6, the bilinear prolongation
// applied to p and the faces, three SOR sweeps at 1.2.  Every stage keeps
// the reference's per-cell operation order; the serial loops become a
// pipeline (the SOR sweeps, the coarse sweeps) or a per-face kernel that
// applies a face's two updates in the loop's order (the correction).  Once
// a solve exits early, *stop makes every later kernel of it return.

// After the three pre-smoothing sweeps: count them and latch the exit when
// the last one's max |div| is below the tolerance.
__global__ void k_mg_check(const DevStats* __restrict__ sm, DevStats* st, int* stop, float tol,
                           int post) {
  if (*stop) return;
  st->sweeps += 3;
  if (post) return;
  float maxDiv = (float)sm->last_maxdiv;
  st->last_maxdiv = sm->last_maxdiv;
  if (maxDiv < tol) *stop = 1;
}

// computePressureResidual (fluid.go:596-628): r = -div - laplacian(p) on
// fluid interior cells, 0 elsewhere.
__global__ void k_mg_residual(const float* __restrict__ U, const float* __restrict__ V,
                              const float* __restrict__ p, const uint8_t* __restrict__ flags,
                              float* __restrict__ r, const int* __restrict__ stop, Grid g) {
  if (*stop) return;
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.NX || j >= g.NY) return;
  const int P = g.P;
  int c = i * P + j;
  uint8_t fl = flags[c];
  float out = 0.0f;
  if ((fl & (F_FLUID | F_INTERIOR)) == (F_FLUID | F_INTERIOR)) {
    float div = U[c + P] - U[c] + V[c + 1] - V[c];
    float sx0 = fbit(fl, F_W), sx1 = fbit(fl, F_E), sy0 = fbit(fl, F_S), sy1 = fbit(fl, F_N);
    float lap = sx0 * (p[c - P] - p[c]) + sx1 * (p[c + P] - p[c]) + sy0 * (p[c - 1] - p[c]) +
                sy1 * (p[c + 1] - p[c]);
    out = -div - lap;
  }
  r[c] = out;
}

// The coarse solid mask: the fine cell (2i, 2j) (fluid.go:672-685).
__device__ __forceinline__ float coarse_s(const uint8_t* __restrict__ flags, int i, int j,
                                          const Grid& g) {
  int fi = 2 * i, fj = 2 * j;
  if (fi >= g.NX || fj >= g.NY) return 0.0f;
  return (flags[fi * g.P + fj] & F_FLUID) ? 1.0f : 0.0f;
}

// restrictResidual (fluid.go:630-660) into cr, with the flag byte of every
// coarse cell into cflags (both cNX rows of cP).
__global__ void k_mg_restrict(const float* __restrict__ r, float* __restrict__ cr,
                              const int* __restrict__ stop, Grid g, int cNX, int cNY, int cP,
                              const uint8_t* __restrict__ flags, uint8_t* __restrict__ cflags) {
  if (*stop) return;
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= cNX || j >= cNY) return;
  float out = 0.0f;
  uint8_t fl = 0;
  int fi = 2 * i, fj = 2 * j;
  const bool interior = i >= 1 && i < cNX - 1 && j >= 1 && j < cNY - 1;
  if (interior && fi < g.NX - 1 && fj < g.NY - 1) {
    const int P = g.P;
    int c = fi * P + fj;
    float center = r[c] * 0.25f;
    float nb = (r[c - P] + r[c + P] + r[c - 1] + r[c + 1]) * 0.125f;
    float cr4 = (r[c - P - 1] + r[c + P - 1] + r[c - P + 1] + r[c + P + 1]) * 0.0625f;
    out = center + nb + cr4;
  }
  if (interior) {
    fl = F_INTERIOR;
    if (coarse_s(flags, i, j, g) != 0.0f) fl |= F_FLUID;
    if (coarse_s(flags, i - 1, j, g) != 0.0f) fl |= F_W;
    if (coarse_s(flags, i + 1, j, g) != 0.0f) fl |= F_E;
    if (coarse_s(flags, i, j - 1, g) != 0.0f) fl |= F_S;
    if (coarse_s(flags, i, j + 1, g) != 0.0f) fl |= F_N;
  }
  cr[i * cP + j] = out;
  cflags[i * cP + j] = fl;
}

// solveCoarseGrid (fluid.go:662-715): 40 lexicographic Gauss-Seidel sweeps
// from zero, in one block, as anti-diagonal wavefronts two diagonals apart
// (k_wave's fallback, like k_lexsor).
constexpr int MG_THREADS = 1024;
__global__ void __launch_bounds__(MG_THREADS)
    k_mg_coarse(const float* __restrict__ cr, float* __restrict__ x,
                const uint8_t* __restrict__ cflags, const int* __restrict__ stop, int cNX, int cNY,
                int cP, int sweeps, float relaxation) {
  if (*stop) return;
  const int ni = cNX - 2, nj = cNY - 2;
  for (int k = threadIdx.x; k < cNX * cP; k += MG_THREADS) x[k] = 0.0f;
  __syncthreads();
  if (ni <= 0 || nj <= 0) return;
  const int D = ni + nj - 1;
  const int L = ni < nj ? ni : nj;
  const float invL = 1.0f / (float)L;
  const long long steps = (long long)D + 2LL * (sweeps - 1);
  for (long long tau = 0; tau < steps; ++tau) {
    // Sweeps t with 0 <= tau - 2t < D, each on diagonal d = tau - 2t + 2; the
    // cells of a step are independent.
    int t_lo = (int)((tau - D + 2) / 2);
    if (t_lo < 0) t_lo = 0;
    while (tau - 2LL * t_lo >= D) ++t_lo;
    int t_hi = (int)(tau / 2);
    if (t_hi > sweeps - 1) t_hi = sweeps - 1;
    const int items = (t_hi - t_lo + 1) * L;
    for (int q = threadIdx.x; q < items; q += MG_THREADS) {
      int k;
      const int t = t_lo + (items < (1 << 24) ? div_small(q, L, invL, k) : (k = q % L, q / L));
      const int d = (int)(tau - 2LL * t) + 2;
      const int i = max(1, d - nj) + k;
      if (i > min(ni, d - 1)) continue;
      const int c = i * cP + (d - i);
      const uint8_t fl = cflags[c];
      if (!flag_active(fl)) continue;
      const float p0 = x[c];
      const float lap = fbit(fl, F_W) * (x[c - cP] - p0) + fbit(fl, F_E) * (x[c + cP] - p0) +
                        fbit(fl, F_S) * (x[c - 1] - p0) + fbit(fl, F_N) * (x[c + 1] - p0);
      const float residual = cr[c] - lap;
      x[c] = p0 + -residual / (float)flag_count(fl) * relaxation;
    }
    __syncthreads();
  }
}

// prolongateCorrection (fluid.go:717-758) at fine cell (i, j).
__device__ __forceinline__ float mg_corr(const float* __restrict__ cc, int i, int j, int cNX,
                                         int cNY, int cP) {
  int ci = i / 2, cj = j / 2;
  if (ci >= cNX - 1 || cj >= cNY - 1) return 0.0f;
  float fI = (float)(i % 2) * 0.5f, fJ = (float)(j % 2) * 0.5f;
  return (1.0f - fI) * (1.0f - fJ) * cc[ci * cP + cj] +
         fI * (1.0f - fJ) * cc[(ci + 1) * cP + cj] +
         (1.0f - fI) * fJ * cc[ci * cP + cj + 1] +
         fI * fJ * cc[(ci + 1) * cP + cj + 1];
}

// applePressureCorrection (fluid.go:1122-1149): p += corr * cp on fluid
// interior cells; face (i, j) of U first gets + S_i corr(i-1, j) from cell
// (i-1, j), then - S_{i-1} corr(i, j) from cell (i, j), as the loop visits
// them; V likewise along j.
__global__ void k_mg_apply(float* __restrict__ U, float* __restrict__ V, float* __restrict__ p,
                           const float* __restrict__ cc, const uint8_t* __restrict__ flags,
                           const int* __restrict__ stop, float cp, Grid g, int cNX, int cNY,
                           int cP) {
  if (*stop) return;
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.NX || j >= g.NY) return;
  const int P = g.P;
  int c = i * P + j;
  auto fluid_int = [&](int a, int b) {
    return a >= 1 && a <= g.NX - 2 && b >= 1 && b <= g.NY - 2 &&
           (flags[a * P + b] & F_FLUID) != 0;
  };
  bool self = fluid_int(i, j);
  float corr = self ? mg_corr(cc, i, j, cNX, cNY, cP) : 0.0f;
  if (self) p[c] += corr * cp;
  uint8_t fl = flags[c];
  if (i >= 1) {
    float u = U[c];
    if (fluid_int(i - 1, j)) u += fbit(fl, F_FLUID) * mg_corr(cc, i - 1, j, cNX, cNY, cP);
    if (self) u -= fbit(fl, F_W) * corr;
    U[c] = u;
  }
  if (j >= 1) {
    float v = V[c];
    if (fluid_int(i, j - 1)) v += fbit(fl, F_FLUID) * mg_corr(cc, i, j - 1, cNX, cNY, cP);
    if (self) v -= fbit(fl, F_S) * corr;
    V[c] = v;
  }
}

}  // namespace

// ------------------------------------------------------------------ host side
static size_t wave_smem(bool gs) {
  return (size_t)WV_W * 4 * (WV_A0 + (gs ? 1 : 2) * WV_A1) + (size_t)WV_A1 * WV_FP;
}
static int wave_strips(int NX, int G) { return (NX + G - 2 + 31) / 32; }

// Sets the pipeline kernels' shared-memory limit and counts the blocks the
// current device holds at once (0: they cannot run).  Outside any capture.
static int wave_blocks() {
  int dev = 0, sms = 0, per[2] = {};
  const int s0 = (int)wave_smem(false), s1 = (int)wave_smem(true), nt = (WV_G + 2) * 32;
  const bool ok =
      cudaGetDevice(&dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
      cudaFuncSetAttribute(k_wave<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, s0) ==
          cudaSuccess &&
      cudaFuncSetAttribute(k_wave<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, s1) ==
          cudaSuccess &&
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[0], k_wave<false>, nt, s0) == cudaSuccess &&
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[1], k_wave<true>, nt, s1) == cudaSuccess;
  cudaGetLastError();
  return ok && per[0] > 0 && per[1] > 0 ? sms : 0;
}

// Bytes of the pipeline's buffers for an NX x NY grid (rows of P), and their
// places in the block: control words, completion words, the SOR's and the
// coarse solve's packets, the speculative pass's fields.
static size_t wave_layout(const fg_fluid* f, size_t* fin, size_t* pkt, size_t* gs, size_t* fields) {
  const int B = wave_strips(f->NX, WV_G), cNX = (f->NX + 1) / 2, cNY = (f->NY + 1) / 2;
  const int cB = wave_strips(cNX, WV_G), cP = (cNY + 31) / 32 * 32;
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  size_t at = up(sizeof(WaveCtl));
  *fin = at;
  at += up((size_t)B * WV_GROUPS * sizeof(unsigned long long));
  *pkt = at;
  at += up((size_t)B * 2 * WV_G * f->P * 16);
  *gs = at;
  at += up((size_t)cB * 2 * WV_G * cP * 8);
  *fields = at;
  return at + 3 * up((size_t)f->NX * f->P * sizeof(float));
}

size_t wave_bytes(const fg_fluid* f) {
  size_t a, b, c, d;
  return wave_layout(f, &a, &b, &c, &d);
}

// (Outside capture: zeroes the tags and control words of a new block.)
cudaError_t wave_init(fg_fluid* f) {
  size_t fin, pkt, gs, fields;
  wave_layout(f, &fin, &pkt, &gs, &fields);
  f->wave_blocks = wave_blocks();
  return cudaMemsetAsync(f->wave, 0, fields, f->stream);
}

static WaveArgs wave_args(fg_fluid* f, bool gs) {
  size_t fin, pkt, gpkt, fields;
  wave_layout(f, &fin, &pkt, &gpkt, &fields);
  char* w = static_cast<char*>(f->wave);
  WaveArgs a = {};
  a.ctl = reinterpret_cast<WaveCtl*>(w);
  a.fin = reinterpret_cast<unsigned long long*>(w + fin);
  a.pkt = w + (gs ? gpkt : pkt);
  const size_t fb = ((size_t)f->NX * f->P * sizeof(float) + 255) & ~(size_t)255;
  for (int k = 0; k < 3; ++k) a.scratch[k] = reinterpret_cast<float*>(w + fields + k * fb);
  a.err = &f->dstats->timeout;
  a.stall = f->stall_tile;
  return a;
}

// One launch: sweeps [t0, t0 + n) of the solve a describes.
static void wave_launch(fg_fluid* f, WaveArgs a, bool gs, int t0, int n) {
  a.t0 = t0;
  a.nsweeps = n;
  a.last = t0 + n == a.iters;
  a.G = std::min(WV_G, n);
  a.B = wave_strips(a.NX, a.G);
  const long long tasks = (long long)a.B * ((n + a.G - 1) / a.G);
  const int blocks =
      a.mode == WV_FINISH ? f->wave_blocks : (int)std::min<long long>(tasks, f->wave_blocks);
  if (gs)
    k_wave<true><<<blocks, (a.G + 2) * 32, wave_smem(true), f->stream>>>(a);
  else
    k_wave<false><<<blocks, (a.G + 2) * 32, wave_smem(false), f->stream>>>(a);
  count(f);
}

// `iters` SOR sweeps on the handle's U, V and p, relaxation relax0 -> relax1.
// A solve of more than WV_SWEEPS sweeps takes several launches.
static void lexsor_solve(fg_fluid* f, int iters, float relax0, float relax1, float cp,
                         bool early_exit, DevStats* st, const int* stop) {
  if (iters <= 0) return;
  if (!f->wave || f->wave_blocks == 0) {
    k_lexsor<<<1, LEX_THREADS, 0, f->stream>>>(f->d[FG_U], f->d[FG_V], f->d[FG_P], f->flags, f->g,
                                                iters, relax0, f->prm.pressure_damping, cp,
                                                f->prm.tolerance, early_exit, st, relax1, stop);
    count(f);
    return;
  }
  WaveArgs a = wave_args(f, false);
  a.flags = f->flags;
  a.NX = f->NX;
  a.NY = f->NY;
  a.P = f->P;
  a.iters = iters;
  a.relax0 = relax0;
  a.relax1 = relax1;
  a.damping = f->prm.pressure_damping;
  a.cp = cp;
  a.tol = f->prm.tolerance;
  a.stop = stop;
  a.st = st;
  float* state[3] = {f->d[FG_U], f->d[FG_V], f->d[FG_P]};
  auto pass = [&](int mode) {
    a.mode = mode;
    for (int t = 0; t < iters; t += WV_SWEEPS) {
      for (int k = 0; k < 3; ++k) {
        a.dst[k] = mode == WV_SPECULATE ? a.scratch[k] : state[k];
        a.src[k] = mode == WV_SPECULATE && t > 0 ? a.scratch[k] : state[k];
      }
      wave_launch(f, a, false, t, std::min(WV_SWEEPS, iters - t));
    }
  };
  if (early_exit) {
    pass(WV_SPECULATE);
    pass(WV_FINISH);
  } else {
    pass(WV_PLAIN);
  }
}

cudaError_t launch_lexsor(fg_fluid* f, int num_iters, float dt) {
  lexsor_solve(f, num_iters, f->prm.relaxation, 1.2f, f->density * f->h / dt,
               f->prm.early_exit != 0, f->dstats, nullptr);
  return cudaGetLastError();
}

// solveCoarseGrid's 40 sweeps from zero.
static void launch_mg_coarse(fg_fluid* f, const int* stop, int cNX, int cNY, int cP,
                             const uint8_t* cflags) {
  if (!f->wave || f->wave_blocks == 0) {
    k_mg_coarse<<<1, MG_THREADS, 0, f->stream>>>(f->err, f->err2, cflags, stop, cNX, cNY, cP, 40,
                                                  1.6f);
    count(f);
    return;
  }
  WaveArgs a = wave_args(f, true);
  a.src[0] = a.dst[0] = f->err2;
  a.src[1] = f->err;
  a.flags = cflags;
  a.NX = cNX;
  a.NY = cNY;
  a.P = cP;
  a.iters = 40;
  a.relax0 = 1.6f;
  a.mode = WV_PLAIN;
  a.stop = stop;
  a.stall = -1;
  wave_launch(f, a, true, 0, 40);
}

cudaError_t launch_multigrid(fg_fluid* f, int num_iters, float dt) {
  float cp = f->density * f->h / dt;  // fluid.go:560
  const int cNX = (f->NX + 1) / 2, cNY = (f->NY + 1) / 2;
  // Scratch: the fine residual in rhs, the coarse right-hand side and
  // solution in err / err2, the stop latch and the smoothers' statistics in
  // the correction solve's control block (unused by this scheme).
  int* stop = reinterpret_cast<int*>(f->ectl);
  DevStats* sm = reinterpret_cast<DevStats*>(reinterpret_cast<char*>(f->ectl) + 64);
  cudaError_t e = cudaMemsetAsync(f->ectl, 0, 64 + sizeof(DevStats), f->stream);
  if (e != cudaSuccess) return e;
  dim3 gr = cell_grid(f), bl(BX, BY);
  dim3 cg((cNY + BX - 1) / BX, (cNX + BY - 1) / BY);
  const int cP = (cNY + 31) / 32 * 32;
  if ((size_t)cNX * cP > (size_t)f->NX * f->P) return cudaErrorInvalidValue;
  uint8_t* cflags = reinterpret_cast<uint8_t*>(f->rhs_e);
  for (int it = 0; it < num_iters; ++it) {
    count(f, 5);
    lexsor_solve(f, 3, 1.5f, 1.5f, cp, false, sm, stop);
    k_mg_check<<<1, 1, 0, f->stream>>>(sm, f->dstats, stop, f->prm.tolerance, 0);
    k_mg_residual<<<gr, bl, 0, f->stream>>>(f->d[FG_U], f->d[FG_V], f->d[FG_P], f->flags, f->rhs,
                                            stop, f->g);
    k_mg_restrict<<<cg, bl, 0, f->stream>>>(f->rhs, f->err, stop, f->g, cNX, cNY, cP, f->flags,
                                            cflags);
    launch_mg_coarse(f, stop, cNX, cNY, cP, cflags);
    k_mg_apply<<<gr, bl, 0, f->stream>>>(f->d[FG_U], f->d[FG_V], f->d[FG_P], f->err2, f->flags,
                                         stop, cp, f->g, cNX, cNY, cP);
    lexsor_solve(f, 3, 1.2f, 1.2f, cp, false, sm, stop);
    k_mg_check<<<1, 1, 0, f->stream>>>(sm, f->dstats, stop, f->prm.tolerance, 1);
  }
  return cudaGetLastError();
}

}  // namespace fg
