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
#include <type_traits>

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
// ring of WV_W columns that a loader warp fills and a storer warp drains, so a
// step costs the shuffle, the arithmetic and its own instructions, where a
// wavefront through L2 with a barrier per anti-diagonal paid a memory round
// trip and the barrier (2.4 us, on one block or eight).
// Chunks of 16 columns: a chunk's waits, packets and report take about 240
// cycles, so 8 columns measured slower in a strip (20x2046, one sweep: 163
// against 147 us) and 8 columns with 16 sweeps a block, whose ring then has
// no slack, slower on large solves (2048^2, 200 sweeps: 2.56 against 2.35 ms).
// Between strips the topmost lane hands each column's new values on as one
// 16-byte packet {u, v, p, tag} in global memory, written and read whole, so
// the receiving warp polls the data itself and no fence or flag stands
// between the two.  Tasks (strip b, group g of sweeps) are claimed by ticket
// in the order of b + 2 g: a task needs (b-1, g), (b, g-1) and (b+1, g-1),
// all of earlier tickets, so whatever number of blocks is resident the oldest
// unfinished task can always proceed.
//
// Bound by the serial chain: NX + NY steps and a packet's flight per strip.
// Measured on a GB300: one sweep takes 53 ns a column along a strip and 3.7 us
// a strip of 32 rows (47 steps and 1.2 us of flight), a group of 8 sweeps 78 ns
// and 4.5 us; every further group 26 us at 300x251, 20 at 30x30.  The chain
// leaves most of the issue slots empty (32 % used on the SMs that have a
// block; per issue 1.95 warps wait on a fixed latency, 0.95 on shared memory).
// Against the wavefront through L2 that it replaced (one block, an 8-block
// cluster or a grid barrier per anti-diagonal), whole passes from the host: the
// app's 300x251 jet with 8 sweeps and the early exit 1386 -> 162 us, two steps
// of a 128x128 jet with 40 sweeps 2893 -> 365 us, a 1024x768 box with BFECC
// 4464 -> 413 us, a 512x512 box with 8 reference V-cycles 45.7 -> 3.3 ms; 200
// sweeps alone at 2048^2 2.34 ms.
constexpr int WV_G = 8;            // sweeps per group (compute warps of a block)
constexpr int WV_C = 16;           // columns per chunk
constexpr int WV_W = 256;          // ring columns
constexpr int WV_M = WV_W - 1;
constexpr int WV_BEFORE = 64;      // columns before the row's start that the sweeps step through
constexpr int WV_PAST = 96;        // columns past its end
constexpr int WV_GROUPS = 256;     // groups per launch (slots of `fin` per strip)
constexpr int WV_SWEEPS = WV_G * WV_GROUPS;
// The ring's rows: the first field's (U; the coarse solution), then V (the
// coarse right-hand side), p (SOR only) and the cells' coefficient offsets.
// Row q of each holds grid row i0 + q - WV_G, so a cell's values lie at
// constant distances; 32 lanes on 32 rows and consecutive columns (a row is
// a multiple of 32 words) never share a bank.
constexpr int WV_A0 = 33 + WV_G, WV_A1 = 32 + WV_G;
template <bool GS>
struct WaveRing {
  static constexpr int O1 = WV_A0 * WV_W, O2 = O1 + WV_A1 * WV_W,
                       OF = GS ? O2 : O2 + WV_A1 * WV_W, WORDS = OF + WV_A1 * WV_W;
};
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
// count are the serial loop's).  The copying launch takes 5.5 us at 128x128, 8
// at 300x251, 10 at 1024x768, 61 at 2048^2, beside 61, 97, 254 and 528 us of a
// makeIncompressible with 8 sweeps.
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
  asm volatile(
      "{\n\t.reg .b64 a;\n\tmov.b64 a, {%1, %2};\n\tst.relaxed.gpu.global.b64 [%0], a;\n\t}" ::"l"(p),
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
    __nanosleep(20);  // (a polling warp takes issue slots from the sweeps)
    if (__all_sync(0xffffffffu, ld_cta(p) >= need)) return true;
    if ((it & 255) == 0 &&
        __any_sync(0xffffffffu, ld_cta(&sh->abort) != 0 || wv_ns() - t0 > WV_WAIT_NS))
      break;
  }
  st_cta(&sh->abort, 1);
  return false;
}

// Per flag byte: the faces' fluid bits as floats, the neighbour count and its
// rounded reciprocal (0 on cells the sweeps leave alone).  A step reads its
// cell's entry a step ahead, so it has no branch and decodes nothing.
struct __align__(16) WaveCoef {
  float W, E, S, N, n, r, pad[2];
};
__device__ __forceinline__ void wv_fill_coef(WaveCoef* lut) {
  for (int f = threadIdx.x - 1; f < 64; f += blockDim.x - 1) {  // (not by thread 0)
    WaveCoef c = {};
    if ((f & (F_FLUID | F_INTERIOR)) == (F_FLUID | F_INTERIOR) && (f & 15)) {
      c.W = fbit(f, F_W);
      c.E = fbit(f, F_E);
      c.S = fbit(f, F_S);
      c.N = fbit(f, F_N);
      c.n = c.W + c.E + c.S + c.N;
      c.r = 1.0f / c.n;
    }
    lut[f] = c;
  }
}
// x / n, n = 1..4, r = 1 / n rounded: the quotient by the reciprocal with
// Markstein's correction (IBM J. Res. Dev. 34, 1990), whose remainder is
// exact for every float and these n; the remainder is taken as n q - x so
// that a zero keeps its sign, and an infinity keeps its first quotient.
// Equal to the division for all 2^32 floats and each n (tests/test_div_count.py).
__device__ __forceinline__ float div_count(float x, float n, float r) {
  float q = x * r;
  const float e = __fmaf_rn(n, q, -x);
  asm("{\n\t.reg .pred p;\n\t.reg .f32 a;\n\tabs.f32 a, %2;\n\tsetp.lt.f32 p, a, 0f7F800000;\n\t"
      "@p fma.rn.f32 %0, %1, %3, %0;\n\t}"
      : "+f"(q)
      : "f"(e), "f"(x), "f"(-r));
  return q;
}
// x = fma(c, y, x), x = x + y, m = max(m, |y|) where r > 0, else unchanged (a
// predicated instruction instead of a select behind it in the serial chain).
__device__ __forceinline__ void fma_if(float& x, float c, float y, float r) {
  asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %3, 0f00000000;\n\t@p fma.rn.f32 %0, %1, %2, %0;\n\t}"
      : "+f"(x)
      : "f"(c), "f"(y), "f"(r));
}
__device__ __forceinline__ void add_if(float& x, float y, float r) {
  asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %2, 0f00000000;\n\t@p add.rn.f32 %0, %0, %1;\n\t}"
      : "+f"(x)
      : "f"(y), "f"(r));
}
__device__ __forceinline__ void max_if(float& m, float y, float r) {
  asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %2, 0f00000000;\n\t@p max.f32 %0, %0, %1;\n\t}"
      : "+f"(m)
      : "f"(fabsf(y)), "f"(r));
}
// The column that lane 0 of a strip would be at in step 0, but for the sweeps'
// offsets (<= 0): lane 31 of the strip below is 31 columns behind its lane 0,
// so this shift by b makes its chunks of columns the ones received here.
__device__ __forceinline__ int wv_lead(int b) { return (b & (WV_C - 1)) - WV_C; }

// One sweep (warp w of the block, sweep t of the solve) of task (b, g).
// D1: the damping is 1 (its product is then the factor itself).
//
// Every step treats its cell alike, active or not, on the grid or off it:
// predicates leave inactive cells as they are, the coefficients are 0 or 1 (so
// each fused multiply-add rounds as the reference's product and sum), and the
// ring holds zero coefficients in the columns before the first and past the
// last, so lanes there change nothing.  A second body without coefficients
// for chunks of full cells was measured slower than this one alone (chunks of
// 8: 20x2046, one sweep, 199 against 163 us; 2048^2, 200 sweeps, 2.56 against
// 2.49 ms): choosing costs more per chunk than it saves, and a strip's first
// and last 33 columns, where the wave enters the next strip, are never full.
template <bool GS, bool D1>
__device__ __forceinline__ void wv_sweep(const WaveArgs& a, WaveShared* sh, const char* lut,
                                         char* ring, int b, int g, int w, int Gt, int nchunks,
                                         unsigned tag) {
  using R = WaveRing<GS>;
  constexpr int RB = 4 * WV_W;  // bytes of a ring row
  const int lane = threadIdx.x & 31;
  const int row = (WV_G - w + lane) * RB;
  const int t = a.t0 + g * a.G + w;
  const float prog_t = (float)t / (float)a.iters;
  const float rel = GS ? a.relax0 : a.relax0 - (a.relax0 - a.relax1) * prog_t;  // fluid.go:169-170
  const float damping = a.damping, cp = a.cp;
  const int NY = a.NY;
  const size_t slot = (size_t)(g & 1) * a.G + w;
  const size_t in_at = ((size_t)(b - 1) * 2 * a.G + slot) * a.P;
  const size_t out_at = ((size_t)b * 2 * a.G + slot) * a.P;
  const uint4* in4 = (const uint4*)a.pkt + in_at;
  const uint2* in2 = (const uint2*)a.pkt + in_at;
  const bool recv = b > 0, send = b + 1 < a.B && b != a.stall;
  float mx = 0.0f;
  // v0: V[i][j], updated by (i, j-1) (SOR); the old P[i][j] (GS).  ue: the
  // last step's new P (GS).  shv: the lower lane's east face after the last
  // step (SOR), its new P (GS).
  float v0 = 0.0f, ue = 0.0f, shv = 0.0f;
  float n1 = 0.0f, n2 = 0.0f, n3 = 0.0f, west = 0.0f;  // the next step's inputs
  float4 k4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);      // its coefficients
  float2 k2 = make_float2(0.0f, 0.0f);
  unsigned nf = 0;                     // the coefficient offset of the step after it
  // The chunk's first step.  The first chunk is the one with step -1, in
  // which lane 0 picks up V[i][0].
  int s = wv_lead(b) - 2 * (w + 1);
  const int n0 = (-1 - s) / WV_C;
  s += n0 * WV_C;
  int j4 = 4 * (s - lane);             // 4 x the step's column
  // Byte offsets in the ring of the step's cell and of the next two columns'.
  int at0 = row | (j4 & (RB - 4)), at1 = row | ((j4 + 4) & (RB - 4)), at2 = 0;
  auto F = [&](int at) -> float& { return *reinterpret_cast<float*>(ring + at); };
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
  // The inputs of the column at c, the next column at cn.
  auto fetch = [&](int c, int cn) {
    n1 = F(c + RB);                             // U[i+1][j]; the old P[i+1][j]
    n2 = GS ? F(cn) : F(cn + 4 * R::O1);        // V[i][j+1]; the old P[i][j+1]
    n3 = GS ? F(c + 4 * R::O1) : F(c + 4 * R::O2);  // p; the right-hand side
  };
  auto coef = [&] {
    k4 = *reinterpret_cast<const float4*>(lut + nf);
    k2 = *reinterpret_cast<const float2*>(lut + nf + 16);
  };
  if (recv && lane < WV_C && (unsigned)(s + lane) < (unsigned)NY) poll(s + lane);
  // The progress of the sweep below (of the loader, for the first sweep) is
  // read in the middle of a chunk for the next one.
  const int* word = w ? &sh->prog[w - 1] : &sh->loaded;
  int seen = 0;
  for (int n = n0; n < nchunks; ++n, s += WV_C) {
    const int need = w ? n + 1 : min(s + WV_C + 2, a.P + WV_PAST);
    if (!__all_sync(0xffffffffu, seen >= need) && !wv_wait(word, need, sh)) return;
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
        const int d = (WV_G - w) * RB | ((4 * c) & (RB - 4));
        if (GS) {
          F(d - RB) = __uint_as_float(pk.x);
        } else {
          F(d) = __uint_as_float(pk.x);
          if (w + 1 < Gt) {
            F(d + 4 * R::O1 - RB) = __uint_as_float(pk.y);
            F(d + 4 * R::O2 - RB) = __uint_as_float(pk.z);
          }
        }
      }
      west = __uint_as_float(pk.x);  // (lane 0's is the first step's)
      __syncwarp();
      if (lane < WV_C && (unsigned)(c + WV_C) < (unsigned)NY) poll(c + WV_C);
    } else {
      west = F(at0 - (GS ? RB : 0));
    }
    if (n == n0) {
      fetch(at0, at1);
      nf = __float_as_uint(F(at0 + 4 * R::OF));
      coef();
      nf = __float_as_uint(F(at1 + 4 * R::OF));
    }
#pragma unroll
    for (int k = 0; k < WV_C; ++k) {
      const float wv = lane == 0 ? west : shv;
      const float x1 = n1, x2 = n2, x3 = n3;
      const float4 c4 = k4;
      const float2 c2 = k2;
      at2 = row | ((j4 + 8) & (RB - 4));
      fetch(at1, at2);
      if (k + 1 < WV_C) west = F(at1 - (GS ? RB : 0));
      coef();
      nf = __float_as_uint(F(at2 + 4 * R::OF));
      if (k == WV_C / 2) seen = ld_cta(word);
      if (GS) {
        float out = v0;
        const float lap =
            c4.x * (wv - v0) + c4.y * (x1 - v0) + c4.z * (ue - v0) + c4.w * (x2 - v0);
        add_if(out, div_count(-(x3 - lap), c2.x, c2.y) * rel, c2.y);
        shv = __shfl_up_sync(0xffffffffu, out, 1);
        F(at0) = out;
        ue = out;
        v0 = x2;
      } else {
        const float div = x1 - wv + x2 - v0;
        float un = wv, en = x1, vn = v0, tn = x2, pn = x3;
        float pp = div_count(-div, c2.x, c2.y);
        pp *= rel;
        if (!D1) pp *= damping;
        fma_if(en, c4.y, pp, c2.y);
        // The next step's west value sets off before this step's stores.
        shv = __shfl_up_sync(0xffffffffu, en, 1);
        fma_if(tn, c4.w, pp, c2.y);
        fma_if(un, -c4.x, pp, c2.y);
        fma_if(vn, -c4.z, pp, c2.y);
        add_if(pn, cp * pp, c2.y);
        max_if(mx, div, c2.y);
        F(at0) = un;
        // (A lower lane's east face is the next lane's `un` one step later; no
        // two lanes store the same word between two barriers of the warp.)
        if (lane == 31) F(at0 + RB) = en;
        F(at0 + 4 * R::O1) = vn;
        F(at0 + 4 * R::O2) = pn;
        v0 = tn;
      }
      at0 = at1;
      at1 = at2;
      j4 += 4;
    }
    __syncwarp();
    // Lane 31's columns of this chunk go to the strip above (read before the
    // chunk is reported, after which the ring may be refilled).
    const int cs = s - 31 + lane;
    const bool out = send && lane < WV_C && (unsigned)cs < (unsigned)NY;
    uint4 x = make_uint4(0, 0, 0, tag);
    if (out) {
      const int d = (WV_G - w + 31) * RB | ((4 * cs) & (RB - 4));
      x.x = __float_as_uint(F(d + (GS ? 0 : RB)));
      if (!GS) {
        x.y = __float_as_uint(F(d + 4 * R::O1));
        x.z = __float_as_uint(F(d + 4 * R::O2));
      }
    }
    __syncwarp();
    if (lane == 0) st_cta(&sh->prog[w], n + 1);
    if (out) {
      if (GS)
        st_pkt2((uint2*)a.pkt + out_at + cs, make_uint2(x.x, tag));
      else
        st_pkt((uint4*)a.pkt + out_at + cs, x);
    }
  }
  if (!GS) {
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
    if (lane == 0 && m) atomicMax(&a.ctl->gmax[g * a.G + w], m);
  }
}

// Copies 32 columns (from column c) of grid rows [i, i + n) of a field to ring
// row q on, 8 lanes a row; rows outside the grid, and everything when !data,
// become zeros.
__device__ __forceinline__ void wv_load_rows(float* ring, int q, const float* src, int i, int n,
                                             int c, int NX, int P, bool data) {
  const int lane = threadIdx.x & 31, r0 = lane >> 3, e = c + (lane & 7) * 4;
  float* d = ring + (q + r0) * WV_W + (e & WV_M);
  const float* p = src + (ptrdiff_t)(i + r0) * P + e;
  i += r0;
#pragma unroll 4
  for (int r = r0; r < n; r += 4, i += 4, d += 4 * WV_W, p += 4 * (ptrdiff_t)P) {
    const bool in = data && (unsigned)i < (unsigned)NX;
    wv_copy16(d, in ? p : src, in);
  }
}

// The loader warp: 32 columns at a time, as far ahead as the ring has room.
template <bool GS>
__device__ void wv_loader(const WaveArgs& a, WaveShared* sh, float* ring, int b, int g, int Gt,
                          int nchunks, unsigned tag) {
  using R = WaveRing<GS>;
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
    const bool all = __all_sync(0xffffffffu, r) != 0;
    // (A vote orders no memory: what the two lanes acquired, before every lane's copies.)
    __syncwarp();
    return all;
  };
  auto publish = [&](int cols) {
    __syncwarp();
    if (lane == 0) st_cta(&sh->loaded, cols);
  };
  // Flag bytes of the next 32 columns (4 a lane), read a block ahead.
  constexpr int NF = (WV_A1 * 8 + 31) / 32;
  unsigned f[NF];
  auto flags = [&](int c) {
    const int r0 = lane >> 3, e = c + (lane & 7) * 4;
    int i = i0 + lo - WV_G + r0;
#pragma unroll
    for (int m = 0; m < NF; ++m, i += 4)
      f[m] = lo + r0 + 4 * m < hi && c < a.P && (unsigned)i < (unsigned)a.NX
                 ? __ldg(reinterpret_cast<const unsigned*>(a.flags + (size_t)i * a.P + e))
                 : 0u;
  };
  // Their coefficient offsets, into the ring.
  auto offsets = [&](int c) {
    const int r0 = lane >> 3;
    float* d = ring + R::OF + (lo + r0) * WV_W + (c & WV_M) + (lane & 7) * 4;
    constexpr unsigned SZ = sizeof(WaveCoef);
#pragma unroll
    for (int m = 0; m < NF; ++m, d += 4 * WV_W)
      if (lo + r0 + 4 * m < hi)
        *reinterpret_cast<uint4*>(d) =
            make_uint4((f[m] & 63u) * SZ, (f[m] >> 8 & 63u) * SZ, (f[m] >> 16 & 63u) * SZ,
                       (f[m] >> 24 & 63u) * SZ);
  };
  // Zero coefficients before column 0 (the ring's last blocks) and in the
  // WV_PAST columns after the row.
  flags(a.P);
  for (int c = WV_W - WV_BEFORE; c < WV_W; c += 32) offsets(c);
  flags(0);
  // Chunks after which no lane of the last sweep is before column 0.
  const int inside = (32 - wv_lead(b) + 2 * Gt + WV_C - 1) / WV_C;
  bool ok = true;
  int copied = 0, known = 0;  // columns issued, columns published
  for (int c = 0; c < a.P + WV_PAST && ok; c += 32) {
    // A block's ring columns are free once the storer has drained them; the
    // last blocks' first columns once the sweeps have left them.
    const bool first = c < WV_W;
    const int* word = first ? &sh->prog[Gt - 1] : &sh->stored;
    const int room = !first ? c + 32 - WV_W : c < WV_W - WV_BEFORE ? 0 : min(inside, nchunks);
    const bool now = (room <= 0 || __all_sync(0xffffffffu, ld_cta(word) >= room)) &&
                     (c >= a.P || ready(c));
    if (!now) {
      if (known < copied) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        publish(known = copied);
      }
      if (room > 0) ok = wv_wait(word, room, sh);
      const unsigned long long t0 = wv_ns();
      for (int it = 1; ok && c < a.P && !ready(c); ++it)
        if ((it & 63) == 0 &&
            (it >= WV_MAX_TRIES ||
             __any_sync(0xffffffffu, ld_cta(&sh->abort) != 0 || wv_ns() - t0 > WV_WAIT_NS))) {
          st_cta(&sh->abort, 1);
          ok = false;
        }
      if (!ok) break;
    }
    if (c >= a.P) {
      // (no fields past the row)
    } else if (GS) {
      // Row 0 and the rows below it hold zeros (strip 0); the right-hand side
      // and the flags reach down to the last sweep's rows.
      const int q0 = b ? WV_G : WV_G - a.G;
      wv_load_rows(ring, q0, s0, i0 + q0 - WV_G, hi + 1 - q0, c, a.NX, a.P, g > 0);
      wv_load_rows(ring + R::O1, lo, s1, i0 + lo - WV_G, hi - lo, c, a.NX, a.P, true);
    } else {
      wv_load_rows(ring, WV_G, s0, i0, 33, c, a.NX, a.P, true);
      wv_load_rows(ring + R::O1, WV_G, s1, i0, 32, c, a.NX, a.P, true);
      wv_load_rows(ring + R::O2, WV_G, s2, i0, 32, c, a.NX, a.P, true);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    copied = c + 32;
    offsets(c);
    flags(c + 32);
    if (copied - known > 64) {  // (up to three blocks in flight)
      asm volatile("cp.async.wait_group 2;" ::: "memory");
      publish(known = copied - 64);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (known < copied) publish(copied);
}

// The storer warp: the group's final values, 32 columns at a time, once its
// last sweep's topmost lane has passed them.
template <bool GS>
__device__ void wv_storer(const WaveArgs& a, WaveShared* sh, const float* ring, int b, int g,
                          int Gt, int nchunks, unsigned tag, bool more) {
  using R = WaveRing<GS>;
  const int lane = threadIdx.x & 31;
  const int i0 = 1 + 32 * b;
  constexpr int NF = GS ? 1 : 3;
  const int first = GS ? 0 : 1;  // (GS: strip 0 also writes row 0's zeros)
  for (int c = 0; c < a.P; c += 32) {
    // Lane 31 passes column c + 31 in step c + 62.
    const int need = min((c + 63 - wv_lead(b) + 2 * Gt + WV_C - 1) / WV_C, nchunks);
    if (!wv_wait(&sh->prog[Gt - 1], need, sh)) return;
#pragma unroll
    for (int fd = 0; fd < NF; ++fd) {
      const float* from = ring + (fd == 0 ? 0 : fd == 1 ? R::O1 : R::O2);
      float* dst = a.dst[fd];
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const int r = m * 4 + (lane >> 3), e = (lane & 7) * 4;
        const int q = WV_G - (Gt - 1) + r, i = i0 - (Gt - 1) + r, j = c + e;
        const float4 v = *reinterpret_cast<const float4*>(from + q * WV_W + (c & WV_M) + e);
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

template <bool GS, bool D1>
__global__ void __launch_bounds__((WV_G + 2) * 32, 1) k_wave(WaveArgs a) {
  extern __shared__ __align__(1024) unsigned char wv_dyn[];
  __shared__ WaveShared sh;
  __shared__ WaveCoef lut[64];
  float* ring = reinterpret_cast<float*>(wv_dyn);
  WaveCtl* ctl = a.ctl;
  const int warp = threadIdx.x >> 5;
  // (Changed only after every block has left.)
  const unsigned epoch = ctl->epoch;
  const int found = ctl->exit_sweep;
  if (a.stop && *a.stop) return;  // (the same in every block)
  int nsw = a.nsweeps;
  bool copy = false;
  if (a.mode == WV_SPECULATE && a.t0 > 0 && found) nsw = 0;
  if (a.mode == WV_FINISH) {
    const bool rerun = found && found < a.iters;
    nsw = rerun ? max(0, min(a.nsweeps, found - a.t0)) : 0;
    copy = !rerun && a.last;
  }
  const int ng = (nsw + a.G - 1) / a.G, ntasks = a.B * ng;
  if (threadIdx.x == 0) sh.abort = 0;
  int key = 0, before = 0;  // ticket decoding (thread 0): tasks with b + 2 g < key
  for (int turn = 0;; ++turn) {
    if (threadIdx.x == 0) {
      sh.b = -1;
      // (With a block per task, no block gets a second one.)
      const int tk = ntasks && (turn == 0 || ntasks > (int)gridDim.x)
                         ? (int)atomicAdd(&ctl->ticket, 1u)
                         : ntasks;
      if (tk < ntasks && !sh.abort && (turn == 0 || !*(volatile int*)&ctl->fail)) {
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
    } else if (turn == 0) {
      wv_fill_coef(lut);
    }
    __syncthreads();
    const int b = sh.b, g = sh.g;
    if (b < 0) break;
    const int Gt = min(a.G, nsw - g * a.G);
    const int nchunks = (a.NY + 31 - wv_lead(b) + 2 * Gt + WV_C - 1) / WV_C;
    const unsigned tag = epoch + 1u + (unsigned)g;
    if (warp == a.G)
      wv_loader<GS>(a, &sh, ring, b, g, Gt, nchunks, tag);
    else if (warp == a.G + 1)
      wv_storer<GS>(a, &sh, ring, b, g, Gt, nchunks, tag, g + 1 < ng);
    else if (warp < Gt)
      wv_sweep<GS, D1>(a, &sh, reinterpret_cast<const char*>(lut),
                       reinterpret_cast<char*>(wv_dyn), b, g, warp, Gt, nchunks, tag);
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
  return sizeof(float) * (gs ? WaveRing<true>::WORDS : WaveRing<false>::WORDS);
}
static int wave_strips(int NX, int G) { return (NX + G - 2 + 31) / 32; }

// The kernel of a launch: the coarse solve, or the SOR with damping 1 or not.
typedef void (*WaveKernel)(WaveArgs);
static WaveKernel wave_kernel(bool gs, bool d1) {
  return gs ? k_wave<true, true> : d1 ? k_wave<false, true> : k_wave<false, false>;
}

// Sets the pipeline kernels' shared-memory limit and counts the blocks the
// current device holds at once (0: they cannot run).  Outside any capture.
static int wave_blocks() {
  int dev = 0, sms = 0;
  bool ok = cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess;
  for (int k = 0; k < 3 && ok; ++k) {
    const bool gs = k == 2;
    WaveKernel fn = wave_kernel(gs, k == 1);
    int per = 0;
    ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)wave_smem(gs)) == cudaSuccess &&
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, (WV_G + 2) * 32, wave_smem(gs)) ==
             cudaSuccess &&
         per > 0;
  }
  cudaGetLastError();
  return ok ? sms : 0;
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
  wave_kernel(gs, a.damping == 1.0f)<<<blocks, (a.G + 2) * 32, wave_smem(gs), f->stream>>>(a);
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
