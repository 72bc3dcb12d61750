// colreg.cuh -- register column transforms with the tensor product (FP32 runs
// of one layer with FFT columns of 64..1024 points, or of two layers with 512
// or 1024), sm_100a.
//
// The column half of get_demag (src/demag.f90:113-127): for each k_x column of
// the 3 NL half spectra M^, the forward FFT along y, H^ = N^ M^ with the
// FP64-built tensor spectrum, and the inverse FFT along y.
//
// A thread works on two adjacent columns at once: their values travel as one
// 16-byte unit through shared memory and as the two lanes of the paired FP32
// instructions (real parts in one pair, imaginary parts in another), so one
// column's instruction stream, addresses and twiddles serve two.  One component
// of N points of a column pair is transformed by NT = N/8 threads holding eight
// elements each, in the stages of regfft.cuh (RegPlan: the Cooley-Tukey plan,
// positions and tables of fft.cuh's in-place passes, so every column kernel
// computes the same transform):
//
//   stage 0: thread t takes rows t + k NT, k < 8, of the staged M^ tile (the
//       zero padding of an open boundary, rows >= N/2, is neither read nor
//       transformed);
//   stages 1..S-1: radix-8 butterflies, each thread reading and writing its own
//       positions of the component's exchange buffer in place;
//   product: thread (component a, t) reads every component at its positions
//       8t..8t+7 of the mixed-radix digit-reversed order and forms H^_a there;
//   the inverse stages run in the reverse order (decimation in time), the first
//       on the product's registers, and the last writes rows < ny of H^ straight
//       to global memory.
//
// The components of a column pair are transformed side by side, by one group
// of G threads each (several column pairs per group where N is short): 3 NL
// groups to a block.  Row p of a column pair sits at unit p + p/8: one pad unit
// in eight keeps the eight lanes of a quarter warp (one 16-byte access each)
// on distinct banks in every stage, and the eight elements of a stage at
// constant offsets from the thread's first (a swizzle would need an xor per
// element and access).
#pragma once
#include "kernels.cuh"

namespace mrm {

constexpr int kCregMinLg = 6, kCregMinLg2 = 9, kCregMaxLg = 10;  // column lengths (kCregMinLg2: two layers)

// ---------------- two columns per thread ----------------
// A pair of FP32 values, one per column, in one 64-bit register (kept as such:
// assembling pairs from scalars costs a move per half).
using F2 = unsigned long long;
MRM_D F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
MRM_D F2 f2(float a) { return f2(a, a); }
MRM_D float2 f2split(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
MRM_D F2 f2add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
MRM_D F2 f2sub(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
MRM_D F2 f2mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
MRM_D F2 f2fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
MRM_D F2 f2neg(F2 a) {
  const float2 v = f2split(a);
  return f2(-v.x, -v.y);
}
struct alignas(16) P2 {
  F2 r, i;  // real and imaginary parts
};
MRM_D P2 padd(P2 a, P2 b) { return {f2add(a.r, b.r), f2add(a.i, b.i)}; }
MRM_D P2 psub(P2 a, P2 b) { return {f2sub(a.r, b.r), f2sub(a.i, b.i)}; }
// a + S i b for S = +1 or -1
template <int S>
MRM_D P2 padd_i(P2 a, P2 b) {
  return S > 0 ? P2{f2sub(a.r, b.i), f2add(a.i, b.r)} : P2{f2add(a.r, b.i), f2sub(a.i, b.r)};
}
// a times the twiddle w = ((wr, wr), (wi, wi)), or its conjugate
template <bool CONJ>
MRM_D P2 ptwiddle(P2 a, P2 w) {
  if (CONJ) return {f2fma(a.r, w.r, f2mul(a.i, w.i)), f2fma(a.i, w.r, f2neg(f2mul(a.r, w.i)))};
  return {f2fma(a.r, w.r, f2neg(f2mul(a.i, w.i))), f2fma(a.i, w.r, f2mul(a.r, w.i))};
}
// shared-memory units of a column pair
MRM_D P2 pload(const float4* p) {
  P2 v;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.r), "=l"(v.i) : "r"(smem_u32(p)));
  return v;
}
MRM_D void pstore(float4* p, P2 v) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(smem_u32(p)), "l"(v.r), "l"(v.i) : "memory");
}

// S = -1 forward, +1 inverse
template <int S>
MRM_D void pdft4(P2& a0, P2& a1, P2& a2, P2& a3) {
  const P2 t0 = padd(a0, a2), t1 = psub(a0, a2), t2 = padd(a1, a3), t3 = psub(a1, a3);
  a0 = padd(t0, t2);
  a2 = psub(t0, t2);
  a1 = padd_i<S>(t1, t3);
  a3 = padd_i<-S>(t1, t3);
}
// the last radix-2 step of an eight-point transform from the transforms e of
// the even and o of the odd elements: the odd ones turned by w8^(S k); the
// factor 1/sqrt 2 of k = 1, 3 joins the sums as a fused multiply-add
template <int S>
MRM_D void pdft8_join(P2 (&v)[8], P2 e0, P2 e1, P2 e2, P2 e3, P2 o0, P2 o1, P2 o2, P2 o3) {
  const F2 h = f2(0.70710678118654752440f), mh = f2(-0.70710678118654752440f);
  v[0] = padd(e0, o0);
  v[4] = psub(e0, o0);
  v[2] = padd_i<S>(e2, o2);
  v[6] = padd_i<-S>(e2, o2);
  // (1 + S i) o1 and (-1 + S i) o3
  const P2 q1 = padd_i<S>(o1, o1), q3 = padd_i<-S>(o3, o3);  // q3 = (1 - S i) o3 = -(-1 + S i) o3
  v[1] = {f2fma(q1.r, h, e1.r), f2fma(q1.i, h, e1.i)};
  v[5] = {f2fma(q1.r, mh, e1.r), f2fma(q1.i, mh, e1.i)};
  v[3] = {f2fma(q3.r, mh, e3.r), f2fma(q3.i, mh, e3.i)};
  v[7] = {f2fma(q3.r, h, e3.r), f2fma(q3.i, h, e3.i)};
}
template <int S>
MRM_D void pdft8(P2 (&v)[8]) {
  P2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  pdft4<S>(e0, e1, e2, e3);
  pdft4<S>(o0, o1, o2, o3);
  pdft8_join<S>(v, e0, e1, e2, e3, o0, o1, o2, o3);
}

// The twiddle m of a thread's butterfly jl in stage STAGE: from the expanded
// pass tables, or from the thread's registers (reg_twiddles).
template <int LGN, int STAGE>
struct TabTwiddles {
  const float4* tw;
  int t;
  MRM_D P2 operator()(int jl, int m) const {
    constexpr int LGD = RegPlan<LGN>::lgd(STAGE), D = 1 << LGD, OFF = pass_tw_off(LGN, LGD);
    const int j0 = STAGE == 0 ? t + (jl << (LGN - 3)) : (t & (D - 1));
    return pload(tw + OFF + (m - 1) * D + j0);
  }
};
template <int LGN, int STAGE>
struct RegTwiddles {
  Cx<float> w[8];
  MRM_D RegTwiddles(int t, const Cx<float>* __restrict__ tw) { reg_twiddles<LGN, STAGE>(w, t, tw); }
  MRM_D P2 operator()(int jl, int m) const {
    constexpr int R = STAGE == 0 ? (1 << RegPlan<LGN>::R0) : 8;
    return P2{f2(w[jl * R + m].x), f2(w[jl * R + m].y)};
  }
};

// Forward stage STAGE on one component's eight elements (decimation in
// frequency: butterfly, then twiddles).  HALF (stage 0): elements of rows >=
// N/2 are zero and not read.
template <int LGN, int STAGE, bool HALF, class TW>
MRM_D void creg_fwd(P2 (&v)[8], const TW& tw) {
  using P = RegPlan<LGN>;
  constexpr int D = 1 << P::lgd(STAGE);
  if constexpr (STAGE == 0 && P::R0 < 3) {
    constexpr int R = 1 << P::R0, NB = 8 / R;
#pragma unroll
    for (int jl = 0; jl < NB; ++jl) {
      P2 u[R];
#pragma unroll
      for (int m = 0; m < (HALF ? R / 2 : R); ++m) u[m] = v[jl + NB * m];
      if constexpr (R == 2) {
        if constexpr (HALF) u[1] = u[0];
        else {
          const P2 a = u[0];
          u[0] = padd(a, u[1]);
          u[1] = psub(a, u[1]);
        }
      } else if constexpr (HALF) {
        const P2 a = u[0], b = u[1];
        u[0] = padd(a, b);
        u[2] = psub(a, b);
        u[1] = padd_i<-1>(a, b);
        u[3] = padd_i<1>(a, b);
      } else {
        pdft4<-1>(u[0], u[1], u[2], u[3]);
      }
      v[jl] = u[0];
#pragma unroll
      for (int m = 1; m < R; ++m) v[jl + NB * m] = ptwiddle<false>(u[m], tw(jl, m));
    }
  } else {
    if constexpr (STAGE == 0 && HALF) {
      // inputs 4..7 zero: the even elements are v0, v2, the odd ones v1, v3
      const P2 a = v[0], b = v[1], c = v[2], d = v[3];
      pdft8_join<-1>(v, padd(a, c), padd_i<-1>(a, c), psub(a, c), padd_i<1>(a, c), padd(b, d), padd_i<-1>(b, d),
                     psub(b, d), padd_i<1>(b, d));
    } else {
      pdft8<-1>(v);
    }
    if constexpr (D > 1) {
#pragma unroll
      for (int m = 1; m < 8; ++m) v[m] = ptwiddle<false>(v[m], tw(0, m));
    }
  }
}

// Inverse stage STAGE (decimation in time: conjugate twiddles, then the
// butterfly with the + sign), unnormalised.
template <int LGN, int STAGE, class TW>
MRM_D void creg_inv(P2 (&v)[8], const TW& tw) {
  using P = RegPlan<LGN>;
  constexpr int D = 1 << P::lgd(STAGE);
  if constexpr (STAGE == 0 && P::R0 < 3) {
    constexpr int R = 1 << P::R0, NB = 8 / R;
#pragma unroll
    for (int jl = 0; jl < NB; ++jl) {
      P2 u[R];
      u[0] = v[jl];
#pragma unroll
      for (int m = 1; m < R; ++m) u[m] = ptwiddle<true>(v[jl + NB * m], tw(jl, m));
      if constexpr (R == 4) {
        pdft4<1>(u[0], u[1], u[2], u[3]);
      } else {
        const P2 a = u[0];
        u[0] = padd(a, u[1]);
        u[1] = psub(a, u[1]);
      }
#pragma unroll
      for (int m = 0; m < R; ++m) v[jl + NB * m] = u[m];
    }
  } else {
    if constexpr (D > 1) {
#pragma unroll
      for (int m = 1; m < 8; ++m) v[m] = ptwiddle<true>(v[m], tw(0, m));
    }
    pdft8<1>(v);
  }
}

// A block's shape: G threads per component group, 3 NL groups; a group holds
// G / (N/8) column pairs, their units interleaved (thread = t * pairs + pair).
MRM_HD constexpr int creg_pairs(int lgpy, int group) { return group >> (lgpy - 3); }
// Shared memory: the expanded twiddles (16 bytes for each of the longest
// columns' table entries), the exchange buffers (G threads x 8 elements x 9/8
// x 16 bytes per group whatever N), then the staged M^ tile.
MRM_HD constexpr int creg_xb_units(int group, int nl) { return 3 * nl * group * 9; }
MRM_HD constexpr int creg_stage_bytes(int nys, int lgpy, int group, int nl) {
  return 3 * nl * nys * 2 * creg_pairs(lgpy, group) * (int)sizeof(Cx<float>);
}
MRM_HD constexpr int creg_smem(int tw_cap, int group, int nl, int stage_bytes) {
  return (tw_cap + creg_xb_units(group, nl)) * (int)sizeof(float4) + stage_bytes;
}

// The tensor of the column pair kp at the product positions: [pair of layers]
// [component: xx yy zz xy xz yz][j < 4][t < NT][position 8t + 2j, 8t + 2j + 1][column],
// reals (the xz and yz spectra are imaginary: the stored real times i; the sign
// of the odd components in the upper half of k_y folded in), so the lanes of a
// warp read consecutive float4.
MRM_HD constexpr size_t creg_tensor_reals(int lgpy, int nl) { return (size_t)nl * nl * 6 * 2 << lgpy; }

// barrier of the G threads of group c (ids are immediates: a kernel reserves
// barriers 0..6)
template <int G>
MRM_D void creg_group_sync(int c) {
  if constexpr (G == 32) {
    __syncwarp();
  } else {
    switch (c) {
      case 0: asm volatile("bar.sync 1, %0;" ::"n"(G) : "memory"); break;
      case 1: asm volatile("bar.sync 2, %0;" ::"n"(G) : "memory"); break;
      case 2: asm volatile("bar.sync 3, %0;" ::"n"(G) : "memory"); break;
      case 3: asm volatile("bar.sync 4, %0;" ::"n"(G) : "memory"); break;
      case 4: asm volatile("bar.sync 5, %0;" ::"n"(G) : "memory"); break;
      default: asm volatile("bar.sync 6, %0;" ::"n"(G) : "memory"); break;
    }
  }
}

template <int LGN, int G, int STAGE, bool INV>
MRM_D void creg_stage(float4* __restrict__ buf, int t, const float4* __restrict__ tw) {
  using P = RegPlan<LGN>;
  constexpr int B = P::dbit(STAGE), PR = G / P::NT, STEP = B >= 3 ? ((1 << B) + (1 << (B - 3))) * PR : PR;
  static_assert(B == 0 || B >= 3, "the padded positions of a stage are equally spaced");
  const int pb = reg_base<B>(t);
  float4* b = buf + (pb + (pb >> 3)) * PR;
  P2 v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = pload(b + k * STEP);
  const TabTwiddles<LGN, STAGE> w{tw, t};
  if constexpr (INV) creg_inv<LGN, STAGE>(v, w);
  else creg_fwd<LGN, STAGE, false>(v, w);
#pragma unroll
  for (int k = 0; k < 8; ++k) pstore(b + k * STEP, v[k]);
}

// The tensor values of a thread's product (layer and component a of H^, its
// positions 8t..8t+7), in pieces hs of four positions and one source layer:
// those of one layer are loaded ahead of the task's transforms, which cover
// their latency (the tensor never changes: the first task's come in before the
// previous kernel has finished), further layers' as the product goes.
// AHEAD: the pieces loaded ahead (both of one layer where the launch bounds
// leave a thread the registers: at most 384 threads per SM).
template <int LGN, int G, int NL, int AHEAD>
struct CregTens {
  static constexpr int PIECES = 2 * NL;
  ulonglong2 v[PIECES][3][2];
  const ulonglong2* tn;
  // k0 < 0: nothing to load
  MRM_D void start(const RunDev<float>& rd, int k0, int nc) {
    constexpr int NT = RegPlan<LGN>::NT, PR = G / NT;
    const int q = threadIdx.x / G, gt = threadIdx.x - q * G, t = gt / PR, pair = gt - t * PR;
    const int kp = k0 < 0 ? 0 : (k0 >> 1) + (2 * pair < nc ? pair : 0);
    tn = reinterpret_cast<const ulonglong2*>(rd.tens + (size_t)kp * creg_tensor_reals(LGN, NL)) + t;
#pragma unroll
    for (int hs = 0; hs < AHEAD; ++hs) load(hs, k0 >= 0);
  }
  MRM_D void load(int hs, bool on = true) {
    constexpr int NT = RegPlan<LGN>::NT;
    const int q = threadIdx.x / G, a = q % 3, o = q / 3, half = hs / NL, s = hs - half * NL;
    // a = q % 3 of layer o = q / 3 (layer pair = source * NL + o)
    const int comp[3] = {a == 0 ? 0 : a == 1 ? 3 : 4, a == 0 ? 3 : a == 1 ? 1 : 5, a == 0 ? 4 : a == 1 ? 5 : 2};
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        v[hs][b][j] = on ? __ldg(tn + ((size_t)((s * NL + o) * 6 + comp[b]) * 4 + 2 * half + j) * NT)
                         : make_ulonglong2(0, 0);
  }
};

// One task (columns k0 .. k0 + nc - 1 of run rd): forward transforms, product,
// inverse transforms.  stg: the task's M^ tiles staged in shared memory
// ([plane][tile][nys][T]); xb: the exchange buffers; `staged_read` runs once
// every thread has its stage-0 elements in registers.
template <int LGN, int G, int NL, int AHEAD, bool HALF, class AFTER>
MRM_D void creg_body(const RunDev<float>& rd, int k0, int nc, CregTens<LGN, G, NL, AHEAD>& tens,
                     const float4* __restrict__ tw, const Cx<float>* __restrict__ stg, float4* __restrict__ xb,
                     const AFTER& staged_read) {
  using P = RegPlan<LGN>;
  constexpr int N = P::N, NT = P::NT, KIN = HALF ? 4 : 8, PR = G / NT, S = P::S, B0 = P::dbit(0);
  constexpr int SEQ = G * 9;  // units of a group's exchange buffer
  constexpr int STEP0 = ((1 << B0) + (1 << (B0 - 3))) * PR;
  const int q = threadIdx.x / G, gt = threadIdx.x - q * G, t = gt / PR, pair = gt - t * PR;
  const bool live = 2 * pair < nc;
  float4* const buf = xb + q * SEQ + pair;
  const int ny = rd.ny;
  P2 v[8];
  {
    // stage 0 from the staged tiles: rows t + kk NT
    const int lgct = rd.lgct, T = 1 << lgct, nys = rd.nys;
    const int ntl = (nc + T - 1) >> lgct;
    const Cx<float>* src = stg + (((size_t)(q * ntl + ((2 * pair) >> lgct)) * nys) << lgct) + ((2 * pair) & (T - 1));
#pragma unroll
    for (int kk = 0; kk < KIN; ++kk) {
      const int j = t + kk * NT;
      if (live && j < ny) {
        const float4 a = *reinterpret_cast<const float4*>(src + ((size_t)j << lgct));
        v[kk] = P2{f2(a.x, a.z), f2(a.y, a.w)};
      } else {
        v[kk] = P2{0, 0};
      }
    }
    creg_fwd<LGN, 0, HALF>(v, TabTwiddles<LGN, 0>{tw, t});
    float4* b = buf + (t + (t >> 3)) * PR;  // positions t + kk NT (the thread's own last reads of the task before)
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) pstore(b + kk * STEP0, v[kk]);
  }
  __syncthreads();
  staged_read();
  creg_stage<LGN, G, 1, false>(buf, t, tw);
  if constexpr (S >= 3) {
    creg_group_sync<G>(q);
    creg_stage<LGN, G, 2, false>(buf, t, tw);
  }
  if constexpr (S >= 4) {
    creg_group_sync<G>(q);
    creg_stage<LGN, G, 3, false>(buf, t, tw);
  }
  // product: H^_a at positions 8t..8t+7
  const int a = q % 3;
  __syncthreads();
  const int at8 = 9 * t * PR + pair;
#pragma unroll
  for (int hs = 0; hs < 2 * NL; ++hs) {
    const int half = hs / NL, s = hs - half * NL;
    if (hs + AHEAD < 2 * NL) tens.load(hs + AHEAD);
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const float4* m = xb + (s * 3 + b) * SEQ + at8 + 4 * half * PR;
      // xz, zx, yz, zy are imaginary
      const bool imag = (a == 2) != (b == 2);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        P2 mk = pload(m + k * PR);
        const F2 tk = (k & 1) ? tens.v[hs][b][k >> 1].y : tens.v[hs][b][k >> 1].x;
        P2& h = v[4 * half + k];
        if (imag) mk = P2{f2neg(mk.i), mk.r};
        if (s == 0 && b == 0) h = P2{f2mul(tk, mk.r), f2mul(tk, mk.i)};
        else h = P2{f2fma(tk, mk.r, h.r), f2fma(tk, mk.i, h.i)};
      }
    }
  }
  creg_inv<LGN, S - 1>(v, TabTwiddles<LGN, S - 1>{tw, t});
  __syncthreads();  // every group has read the products' inputs
  {
    float4* b = buf + 9 * t * PR;
#pragma unroll
    for (int k = 0; k < 8; ++k) pstore(b + k * PR, v[k]);
  }
  creg_group_sync<G>(q);
  if constexpr (S >= 4) {
    creg_stage<LGN, G, 2, true>(buf, t, tw);
    creg_group_sync<G>(q);
  }
  if constexpr (S >= 3) {
    creg_stage<LGN, G, 1, true>(buf, t, tw);
    creg_group_sync<G>(q);
  }
  // inverse stage 0 and the H^ rows, row-major [plane][ny][phs] (a last odd
  // column's partner is the row's padding)
  const float4* b = buf + (t + (t >> 3)) * PR;
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) v[kk] = pload(b + kk * STEP0);
  creg_inv<LGN, 0>(v, TabTwiddles<LGN, 0>{tw, t});
  if (live) {
    const int phs = rd.phs;
    Cx<float>* dst = rd.spech + (size_t)q * ny * phs + k0 + 2 * pair;
#pragma unroll
    for (int kk = 0; kk < KIN; ++kk) {
      const int j = t + kk * NT;
      if (j < ny) {
        const float2 re = f2split(v[kk].r), im = f2split(v[kk].i);
        *reinterpret_cast<float4*>(dst + (size_t)j * phs) = make_float4(re.x, im.x, re.y, im.y);
      }
    }
  }
}

// A task (run, first column k0, columns nc <= 2 G / (py/8), whole M^ tiles but
// for the run's last) is checked against the compiled shape and the launch's
// shared memory.
MRM_D bool creg_task_ok(const RunDev<float>& rd, int k0, int nc, int group, int nl, int tw_cap, int stage_cap) {
  const int lgpy = rd.lgpy, T = 1 << rd.lgct, ph = (rd.px >> 1) + 1;
  return lgpy >= (nl == 1 ? kCregMinLg : kCregMinLg2) && lgpy <= kCregMaxLg && (8 * group >> lgpy) >= 1 && rd.nl == nl && nc >= 1 && k0 >= 0 &&
         k0 + nc <= ph && nc <= 2 * creg_pairs(lgpy, group) && T >= 2 && (k0 & (T - 1)) == 0 &&
         col_tw_count(lgpy) <= tw_cap && T <= 2 * creg_pairs(lgpy, group) &&
         creg_stage_bytes(rd.nys, lgpy, group, nl) <= stage_cap;
}

// Persistent blocks: block b takes tasks b, b + B, b + 2B, ... (B blocks).
// While a task is transformed, the next task's M^ tiles and the descriptor
// (RunDev up to its layers) of the task after that are on their way into
// shared memory, by bulk copies that one thread issues as soon as every thread
// has read the current tiles: neither the tiles nor the chain task -> run ->
// address is waited for, and the block reads the run's sizes and strides from
// shared memory.  The first task's descriptor, twiddles and tensor come in
// before the previous kernel has finished.  The twiddles are expanded again
// only when the next task's column length differs.
// Bound, in a single run, by the latency of one task's chain of stages (129
// tasks on 148 SMs at 256 x 256): with the tensor loaded ahead and the first
// descriptor before the dependency wait, at 168 registers and two blocks per SM,
// a 256 x 256 run takes 38.2 us per Heun step, and 48.0 without (80 registers
// spill those loads).  On a batch by the shared-memory pipe (78 % of its
// wavefronts): see below.
//
// Whether a task has work (its run is active and due) is thread 0's verdict,
// taken when it issues the tiles, in a word of its own per slot that is read
// only behind landed() of that task.  Everything read earlier, the choice of
// the loop among it, is constant while the kernel runs, so every thread of the
// block takes the same path and meets the same barriers: a task without work
// meets one, in landed().
struct CregTasks {
  alignas(16) unsigned char hdr[3][kRunHdrBytes];  // run headers of three consecutive tasks
  int2 cols[3];                                    // their first column and columns
  int work[3];                                     // their tiles are on the way (thread 0's verdict)
  uint64_t bar;
};

struct CregLoop {
  const RunDev<float>* runs;
  const Task* tasks;
  CregTasks* ct;
  Cx<float>* stg;
  int* err;
  int ntasks, istep, flags, tw_cap, stage_cap;
  int i, r;         // the current task's index and slot
  uint32_t phase;
  bool first;       // the current task is the block's first: its tiles are not under way
  Task tnext;       // thread 0: the task whose header is copied next

  MRM_D const RunDev<float>& rd(int slot) const { return *reinterpret_cast<const RunDev<float>*>(ct->hdr[slot]); }
  MRM_D int next_slot(int slot) const { return slot == 2 ? 0 : slot + 1; }
  // thread 0: the run header of a task into a slot
  MRM_D void start_header(int slot, const Task& tk) {
    ct->cols[slot] = make_int2(tk.y, tk.z);
    bulk_copy(&ct->bar, ct->hdr[slot], runs + tk.x, (uint32_t)kRunHdrBytes);
  }
  // thread 0: the tiles of the task in the slot (its header has landed) into the
  // staging area
  MRM_D void start_tile(int slot, long long step) {
    const RunDev<float>& h = rd(slot);
    const int2 kc = ct->cols[slot];
    const bool live = h.active && h.demag && ((flags & kFlagForce) || step_due(h, step + istep));
    const bool ok = task_ok(slot);
    if (live && !ok) atomicOr(err, kErrShape);
    ct->work[slot] = live && ok;
    if (!(live && ok)) return;
    const int lgct = h.lgct, T = 1 << lgct, ph = (h.px >> 1) + 1, ntile = (ph + T - 1) >> lgct;
    const int ntl = (kc.y + T - 1) >> lgct, plane = (h.nys << lgct) * ntl;
    const Cx<float>* src = h.specx + (((size_t)(kc.x >> lgct) * h.nys) << lgct);
    const size_t pstride = ((size_t)ntile * h.nys) << lgct;
    for (int q = 0; q < 3 * nl; ++q)
      bulk_copy(&ct->bar, stg + q * plane, src + q * pstride, (uint32_t)(plane * sizeof(Cx<float>)));
  }
  int group, nl;    // the compiled shape
  // (from the lengths and the table entry alone: the same for every thread at
  // any time once the header has landed)
  MRM_D bool task_ok(int slot) const {
    const int2 kc = ct->cols[slot];
    return creg_task_ok(rd(slot), kc.x, kc.y, group, nl, tw_cap, stage_cap);
  }
  // thread 0: the tiles of task index `at` in the slot and the header of the next,
  // one phase of the barrier
  MRM_D void issue(int slot, int at, long long step) {
    const int stride = (int)gridDim.x;
    start_tile(slot, step);
    if (at + stride < ntasks) {
      start_header(next_slot(slot), tnext);
      if (at + 2 * stride < ntasks) tnext = tasks[at + 2 * stride];
    }
    mbar_arrive(&ct->bar);
  }
  // (the header's step counter is the one of the launch: it was copied after the
  // dependency wait)
  MRM_D void issue_next() {
    if (threadIdx.x == 0 && i + (int)gridDim.x < ntasks) issue(next_slot(r), i + (int)gridDim.x, rd(next_slot(r)).step);
  }
  MRM_D bool landed() {
    const bool ok = mbar_wait(&ct->bar, phase);
    phase ^= 1;
    if (!__syncthreads_or(!ok)) return true;
    if (threadIdx.x == 0) atomicOr(err, kErrBarrierTimeout);
    mbar_wait(&ct->bar, phase ^ 1);
    return false;
  }
  // the dependency wait, then the first task's tiles (its header came in before
  // the wait: the step counter is read again)
  MRM_D void begin() {
    if (!first) return;
    first = false;
    pdl_wait();
    if (threadIdx.x == 0) issue(r, i, *reinterpret_cast<const volatile long long*>(&runs[tasks[i].x].step));
  }
  MRM_D void advance() {
    i += (int)gridDim.x;
    r = next_slot(r);
  }
};

// The block's tasks from the current one on for as long as they have this
// column length and padding (the current one does); false: a copy did not land.
template <int LGN, int G, int NL, int AHEAD, bool HALF>
MRM_D bool creg_run(CregLoop& c, const float4* tw, float4* xb) {
  if constexpr ((1 << (LGN - 3)) <= G) {
    while (true) {
      const RunDev<float>& rd = c.rd(c.r);
      CregTens<LGN, G, NL, AHEAD> tens;
      tens.start(rd, rd.active && rd.demag ? c.ct->cols[c.r].x : -1, c.ct->cols[c.r].y);
      c.begin();
      if (!c.landed()) return false;
      const int2 kc = c.ct->cols[c.r];
      if (!c.ct->work[c.r]) {
        c.issue_next();  // (no tile of this task was copied, and every thread is past the last one's)
      } else {
        creg_body<LGN, G, NL, AHEAD, HALF>(rd, kc.x, kc.y, tens, tw, c.stg, xb, [&]() { c.issue_next(); });
      }
      c.advance();
      if (c.i >= c.ntasks) return true;
      const RunDev<float>& rn = c.rd(c.r);
      if (rn.lgpy != LGN || (rn.py >= 2 * rn.ny) != HALF || !c.task_ok(c.r)) return true;
    }
  }
  return true;
}

template <int G, int NL, int MINB>
__global__ void __launch_bounds__(3 * NL * G, MINB)
    creg_kernel(const RunDev<float>* __restrict__ runs, const Task* __restrict__ tasks, int ntasks,
                const Cx<float>* __restrict__ twg, int istep, int flags, int tw_cap, int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ CregTasks ct;
  pdl_launch_dependents();
  float4* tws = reinterpret_cast<float4*>(smem_raw);
  float4* xb = tws + tw_cap;
  Cx<float>* stg = reinterpret_cast<Cx<float>*>(xb + creg_xb_units(G, NL));
  const int stage_cap = (int)dynamic_smem_bytes() - (tw_cap + creg_xb_units(G, NL)) * (int)sizeof(float4);
  CregLoop c;
  c.runs = runs;
  c.tasks = tasks;
  c.ct = &ct;
  c.stg = stg;
  c.err = err;
  c.ntasks = ntasks;
  c.istep = istep;
  c.flags = flags;
  c.tw_cap = tw_cap;
  c.stage_cap = stage_cap;
  c.i = blockIdx.x;
  c.r = 0;
  c.phase = 0;
  c.first = true;
  c.tnext = Task{};
  c.group = G;
  c.nl = NL;
  if (c.i >= ntasks) {
    pdl_wait();
    return;
  }
  if (threadIdx.x == 0) {
    mbar_init(&ct.bar, 1);
    mbar_fence_init();
    // phase 0: the header of the block's first task (but for the step counter, a
    // run's header never changes while kernels of the engine run)
    c.start_header(0, tasks[c.i]);
    mbar_arrive(&ct.bar);
    if (c.i + (int)gridDim.x < ntasks) c.tnext = tasks[c.i + gridDim.x];
  }
  __syncthreads();
  if (!c.landed()) return;
  int tw_lg = -1;
  // the pass tables of columns of 2^lg points, each entry as (re, re, im, im)
  auto expand_twiddles = [&](int lg, int off) {
    const int n = min(col_tw_count(lg), tw_cap);
    for (int e = threadIdx.x; e < n; e += 3 * NL * G) {
      const Cx<float> w = twg[off + e];
      tws[e] = make_float4(w.x, w.x, w.y, w.y);
    }
    tw_lg = lg;
  };
  bool ok = true;
  while (ok && c.i < ntasks) {
    const RunDev<float>& rd = c.rd(c.r);
    if (!c.task_ok(c.r)) {  // (start_tile reports it and copies nothing)
      c.begin();
      ok = c.landed();
      if (!ok) return;
      c.issue_next();
      c.advance();
      continue;
    }
    const int lgpy = rd.lgpy;
    if (lgpy != tw_lg) {
      __syncthreads();  // every thread is past its last use of the tables
      expand_twiddles(lgpy, rd.tw_col);
      __syncthreads();
    }
    const bool half = rd.py >= 2 * rd.ny;
    auto go = [&](auto lg) {
      constexpr int LGN = decltype(lg)::value, AHEAD = NL == 1 && 3 * NL * G * MINB <= 384 ? 2 : 1;
      ok = half ? creg_run<LGN, G, NL, AHEAD, true>(c, tws, xb) : creg_run<LGN, G, NL, AHEAD, false>(c, tws, xb);
    };
    if constexpr (NL == 1) {
      switch (lgpy) {
        case 6: go(IntC<6>{}); break;
        case 7: go(IntC<7>{}); break;
        case 8: go(IntC<8>{}); break;
        case 9: go(IntC<9>{}); break;
        default: go(IntC<10>{}); break;
      }
    } else {
      if (lgpy == 9) go(IntC<9>{});
      else go(IntC<10>{});
    }
  }
}

// ---------------- components in turn ----------------
// The same transforms with one group of G threads taking the three components
// of its column pairs in turn (runs of one layer): the twiddles of a stage are
// loaded once for the three, and the last forward stage, the product and the
// first inverse stage run in registers, so a component passes through shared
// memory eight times instead of twelve.  It moves about half the shared-memory
// wavefronts of the kernel above, which is what binds that one on a batch; the
// latter has a third of its latency per task, which is what a single run waits
// for.
MRM_HD constexpr int cser_smem(int tw_cap, int group) {
  return tw_cap * (int)sizeof(Cx<float>) + creg_xb_units(group, 1) * (int)sizeof(float4);
}

template <int LGN, int G, int STAGE, bool INV>
MRM_D void cser_stage(float4* __restrict__ buf, int t, const Cx<float>* __restrict__ tw) {
  using P = RegPlan<LGN>;
  constexpr int B = P::dbit(STAGE), PR = G / P::NT, STEP = B >= 3 ? ((1 << B) + (1 << (B - 3))) * PR : PR;
  static_assert(B == 0 || B >= 3, "the padded positions of a stage are equally spaced");
  const int pb = reg_base<B>(t);
  const RegTwiddles<LGN, STAGE> w(t, tw);
#pragma unroll 1
  for (int q = 0; q < 3; ++q) {
    float4* b = buf + q * (G * 9) + (pb + (pb >> 3)) * PR;
    P2 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = pload(b + k * STEP);
    if constexpr (INV) creg_inv<LGN, STAGE>(v, w);
    else creg_fwd<LGN, STAGE, false>(v, w);
#pragma unroll
    for (int k = 0; k < 8; ++k) pstore(b + k * STEP, v[k]);
  }
}

// The thread's stage-0 inputs of a task, straight from the M^ tiles: rows
// t + kk NT of its column pair (two columns to a 16-byte unit) of each component.
template <int LGN, int G, bool HALF>
struct CserIn {
  static constexpr int KIN = HALF ? 4 : 8;
  float4 v[3][KIN];
  MRM_D void load(const RunDev<float>& rd, int k0, int nc) {
    using P = RegPlan<LGN>;
    constexpr int NT = P::NT, PR = G / NT;
    const int t = threadIdx.x / PR, pair = threadIdx.x - t * PR, k = k0 + 2 * pair;
    const bool live = 2 * pair < nc;
    const int lgct = rd.lgct, T = 1 << lgct, ny = rd.ny, nys = rd.nys, ntile = (((rd.px >> 1) + 1) + T - 1) >> lgct;
    const size_t pstride = ((size_t)ntile * nys) << lgct;
    const Cx<float>* src = rd.specx + (((size_t)((live ? k : k0) >> lgct) * nys) << lgct) + (k & (T - 1));
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int kk = 0; kk < KIN; ++kk) {
        const int j = t + kk * NT;
        v[q][kk] = live && j < ny ? *reinterpret_cast<const float4*>(src + q * pstride + ((size_t)j << lgct))
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
      }
  }
};

template <int LGN, int G, bool HALF>
MRM_D void cser_body(const RunDev<float>& rd, int k0, int nc, const Cx<float>* __restrict__ tw,
                     float4* __restrict__ xb) {
  using P = RegPlan<LGN>;
  constexpr int NT = P::NT, KIN = HALF ? 4 : 8, PR = G / NT, S = P::S, B0 = P::dbit(0);
  constexpr int SEQ = G * 9, STEP0 = ((1 << B0) + (1 << (B0 - 3))) * PR;
  const int t = threadIdx.x / PR, pair = threadIdx.x - t * PR, k = k0 + 2 * pair;
  const bool live = 2 * pair < nc;
  float4* const buf = xb + pair;
  {
    CserIn<LGN, G, HALF> in;
    in.load(rd, k0, nc);
    const RegTwiddles<LGN, 0> w(t, tw);
    float4* b = buf + (t + (t >> 3)) * PR;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      P2 v[8];
#pragma unroll
      for (int kk = 0; kk < KIN; ++kk) {
        const float4 x = in.v[q][kk];
        v[kk] = P2{f2(x.x, x.z), f2(x.y, x.w)};
      }
      creg_fwd<LGN, 0, HALF>(v, w);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) pstore(b + q * SEQ + kk * STEP0, v[kk]);
    }
  }
  __syncthreads();
  if constexpr (S >= 3) {
    cser_stage<LGN, G, 1, false>(buf, t, tw);
    __syncthreads();
  }
  if constexpr (S >= 4) {
    cser_stage<LGN, G, 2, false>(buf, t, tw);
    __syncthreads();
  }
  {
    // last forward stage (no twiddles), product, first inverse stage at the
    // thread's own positions 8t..8t+7; the tensor one chunk (of two positions) ahead
    const ulonglong2* tn = reinterpret_cast<const ulonglong2*>(rd.tens + (size_t)((live ? k : k0) >> 1) *
                                                                             creg_tensor_reals(LGN, 1)) + t;
    ulonglong2 tv[2][6];
    auto tens_load = [&](int j) {
#pragma unroll
      for (int c = 0; c < 6; ++c) tv[j & 1][c] = __ldg(tn + (c * 4 + j) * NT);
    };
    tens_load(0);
    float4* b = buf + 9 * t * PR;
    P2 v[3][8];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) v[q][kk] = pload(b + q * SEQ + kk * PR);
      pdft8<-1>(v[q]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j < 3) tens_load(j + 1);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        auto tc = [&](int c) { return h ? tv[j & 1][c].y : tv[j & 1][c].x; };
        const F2 xx = tc(0), yy = tc(1), zz = tc(2), xy = tc(3), xz = tc(4), yz = tc(5);
        P2 &ax = v[0][2 * j + h], &ay = v[1][2 * j + h], &az = v[2][2 * j + h];
        const P2 x = ax, y = ay, z = az;
        // (xz and yz are imaginary; the sums in the order of the kernel above)
        const F2 xi = f2neg(x.i), yi = f2neg(y.i), zi = f2neg(z.i);
        ax = P2{f2fma(xz, zi, f2fma(xy, y.r, f2mul(xx, x.r))), f2fma(xz, z.r, f2fma(xy, y.i, f2mul(xx, x.i)))};
        ay = P2{f2fma(yz, zi, f2fma(yy, y.r, f2mul(xy, x.r))), f2fma(yz, z.r, f2fma(yy, y.i, f2mul(xy, x.i)))};
        az = P2{f2fma(zz, z.r, f2fma(yz, yi, f2mul(xz, xi))), f2fma(zz, z.i, f2fma(yz, y.r, f2mul(xz, x.r)))};
      }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      pdft8<1>(v[q]);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) pstore(b + q * SEQ + kk * PR, v[q][kk]);
    }
  }
  if constexpr (S >= 4) {
    __syncthreads();
    cser_stage<LGN, G, 2, true>(buf, t, tw);
  }
  if constexpr (S >= 3) {
    __syncthreads();
    cser_stage<LGN, G, 1, true>(buf, t, tw);
  }
  __syncthreads();
  // inverse stage 0 and the H^ rows (a last odd column's partner is the row's padding)
  const RegTwiddles<LGN, 0> w(t, tw);
  const int phs = rd.phs, ny = rd.ny;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const float4* b = buf + q * SEQ + (t + (t >> 3)) * PR;
    P2 v[8];
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) v[kk] = pload(b + kk * STEP0);
    creg_inv<LGN, 0>(v, w);
    if (live) {
      Cx<float>* dst = rd.spech + (size_t)q * ny * phs + k;
#pragma unroll
      for (int kk = 0; kk < KIN; ++kk) {
        const int j = t + kk * NT;
        if (j < ny) {
          const float2 re = f2split(v[kk].r), im = f2split(v[kk].i);
          *reinterpret_cast<float4*>(dst + (size_t)j * phs) = make_float4(re.x, im.x, re.y, im.y);
        }
      }
    }
  }
}

template <int LGN, int G>
MRM_D void cser_column(const RunDev<float>& rd, int k0, int nc, const Cx<float>* tw, float4* xb) {
  if constexpr ((1 << (LGN - 3)) <= G) {
    if (rd.py >= 2 * rd.ny) cser_body<LGN, G, true>(rd, k0, nc, tw, xb);
    else cser_body<LGN, G, false>(rd, k0, nc, tw, xb);
  }
}

// Persistent blocks: block b takes tasks b, b + B, b + 2B, ... (B blocks), its
// next task's table entry loaded while the current one runs.
// Measured on 32 runs of 256 x 256 grains, per launch: 72 us (22.7 M warp
// instructions; 168 registers, 12 warps per SM, so bound by latency: a third of
// its stalls are global loads, a fifth shared ones), 86 us with the components
// side by side, 94 us with one column per thread group and 8-byte accesses
// (36 M); eight runs of 512 x 512 87 us, and 103 in the last form.  Loading the
// next task's inputs ahead spills (76 us); the tensor two chunks ahead instead
// of one changes nothing.
template <int G, int MINB>
__global__ void __launch_bounds__(G, MINB)
    cser_kernel(const RunDev<float>* __restrict__ runs, const Task* __restrict__ tasks, int ntasks,
                const Cx<float>* __restrict__ twg, int istep, int flags, int tw_cap, int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_launch_dependents();
  float4* xb = reinterpret_cast<float4*>(smem_raw);
  Cx<float>* tws = reinterpret_cast<Cx<float>*>(xb + creg_xb_units(G, 1));
  const int tw_room =
      min(tw_cap, ((int)dynamic_smem_bytes() - creg_xb_units(G, 1) * (int)sizeof(float4)) / (int)sizeof(Cx<float>));
  int i = blockIdx.x, tw_lg = -1;
  auto copy_twiddles = [&](int lg, int off) {
    const int n = min(col_tw_count(lg), tw_room);
    for (int e = threadIdx.x; e < n; e += G) tws[e] = twg[off + e];
    tw_lg = lg;
  };
  if (i >= ntasks) return;
  Task tk = tasks[i];
  copy_twiddles(runs[tk.x].lgpy, runs[tk.x].tw_col);  // (a run's never change)
  __syncthreads();
  pdl_wait();  // every task's M^ tiles come from the previous kernel
  while (true) {
    const RunDev<float>& rd = runs[tk.x];
    const int k0 = tk.y, nc = tk.z;
    i += gridDim.x;
    if (i < ntasks) tk = tasks[i];
    const int lgpy = rd.lgpy, T = 1 << rd.lgct, ph = (rd.px >> 1) + 1;
    // (the step counter does not change while this kernel is resident: advance_kernel)
    const bool work = rd.active && rd.demag && ((flags & kFlagForce) || step_due(rd, rd.step + istep));
    const bool ok = lgpy >= kCregMinLg && lgpy <= kCregMaxLg && (8 * G >> lgpy) >= 1 && rd.nl == 1 && nc >= 1 &&
                    k0 >= 0 && (k0 & 1) == 0 && k0 + nc <= ph && nc <= 2 * creg_pairs(lgpy, G) && T >= 2 &&
                    col_tw_count(lgpy) <= tw_room;
    if (work && !ok && threadIdx.x == 0) atomicOr(err, kErrShape);
    if (work && ok) {
      if (lgpy != tw_lg) {
        __syncthreads();  // every thread is past its last use of the tables
        copy_twiddles(lgpy, rd.tw_col);
        __syncthreads();
      }
      switch (lgpy) {
        case 6: cser_column<6, G>(rd, k0, nc, tws, xb); break;
        case 7: cser_column<7, G>(rd, k0, nc, tws, xb); break;
        case 8: cser_column<8, G>(rd, k0, nc, tws, xb); break;
        case 9: cser_column<9, G>(rd, k0, nc, tws, xb); break;
        default: cser_column<10, G>(rd, k0, nc, tws, xb); break;
      }
    }
    if (i >= ntasks) return;
  }
}

}  // namespace mrm
