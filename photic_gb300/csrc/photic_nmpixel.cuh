// photic_nmpixel.cuh -- the resumable Nelder-Mead of photic_nm.cuh for the
// six unknowns of a single-scene pixel, one lane a pixel, written for a
// small footprint in the instruction cache.
//
// The kernels that run it (photic_invert.cu, photic_lut.cu) evaluate about
// two thousand instructions of cost a trip, and their warps are at
// different places of the code: past the 32 KB that the instruction cache
// streams at full rate a warp waited for instructions as often as for
// anything else (3.8 of 8.5 clocks between two instructions, ncu).  So the
// vectors live in shared memory ([slot][thread], conflict-free) beside the
// vertices, loops over the coordinates are rolled, and everything that
// several phases do is written once: the switch only decides (a vertex
// replaced, made or shrunk, the next point) and the stages below it act.
// The centroid's sums run on the integer pipe (sf::sum_less_one): on the
// FP64 pipe they were a fifth of a trip.  The point under evaluation doubles
// as the trial of an expansion or contraction and as the minimiser that the
// probes move.
//
// The sequence of points, comparisons and counters is nelmin's
// (model/asa047.c:10-502).
#pragma once
#include <stdint.h>

#include "photic_nm.cuh"
#include "photic_softfp.cuh"

namespace photic {

template <class P, int BS>
struct NmPixel {
  using T = typename P::T;
  static constexpr int N = 6;
  // slots of the lane's shared memory
  static constexpr int kV = 0, kF = kV + (N + 1) * N, kX = kF + N + 1, kRefl = kX + N,
                       kCen = kRefl + N, kStep = kCen + N, kSlots = kStep + N;
  T *w;  // shared: slot s at w[s * BS]
  T ylo, fr, scale, var_limit;
  long long floor_lo;
  int32_t phase, jj, hi, lo, icount, numres, ifault, countdown, kcount, konvge;

  __device__ __forceinline__ T &V(int j, int i) { return w[(kV + j * N + i) * BS]; }
  __device__ __forceinline__ T &F(int j) { return w[(kF + j) * BS]; }
  __device__ __forceinline__ T &x(int i) { return w[(kX + i) * BS]; }
  __device__ __forceinline__ T &refl(int i) { return w[(kRefl + i) * BS]; }
  __device__ __forceinline__ T &cen(int i) { return w[(kCen + i) * BS]; }
  __device__ __forceinline__ T &step(int i) { return w[(kStep + i) * BS]; }

  __device__ __forceinline__ void set_start(const T (&start)[N], const T (&steps)[N]) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      x(i) = start[i];
      step(i) = steps[i];
    }
  }

  // Begin a nelmin call from x (the start) and step (model/asa047.c:161-170).
  __device__ __forceinline__ void begin(T var_limit_, int32_t konvge_, int32_t kcount_) {
    konvge = konvge_;
    kcount = kcount_;
    countdown = konvge_;
    icount = 0;
    numres = 0;
    ifault = 0;
    scale = P::one();
    var_limit = var_limit_;
    restart_simplex();
  }

  // Vertex N is the start point.
  __device__ __forceinline__ void restart_simplex() {
#pragma unroll 1
    for (int i = 0; i < N; i++) V(N, i) = x(i);
    phase = PH_INIT_BASE;
  }

  // Top of the inner loop (model/asa047.c:213-250).  false: the loop ends.
  __device__ __forceinline__ bool inner_top() {
    if (kcount <= icount) return false;
    T yhi = F(0);
    hi = 0;
#pragma unroll 1
    for (int j = 1; j <= N; j++) {
      const T fj = F(j);
      if (P::lt(yhi, fj)) {
        yhi = fj;
        hi = j;
      }
    }
#pragma unroll 1
    for (int i = 0; i < N; i++) {
      T z;
      if (!P::sum_less_one(&V(0, i), N * BS, N + 1, hi, z)) {
        z = P::zero();
#pragma unroll 1
        for (int j = 0; j <= N; j++) z = P::add(z, V(j, i));
        z = P::sub(z, V(hi, i));
      }
      cen(i) = P::div_n(z, N);
    }
    phase = PH_REFLECT;
    return true;
  }

  // End of an iteration (model/asa047.c:395-434).  true: the variance test
  // ends the inner loop.
  __device__ __forceinline__ bool iteration_end() {
    const T fh = F(hi);
    if (P::lt(fh, ylo)) {
      ylo = fh;
      lo = hi;
    }
    countdown--;
    if (countdown > 0 || icount > kcount) return false;
    countdown = konvge;
    T z = P::zero();
#pragma unroll 1
    for (int j = 0; j <= N; j++) z = P::add(z, F(j));
    const T mean = P::div_n(z, N + 1);
    z = P::zero();
#pragma unroll 1
    for (int j = 0; j <= N; j++) {
      const T d = P::sub(F(j), mean);
      z = P::add(z, P::mul(d, d));
    }
    return P::le(z, var_limit);
  }

  // Consume the cost y of x and advance to the next point.  Returns true
  // when the nelmin call has returned (x, F(lo), icount, numres, ifault hold
  // its results).
  __device__ __forceinline__ bool step_machine(T y) {
    enum { CS_NONE = -1, CS_READY, CS_TOP, CS_ITER_END, CS_END_INNER, CS_PROBE_PLUS,
           CS_PROBE_END, CS_NM_DONE };
    int cs = CS_NONE, pk = PK_NONE, rep = 0, vert = -1, shr = -1;
    icount++;
    switch (phase) {
      case PH_INIT_BASE:
        F(N) = y;
        vert = 0;
        break;
      case PH_INIT_VERT:
        F(jj) = y;
        if (jj + 1 < N) vert = jj + 1;
        else cs = CS_READY;
        break;
      case PH_REFLECT:
        fr = y;
        if (P::lt(fr, ylo)) {
          pk = PK_EXPAND;
          phase = PH_EXPAND;
        } else {
          int worse = 0;
#pragma unroll 1
          for (int j = 0; j <= N; j++)
            if (P::lt(fr, F(j))) worse++;
          if (worse > 1) {
            rep = 1;
          } else if (worse == 0) {
            pk = PK_CONTRACT_IN;
            phase = PH_CONTRACT_IN;
          } else {
            pk = PK_CONTRACT_OUT;
            phase = PH_CONTRACT_OUT;
          }
        }
        break;
      case PH_EXPAND:
        rep = P::lt(fr, y) ? 1 : 2;
        break;
      case PH_CONTRACT_IN:
        // shrink every vertex towards the best (model/asa047.c:331-351)
        if (P::lt(F(hi), y)) shr = 0;
        else rep = 2;
        break;
      case PH_SHRINK:
        F(jj) = y;
        if (jj < N) shr = jj + 1;
        else cs = CS_READY;
        break;
      case PH_CONTRACT_OUT:
        rep = P::le(y, fr) ? 2 : 1;
        break;
      case PH_PROBE_PLUS:
      case PH_PROBE_MINUS:
        if (P::trunc10(y) < floor_lo) {
          ifault = 2;
          cs = CS_PROBE_END;
        } else {
          const T del = P::eps_step(step(jj));
          T v = x(jj);
          if (phase == PH_PROBE_PLUS) {
            v = P::sub(P::sub(v, del), del);
            phase = PH_PROBE_MINUS;
          } else {
            v = P::add(v, del);  // back to the centre
            cs = jj + 1 < N ? CS_PROBE_PLUS : CS_PROBE_END;
          }
          x(jj) = v;
          if (cs != CS_NONE) jj++;
        }
        break;
      default:
        icount--;
        break;
    }
    // Vertex `vert`: the start moved by step * scale along its coordinate
    // (model/asa047.c:181-194); `shr`: the vertex half way to the best;
    // `rep`: the worst replaced by the reflection (1) or by x (2).
    if (vert >= 0 || shr >= 0 || rep) {
      const int at = rep ? hi : (vert >= 0 ? vert : shr);
#pragma unroll 1
      for (int i = 0; i < N; i++) {
        T s;
        if (rep) {
          s = rep == 1 ? refl(i) : x(i);
        } else if (vert >= 0) {
          s = V(N, i);
          if (i == vert) s = P::add(s, P::mul(step(i), scale));
          x(i) = s;
        } else {
          s = P::half(P::add(V(shr, i), V(lo, i)));
          x(i) = s;
        }
        V(at, i) = s;
      }
      if (rep) {
        F(hi) = rep == 1 ? fr : y;
        cs = CS_ITER_END;
      } else {
        jj = at;
        phase = vert >= 0 ? PH_INIT_VERT : PH_SHRINK;
      }
    }
    // The transitions between the stages only go forward.
    if (cs == CS_READY) {
      ylo = F(0);
      lo = 0;
#pragma unroll 1
      for (int j = 1; j <= N; j++) {
        const T fj = F(j);
        if (P::lt(fj, ylo)) {
          ylo = fj;
          lo = j;
        }
      }
      cs = CS_TOP;
    }
    if (cs == CS_ITER_END) cs = iteration_end() ? CS_END_INNER : CS_TOP;
    if (cs == CS_TOP) {
      if (inner_top()) {
        pk = PK_REFL;
        cs = CS_NONE;
      } else {
        cs = CS_END_INNER;
      }
    }
    // The pending point cen + c (a - b), the same expression for every kind
    // (photic_nm.cuh).
    if (pk != PK_NONE) {
      const float c = pk == PK_EXPAND ? 2.0f : (pk == PK_REFL ? 1.0f : 0.5f);
#pragma unroll 1
      for (int i = 0; i < N; i++) {
        const T ce = cen(i);
        const T a = pk == PK_REFL ? ce : (pk == PK_CONTRACT_IN ? V(hi, i) : refl(i));
        const T b = pk == PK_REFL ? V(hi, i) : ce;
        const T p = P::add_scaled2(ce, P::sub(a, b), c);
        x(i) = p;
        if (pk == PK_REFL) refl(i) = p;
      }
    }
    if (cs == CS_END_INNER) {
#pragma unroll 1
      for (int i = 0; i < N; i++) x(i) = V(lo, i);
      floor_lo = P::trunc10(F(lo));
      ifault = kcount < icount ? 2 : 0;
      jj = 0;
      cs = ifault ? CS_NM_DONE : CS_PROBE_PLUS;
    }
    if (cs == CS_PROBE_PLUS) {
      x(jj) = P::add(x(jj), P::eps_step(step(jj)));
      phase = PH_PROBE_PLUS;
    }
    if (cs == CS_PROBE_END) {
      if (ifault == 0) {
        cs = CS_NM_DONE;
      } else {
        // restart from the probe point with a 1e-6 simplex
        scale = P::eps_scale();
        numres++;
        restart_simplex();
      }
    }
    return cs == CS_NM_DONE;
  }
};

}  // namespace photic
