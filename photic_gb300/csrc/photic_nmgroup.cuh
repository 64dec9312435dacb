// photic_nmgroup.cuh -- Nelder-Mead (model/asa047.c:10-502) for a group of
// G lanes sharing one pixel: the resumable state machine of photic_nm.cuh
// with the coordinate loops cut to each lane's own coordinates.  Lane l owns
// coordinate l (and l + G, ... up to C slots) of every vertex, the centroid
// and the trial points; the vertex costs and every decision taken on them
// are replicated in all lanes of the group, each lane keeping its own copy
// of the costs -- or, with kSharedF, one copy for the group, which every
// write reaches between two barriers of the group's lanes.  The simplex size is a
// template constant (NT > 0) or set at run time (NT = 0, member nrt), for
// pixels whose parameter count varies.
#pragma once
#include <stdint.h>

#include "photic_fp64.cuh"
#include "photic_nm.cuh"

namespace photic {

// Group-distributed Nelder-Mead: the state machine of NmLane with the
// coordinate loops cut to the lane's own coordinates.
template <int NT, int C, int G, int CG, bool kSharedF = false>
struct NmGroup {
  int nrt;             // the simplex size when NT <= 0 (set before begin)
  double *V, *Fv, *X;  // shared: V[j * CG + i], this lane's costs Fv[j * G] (or the
                       // group's Fv[j] with kSharedF), X[i]
  int gl;              // lane within the group
  unsigned gmask;      // the group's lanes
  double cen[C], refl[C], trial[C], xmin[C], start[C], step[C];
  double ylo, fr, scale, var_limit;
  // 1 / n as hi + lo for the centroid's division, RN(1 / (n + 1)) for the
  // variance test's
  double inv_n, inv_n_lo, inv_n1;
  long long floor_lo;
  int32_t phase, jj, hi, lo, icount, numres, ifault, countdown, kcount, konvge;
  // The centroid sums every coordinate over the vertices in order, and an
  // iteration changes one vertex: ck holds the sums before vertices kCkStep,
  // 2 kCkStep, ..., the first ck_valid of them up to date, so that the sum
  // resumes at the changed vertex's block instead of at vertex 0 (the same
  // additions in the same order; half of them on average).
  static constexpr int kCkStep = 8;
  static constexpr int kCk = ((NT > 0 ? NT : C * G) + kCkStep) / kCkStep;
  double ck[C][kCk];
  int32_t ck_valid;

  static __device__ __forceinline__ bool lt(double a, double b) {
    return NT > 0 ? sf::lt_call(a, b) : sf::lt(a, b);
  }
  static __device__ __forceinline__ bool le(double a, double b) {
    return NT > 0 ? sf::le_call(a, b) : sf::le(a, b);
  }
  __device__ __forceinline__ int dim() const { return NT > 0 ? NT : nrt; }
  __device__ __forceinline__ int coord(int t) const { return gl + t * G; }
  __device__ __forceinline__ bool own(int t) const { return coord(t) < dim(); }
  // Whether slot t holds a coordinate on any lane, and the coordinate that a
  // lane reads for it (a lane without one reads its group's first).
  __device__ __forceinline__ bool slot_used(int t) const { return t == 0 || t * G < dim(); }
  __device__ __forceinline__ int column(int t) const { return own(t) ? coord(t) : t * G; }
  // The slot holding coordinate i on this lane, -1 if another lane owns it.
  // (Matching i against coord(t) slot by slot instead lost the match on
  // the second slot in the compiled kernel: the stepped vertex of the last
  // coordinate came out unstepped.)
  __device__ __forceinline__ int slot_of(int i) const { return (i % G) == gl ? i / G : -1; }
  __device__ __forceinline__ double &Vv(int j, int i) { return V[j * CG + i]; }
  __device__ __forceinline__ double &F(int j) { return Fv[kSharedF ? j : j * G]; }
  // A cost write.  With one copy for the warp, every lane has made the
  // step's reads before any lane writes, and sees the write after it:
  // the lanes take the same decisions, so they all reach both barriers.
  __device__ __forceinline__ void setF(int j, double y) {
    if constexpr (kSharedF) {
#if defined(__CUDA_ARCH__)
      __syncwarp(gmask);
#endif
      Fv[j] = y;
#if defined(__CUDA_ARCH__)
      __syncwarp(gmask);
#endif
    } else {
      Fv[j * G] = y;
    }
  }

  // Every slot gets a defined value, also those of coordinates the lane
  // does not own (they are computed on but never stored).
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int t = 0; t < C; t++) {
      cen[t] = 0.0;
      refl[t] = 0.0;
      trial[t] = 0.0;
      xmin[t] = 0.0;
      start[t] = 0.0;
      step[t] = 0.0;
    }
    ylo = fr = 0.0;
    inv_n = inv_n1 = 1.0;
    inv_n_lo = 0.0;
    scale = 1.0;
    floor_lo = 0;
    phase = jj = hi = lo = icount = numres = ifault = countdown = ck_valid = 0;
  }

  __device__ __forceinline__ void begin(double var_limit_, int32_t konvge_, int32_t kcount_) {
    konvge = konvge_;
    kcount = kcount_;
    countdown = konvge_;
    icount = 0;
    numres = 0;
    ifault = 0;
    scale = 1.0;
    var_limit = var_limit_;
    inv_n = 1.0 / (double)dim();
    inv_n_lo = fm::recip_lo((double)dim(), inv_n);
    inv_n1 = 1.0 / (double)(dim() + 1);
    restart_simplex();
  }

  __device__ __forceinline__ void restart_simplex() {
#pragma unroll
    for (int t = 0; t < C; t++)
      if (own(t)) {
        X[coord(t)] = start[t];
        Vv(dim(), coord(t)) = start[t];
      }
    ck_valid = 0;
    phase = PH_INIT_BASE;
  }

  __device__ __forceinline__ void make_vertex(int j) {
    const int ts = slot_of(j);
#pragma unroll
    for (int t = 0; t < C; t++)
      if (own(t)) {
        const int i = coord(t);
        double s = start[t];
        if (t == ts) s = start[t] + step[t] * scale;
        X[i] = s;
        Vv(j, i) = s;
      }
    jj = j;
    phase = PH_INIT_VERT;
  }

  __device__ __forceinline__ void find_lo() {
    ylo = F(0);
    lo = 0;
#pragma unroll 1
    for (int j = 1; j <= dim(); j++) {
      const double fj = F(j);
      if (lt(fj, ylo)) {
        ylo = fj;
        lo = j;
      }
    }
  }

  // The worst vertex: the first index of the largest cost, a NaN cost
  // never replacing the running one (a NaN at index 0 is kept, model/
  // asa047.c:221-231).  With one cost copy for the warp, each lane scans
  // the vertices j = lane, lane + 32, ..., and the warp reduces the costs'
  // order keys, then the indices that have the largest.
  __device__ __forceinline__ int worst_vertex() {
    if constexpr (kSharedF) {
#if defined(__CUDA_ARCH__)
      if (sf::order_key(F(0)) == 0) return 0;
      uint64_t v = 0;
      int idx = 0x7fffffff;
#pragma unroll 1
      for (int j = gl; j <= dim(); j += G) {
        const uint64_t f = sf::order_key(F(j));
        if (f > v) {
          v = f;
          idx = j;
        }
      }
      const uint32_t h = __reduce_max_sync(gmask, (uint32_t)(v >> 32));
      const uint32_t l = __reduce_max_sync(gmask, (uint32_t)(v >> 32) == h ? (uint32_t)v : 0u);
      if (v != ((uint64_t)h << 32 | l)) idx = 0x7fffffff;
      idx = __reduce_min_sync(gmask, idx);
      return idx;
#endif
    }
    double yhi = F(0);
    int h = 0;
#pragma unroll 1
    for (int j = 1; j <= dim(); j++) {
      const double fj = F(j);
      if (lt(yhi, fj)) {
        yhi = fj;
        h = j;
      }
    }
    return h;
  }

  // How many vertices cost more than fr (model/asa047.c:294-301): a count,
  // so with one cost copy the lanes count their vertices and the warp adds.
  __device__ __forceinline__ int count_worse(double fr_) {
    if constexpr (kSharedF) {
#if defined(__CUDA_ARCH__)
      int c = 0;
      const uint64_t kf = sf::order_key(fr_);
#pragma unroll 1
      for (int j = gl; j <= dim(); j += G)
        if (kf != 0 && kf < sf::order_key(F(j))) c++;
      return (int)__reduce_add_sync(gmask, (unsigned)c);
#endif
    }
    int worse = 0;
#pragma unroll 1
    for (int j = 0; j <= dim(); j++)
      if (lt(fr_, F(j))) worse++;
    return worse;
  }

  __device__ __forceinline__ bool inner_top() {
    if (kcount <= icount) return false;
    hi = worst_vertex();
    double z[C];
    int m = ck_valid;
#pragma unroll
    for (int t = 0; t < C; t++) z[t] = m > 0 ? ck[t][m - 1] : 0.0;
    int j = m * kCkStep;
#pragma unroll 1
    for (; j + kCkStep <= dim() + 1; j += kCkStep, m++) {
#pragma unroll
      for (int t = 0; t < C; t++)
        if (slot_used(t)) {
#pragma unroll
          for (int i = 0; i < kCkStep; i++) z[t] = z[t] + Vv(j + i, column(t));
          ck[t][m] = z[t];
        }
    }
    ck_valid = m;
#pragma unroll 1
    for (; j <= dim(); j++) {
#pragma unroll
      for (int t = 0; t < C; t++)
        if (slot_used(t)) z[t] = z[t] + Vv(j, column(t));
    }
#pragma unroll
    for (int t = 0; t < C; t++)
      if (slot_used(t)) {
        z[t] = z[t] - Vv(hi, column(t));
        cen[t] = fm::div_const(z[t], (double)dim(), inv_n, inv_n_lo);
      }
    phase = PH_REFLECT;
    return true;
  }

  // Each lane keeps its own copy of the vertex costs (the same values in
  // every lane of the group), so no lane ever reads a cost another lane is
  // writing, whatever the lanes' relative progress; or one shared copy
  // written between barriers (setF).
  __device__ __forceinline__ void replace_hi(bool reflection, double y) {
#pragma unroll
    for (int t = 0; t < C; t++)
      if (own(t)) Vv(hi, coord(t)) = reflection ? refl[t] : trial[t];
    if (hi / kCkStep < ck_valid) ck_valid = hi / kCkStep;
    setF(hi, y);
  }

  // The pending point of the iteration, cen + c (a - b) (photic_nm.cuh): the
  // reflection, the expansion or a contraction, written once.
  __device__ __forceinline__ void make_point(int pk) {
    const float c = pk == PK_EXPAND ? 2.0f : (pk == PK_REFL ? 1.0f : 0.5f);
#pragma unroll
    for (int t = 0; t < C; t++)
      if (slot_used(t)) {
        const double w = Vv(hi, column(t));
        const double a = pk == PK_REFL ? cen[t] : (pk == PK_CONTRACT_IN ? w : refl[t]);
        const double b = pk == PK_REFL ? w : cen[t];
        const double p = sf::add_scaled2(cen[t], a - b, c);
        if (pk == PK_REFL) refl[t] = p;
        else trial[t] = p;
        if (own(t)) X[coord(t)] = p;
      }
  }

  __device__ __forceinline__ bool iteration_end() {
    const double fh = F(hi);
    if (lt(fh, ylo)) {
      ylo = fh;
      lo = hi;
    }
    countdown--;
    if (countdown > 0) return false;
    if (icount <= kcount) {
      countdown = konvge;
      double z = 0.0;
#pragma unroll 1
      for (int j = 0; j <= dim(); j++) z = z + F(j);
      const double mean = fm::div_by(z, (double)(dim() + 1), inv_n1);
      z = 0.0;
#pragma unroll 1
      for (int j = 0; j <= dim(); j++) {
        const double d = F(j) - mean;
        z = z + d * d;
      }
      if (le(z, var_limit)) return true;
    }
    return false;
  }

  __device__ __forceinline__ void set_x_from(const double (&p)[C]) {
#pragma unroll
    for (int t = 0; t < C; t++)
      if (own(t)) X[coord(t)] = p[t];
  }

  // xmin[jj] += sgn * del on the lane that owns coordinate jj.
  __device__ __forceinline__ void probe_move(int sgn_twice) {
    const int ts = slot_of(jj);
#pragma unroll
    for (int t = 0; t < C; t++)
      if (t == ts) {
        const double del = step[t] * 1.0e-6;
        if (sgn_twice > 0) xmin[t] = xmin[t] + del;
        else if (sgn_twice < 0) xmin[t] = (xmin[t] - del) - del;
        else xmin[t] = xmin[t] + del;  // back to the centre after the minus probe
      }
  }

  // Consume the cost y of the point at X and stage the next one.  Returns
  // true when the nelmin call has returned.  As in photic_nm.cuh the switch
  // only decides; what it decides on (a vertex replaced, a vertex shrunk, the
  // next point) is written once below it, and the transitions between the
  // stages only go forward.
  __device__ __forceinline__ bool step_machine(double y) {
    enum { CS_NONE = -1, CS_READY, CS_TOP, CS_ITER_END, CS_END_INNER, CS_PROBE_PLUS,
           CS_PROBE_END, CS_NM_DONE };
    int cs = CS_NONE, pk = PK_NONE, rep = 0, vert = -1, shr = -1;
    icount++;
    switch (phase) {
      case PH_INIT_BASE:
        setF(dim(), y);
        vert = 0;
        break;
      case PH_INIT_VERT:
        setF(jj, y);
        if (jj + 1 < dim()) vert = jj + 1;
        else cs = CS_READY;
        break;
      case PH_REFLECT:
        fr = y;
        if (lt(fr, ylo)) {
          pk = PK_EXPAND;
          phase = PH_EXPAND;
        } else {
          const int worse = count_worse(fr);
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
        rep = lt(fr, y) ? 1 : 2;
        break;
      case PH_CONTRACT_IN:
        // shrink every vertex towards the best (model/asa047.c:331-351)
        if (lt(F(hi), y)) shr = 0;
        else rep = 2;
        break;
      case PH_SHRINK:
        setF(jj, y);
        if (jj < dim()) shr = jj + 1;
        else cs = CS_READY;
        break;
      case PH_CONTRACT_OUT:
        rep = le(y, fr) ? 2 : 1;
        break;
      case PH_PROBE_PLUS:
      case PH_PROBE_MINUS:
        if (trunc10(y) < floor_lo) {
          ifault = 2;
          cs = CS_PROBE_END;
        } else if (phase == PH_PROBE_PLUS) {
          probe_move(-1);
          set_x_from(xmin);
          phase = PH_PROBE_MINUS;
        } else {
          probe_move(0);
          jj++;
          cs = (jj < dim()) ? CS_PROBE_PLUS : CS_PROBE_END;
        }
        break;
      default:
        icount--;
        break;
    }
    if (vert >= 0) make_vertex(vert);
    if (shr >= 0) {
#pragma unroll
      for (int t = 0; t < C; t++)
        if (own(t)) {
          const int i = coord(t);
          const double s = (Vv(shr, i) + Vv(lo, i)) * 0.5;
          Vv(shr, i) = s;
          X[i] = s;
        }
      ck_valid = 0;
      jj = shr;
      phase = PH_SHRINK;
    }
    if (rep) {
      replace_hi(rep == 1, rep == 1 ? fr : y);
      cs = CS_ITER_END;
    }
    if (cs == CS_READY) {
      find_lo();
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
    if (pk != PK_NONE) make_point(pk);
    if (cs == CS_END_INNER) {
#pragma unroll
      for (int t = 0; t < C; t++)
        if (own(t)) xmin[t] = Vv(lo, coord(t));
      floor_lo = trunc10(F(lo));
      if (kcount < icount) {
        ifault = 2;
        cs = CS_NM_DONE;
      } else {
        ifault = 0;
        jj = 0;
        cs = CS_PROBE_PLUS;
      }
    }
    if (cs == CS_PROBE_PLUS) {
      probe_move(+1);
      set_x_from(xmin);
      phase = PH_PROBE_PLUS;
    }
    if (cs == CS_PROBE_END) {
      if (ifault == 0) {
        cs = CS_NM_DONE;
      } else {
#pragma unroll
        for (int t = 0; t < C; t++) start[t] = xmin[t];
        scale = 1.0e-6;
        numres++;
        restart_simplex();
      }
    }
    return cs == CS_NM_DONE;
  }
};

}  // namespace photic
