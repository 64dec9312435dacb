// photic_invert.cu -- persistent, work-queue batched inversion of
// single-scene pixels (the plain method).
//
// One lane owns one pixel at a time and runs the whole per-pixel driver of
// samodel_optimise (model/samodel.c:1768-2115) with its cold depth starts
// and early exit (model/samodel.c:2243-2407) on the resumable Nelder-Mead
// of photic_nm.cuh.  Every loop trip all lanes that hold a pixel evaluate
// the cost together; when a lane's pixel is finished it takes the next one
// from its warp's chunk, and a warp whose chunk is used up claims the next
// 32 pixels with one atomic and stages their spectra through shared memory
// with coalesced (float4 when the layout allows) loads.  Ragged iteration
// counts (a few hundred to several thousand evaluations per pixel) thus
// never leave a lane idle while work remains.  A pixel's depth starts are
// positions of the queue of their own while the scene is small enough to
// keep their results (see invert_kernel): a launch then ends with single
// starts of at most kcount evaluations instead of with pixels of eight.
//
// The arithmetic is a policy: PrecF64 (IEEE double, reference operation
// order, --fmad=false), PrecF32 (the forward model in float with the
// special-function unit, the simplex in double) or PrecDF (double-float on
// the FP32 pipes).
//
// Scratch: one 64-bit queue head per call (stream-ordered allocation in
// photic_host.cu) and the per-device sticky error word.
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "photic_dfcost.cuh"
#include "photic_fp64.cuh"
#include "photic_kernels.h"
#include "photic_nm.cuh"
#include "photic_nmgroup.cuh"
#include "photic_prec64.cuh"
#include "photic_starts.cuh"

namespace photic {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kN = 6;  // H, 100B, q, 100P, 100G, 100X

// ---------------------------------------------------------------------------
// Precision policies (PrecF64 is in photic_prec64.cuh)
// ---------------------------------------------------------------------------
// Single-precision forward model (FP32 with the special-function unit):
// the cost of a double parameter vector evaluated in float with the
// special-function unit's exp and log and approximate divisions, returned as
// a double; the simplex, its decisions, the convergence and local-minimum
// tests and the final re-evaluation at the kept optimum stay in FP64.
template <int NB>
struct PixelF32 {
  PixelF64<NB> d;        // the double set-up (cold starts, details)
  float rrs[NB], pw[NB];
  float mean;
};

struct PrecF32 : PrecF64 {
  static constexpr bool kFused = false;  // its products come from an FP64 evaluation
  template <int NB>
  using Pixel = PixelF32<NB>;
  template <int NB>
  static __device__ __forceinline__ void setup(const InvertArgs &a, const float *r, Pixel<NB> &px) {
    PrecF64::setup<NB>(a, r, px.d);
#pragma unroll
    for (int b = 0; b < NB; b++) {
      px.rrs[b] = (float)px.d.rrs[b];
      px.pw[b] = (float)px.d.pw[b];
    }
    px.mean = (float)px.d.mean;
  }
  template <int NB>
  static __device__ __forceinline__ void cold_start(const InvertArgs &a, const Pixel<NB> &px,
                                                    T *start, T *step) {
    cold_start_f64<NB>(a.fp, px.d, start, step);
  }
  // samodel_error (model/samodel.c:2432-2759) over samodel_Rrs (:2846-2949)
  // for one region, scene and bottom type, in float
  template <int NB>
  static __device__ __forceinline__ T cost(const InvertArgs &a, const Pixel<NB> &px, const T *x) {
    const FitParams &fp = a.fp;
    const SceneConsts &sc = a.sc;
    const int nb = fp.n_bands;
    const float H = fabsf((float)x[0]);
    const float B = 0.01f * fabsf((float)x[1]);
    const float qa = fabsf((float)x[2]);
    const float q = qa / qa;
    const float P = 0.01f * fabsf((float)x[3]);
    const float G = 0.01f * fabsf((float)x[4]);
    const float X = 0.01f * fabsf((float)x[5]);
    const float lnP = __logf(P);
    const float qB = q * B;
    const float ss = (float)sc.sec_sun, sv = (float)sc.sec_view;
    float err = 0.0f, K_min = 1.0e4f;
#pragma unroll
    for (int b = 0; b < NB; b++) {
      if (b < nb) {
        const float rho = qB * (float)sc.refl[b];
        const float a_phi = ((float)sc.a0[b] + (float)sc.a1[b] * lnP) * P;
        const float a_g = G * (float)sc.eS[b];
        const float aa = (float)sc.aw[b] + a_phi + a_g;
        const float bb = (float)sc.bbw[b] + X * px.pw[b];
        const float u = __fdividef(bb, aa + bb);
        float K = aa + bb;
        K = fminf(fmaxf(K, 0.0f), 2.5f);
        const float rrs_dp = (0.084f + 0.170f * u) * u;
        const float DuC = 1.03f * sqrtf(1.0f + 2.4f * u);
        const float DuB = 1.04f * sqrtf(1.0f + 5.4f * u);
        const float rrs_C = rrs_dp * (1.0f - __expf(-(ss + DuC * sv) * K * H));
        const float rrs_B = rho * 0.31830988618f * __expf(-(ss + DuB * sv) * K * H);
        const float rrs = rrs_C + rrs_B;
        const float Rm = __fdividef(0.5f * rrs, 1.0f - 1.5f * rrs);
        const float d = Rm - px.rrs[b];
        err += d * d;
        if (K != 0.0f && K < K_min) K_min = K;
      }
    }
    const float E = __fdividef(100.0f * sqrtf(err / (float)nb), px.mean);
    float Ke = 0.0f;
    int c = -1;
    const KPenalty &kp = fp.kp;
    if (H < 1.0f && K_min < (float)kp.k_thr[0]) c = 0;
    else if (H < 2.0f && K_min < (float)kp.k_thr[1]) c = 1;
    else if (H < 3.0f && K_min < (float)kp.k_thr[2]) c = 2;
    else if (H < 4.0f && K_min < (float)kp.k_thr[3]) c = 3;
    else if (H < 5.0f && K_min < (float)kp.k_thr[4]) c = 4;
    if (c >= 0) {
      float it = (float)kp.inv_t[0];
      for (int i = 1; i < 5; i++)
        if (i == c) it = (float)kp.inv_t[i];
      const float d = __fdividef(1.0f, 0.01f + K_min) - it;
      Ke = 100.0f * d * d;
    }
    if (K_min > 0.7f) {
      const float d = 4.0f * (K_min - 0.7f);
      Ke += 100.0f * d * d;
    }
    return (double)((80.0f * E + 15.0f * Ke) * (1.0f / 120.0f));
  }
  template <int NB>
  static __device__ __forceinline__ void details(const InvertArgs &a, const Pixel<NB> &px,
                                                 const T *x, Details &d) {
    PrecF64::details<NB>(a, px.d, x, d);
  }
};

struct PrecDF {
  static constexpr bool kFused = false;
  using T = df64;
  template <int NB>
  using Pixel = PixelDF<NB>;
  struct Details {
    double rrs_error, model_error, bottom_albedo, K_min, iod;
  };
  static __device__ __forceinline__ T zero() { return df64{0.0f, 0.0f}; }
  static __device__ __forceinline__ T one() { return df64{1.0f, 0.0f}; }
  static __device__ __forceinline__ T add(T a, T b) { return df_add(a, b); }
  static __device__ __forceinline__ T sub(T a, T b) { return df_sub(a, b); }
  static __device__ __forceinline__ T mul(T a, T b) { return df_mul(a, b); }
  static __device__ __forceinline__ T mul2(T a) { return df64{2.0f * a.hi, 2.0f * a.lo}; }
  static __device__ __forceinline__ T half(T a) { return df64{0.5f * a.hi, 0.5f * a.lo}; }
  static __device__ __forceinline__ T scale2(T a, float c) { return df64{c * a.hi, c * a.lo}; }
  static __device__ __forceinline__ T add_scaled2(T a, T b, float c) { return add(a, scale2(b, c)); }
  static __device__ __forceinline__ bool sum_less_one(const T *, int, int, int, T &) { return false; }
  static __device__ __forceinline__ T div_n(T a, int n) { return df_div_f(a, (float)n); }
  static __device__ __forceinline__ bool lt(T a, T b) { return df_lt(a, b); }
  static __device__ __forceinline__ bool le(T a, T b) { return df_le(a, b); }
  static __device__ __forceinline__ T eps_step(T s) { return df_mul(s, DFK(1.0e-6)); }
  static __device__ __forceinline__ T eps_scale() { return DFK(1.0e-6); }
  static __device__ __forceinline__ long long trunc10(T y) { return df_trunc10(y); }
  static __device__ __forceinline__ T from_double(double d) { return df_from_double(d); }
  static __device__ __forceinline__ double to_double(T a) { return df_to_double(a); }
  static __device__ __forceinline__ T var_limit(const InvertArgs &a) { return dp(a.ds.reqmin_n); }
  static __device__ __forceinline__ T hstart(const InvertArgs &a, int k) {
    return dp(a.ds.hstarts[k]);
  }
  static __device__ __forceinline__ T h_step(T h) { return df_mul_f(h, 1.25f); }
  template <int NB>
  static __device__ __forceinline__ void setup(const InvertArgs &a, const float *r, Pixel<NB> &px) {
    pixel_setup_df<NB>(a.fp, a.ds, r, px);
  }
  template <int NB>
  static __device__ __forceinline__ void cold_start(const InvertArgs &a, const Pixel<NB> &px,
                                                    T *start, T *step) {
    cold_start_df<NB>(a.fp, a.ds, px, start, step);
  }
  template <int NB>
  static __device__ __forceinline__ T cost(const InvertArgs &a, const Pixel<NB> &px, const T *x) {
    return cost_df<false, NB>(a.fp, a.ds, px, x, nullptr);
  }
  template <int NB>
  static __device__ __forceinline__ void details(const InvertArgs &a, const Pixel<NB> &px,
                                                 const T *x, Details &d) {
    CostDetailsDF det;
    cost_df<true, NB>(a.fp, a.ds, px, x, &det);
    d.rrs_error = df_to_double(det.rrs_error);
    d.model_error = df_to_double(det.model_error);
    d.bottom_albedo = df_to_double(det.bottom_albedo);
    d.K_min = df_to_double(det.K_min);
    d.iod = df_to_double(det.iod);
  }
};

// One start's nelmin result, kept until the pixel's starts are compared.
template <class P>
struct StartRecord {
  typename P::T y;
  int32_t evals;  // -1: the start hit the defensive evaluation cap
  int32_t fault;
  typename P::T x[kN];
};

template <class P, int NB>
__device__ __forceinline__ void write_fit(const photic_outputs &o, int64_t p,
                                          const typename P::T *x,
                                          const typename P::Details &det, int32_t total,
                                          int32_t kept_evals, int32_t kept_start,
                                          int32_t kept_fault) {
  const double H = fabs(P::to_double(x[0]));
  if (o.depth) o.depth[p] = (float)H;
  if (o.depth_f64) o.depth_f64[p] = H;
  if (o.P) o.P[p] = (float)(0.01 * fabs(P::to_double(x[3])));
  if (o.G) o.G[p] = (float)(0.01 * fabs(P::to_double(x[4])));
  if (o.X) o.X[p] = (float)(0.01 * fabs(P::to_double(x[5])));
  if (o.bottom_albedo) o.bottom_albedo[p] = (float)det.bottom_albedo;
  if (o.model_error) o.model_error[p] = (float)det.model_error;
  if (o.rrs_error) o.rrs_error[p] = (float)det.rrs_error;
  if (o.K_min) o.K_min[p] = (float)det.K_min;
  if (o.iod) o.iod[p] = (float)det.iod;
  if (o.evals) o.evals[p] = total;
  if (o.evals_kept) o.evals_kept[p] = kept_evals;
  if (o.params)
    for (int i = 0; i < kN; i++) o.params[p * kN + i] = P::to_double(x[i]);
  if (o.status)
    o.status[p] = PHOTIC_PX_FITTED | (kept_fault == 0 ? PHOTIC_PX_CONVERGED : 0) |
                  (kept_start << 16);
}

__device__ __forceinline__ int64_t pixel_at(const InvertArgs &args, int64_t q) {
  return args.order ? (int64_t)args.order[q] : args.pixels ? args.pixels[q] : q;
}

// What the lookup-table loop reports of the pixel at position q.
__device__ __forceinline__ void write_single_chain(const InvertArgs &args, int64_t q, int64_t p,
                                                   double model_error) {
  if (args.source) args.source[p] = -1;
  if (args.chain_stats) single_chain_stats(args.chain_stats + q * 4, 1.5, model_error);
}

// A pixel that ended invalid: no fit, and in the loop a chain that moved no
// threshold.
__device__ __forceinline__ void write_invalid(const InvertArgs &args, int64_t q, int64_t p) {
  if (args.out.status) args.out.status[p] = PHOTIC_PX_INVALID;
  if (args.pixels && args.chain_stats) {
    double *const cs = args.chain_stats + q * 4;
    cs[0] = cs[1] = 0.0;
    cs[2] = cs[3] = 1.5;
  }
}

template <int NB>
__device__ __forceinline__ void load_spectrum(const InvertArgs &args, int64_t p, float (&r)[NB]) {
  if (NB == 4 && args.vec4) {
    const float4 v4 = __ldg(reinterpret_cast<const float4 *>(args.rrs) + p);
    r[0] = v4.x;
    r[1] = v4.y;
    r[2] = v4.z;
    r[3] = v4.w;
  } else {
#pragma unroll
    for (int b = 0; b < NB; b++)
      r[b] = b < args.fp.n_bands ? __ldg(args.rrs + p * args.pixel_stride + b * args.band_stride)
                                 : 0.0f;
  }
}

// The end of a launch.  Starts run for 100 to 2 000 evaluations, so once the
// queue is empty warps thin out, and a warp with one start left takes as long
// a trip as a full one.  A warp therefore first takes up starts that others
// have handed on, and one that still has no more than args.give hands on its
// own and ends; when no more than args.few_left are left in all, every warp
// does, and groups of lanes finish them (invert_few_kernel).  Nothing waits:
// a warp takes the next records in order that are ready, or none.  1024 x 320
// pixels 307 -> 299 ms, 20 011 of eight bands 112 -> 83, a 701 x 997 tile of
// seeds 278 -> 264; four lookup-table loops over 509 x 400, whose rarest
// starts take 5 000 evaluations, 115 to 153 ms -> 111 to 146.
// counted: the warp's starts in LeftStarts::live, -1 before its first call.
// true: the warp ends.
template <int BS, class Px>
__device__ __forceinline__ bool hand_on(const InvertArgs &args, NmPixel<PrecF64, BS> &m, Px &px,
                                        int lane, double var_limit, bool &has, int64_t &item,
                                        int32_t &start_k, int32_t &guard, int &counted) {
  using Nm = NmPixel<PrecF64, BS>;
  constexpr int kPx = 2 * (int)(sizeof px.rrs / sizeof(double)) + 1;
  LeftStarts &q = *args.left;
  unsigned char *const mem = reinterpret_cast<unsigned char *>(args.left);
  int32_t *const ready = reinterpret_cast<int32_t *>(mem + left_ready_offset());
  LeftStart *const rec = reinterpret_cast<LeftStart *>(mem + left_record_offset(args.left_slots));
  double *const mine = reinterpret_cast<double *>(&px);

  int n = __popc(__ballot_sync(kFull, has));
  unsigned head = 0;
  bool few = false;
  if (lane == 0) {
    if (counted < 0) {
      atomicAdd(&q.live, n);
      __threadfence();
      atomicAdd(&q.warps_out, 1);
    } else if (n != counted) {
      atomicSub(&q.live, counted - n);
    }
    few = __ldcg(&q.warps_out) == (int)(gridDim.x * (BS / 32)) && __ldcg(&q.live) <= args.few_left;
    head = __ldcg(&q.taken);
  }
  head = __shfl_sync(kFull, head, 0);
  few = __shfl_sync(kFull, few, 0);

  if (n < 32 && !few) {
    const unsigned at = head + lane;
    const bool full = at < (unsigned)args.left_slots && __ldcg(ready + at) != 0;
    const unsigned waiting = __ballot_sync(kFull, full);
    const int run = waiting == kFull ? 32 : __ffs(~waiting) - 1;
    const int k = run < 32 - n ? run : 32 - n;
    if (k > 0) {
      __threadfence();
      __syncwarp();  // another lane reads the record than saw its flag: votes order no memory
      bool won = false;
      if (lane == 0) won = atomicCAS(&q.taken, head, head + k) == head;
      won = __shfl_sync(kFull, won, 0);
      const unsigned idle = __ballot_sync(kFull, !has);
      const int rank = __popc(idle & ((1u << lane) - 1u));
      if (won && !has && rank < k) {
        const LeftStart &d = rec[head + rank];
#pragma unroll 1
        for (int i = 0; i < Nm::kSlots; i++) m.w[i * BS] = __ldcg(d.slots + i);
#pragma unroll
        for (int i = 0; i < kPx; i++) mine[i] = __ldcg(d.px + i);
        m.ylo = __ldcg(&d.ylo);
        m.fr = __ldcg(&d.fr);
        m.scale = __ldcg(&d.scale);
        m.floor_lo = __ldcg(&d.floor_lo);
        m.phase = __ldcg(&d.phase);
        m.jj = __ldcg(&d.jj);
        m.hi = __ldcg(&d.hi);
        m.lo = __ldcg(&d.lo);
        m.icount = __ldcg(&d.icount);
        m.numres = __ldcg(&d.numres);
        m.ifault = __ldcg(&d.ifault);
        m.countdown = __ldcg(&d.countdown);
        m.var_limit = var_limit;
        m.konvge = args.fp.konvge;
        m.kcount = args.fp.kcount;
        item = __ldcg(&d.item);
        start_k = __ldcg(&d.start_k);
        guard = __ldcg(&d.guard);
        has = true;
      }
      if (won) n += k;
    }
  }
  counted = n;

  // starts in sequence (item < 0) stay with their warp
  if ((n > args.give && !few) || __any_sync(kFull, has && item < 0)) return false;
  unsigned base = 0;
  if (lane == 0 && n > 0) base = atomicAdd(&q.given, (unsigned)n);
  base = __shfl_sync(kFull, base, 0);
  const unsigned busy = __ballot_sync(kFull, has);
  const unsigned at = base + __popc(busy & ((1u << lane) - 1u));
  if (has && at < (unsigned)args.left_slots) {
    LeftStart &d = rec[at];
#pragma unroll 1
    for (int i = 0; i < Nm::kSlots; i++) d.slots[i] = m.w[i * BS];
#pragma unroll
    for (int i = 0; i < kPx; i++) d.px[i] = mine[i];
    d.ylo = m.ylo;
    d.fr = m.fr;
    d.scale = m.scale;
    d.floor_lo = m.floor_lo;
    d.item = item;
    d.phase = m.phase;
    d.jj = m.jj;
    d.hi = m.hi;
    d.lo = m.lo;
    d.icount = m.icount;
    d.numres = m.numres;
    d.ifault = m.ifault;
    d.countdown = m.countdown;
    d.start_k = start_k;
    d.guard = guard;
    __threadfence();
    atomicExch(ready + at, 1);
  }
  return true;
}

// The queue's positions: the first n_seq are pixels, each lane running a
// pixel's starts one after the other; then, for the other n_par pixels, every
// start is a position of its own (start-major: the first starts of all these
// pixels, then the second starts, ...), its result goes to a record, and
// finish_kernel compares a pixel's records in the order of the starts.  The
// result is the sequential one: a start is left out once an earlier start of
// its pixel has met the early exit (exit_k), where the sequential loop would
// have ended at that start or before.  A launch lasts at least as long as its
// longest position, and a pixel whose starts all fail takes eight times a
// start: 256 pixels 131 -> 34 ms, 20 011 eight-band pixels 470 -> 124 ms, a
// 1024 x 320 scene 601 -> 443 ms, a 701 x 997 tile of seeds 382 -> 363 ms.
template <class P, int NB, int BS>
__global__ void __launch_bounds__(BS) invert_kernel(const __grid_constant__ InvertArgs args) {
  using T = typename P::T;
  const FitParams &fp = args.fp;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *snm = reinterpret_cast<T *>(smem_raw);          // [NmPixel's slots][BS]
  T *sbest = snm + NmPixel<P, BS>::kSlots * BS;      // [N][BS]
  using Px = typename P::template Pixel<NB>;
  Px *spx = reinterpret_cast<Px *>(sbest + kN * BS);  // [BS/32][32] set-ups of the chunk
  int64_t *spos = reinterpret_cast<int64_t *>(spx + BS);  // [BS/32][32] their positions

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  Px *wpx = spx + warp * 32;
  int64_t *wpos = spos + warp * 32;
  const unsigned lt_mask = (1u << lane) - 1u;
  StartRecord<P> *const rec = reinterpret_cast<StartRecord<P> *>(args.records);
  const int64_t total_pos = args.n_seq + args.n_par * fp.n_hstarts;

  NmPixel<P, BS> m;
  m.w = snm + tid;
  m.phase = PH_INIT_BASE;
  T *best = sbest + tid;
  Px px;
  const T var_limit = P::var_limit(args);
  const photic_outputs &o = args.out;

  int64_t pixel = -1, item = -1;  // item: pixel number within the n_par, or -1
  int64_t position = 0;
  int32_t start_k = 0, n_starts = 0, total = 0, kept_evals = 0, kept_start = 0, kept_fault = 0;
  int32_t guard = 0;
  T lowest = P::zero();

  bool has = false, open = true;
  int chunk_next = 0, chunk_end = 0, counted = -1;
  const int32_t guard_cap = (fp.n_hstarts + 1) * (fp.kcount + 8 * kN + 16);

  for (;;) {
    // ---- hand out positions to lanes that have none ----------------------
    unsigned need = __ballot_sync(kFull, !has && open);
    while (need) {
      if (chunk_next >= chunk_end) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(args.queue, (unsigned long long)args.claim);
        base = __shfl_sync(kFull, base, 0);
        if (base >= (unsigned long long)total_pos) {
          open = false;
          break;
        }
        __syncwarp();
        // Every lane looks at one position of the chunk: masked pixels are
        // written, starts that are not needed dropped, the others set up
        // (interpolated Rrs, Y and (440/lambda)^Y, model/samodel.c:1783-1799,
        // 2897-2902) with the whole warp, instead of each lane alone when it
        // takes the pixel.
        const int64_t w = (int64_t)base + lane;
        bool live = lane < args.claim && w < total_pos;
        int64_t p = 0;
        float r[NB];
        if (live) {
          int64_t q = w;
          int k = 0;
          if (w >= args.n_seq) {
            k = (int)((w - args.n_seq) / args.n_par);
            q = args.n_seq + (w - args.n_seq) % args.n_par;
          }
          p = pixel_at(args, q);
          if (k > 0)
            live = __ldcg(args.exit_k + (q - args.n_seq)) >= k &&
                   (args.seeds == nullptr || isnan(args.seeds[p * kN]));
          if (live) {
            load_spectrum<NB>(args, p, r);
            bool masked = false;
#pragma unroll
            for (int b = 0; b < NB; b++)
              if (b < fp.n_bands && !args.no_mask && band_masked(r[b], fp.nodata)) masked = true;
            if (masked) {
              live = false;
              if (k == 0) {
                write_masked(o, p);
                if (w >= args.n_seq) args.exit_k[q - args.n_seq] = -1;
              }
            }
          }
        }
        const unsigned alive = __ballot_sync(kFull, live);
        if (live) {
          const int slot = __popc(alive & lt_mask);
          P::template setup<NB>(args, r, wpx[slot]);
          wpos[slot] = w;
        }
        chunk_next = 0;
        chunk_end = __popc(alive);
        __syncwarp();
        if (chunk_end == 0) continue;
      }
      const int rank = __popc(need & lt_mask);
      const bool mine = ((need >> lane) & 1u) && rank < chunk_end - chunk_next;
      const unsigned taken = __ballot_sync(kFull, mine);
      if (mine) {
        const int slot = chunk_next + rank;
        const int64_t w = wpos[slot];
        int64_t q = w;
        start_k = 0;
        item = -1;
        if (w >= args.n_seq) {
          item = (w - args.n_seq) % args.n_par;
          start_k = (int32_t)((w - args.n_seq) / args.n_par);
          q = args.n_seq + item;
        }
        position = q;
        pixel = pixel_at(args, q);
        px = wpx[slot];
        total = kept_evals = kept_start = kept_fault = guard = 0;
        lowest = P::from_double(1.0e4);
        bool seeded = false;
        T start[kN], step[kN];
#pragma unroll
        for (int i = 0; i < kN; i++) best[i * BS] = P::zero();
        if (args.seeds != nullptr) {
          const double *sd = args.seeds + pixel * kN;
          if (!isnan(sd[0])) {
            const double rel[kN] = {1.25, 1.5, 0.5, 2.0, 2.0, 2.0};
            seeded = true;
#pragma unroll
            for (int i = 0; i < kN; i++) {
              start[i] = P::from_double(sd[i]);
              step[i] = P::from_double((rel[i] * fp.seed_step_scale) * sd[i]);
            }
          }
        }
        n_starts = seeded ? 1 : fp.n_hstarts;
        if (!seeded) {
          P::template cold_start<NB>(args, px, start, step);
          start[0] = P::hstart(args, start_k);
          step[0] = P::h_step(start[0]);
        }
        m.set_start(start, step);
        m.begin(var_limit, fp.konvge, fp.kcount);
        has = true;
      }
      chunk_next += __popc(taken);
      need &= ~taken;
    }
    if constexpr (std::is_same<P, PrecF64>::value) {
      if (!open && args.left != nullptr) {
        if (hand_on(args, m, px, lane, var_limit, has, item, start_k, guard, counted)) break;
      }
    }
    if (!__any_sync(kFull, has)) break;

    // ---- one cost evaluation per lane, then the bookkeeping --------------
    if (has) {
      const bool fin = m.phase == PH_FINAL;
      typename P::Details det;
      T y = P::zero(), x[kN];
#pragma unroll
      for (int i = 0; i < kN; i++) x[i] = m.x(i);
      if constexpr (P::kFused) {
        // the kept optimum is evaluated together with the other lanes' points
        typename P::template Keep<NB> keep;
        keep.want = fin;
        y = P::template cost_keep<NB>(args, px, x, keep);
        if (fin) P::template details_from_keep<NB>(args, keep, y, det);
      } else {
        if (fin) P::template details<NB>(args, px, x, det);
        else y = P::template cost<NB>(args, px, x);
      }
      if (fin) {
        write_fit<P, NB>(o, pixel, x, det, total, kept_evals, kept_start, kept_fault);
        if (args.pixels) write_single_chain(args, position, pixel, det.model_error);
        has = false;
      } else if (++guard > guard_cap) {
        // Defensive cap: each nelmin call is bounded by kcount, so
        // reaching this means a defect; flag it instead of spinning.
        atomicOr(args.error, PHOTIC_DEVERR_EVAL_CAP);
        if (item >= 0) rec[item * fp.n_hstarts + start_k].evals = -1;
        else write_invalid(args, position, pixel);
        has = false;
      } else if (m.step_machine(y)) {
        const T ynewlo = m.F(m.lo);
        if (item >= 0) {
          // a start on its own: its record, and the early exit for the
          // pixel's later starts (model/samodel.c:2404)
          StartRecord<P> &rc = rec[item * fp.n_hstarts + start_k];
          rc.y = ynewlo;
          rc.evals = m.icount;
          rc.fault = m.ifault;
#pragma unroll
          for (int i = 0; i < kN; i++) rc.x[i] = m.x(i);
          if (P::lt(ynewlo, P::from_double(args.early_exit)) && P::lt(ynewlo, P::from_double(1.0e4)))
            atomicMin(args.exit_k + item, start_k);
          has = false;
        } else {
          // nelmin returned: keep the best start (model/samodel.c:2380-2405)
          total += m.icount;
          bool finish = false;
          if (P::lt(ynewlo, lowest)) {
            lowest = ynewlo;
#pragma unroll
            for (int i = 0; i < kN; i++) best[i * BS] = m.x(i);
            kept_evals = m.icount;
            kept_start = start_k;
            kept_fault = m.ifault;
            if (P::lt(lowest, P::from_double(args.early_exit))) finish = true;
          }
          start_k++;
          if (!finish && start_k < n_starts) {
            T start[kN], step[kN];
            P::template cold_start<NB>(args, px, start, step);
            start[0] = P::hstart(args, start_k);
            step[0] = P::h_step(start[0]);
            m.set_start(start, step);
            m.begin(var_limit, fp.konvge, fp.kcount);
          } else {
#pragma unroll
            for (int i = 0; i < kN; i++) m.x(i) = best[i * BS];
            m.phase = PH_FINAL;
          }
        }
      } else if (item >= 0 && start_k > 0 && (guard & 63) == 0 &&
                 __ldcg(args.exit_k + item) < start_k) {
        has = false;  // an earlier start has ended the pixel
      }
    }
  }
}

// A band's term (band_term) from two lanes of the group `mask`: a lane with
// `bottom` set evaluates the bottom's path, the lane `apart` below it the
// columns' and the term (valid there).
__device__ __forceinline__ void band_term_pair(const SceneConsts &sc, int b, double sec_sun,
                                               bool bottom, int apart, unsigned mask, double mean,
                                               double H, double rho, double P, double lnP, double G, double X,
                                               double pw, double r, BandTerm &t) {
  double u, K;
  bool ok = band_medium(sc, b, P, lnP, G, X, pw, u, K), deep;
  double Du = (bottom ? 1.04 : 1.03) * sf::sqrt_mid(1.0 + (bottom ? 5.4 : 2.4) * u);
  if (sc.sec_view != 1.0) Du = Du * sc.sec_view;
  const double e = path_loss((sec_sun + Du) * K * H, deep, ok);
  const double eB = __shfl_down_sync(mask, e, apart);
  const int fB = __shfl_down_sync(mask, (ok ? 1 : 0) | (deep ? 2 : 0), apart);
  if (bottom) return;
  ok = band_close(u, K, e, eB, (fB & 2) != 0, rho, r, t) && ok && (fB & 1) != 0;
  if (!ok) band_term_again(sc, b, sec_sun, false, mean, H, rho, P, lnP, G, X, pw, r, t);
}

// The same queue of starts for few positions: a group of eight lanes a start,
// band b on lane b (of up to four bands its bottom path on lane b + 4),
// coordinate i of the simplex on lane i (NmGroup).  A launch of few positions
// lasts as long as one start's chain of up to kcount evaluations, and one
// lane's evaluation takes four times a band's FP64 instructions and six
// coordinates' (342 a trip, here about 115, at 64 clocks each for a warp alone
// on its SM quarter): 256 pixels 35 -> 14.6 ms, and with the bottom path on its
// own lane 12.9.  A full device is better used by a lane a start (few_starts,
// photic_host.cu).
//
// kLeft: the starts that the warps of the lane kernel have handed on and none
// has taken up, each from the state it was left in.
constexpr int kFewLanes = 8, kFewBlock = 128;
template <int NB, bool kLeft>
__global__ void __launch_bounds__(kFewBlock) invert_few_kernel(const __grid_constant__ InvertArgs args) {
  constexpr int G = kFewLanes;
  using Nm = NmGroup<kN, 1, G, G, true>;
  constexpr int kV = (kN + 1) * G, kF = kN + 2;
  // up to four bands: band gl % 4, the lanes from 4 on its bottom path
  constexpr int kPaths = G / 2;
  constexpr bool kPair = NB <= kPaths;
  __shared__ double smem[kFewBlock / G][kV + kF + 3 * G];
  const FitParams &fp = args.fp;
  const SceneConsts &sc = args.sc;
  const int nb = fp.n_bands;
  const int gl = threadIdx.x % G;
  const int band = kPair ? (gl % kPaths < nb ? gl % kPaths : 0) : (gl < nb ? gl : 0);
  double *base = smem[threadIdx.x / G];
  double *X = base + kV + kF, *dd = X + G, *kk = dd + G;
  Nm m;
  m.V = base;
  m.Fv = base + kV;
  m.X = X;
  m.gl = gl;
  m.clear();
  const unsigned gmask = ((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1));
  m.gmask = gmask;
  StartRecord<PrecF64> *const rec = reinterpret_cast<StartRecord<PrecF64> *>(args.records);
  const int64_t total_pos = kLeft ? (int64_t)__ldcg(&args.left->given) : args.n_par * fp.n_hstarts;
  const double var_limit = fp.reqmin * (double)kN;
  const int32_t guard_cap = (fp.n_hstarts + 1) * (fp.kcount + 8 * kN + 16);

  bool has = false, open = true;
  int64_t item = 0;
  int32_t start_k = 0, guard = 0;
  double my_rrs = 0.0, my_pw = 0.0, mean = 0.0;

  for (;;) {
    bool fresh = false;
    int64_t p = 0;
    const LeftStart *left = nullptr;
    float r[NB];
    do {
      unsigned long long w = ~0ull;
      const bool ask = !has && open && !fresh;
      if (ask && gl == 0)
        w = kLeft ? (unsigned long long)atomicAdd(&args.left->taken, 1u)
                  : atomicAdd(args.queue, 1ull);
      w = __shfl_sync(kFull, w, 0, G);
      if (ask) {
        if (kLeft && w < (unsigned long long)total_pos) {
          left = reinterpret_cast<const LeftStart *>(
                     reinterpret_cast<const unsigned char *>(args.left) +
                     left_record_offset(args.left_slots)) + w;
          start_k = left->start_k;
          item = left->item;
          fresh = start_wanted(args.exit_k + item, start_k, gmask, G, gl);
        } else if (w < (unsigned long long)total_pos) {
          start_k = (int32_t)((int64_t)w / args.n_par);
          item = (int64_t)w % args.n_par;
          p = pixel_at(args, item);
          fresh = start_k == 0 || (start_wanted(args.exit_k + item, start_k, gmask, G, gl) &&
                                   (args.seeds == nullptr || isnan(args.seeds[p * kN])));
          if (fresh) {
            load_spectrum<NB>(args, p, r);
#pragma unroll
            for (int b = 0; b < NB; b++)
              if (b < nb && !args.no_mask && band_masked(r[b], fp.nodata)) fresh = false;
            if (!fresh && start_k == 0 && gl == 0) {
              write_masked(args.out, p);
              args.exit_k[item] = -1;
            }
          }
        } else {
          open = false;
        }
      }
    } while (__any_sync(kFull, !has && open && !fresh));
    if (!__any_sync(kFull, has || fresh)) break;

    if (kLeft && fresh) {
      using Px = NmPixel<PrecF64, 1>;
      const int i = gl < kN ? gl : 0;  // a lane without a coordinate holds the first's
      mean = left->px[2 * NB];
      my_rrs = left->px[band];
      my_pw = left->px[NB + band];
      m.start[0] = left->slots[Px::kV + kN * kN + i];  // vertex N while the simplex is set up
      m.begin(var_limit, fp.konvge, fp.kcount);
      __syncwarp(gmask);
      if (gl < kN) {
#pragma unroll 1
        for (int j = 0; j <= kN; j++) m.V[j * G + gl] = left->slots[Px::kV + j * kN + gl];
        X[gl] = left->slots[Px::kX + gl];
      }
      if (gl <= kN) m.Fv[gl] = left->slots[Px::kF + gl];
      m.step[0] = left->slots[Px::kStep + i];
      m.refl[0] = left->slots[Px::kRefl + i];
      m.cen[0] = left->slots[Px::kCen + i];
      m.xmin[0] = m.trial[0] = left->slots[Px::kX + i];
      m.ylo = left->ylo;
      m.fr = left->fr;
      m.scale = left->scale;
      m.floor_lo = left->floor_lo;
      m.phase = left->phase;
      m.jj = left->jj;
      m.hi = left->hi;
      m.lo = left->lo;
      m.icount = left->icount;
      m.numres = left->numres;
      m.ifault = left->ifault;
      m.countdown = left->countdown;
      guard = left->guard;
      has = true;
    } else if (fresh) {
      PixelF64<NB> px;
      double rd[NB];
#pragma unroll
      for (int b = 0; b < NB; b++) rd[b] = (double)r[b];
      const double Y = pixel_shape_f64<NB>(fp, rd, px);
      mean = px.mean;
#pragma unroll
      for (int b = 0; b < NB; b++)
        if (b == band) my_rrs = px.rrs[b];
      my_pw = pow_call(sc.ratio440[band], Y);
      double start[kN], step[kN];
      bool seeded = false;
      if (args.seeds != nullptr) {
        const double *sd = args.seeds + p * kN;
        if (!isnan(sd[0])) {
          const double rel[kN] = {1.25, 1.5, 0.5, 2.0, 2.0, 2.0};
          seeded = true;
#pragma unroll
          for (int i = 0; i < kN; i++) {
            start[i] = sd[i];
            step[i] = (rel[i] * fp.seed_step_scale) * sd[i];
          }
        }
      }
      if (!seeded) {
        cold_start_f64<NB>(fp, px, start, step);
        start[0] = fp.hstarts[start_k];
        step[0] = PrecF64::h_step(start[0]);
      }
      m.start[0] = 0.0;
      m.step[0] = 0.0;
#pragma unroll
      for (int i = 0; i < kN; i++)
        if (i == gl) {
          m.start[0] = start[i];
          m.step[0] = step[i];
        }
      guard = 0;
      m.begin(var_limit, fp.konvge, fp.kcount);
      has = true;
    }
    __syncwarp();
    // ---- one evaluation per group at X: a band a lane, then the sum and the
    // rest of the cost on every lane
    if (has && (kPair || gl < nb)) {
      const double H = fabs(X[0]), B = 0.01 * fabs(X[1]);
      const double qB = fm::self_ratio(fabs(X[2])) * B;
      const double P = 0.01 * fabs(X[3]), Gg = 0.01 * fabs(X[4]), Xx = 0.01 * fabs(X[5]);
      BandTerm t;
      if constexpr (kPair)
        band_term_pair(sc, band, sc.sec_sun, gl >= kPaths, kPaths, gmask, mean, H,
                       qB * sc.refl[band], P, log(P), Gg, Xx, my_pw, my_rrs, t);
      else
        band_term(sc, gl, sc.sec_sun, false, mean, H, qB * sc.refl[gl], P, log(P), Gg, Xx, my_pw,
                  my_rrs, t);
      if (gl < nb) {
        dd[gl] = t.dd;
        kk[gl] = t.K;
      }
    }
    __syncwarp();
    if (has) {
      double err = 0.0, K_min = 1.0e4, E;
#pragma unroll
      for (int b = 0; b < NB; b++)
        if (b < nb) {
          err = err + dd[b];
          const double K = kk[b];
          if (k_counts(K) && sf::lt(K, K_min)) K_min = K;
        }
      const double y = cost_total_f64(fp, err, K_min, mean, fabs(X[0]), E);
      __syncwarp(gmask);  // every lane has read X, dd and kk
      const bool capped = ++guard > guard_cap;
      if (capped && gl == 0) atomicOr(args.error, PHOTIC_DEVERR_EVAL_CAP);
      if (start_k > 0 && (guard & 63) == 0 &&
          !start_wanted(args.exit_k + item, start_k, gmask, G, gl)) {
        has = false;  // an earlier start has ended the pixel
      } else if (capped || m.step_machine(y)) {
        const double ynewlo = m.F(m.lo);
        StartRecord<PrecF64> &rc = rec[item * fp.n_hstarts + start_k];
        if (gl < kN) rc.x[gl] = m.xmin[0];
        if (gl == 0) {
          rc.y = ynewlo;
          rc.evals = capped ? -1 : m.icount;
          rc.fault = m.ifault;
          if (!capped && sf::lt(ynewlo, args.early_exit) && sf::lt(ynewlo, 1.0e4))
            atomicMin(args.exit_k + item, start_k);
        }
        has = false;
      }
    }
    __syncwarp();
  }
}

// The n_par pixels after their starts have run: the records compared in the
// order of the starts, as the sequential loop does (model/samodel.c:
// 2380-2405), and the products at the kept optimum.
template <class P, int NB>
__global__ void __launch_bounds__(128) finish_kernel(const __grid_constant__ InvertArgs args) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= args.n_par || args.exit_k[i] < 0) return;
  const FitParams &fp = args.fp;
  const int64_t q = args.n_seq + i;
  const int64_t p = pixel_at(args, q);
  const bool seeded = args.seeds != nullptr && !isnan(args.seeds[p * kN]);
  const int n_starts = seeded ? 1 : fp.n_hstarts;
  const StartRecord<P> *rec = reinterpret_cast<const StartRecord<P> *>(args.records) +
                              i * fp.n_hstarts;
  typename P::T lowest = P::from_double(1.0e4), x[kN];
#pragma unroll
  for (int c = 0; c < kN; c++) x[c] = P::zero();
  int32_t total = 0, kept_evals = 0, kept_start = 0, kept_fault = 0;
  for (int k = 0; k < n_starts; k++) {
    if (rec[k].evals < 0) {
      write_invalid(args, q, p);
      return;
    }
    total += rec[k].evals;
    if (P::lt(rec[k].y, lowest)) {
      lowest = rec[k].y;
#pragma unroll
      for (int c = 0; c < kN; c++) x[c] = rec[k].x[c];
      kept_evals = rec[k].evals;
      kept_start = k;
      kept_fault = rec[k].fault;
      if (P::lt(lowest, P::from_double(args.early_exit))) break;
    }
  }
  float r[NB];
  load_spectrum<NB>(args, p, r);
  typename P::template Pixel<NB> px;
  P::template setup<NB>(args, r, px);
  typename P::Details det;
  if constexpr (P::kFused) {
    typename P::template Keep<NB> keep;
    keep.want = true;
    const typename P::T y = P::template cost_keep<NB>(args, px, x, keep);
    P::template details_from_keep<NB>(args, keep, y, det);
  } else {
    P::template details<NB>(args, px, x, det);
  }
  write_fit<P, NB>(args.out, p, x, det, total, kept_evals, kept_start, kept_fault);
  if (args.pixels) write_single_chain(args, q, p, det.model_error);
}

// Groups of lanes for up to `positions` starts.
template <int NB, bool kLeft>
cudaError_t launch_few_kernel(const InvertArgs &a, int64_t positions, cudaStream_t s) {
  auto k = invert_few_kernel<NB, kLeft>;
  int occ = 0, dev = 0, sms = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, kFewBlock, 0);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorInvalidConfiguration;
  // one block (a warp a quarter) per SM first
  constexpr int kGroups = kFewBlock / kFewLanes;
  int64_t per_sm = (positions + (int64_t)sms * kGroups - 1) / ((int64_t)sms * kGroups);
  if (per_sm > occ) per_sm = occ;
  const int64_t need = (positions + kGroups - 1) / kGroups;
  const int64_t grid = per_sm * sms < need ? per_sm * sms : need;
  k<<<(unsigned)grid, kFewBlock, 0, s>>>(a);
  return cudaGetLastError();
}

template <class P, int NB, int BS>
cudaError_t launch_one(const InvertArgs &a, int grid, cudaStream_t s, int *occupancy) {
  const size_t smem =
      invert_smem_bytes(BS) + (size_t)BS * sizeof(typename P::template Pixel<NB>);
  auto k = invert_kernel<P, NB, BS>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  if (occupancy) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occupancy, k, BS, smem);
  static_assert(sizeof(StartRecord<P>) == kStartRecordBytes, "record size");
  k<<<grid, BS, smem, s>>>(a);
  if constexpr (std::is_same<P, PrecF64>::value) {
    if (a.left != nullptr) {
      e = launch_few_kernel<NB, true>(a, (int64_t)grid * BS, s);
      if (e != cudaSuccess) return e;
    }
  }
  if (a.n_par > 0)
    finish_kernel<P, NB><<<(unsigned)((a.n_par + 127) / 128), 128, 0, s>>>(a);
  return cudaGetLastError();
}

template <class P, int NB>
cudaError_t launch_block(const InvertArgs &a, int block, int grid, cudaStream_t s, int *occ) {
  switch (block) {
    case 64: return launch_one<P, NB, 64>(a, grid, s, occ);
    case 256: return launch_one<P, NB, 256>(a, grid, s, occ);
    default: return launch_one<P, NB, 128>(a, grid, s, occ);
  }
}

template <class P>
cudaError_t launch_prec(const InvertArgs &a, int block, int grid, cudaStream_t s, int *occ) {
  if (a.fp.n_bands == 4) return launch_block<P, 4>(a, block, grid, s, occ);
  return launch_block<P, 8>(a, block, grid, s, occ);
}

}  // namespace

// Shared memory of the simplex and the staged positions; launch_one adds the
// chunk's pixel set-ups, whose size depends on the precision policy.
size_t invert_smem_bytes(int block) {
  // double and double-float both take 8 bytes per value
  return (size_t)block * 8 * (NmPixel<PrecF64, 32>::kSlots + kN + 1);
}

namespace {

template <int NB>
cudaError_t launch_few(const InvertArgs &a, cudaStream_t s) {
  cudaError_t e = launch_few_kernel<NB, false>(a, a.n_par * a.fp.n_hstarts, s);
  if (e != cudaSuccess) return e;
  finish_kernel<PrecF64, NB><<<(unsigned)((a.n_par + 127) / 128), 128, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_invert_few(const InvertArgs &a, cudaStream_t s) {
  return a.fp.n_bands <= 4 ? launch_few<4>(a, s) : launch_few<8>(a, s);
}

cudaError_t launch_invert(const InvertArgs &a, int precision, int block, int grid,
                          cudaStream_t s) {
  if (precision == PHOTIC_PREC_DF64) return launch_prec<PrecDF>(a, block, grid, s, nullptr);
  if (precision == PHOTIC_PREC_FP32) return launch_prec<PrecF32>(a, block, grid, s, nullptr);
  return launch_prec<PrecF64>(a, block, grid, s, nullptr);
}

int invert_blocks_per_sm(const InvertArgs &a, int precision, int block) {
  int n = 0;
  cudaError_t e = precision == PHOTIC_PREC_DF64   ? launch_prec<PrecDF>(a, block, 0, 0, &n)
                  : precision == PHOTIC_PREC_FP32 ? launch_prec<PrecF32>(a, block, 0, 0, &n)
                                                  : launch_prec<PrecF64>(a, block, 0, 0, &n);
  return e == cudaSuccess ? n : 0;
}

}  // namespace photic
