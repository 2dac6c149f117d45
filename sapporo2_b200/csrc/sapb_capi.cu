// C ABI over the device code: device state, staging, launch planning.
// Declared in include/sapporo_b200.h.
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <math.h>

#include <algorithm>
#include <climits>
#include <new>

#include "../../include/sapporo_b200.h"
#include "sapb_dev.h"
#include "sapb_launch.h"

using namespace sapb;

static char g_err[512];

// Pushes of up to this many j records are copied to a pinned buffer of their
// own, which the scatter kernel reads over the bus: the caller's staging is
// free when the call returns, without a copy to the device and a wait for it.  Larger
// ones are copied and waited for: their copy takes longer than the wait.
constexpr int kSmallPush = 512;
// Host force calls of up to this many i read their records from pinned memory
// inside the predictor's launch and write their results to pinned memory from
// the reduction; larger ones use the copy engines, which run beside kernels.
// Both together: 48 j pushed, 48 i on 16384 j through the class 103 -> 87 us;
// 2001 and 2001 on 100003, 708 -> 692.
constexpr int kDirectCall = 16384;

// Default accuracy bound of the single-float position difference on far
// tiles (relative to the pair distance).
constexpr double kSpatialDelta = 1e-6;

static int fail(sapb_dev *d, int code, const char *fmt, ...) {
  char *buf = d ? d->err : g_err;
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, 512, fmt, ap);
  va_end(ap);
  return code;
}

int sapb_fail(sapb_dev *d, int code, const char *fmt, ...) {
  char *buf = d ? d->err : g_err;
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, 512, fmt, ap);
  va_end(ap);
  return code;
}

#define CK(d, call)                                                                       \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      return fail((d), SAPB_ECUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_),       \
                  __FILE__, __LINE__);                                                    \
  } while (0)

static size_t pred_bytes_per_j(int order, int prec) {
  return prec == DOUBLE ? 32u * pred_fields64(order) : 16u * pred_fields(order);
}
static int nplanes(int order) {  // FP64 planes: t m eps + 3*(x v a j) [+ 3*(s c)]
  return 3 + 12 + (order >= SIXTH ? 6 : 0);
}

static void free_j(sapb_dev *d) {
  if (d->jpool) cudaFree(d->jpool);
  if (d->jid) cudaFree(d->jid);
  if (d->pred) cudaFree(d->pred);
  d->jpool = nullptr;
  d->jid = nullptr;
  d->pred = nullptr;
  d->cap = 0;
}

static void bind_planes(JState &js, double *pool, int *id, int cap, int order) {
  double *p = pool;
  js.t = p; p += cap;
  js.m = p; p += cap;
  js.eps = p; p += cap;
  for (int d = 0; d < 3; d++) { js.x[d] = p; p += cap; }
  for (int d = 0; d < 3; d++) { js.v[d] = p; p += cap; }
  for (int d = 0; d < 3; d++) { js.a[d] = p; p += cap; }
  for (int d = 0; d < 3; d++) { js.j[d] = p; p += cap; }
  for (int d = 0; d < 3; d++) {
    js.s[d] = order >= SIXTH ? p : nullptr;
    if (order >= SIXTH) p += cap;
  }
  for (int d = 0; d < 3; d++) {
    js.c[d] = order >= SIXTH ? p : nullptr;
    if (order >= SIXTH) p += cap;
  }
  js.id = id;
}

// Grows j storage to new_cap, copying the first old cap entries of every
// plane and of the predicted records.
static int grow_j(sapb_dev *d, int new_cap) {
  if (new_cap <= d->cap) return SAPB_OK;
  // grow the device store by at least half: callers that stage addresses in
  // order step their bound up by 10 % at a time (the reference's
  // increase_jMemory), which would otherwise reallocate and copy the whole
  // store ~44 times on the way from 16384 to 2^20
  if (d->cap > 0) new_cap = (int)std::min<long long>(INT_MAX / 2, std::max<long long>(new_cap, (long long)d->cap + d->cap / 2));
  const int np = nplanes(d->order);
  double *pool = nullptr;
  int *id = nullptr;
  void *pred = nullptr;
  const size_t pb = pred_bytes_per_j(d->order, d->prec);
  {  // refuse up front what cannot fit (no attempt, no partial allocation)
    const size_t need = ((size_t)np * 8 + 4 + pb) * (size_t)new_cap;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && need > free_b)
      return fail(d, SAPB_ENOMEM,
                  "cannot allocate j storage for %d particles: %.1f GB needed, %.1f GB free",
                  new_cap, need / 1e9, free_b / 1e9);
  }
  if (cudaMalloc(&pool, sizeof(double) * np * (size_t)new_cap) != cudaSuccess ||
      cudaMalloc(&id, sizeof(int) * (size_t)new_cap) != cudaSuccess ||
      cudaMalloc(&pred, pb * (size_t)new_cap) != cudaSuccess) {
    cudaGetLastError();
    if (pool) cudaFree(pool);
    if (id) cudaFree(id);
    if (pred) cudaFree(pred);
    return fail(d, SAPB_ENOMEM, "cannot allocate j storage for %d particles", new_cap);
  }
  CK(d, cudaMemsetAsync(pool, 0, sizeof(double) * np * (size_t)new_cap, d->stream));
  CK(d, cudaMemsetAsync(id, 0, sizeof(int) * (size_t)new_cap, d->stream));
  CK(d, cudaMemsetAsync(pred, 0, pb * (size_t)new_cap, d->stream));
  if (d->cap > 0) {
    for (int k = 0; k < np; k++)
      CK(d, cudaMemcpyAsync(pool + (size_t)k * new_cap, d->jpool + (size_t)k * d->cap,
                            sizeof(double) * d->cap, cudaMemcpyDeviceToDevice, d->stream));
    CK(d, cudaMemcpyAsync(id, d->jid, sizeof(int) * d->cap, cudaMemcpyDeviceToDevice, d->stream));
    CK(d, cudaMemcpyAsync(pred, d->pred, pb * d->cap, cudaMemcpyDeviceToDevice, d->stream));
    CK(d, cudaStreamSynchronize(d->stream));
  }
  free_j(d);
  d->jpool = pool;
  d->jid = id;
  d->pred = pred;
  d->pred_gen++;
  d->cap = new_cap;
  bind_planes(d->js, pool, id, new_cap, d->order);
  return SAPB_OK;
}

static int ensure_i(sapb_dev *d, int ni) {
  if (ni <= d->i_cap) return SAPB_OK;
  const int cap = std::max(ni, d->n_pipes);
  const int is = i_stride(d->order);
  double *ih = nullptr, *id = nullptr, *rh = nullptr, *rd = nullptr;
  int *cnt = nullptr, *lst = nullptr;
  bool ok = cudaHostAlloc(&ih, sizeof(double) * is * (size_t)cap, cudaHostAllocDefault) ==
                cudaSuccess &&
            cudaMalloc(&id, sizeof(double) * is * (size_t)cap) == cudaSuccess &&
            cudaHostAlloc(&rh, sizeof(double) * kResStride * (size_t)cap,
                          cudaHostAllocDefault) == cudaSuccess &&
            cudaMalloc(&rd, sizeof(double) * kResStride * (size_t)cap) == cudaSuccess &&
            cudaMalloc(&cnt, sizeof(int) * (size_t)cap) == cudaSuccess &&
            cudaMalloc(&lst, sizeof(int) * kNgbPB * (size_t)cap) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    if (ih) cudaFreeHost(ih);
    if (rh) cudaFreeHost(rh);
    if (id) cudaFree(id);
    if (rd) cudaFree(rd);
    if (cnt) cudaFree(cnt);
    if (lst) cudaFree(lst);
    return fail(d, SAPB_ENOMEM, "cannot allocate i buffers for %d particles", cap);
  }
  cudaStreamSynchronize(d->stream);  // a call in flight may still use the old buffers
  if (d->irec_h) {
    memcpy(ih, d->irec_h, sizeof(double) * is * (size_t)d->i_cap);
    cudaFreeHost(d->irec_h);
  }
  if (d->res_h) cudaFreeHost(d->res_h);
  if (d->irec_d) cudaFree(d->irec_d);
  if (d->res_d) cudaFree(d->res_d);
  if (d->ngb_count_d) cudaFree(d->ngb_count_d);
  if (d->ngb_list_d) cudaFree(d->ngb_list_d);
  d->irec_h = ih;
  d->irec_d = id;
  d->res_h = rh;
  d->res_d = rd;
  d->ngb_count_d = cnt;
  d->ngb_list_d = lst;
  d->i_cap = cap;
  CK(d, cudaMemsetAsync(cnt, 0, sizeof(int) * (size_t)cap, d->stream));
  return SAPB_OK;
}

// Room for `doubles` of scratch: the block that sapb_open allocates, or for more
// a block grown on demand.  The small one stays when the large one comes: freed
// inside the first call that needs more, it took 0.4 ms of that call (first pass
// of 16384 x 16384 on a new handle 1.25 ms, 0.85 without).
constexpr size_t kPartOpen = 1 << 18;  // 2 MB
static int ensure_part(sapb_dev *d, size_t doubles, double **room) {
  *room = d->part0_d;
  if (doubles <= kPartOpen) return SAPB_OK;
  if (doubles > d->part_cap) {
    if (d->part_d) cudaFree(d->part_d);
    d->part_d = nullptr;
    d->part_cap = 0;
    const size_t want = doubles + doubles / 4;
    if (cudaMalloc(&d->part_d, sizeof(double) * want) != cudaSuccess) {
      cudaGetLastError();
      return fail(d, SAPB_ENOMEM, "cannot allocate %zu bytes of partial sums", sizeof(double) * want);
    }
    d->part_cap = want;
  }
  *room = d->part_d;
  return SAPB_OK;
}

// ---------------------------------------------------------------------
// Launch planner: threads-per-i, i per thread and the number of j slices
// (cost model in make_plan below).
// ---------------------------------------------------------------------
struct Plan {
  int tpi, ip, ns, i_tiles, slice_tiles;
};
// Where a call's results go: the caller's device buffer; or, for host calls,
// device memory and a copy, or pinned memory straight from the reduction.
enum class Call { device, copied, pinned };

// resident blocks per SM of a force-kernel shape (occupancy API)
static int blocks_per_sm(int order, int prec, int tpi, int ip) {
  return std::max(1, force_blocks_per_sm(order, prec, tpi, ip));
}

// Launch shape for ni i-particles and nj j.
//
// Threads per i and i per thread come from shape_mixed or shape_fp64.  The
// number of j-slices S minimises the cost of
// B = i-tiles x S blocks in R = SMs x resident blocks slots: a block costs
// its tiles plus `block` for its start and end; up to one wave the call
// takes as long as its longest block, beyond that as long as the slots take
// for all blocks, plus `tail` of the part of the last wave that stays empty.
// With a share u of an SM's slots in use a tile takes sqrt(u) of its time on
// a full SM (latency, not the pipe, bounds a block there).  Each slice adds
// its records to the reduction, and kSliceS to that kernel's chain of loads.
// More slices are taken only where they cost less than `more` of fewer: other
// calls on the GPU pay for every block's start.
//
// Host calls wait for their results and have the GPU to themselves: kAlone.
// Device-resident ones may run beside others: for them the constants are a
// compromise between a call alone and calls of three streams back to back, over
// 44 calls from 1024 x 1024 to 16384 i on 2^20 j with 1 to 64 slices each: back
// to back within 1 % of the best number on average (2.7 % at most), alone within
// 2.2 %.  With kAlone's they took up to four times the slices: 5000 i on 65536 j
// at 4th order ran in 22, 398 us back to back and 522 alone, against 378 and 551
// in 7; 8192 x 8192 at 6th order in 5, 148 and 200 against 142 and 213 in 3.
struct SliceCost {
  double block, tail, more;
};
constexpr SliceCost kAloneAddress{0.3, 0.6, 0.96};
constexpr SliceCost kAloneSpatial{0.3, 0.6, 1.0 - 1e-9};
constexpr SliceCost kCostAddress{1.0, 0.45, 0.97};
constexpr SliceCost kCostSpatial{1.0, 1.0, 1.0 - 1e-9};  // near tiles run longer: whole waves
constexpr SliceCost kCostFp64{0.3, 0.6, 0.99};
constexpr double kSliceS = 5e-8;
// A call with one slice on the device's own buffers launches no reduction
// (run_force): that kernel's launch, its wait for the force kernel and its run.
// (Mixed, 6th order, 1024 x 1024: one slice 45 us a pass, 58 alone, four 48 and
// 58; FP64 keeps the smaller figure, with 12 us 8192 x 8192 at 4th order would go
// from 8 slices to one, 186 -> 176 us beside other calls but 232 -> 262 alone.)
constexpr double kReduceMixed = 1.2e-5, kReduceFp64 = 1e-5;
extern "C" {
static bool use_spatial(const sapb_dev *d, int ni, int nj);  // defined with the C ABI below
}

// Spatial mode pays for its per-call work (the i sort and bounds, the j
// gather after each prediction) from about 2^28 pairs, 1024 i and 65536 j on
// (B200, predict + force per call, neighbour lists on, i a random subset of
// the j: 1.04-1.06 x at 2^28 with 65536 to 262144 j, 1.07-1.12 x from 2^31;
// 0.89-0.95 x at 2^28 with 16384 or 32768 j, 0.91-1.00 x at 2^26 and 2^27;
// block-step active sets, which are spatially clustered, gain more);
// smaller calls run in address order.
constexpr double kSpatialMinPairs = 268435456.0;  // 2^28
constexpr int kSpatialMinI = 1024;
constexpr int kSpatialMinJ = 65536;

struct Shape {
  int tpi, ip;
};
constexpr int kMaxSlices = 65535;  // slices are blockIdx.y

// Mixed precision.  The fewer threads per i, the longer the FP32 sums before
// they are folded to FP64 (256 / TPI records): the acceleration's relative
// error, rms against FP64 (4000 i on 262144 j, spatial mode), is 2.5e-8 with
// (16,1), 3.1e-8 with (8,2), 3.2e-8 with (4,2), 3.6e-8 with (2,4) or (2,2) and
// 5.1e-8 with (1,4).  Time steps of tight binaries follow that rounding, so a
// shape gives way to a faster one only where that has as many threads per i.
// (Families with fewer below 1024 and 8192 i, (8,1) for (32,1), (4,2) for (8,2),
// were 1-30 % faster, with errors up to 1.9 times as large.)
//
// Free choice among all shapes, or below 2^32 pairs and 2^19 j in address order
// among those of the call's size (two i per thread with about 65536 / ni
// threads per i from 1024 i on: 16384 x 16384, 4th order, 0.45 ms against
// 0.66 for the free choice; 8 or more threads per i below), by the time of whole
// waves of blocks of four tiles or more, a tile more for a block's start.
static Shape shape_mixed(const sapb_dev *d, int ni, int nj, Call call, bool lists) {
  static const Shape shapes[] = {{1, 4}, {2, 4}, {1, 2}, {2, 2}, {4, 2}, {8, 2}, {16, 1}, {32, 1}};
  // throughput of a full GPU: 537.8, 534.6, 521.8, 516.1, 510.4 and 491.2 G
  // interactions/s at N = 2^20, 6th order; the last two are estimates for few i
  static const double eff[] = {1.0, 0.994, 0.970, 0.960, 0.949, 0.913, 0.85, 0.85};
  const bool spatial = use_spatial(d, ni, nj);
  // spatial mode asked for at any size: few i take the shapes of address order
  // (6th order, 1 i on 131072 j, host call: 77 us against 156 with (1,4)), but
  // not the one-i ones, whose kernels know no far tiles
  const bool ordered = spatial && ni >= kSpatialMinI && nj >= kSpatialMinJ;
  int first = 0, last = 7;
  if ((double)ni * nj < 4294967296.0 && nj < (1 << 19) && !ordered) {
    int t = 2;
    while (t < 8 && (long)t * 2 * ni <= 65536) t *= 2;
    first = ni < 1024 ? 5 : (t == 2 ? 3 : (t == 4 ? 4 : 5));
    if (ni >= 1024) last = first;
  }
  if (spatial) last = std::min(last, 5);
  const int tj = force_tile_j(), ntiles = std::max(1, (nj + tj - 1) / tj);
  const int max_ns = std::max(1, ntiles / 4);
  const double sm_rate = d->order >= SIXTH ? 3.6e9 : 5.6e9;
  Shape best = shapes[first];
  double best_t = 1e300;
  for (int q = first; q <= last; q++) {
    const int ti = force_tile_i(shapes[q].tpi, shapes[q].ip);
    const int i_tiles = std::max(1, (ni + ti - 1) / ti);
    // the one-i shapes run four blocks on an SM at 6th order, but each does less
    // than a quarter of one's work (65536 j, 1000 i: (16,1) 178 us, (32,1) 225):
    // counted as the three they would be with a third stage of tiles
    const int bps = shapes[q].ip == 1 && d->order >= SIXTH
                        ? 3
                        : blocks_per_sm(d->order, d->prec, shapes[q].tpi, shapes[q].ip);
    const long slots = (long)d->num_sms * bps;
    const double tile_time = 128.0 * ti * bps / (eff[q] * sm_rate);
    auto consider = [&](int ns) {
      const int st = (ntiles + ns - 1) / ns, used = (ntiles + st - 1) / st;
      const long waves = ((long)i_tiles * used + slots - 1) / slots;
      double t = (double)waves * (st + 1.0) * tile_time;
      if (used > 1) t += 5e-6 + (double)used * ni * kResStride * 8.0 / 4.0e12;
      if (t < best_t * (1.0 - 1e-9)) {
        best_t = t;
        best = shapes[q];
      }
    };
    if (d->nslices) {
      consider(std::min(d->nslices, max_ns));
      continue;
    }
    consider(1);
    consider(max_ns);
    for (int k = 1; k <= 64; k++) {  // just below k whole waves
      const long ns = k * slots / i_tiles;
      if (ns > max_ns) break;
      if (ns >= 1) consider((int)ns);
    }
  }
  // Host calls in spatial mode, below 2^19 j and 60000 i: at least four threads
  // per i.  Block steps of one system mix calls of all widths, and where shapes
  // change between them the sums of a tile err differently from step to step,
  // which the corrector's third differences amplify: 200 block steps of 262144
  // bodies with tight binaries, eight seeds, reach t > 3e-3 in five with (4,2)
  // and in three with the fastest shapes (in FP64 in both of those tried).  It
  // costs 1-2 % at 12983 i on 131072 j and 5-7 % of the force time at 32768 i on
  // 262144 j, less with the host's share of such a call.  From 2^19 j on, where
  // the force is all of a call's time, the fastest shape wins (16384 i on 2^20 j,
  // 6th order: (4,2) 29.6 ms, (1,4) 28.0), as it does for callers with their own
  // device buffers, who can set a shape; with lists, whose scans weigh on near
  // tiles, (4,2) is within 1.4 % of it up to 2^31 pairs, and ahead at 8192 i on
  // 131072 j, 6th order (2.13 ms, (2,4) 2.16), and stays.
  const bool four = call != Call::device ? nj < (1 << 19)
                                         : lists && (double)ni * nj < 2147483648.0;
  if (four && ordered && ni < 60000 && best.tpi < 4)
    return {4, 2};
  return best;
}

// FP64: one i per thread, four blocks per SM (50021 x 50021, 6th order, (8,2)
// at three blocks 10.00 ms a pass, (8,1) 9.87).  (16,1) below 1000 i, where it
// is up to 6 % faster in a call alone (999 i on 32768 j, 6th order, 181 us
// against 192; 136 against 131 beside other calls) and alike on fewer j; below
// 4096 x 4096, where it needs one slice and no reduction ((16,1) 36 us and 65
// alone at 2518 x 2518, 4th order, (8,1) 39 and 59, 77 in one slice); and below
// 2500 i on at most 16384 j, the family that the planner's test fixes at 2048 x
// 16384 (4th order (16,1) 100 us, 143 alone; (8,1) 92 and 141).  Calls from
// 16384 i on 65536 j keep (8,2), fixed there as well; (8,1) measured 8.67 ms
// against 8.93 at 16384 x 131072.  The largest 6th-order calls, 65536 i and 2^32
// pairs on, take (2,2): 262144 x 262144 265.5 ms, (8,2) 274.0, (8,1) 271.1; at 4th
// order (8,2) is as fast.
static Shape shape_fp64(int order, int ni, int nj) {
  if (order >= SIXTH && ni >= 65536 && (double)ni * nj >= 4294967296.0) return {2, 2};
  if (ni < 1000 || (ni < 2500 && nj <= 16384) || (ni < 4096 && nj < 4096)) return {16, 1};
  return ni >= 16384 && nj >= 65536 ? Shape{8, 2} : Shape{8, 1};
}

static Plan make_plan(const sapb_dev *d, int ni, int nj, Call call, bool lists) {
  const int tj = force_tile_j();
  const int ntiles = std::max(1, (nj + tj - 1) / tj);
  // pairs per SM and second of a full GPU (B200, order of magnitude): only
  // the balance between force and reduction depends on them
  const double sm_rate = d->prec == DOUBLE ? (d->order >= SIXTH ? 1.7e9 : 2.4e9)
                                           : (d->order >= SIXTH ? 3.6e9 : 5.6e9);
  // one tile or more per slice; partial records up to 256 MB
  const int max_ns = (int)std::max(
      1.0, std::min<double>(std::min(ntiles, kMaxSlices), 268435456.0 / (96.0 * ni)));
  Plan best{1, 2, 1, 1, ntiles};
  double best_t = 1e300;
  const bool spatial = use_spatial(d, ni, nj), alone = call != Call::device;
  const SliceCost cost = d->prec == DOUBLE ? kCostFp64
                         : spatial         ? (alone ? kAloneSpatial : kCostSpatial)
                                           : (alone ? kAloneAddress : kCostAddress);
  const double reduce = call == Call::pinned ? 0.0 : d->prec == DOUBLE ? kReduceFp64 : kReduceMixed;
  const Shape sh = d->tpi ? Shape{d->tpi, d->ip}
                          : d->prec == DOUBLE ? shape_fp64(d->order, ni, nj) : shape_mixed(d, ni, nj, call, lists);
  const int tpi = sh.tpi, ip = sh.ip;
  const int ti = force_tile_i(tpi, ip);
  const int i_tiles = (ni + ti - 1) / ti;
  const int bps = blocks_per_sm(d->order, d->prec, tpi, ip);
  // a one-i shape of mixed precision has less arithmetic to hide a tile's loads
  // and folds behind (60000 x 60000: (16,1) 6.4 ms, (32,1) 8.2, (2,2) 4.2)
  const double slow = d->prec == DOUBLE || ip > 1 ? 1.0 : (tpi < 32 ? 1.45 : 1.85);
  const double tile_time = slow * (double)tj * ti * bps / sm_rate;
  auto consider = [&](int ns) {
    const int st = (ntiles + ns - 1) / ns;  // tiles of the longest slice
    const double B = (double)i_tiles * ns, sms = d->num_sms, w = B / (sms * bps);
    double tiles = st + cost.block;
    if (w > 1.0) {
      const double mean = w > 2.0 ? (double)ntiles / ns : st;
      tiles = (w + cost.tail * (ceil(w) - w)) * (mean + cost.block);
    }
    const double used = std::min<double>(bps, ceil(B / sms)) / bps;
    double t = tiles * sqrt(used) * tile_time;
    if (ns > 1)
      t += ns * (kSliceS + (double)ni * kResStride * 8.0 / 4.0e12) + reduce;
    if (t < best_t * (best_t < 1e299 ? cost.more : 1.0)) {
      best_t = t;
      best = Plan{tpi, ip, ns, i_tiles, st};
    }
  };
  if (d->nslices) {
    // as the caller asks, in slices of four tiles or more, none empty
    const int ns = std::min(std::min(d->nslices, std::max(1, ntiles / 4)), kMaxSlices);
    const int st = (ntiles + ns - 1) / ns;
    consider((ntiles + st - 1) / st);
  } else {
    // the fewest slices for each length of the longest one
    for (int ns = 1; ns <= max_ns;) {
      consider(ns);
      const int st = (ntiles + ns - 1) / ns;
      ns = st > 1 ? (ntiles + st - 2) / (st - 1) : max_ns + 1;
    }
  }
  return best;
}

// ---------------------------------------------------------------------
// Fixed scratch of sapb_force_device_noalloc.  Every GPU that loads this
// library holds these 32 MiB until the process exits.  Host code must not
// use the symbol itself (in host code it names a host-side stand-in, not
// device memory): its device address is resolved once per device with
// cudaGetSymbolAddress, with that device current, and passed to the kernels.
// ---------------------------------------------------------------------
static __device__ __align__(256) double g_noalloc_scratch[SAPB_NOALLOC_SCRATCH_BYTES / 8];

constexpr int kMaxDevices = 64;
static double *g_noalloc_ptr[kMaxDevices];

// Resolves the scratch address for the current device (once per device).
static int noalloc_setup(sapb_dev *d) {
  if (d->device < 0 || d->device >= kMaxDevices)
    return fail(d, SAPB_EINVAL, "device ordinal %d beyond the no-allocation table", d->device);
  if (g_noalloc_ptr[d->device]) return SAPB_OK;
  CK(d, cudaSetDevice(d->device));
  void *ptr = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
  if (e != cudaSuccess || !ptr)
    return fail(d, SAPB_ECUDA, "cudaGetSymbolAddress(no-allocation scratch): %s",
                cudaGetErrorString(e));
  g_noalloc_ptr[d->device] = static_cast<double *>(ptr);
  return SAPB_OK;
}

// ---------------------------------------------------------------------
extern "C" {

const char *sapb_version(void) { return "sapporo-b200 0.1 (sm_100a)"; }

const char *sapb_error_string(int code) {
  switch (code) {
    case SAPB_OK: return "ok";
    case SAPB_ECUDA: return "CUDA runtime error";
    case SAPB_EINVAL: return "invalid argument";
    case SAPB_ENOMEM: return "out of memory";
    case SAPB_ETIMEOUT: return "device wait timed out";
    case SAPB_ENODEV: return "no CUDA device";
    default: return "unknown error";
  }
}

const char *sapb_last_error(const sapb_dev *d) { return d ? d->err : g_err; }

int sapb_device_count(int *count) {
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *count = 0;
    return fail(nullptr, SAPB_ENODEV, "cudaGetDeviceCount: %s", cudaGetErrorString(e));
  }
  *count = n;
  return SAPB_OK;
}

int sapb_open(sapb_dev **out, int device, int order, int precision, int n_pipes,
              int nj_reserve) {
  if (!out) return fail(nullptr, SAPB_EINVAL, "null handle pointer");
  *out = nullptr;
  if (order != GRAPE5 && order != FOURTH && order != SIXTH)
    return fail(nullptr, SAPB_EINVAL, "order %d not supported (GRAPE-5=0, 4th=1, 6th=2)",
                order);
  if (precision != DOUBLESINGLE && precision != DOUBLE)
    return fail(nullptr, SAPB_EINVAL, "precision %d not supported (DS=1, DOUBLE=2)", precision);
  int ndev = 0;
  if (sapb_device_count(&ndev) != SAPB_OK || ndev == 0)
    return fail(nullptr, SAPB_ENODEV, "no CUDA device available");
  if (device < 0 || device >= ndev)
    return fail(nullptr, SAPB_EINVAL, "device %d out of range (%d devices)", device, ndev);
  sapb_dev *d = new (std::nothrow) sapb_dev();
  if (!d) return fail(nullptr, SAPB_ENOMEM, "host allocation failed");
  d->device = device;
  d->order = order;
  d->prec = precision;
  d->n_pipes = n_pipes > 0 ? n_pipes : SAPB_NPIPES;
  d->sp.far_c = (float)(0x1p-23 / kSpatialDelta);
  if (const char *e = getenv("SAPPORO_B200_SPATIAL")) d->sp.mode = atoi(e) == 0 ? 0 : (atoi(e) >= 2 ? 2 : 1);
  if (const char *e = getenv("SAPPORO_B200_NEAR")) {
    const double k = atof(e);
    if (k >= 0.0 && k <= 1e6) d->near_k = k;
  }
  int rc = SAPB_OK;
  do {
    if (cudaSetDevice(device) != cudaSuccess) { rc = fail(d, SAPB_ECUDA, "cudaSetDevice(%d)", device); break; }
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) { rc = fail(d, SAPB_ECUDA, "cudaGetDeviceProperties"); break; }
    d->num_sms = prop.multiProcessorCount;
    if (prop.major < 10) {
      rc = fail(d, SAPB_ENODEV, "device %d is sm_%d%d; this library targets sm_100a", device,
                prop.major, prop.minor);
      break;
    }
    if (cudaStreamCreateWithFlags(&d->own_stream, cudaStreamNonBlocking) != cudaSuccess) { rc = fail(d, SAPB_ECUDA, "stream"); break; }
    d->stream = d->own_stream;
    if (cudaEventCreateWithFlags(&d->done, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&d->pushed, cudaEventDisableTiming) != cudaSuccess) {
      rc = fail(d, SAPB_ECUDA, "event");
      break;
    }
    if (cudaMalloc(&d->status_d, sizeof(int)) != cudaSuccess ||
        cudaHostAlloc(&d->push_h, sizeof(double) * stage_stride(order) * kSmallPush,
                      cudaHostAllocDefault) != cudaSuccess ||
        cudaHostAlloc(&d->status_h, sizeof(int), cudaHostAllocDefault) != cudaSuccess) {
      rc = fail(d, SAPB_ENOMEM, "status word");
      break;
    }
    *d->status_h = 0;
    if (cudaMemsetAsync(d->status_d, 0, sizeof(int), d->stream) != cudaSuccess) { rc = fail(d, SAPB_ECUDA, "memset"); break; }
    rc = grow_j(d, nj_reserve > 0 ? nj_reserve : 16384);
    if (rc) break;
    rc = ensure_i(d, d->n_pipes);
    if (rc) break;
    // the first small calls find their partial sums' room
    if (cudaMalloc(&d->part0_d, sizeof(double) * kPartOpen) != cudaSuccess) {
      rc = fail(d, SAPB_ENOMEM, "partial sums");
      break;
    }
    rc = noalloc_setup(d);
    if (rc) break;
    if (cudaStreamSynchronize(d->stream) != cudaSuccess) { rc = fail(d, SAPB_ECUDA, "sync"); break; }
  } while (0);
  if (rc != SAPB_OK) {
    snprintf(g_err, sizeof g_err, "%s", d->err);
    sapb_close(d);
    cudaGetLastError();
    return rc;
  }
  *out = d;
  return SAPB_OK;
}

int sapb_close(sapb_dev *d) {
  if (!d) return SAPB_OK;
  cudaSetDevice(d->device);
  if (d->stream) cudaStreamSynchronize(d->stream);
  free_j(d);
  spatial_free(d);
  if (d->stage_h) cudaFreeHost(d->stage_h);
  if (d->stage_d) cudaFree(d->stage_d);
  if (d->irec_h) cudaFreeHost(d->irec_h);
  if (d->irec_d) cudaFree(d->irec_d);
  if (d->res_h) cudaFreeHost(d->res_h);
  if (d->res_d) cudaFree(d->res_d);
  if (d->ngb_count_d) cudaFree(d->ngb_count_d);
  if (d->ngb_list_d) cudaFree(d->ngb_list_d);
  if (d->part0_d) cudaFree(d->part0_d);
  if (d->part_d) cudaFree(d->part_d);
  if (d->status_d) cudaFree(d->status_d);
  if (d->status_h) cudaFreeHost(d->status_h);
  if (d->push_h) cudaFreeHost(d->push_h);
  if (d->done) cudaEventDestroy(d->done);
  if (d->pushed) cudaEventDestroy(d->pushed);
  if (d->own_stream) cudaStreamDestroy(d->own_stream);
  delete d;
  return SAPB_OK;
}

int sapb_info(const sapb_dev *d, int *order, int *precision, int *n_pipes, int *j_capacity,
              int *num_sms) {
  if (!d) return fail(nullptr, SAPB_EINVAL, "null device");
  if (order) *order = d->order;
  if (precision) *precision = d->prec;
  if (n_pipes) *n_pipes = d->n_pipes;
  if (j_capacity) *j_capacity = d->cap;
  if (num_sms) *num_sms = d->num_sms;
  return SAPB_OK;
}

int sapb_set_stream(sapb_dev *d, void *stream) {
  if (!d) return fail(nullptr, SAPB_EINVAL, "null device");
  CK(d, cudaStreamSynchronize(d->stream));
  d->stream = stream ? (cudaStream_t)stream : d->own_stream;
  return SAPB_OK;
}

int sapb_reserve_j(sapb_dev *d, int nj_capacity) {
  if (!d || nj_capacity < 0) return fail(d, SAPB_EINVAL, "bad capacity");
  CK(d, cudaSetDevice(d->device));
  return grow_j(d, nj_capacity);
}

int sapb_j_stage_stride(const sapb_dev *d) { return d ? stage_stride(d->order) : 0; }
int sapb_i_stage_stride(const sapb_dev *d) { return d ? i_stride(d->order) : 0; }

double *sapb_j_stage(sapb_dev *d, int n) {
  if (!d || n < 0) return nullptr;
  if (n <= d->stage_cap) return d->stage_h;
  const int ss = stage_stride(d->order);
  const int cap = std::max(n, d->stage_cap + d->stage_cap / 2 + 1024);
  double *h = nullptr, *dd = nullptr;
  cudaSetDevice(d->device);
  if (cudaHostAlloc(&h, sizeof(double) * ss * (size_t)cap, cudaHostAllocDefault) != cudaSuccess ||
      cudaMalloc(&dd, sizeof(double) * ss * (size_t)cap) != cudaSuccess) {
    cudaGetLastError();
    if (h) cudaFreeHost(h);
    fail(d, SAPB_ENOMEM, "cannot allocate staging for %d j records", cap);
    return nullptr;
  }
  if (d->stage_h) {
    cudaStreamSynchronize(d->stream);  // a pending push may still read the old buffer
    memcpy(h, d->stage_h, sizeof(double) * ss * (size_t)d->stage_cap);
    cudaFreeHost(d->stage_h);
    cudaFree(d->stage_d);
  }
  d->stage_h = h;
  d->stage_d = dd;
  d->stage_cap = cap;
  return h;
}

int sapb_push_j(sapb_dev *d, int n) {
  if (!d || n < 0 || n > d->stage_cap) return fail(d, SAPB_EINVAL, "push of %d records", n);
  if (n == 0) return SAPB_OK;
  CK(d, cudaSetDevice(d->device));
  // A captured push would read the staging at each replay, after the host has
  // written other records there: refused, before anything is queued.
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  CK(d, cudaStreamIsCapturing(d->stream, &capture));
  if (capture != cudaStreamCaptureStatusNone)
    return fail(d, SAPB_ECUDA, "push of %d records on a stream that is being captured", n);
  // grow the j store to cover the highest staged address
  int maxaddr = -1;
  const int ss = stage_stride(d->order);
  for (int k = 0; k < n; k++) {
    int addr;
    memcpy(&addr, d->stage_h + (size_t)k * ss, sizeof(int));
    if (addr < 0) return fail(d, SAPB_EINVAL, "negative j address %d", addr);
    maxaddr = std::max(maxaddr, addr);
  }
  if (maxaddr >= d->cap) {
    int rc = grow_j(d, std::max(maxaddr + 1, (int)(d->cap * 1.1) + 1));
    if (rc) return rc;
  }
  if (n <= kSmallPush) {
    if (d->push_busy) CK(d, cudaEventSynchronize(d->pushed));
    memcpy(d->push_h, d->stage_h, sizeof(double) * ss * (size_t)n);
    CK(d, launch_scatter(d->order, d->prec, d->push_h, n, d->cap, d->js, d->pred, d->status_d,
                         d->stream));
    d->pred_gen++;
    CK(d, cudaEventRecord(d->pushed, d->stream));
    d->push_busy = true;
    return SAPB_OK;
  }
  CK(d, cudaMemcpyAsync(d->stage_d, d->stage_h, sizeof(double) * ss * (size_t)n,
                        cudaMemcpyHostToDevice, d->stream));
  CK(d, launch_scatter(d->order, d->prec, d->stage_d, n, d->cap, d->js, d->pred, d->status_d,
                       d->stream));
  d->pred_gen++;
  // the host may overwrite the staging buffer once the copy has been consumed
  CK(d, cudaStreamSynchronize(d->stream));
  return SAPB_OK;
}

int sapb_predict(sapb_dev *d, int nj, double ti) {
  if (!d || nj < 0 || nj > d->cap) return fail(d, SAPB_EINVAL, "predict of %d j (capacity %d)", nj, d ? d->cap : 0);
  CK(d, cudaSetDevice(d->device));
  CK(d, launch_predict(d->order, d->prec, nj, ti, d->js, d->pred, CallPrep{}, d->stream));
  d->pred_gen++;
  return SAPB_OK;
}

double *sapb_i_stage(sapb_dev *d, int ni) {
  if (!d || ni < 0) return nullptr;
  cudaSetDevice(d->device);
  if (d->pending) {  // do not hand out a buffer an in-flight copy still reads
    cudaEventSynchronize(d->done);
  }
  if (ensure_i(d, ni) != SAPB_OK) return nullptr;
  return d->irec_h;
}

static bool use_spatial(const sapb_dev *d, int ni, int nj) {
  if (d->prec != DOUBLESINGLE || d->sp.mode == 0) return false;
  if (d->sp.mode == 2) return true;
  return ni >= kSpatialMinI && nj >= kSpatialMinJ && (double)ni * nj >= kSpatialMinPairs;
}

// Near-pair radius^2 of a mixed-precision call (FP32, compared with the
// kernels' double-single ds2); 0 turns the FP64 near-pair sums off.
static float near_r2(const sapb_dev *d, double eps2) {
  if (d->prec == DOUBLE || d->order == GRAPE5) return 0.0f;
  return (float)(d->near_k * eps2);
}

// Lists from one bit per record (two ALU operations per pair, gathered per 32
// records) instead of rescans of the tiles that hold a neighbour: the bits win
// where a tile holds neighbours of many of a warp's i, i.e. with few j in
// address order (B200, about 32 neighbours: 16384 x 16384, 4th order, 437 us
// against 530, and 390 without lists), and lose where few do (16384 i on
// 131072 j, 6th order, 4.51 ms against 4.44) or where the spatial order puts a
// warp's neighbours into a few tiles (8192 i on 131072 j 2.21 against 2.15).
constexpr int kListBitsMaxJ = 65536;

// `out`: where the results go, res_dev or (Call::pinned) pinned host memory, and
// then the error word to status_h; the list counts are clear already there.
static int run_force(sapb_dev *d, int nj, int ni, const double *i_dev, double eps2, int flags,
                     double *res_dev, int *cnt_dev, int *list_dev, double *out, Call call) {
  if (nj <= 0 || nj > d->cap) return fail(d, SAPB_EINVAL, "nj = %d (capacity %d)", nj, d->cap);
  const bool direct = call == Call::pinned;
  const bool list = (flags & SAPB_F_NGB_LIST) != 0;
  Plan P = make_plan(d, ni, nj, call, list);
  double *part = nullptr;
  if (P.ns > 1) {
    const int rc = ensure_part(d, (size_t)P.ns * ni * kResStride, &part);
    // no room for the partial sums of a planned split: one slice needs none
    // (a split that the caller fixed is refused)
    if (rc && (rc != SAPB_ENOMEM || d->nslices)) return rc;
    if (rc) P.ns = 1;
  }
  if (list && !direct) CK(d, cudaMemsetAsync(cnt_dev, 0, sizeof(int) * (size_t)ni, d->stream));
  ForceArgs A{};
  A.pred = d->pred;
  // (one-i shapes set by the caller ignore the boxes: nothing to prepare)
  bool spatial = use_spatial(d, ni, nj) && P.ip % 2 == 0;
  if (spatial) {
    const int rc = spatial_prepare(d, nj, ni, i_dev);
    if (rc == SAPB_ENOMEM) spatial = false;  // no room for its buffers: address order
    else if (rc) return rc;
  }
  if (spatial) {
    A.pred = d->sp.spred;
    A.iperm = d->sp.iidx[1];
    A.ibound = d->sp.ibound;
    A.tbox = d->sp.tbox;
    A.far_c = d->sp.far_c;
    A.stats = d->sp.stats;
  }
  A.nj = nj;
  A.irec = i_dev;
  A.ni = ni;
  A.eps2 = eps2;
  A.near_r2 = near_r2(d, eps2);
  A.nslices = P.ns;
  A.i_tiles = P.i_tiles;
  A.do_list = list ? 1 : 0;
  A.list_bits = list && !spatial && d->prec != DOUBLE && nj < kListBitsMaxJ;
  A.ngb_count = cnt_dev;
  A.ngb_list = list_dev;
  A.status = d->status_d;
  A.out = P.ns > 1 ? part : res_dev;
  // One slice on the device's own buffers needs no reduction: each i's thread
  // looks its nearest neighbour up in its row of the tile, at most 32 records
  // with 8 threads per i (with fewer the reduction's lanes are faster).  1024 x
  // 1024, a pass: 42 us instead of 46 (4th order), 38 instead of 41 (FP64).
  A.finish = P.ns == 1 && P.tpi >= 8 && !direct;
  CK(d, launch_force(d->order, d->prec, A, P.tpi, P.ip, d->stream));
  if (A.finish) return SAPB_OK;
  const ReduceArgs R{A.out, P.ns, ni, out, A.pred, nj, P.tpi, i_dev, A.iperm, d->status_d,
                     direct ? d->status_h : nullptr};
  CK(d, launch_reduce(d->order, d->prec, R, d->num_sms, d->stream));
  return SAPB_OK;
}

int sapb_force(sapb_dev *d, int nj, int ni, double eps2, double ti, int flags) {
  if (!d) return fail(nullptr, SAPB_EINVAL, "null device");
  if (ni < 0 || ni > d->i_cap) return fail(d, SAPB_EINVAL, "ni = %d (staged capacity %d)", ni, d->i_cap);
  CK(d, cudaSetDevice(d->device));
  const bool predict = (flags & SAPB_F_PREDICT) != 0;
  const int words = i_stride(d->order) * ni;
  if (ni == 0 || ni > kDirectCall) {
    if (predict) {
      int rc = sapb_predict(d, nj, ti);
      if (rc) return rc;
    }
    d->last_ni = ni;
    if (ni == 0) return SAPB_OK;
    CK(d, cudaMemcpyAsync(d->irec_d, d->irec_h, sizeof(double) * (size_t)words,
                          cudaMemcpyHostToDevice, d->stream));
    int rc = run_force(d, nj, ni, d->irec_d, eps2, flags, d->res_d, d->ngb_count_d, d->ngb_list_d,
                       d->res_d, Call::copied);
    if (rc) return rc;
    CK(d, cudaMemcpyAsync(d->res_h, d->res_d, sizeof(double) * kResStride * (size_t)ni,
                          cudaMemcpyDeviceToHost, d->stream));
    CK(d, cudaMemcpyAsync(d->status_h, d->status_d, sizeof(int), cudaMemcpyDeviceToHost, d->stream));
  } else {
    if (nj < 0 || nj > d->cap) return fail(d, SAPB_EINVAL, "nj = %d (capacity %d)", nj, d->cap);
    d->last_ni = ni;
    CallPrep prep;
    prep.src = d->irec_h;
    prep.dst = d->irec_d;
    prep.words = words;
    prep.ni = ni;
    if (flags & SAPB_F_NGB_LIST) prep.count = d->ngb_count_d;
    CK(d, launch_predict(d->order, d->prec, predict ? nj : 0, ti, d->js, d->pred, prep, d->stream));
    if (predict) d->pred_gen++;
    int rc = run_force(d, nj, ni, d->irec_d, eps2, flags, d->res_d, d->ngb_count_d, d->ngb_list_d,
                       d->res_h, Call::pinned);
    if (rc) return rc;
  }
  CK(d, cudaEventRecord(d->done, d->stream));
  d->pending = true;
  return SAPB_OK;
}

int sapb_results(sapb_dev *d, const double **results, int *ni) {
  if (!d) return fail(nullptr, SAPB_EINVAL, "null device");
  CK(d, cudaSetDevice(d->device));
  if (d->pending) {
    CK(d, cudaEventSynchronize(d->done));
    d->pending = false;
  }
  if (results) *results = d->res_h;
  if (ni) *ni = d->last_ni;
  if (*d->status_h) {
    const int s = *d->status_h;
    *d->status_h = 0;
    cudaMemsetAsync(d->status_d, 0, sizeof(int), d->stream);
    if (s & kErrWaitTimeout) return fail(d, SAPB_ETIMEOUT, "force kernel: bounded wait for a j tile timed out");
    return fail(d, SAPB_EINVAL, "device reported status 0x%x", s);
  }
  return SAPB_OK;
}

int sapb_ngb_fetch(sapb_dev *d, int *counts, int *lists, int ni) {
  if (!d || ni < 0 || ni > d->i_cap) return fail(d, SAPB_EINVAL, "bad ni %d", ni);
  CK(d, cudaSetDevice(d->device));
  if (ni == 0) return SAPB_OK;
  if (counts)
    CK(d, cudaMemcpyAsync(counts, d->ngb_count_d, sizeof(int) * (size_t)ni,
                          cudaMemcpyDeviceToHost, d->stream));
  if (lists)
    CK(d, cudaMemcpyAsync(lists, d->ngb_list_d, sizeof(int) * kNgbPB * (size_t)ni,
                          cudaMemcpyDeviceToHost, d->stream));
  CK(d, cudaStreamSynchronize(d->stream));
  return SAPB_OK;
}

int sapb_force_device(sapb_dev *d, int nj, int ni, const double *i_dev, double eps2, int flags,
                      double *res_dev, int *ngb_count_dev, int *ngb_list_dev) {
  if (!d || !i_dev || !res_dev || ni < 0) return fail(d, SAPB_EINVAL, "bad arguments");
  if ((flags & SAPB_F_NGB_LIST) && (!ngb_count_dev || !ngb_list_dev))
    return fail(d, SAPB_EINVAL, "neighbour lists requested without buffers");
  CK(d, cudaSetDevice(d->device));
  if (ni == 0) return SAPB_OK;
  return run_force(d, nj, ni, i_dev, eps2, flags, res_dev, ngb_count_dev, ngb_list_dev, res_dev,
                   Call::device);
}

int sapb_wait_selftest(sapb_dev *d, int limit_ms) {
  if (!d || limit_ms < 1 || limit_ms > 2000)
    return fail(d, SAPB_EINVAL, "wait self-test limit %d ms (1..2000)", limit_ms);
  CK(d, cudaSetDevice(d->device));
  CK(d, cudaMemsetAsync(d->status_d, 0, sizeof(int), d->stream));
  CK(d, launch_wait_selftest((uint64_t)limit_ms * 1000000ull, d->status_d, d->stream));
  int s = 0;
  CK(d, cudaMemcpyAsync(&s, d->status_d, sizeof(int), cudaMemcpyDeviceToHost, d->stream));
  CK(d, cudaStreamSynchronize(d->stream));
  CK(d, cudaMemsetAsync(d->status_d, 0, sizeof(int), d->stream));
  if (s & kErrWaitTimeout)
    return fail(d, SAPB_ETIMEOUT, "self-test: the bounded device wait gave up after %d ms",
                limit_ms);
  return fail(d, SAPB_ECUDA, "self-test: the wait on a barrier nothing arrives at returned");
}

int sapb_force_device_noalloc(sapb_dev *d, int nj, int ni, const double *i_dev, double eps2,
                              int flags, double *res_dev, int *ngb_count_dev,
                              int *ngb_list_dev) {
  if (!d || !i_dev || !res_dev || ni < 0) return fail(d, SAPB_EINVAL, "bad arguments");
  if ((flags & SAPB_F_NGB_LIST) && (!ngb_count_dev || !ngb_list_dev))
    return fail(d, SAPB_EINVAL, "neighbour lists requested without buffers");
  const size_t cap_records = SAPB_NOALLOC_SCRATCH_BYTES / (sizeof(double) * kResStride);
  if ((size_t)ni > cap_records)
    return fail(d, SAPB_EINVAL,
                "sapb_force_device_noalloc: ni = %d exceeds the fixed scratch (at most %zu "
                "i-particles per call)", ni, cap_records);
  CK(d, cudaSetDevice(d->device));
  if (ni == 0) return SAPB_OK;  // as sapb_force_device: an empty call does nothing
  if (nj <= 0 || nj > d->cap) return fail(d, SAPB_EINVAL, "nj = %d (capacity %d)", nj, d->cap);
  int rc = noalloc_setup(d);  // normally already done by sapb_open
  if (rc) return rc;
  double *scratch = g_noalloc_ptr[d->device];
  // Same plan as sapb_force_device, with the j-split capped so that the
  // per-slice partial records fit the fixed scratch.
  const bool list = (flags & SAPB_F_NGB_LIST) != 0;
  Plan P = make_plan(d, ni, nj, Call::device, list);
  const int tj = force_tile_j();
  const int ntiles = (nj + tj - 1) / tj;
  const int max_ns = (int)std::max<size_t>(1, cap_records / (size_t)ni);
  if (P.ns > max_ns) {
    P.slice_tiles = (ntiles + max_ns - 1) / max_ns;
    P.ns = (ntiles + P.slice_tiles - 1) / P.slice_tiles;
  }
  if (list) CK(d, cudaMemsetAsync(ngb_count_dev, 0, sizeof(int) * (size_t)ni, d->stream));
  ForceArgs A{};
  A.pred = d->pred;
  A.nj = nj;
  A.irec = i_dev;
  A.ni = ni;
  A.eps2 = eps2;
  A.near_r2 = near_r2(d, eps2);
  A.nslices = P.ns;
  A.i_tiles = P.i_tiles;
  A.do_list = list ? 1 : 0;
  A.list_bits = list && d->prec != DOUBLE && nj < kListBitsMaxJ;
  A.ngb_count = ngb_count_dev;
  A.ngb_list = ngb_list_dev;
  A.status = d->status_d;
  A.out = scratch;  // every (slice, valid i) record is written before it is read
  CK(d, launch_force(d->order, d->prec, A, P.tpi, P.ip, d->stream));
  const ReduceArgs R{scratch, P.ns, ni, res_dev, A.pred, nj, P.tpi, i_dev, nullptr, nullptr,
                     nullptr};
  CK(d, launch_reduce(d->order, d->prec, R, d->num_sms, d->stream));
  return SAPB_OK;
}

int sapb_set_spatial(sapb_dev *d, int mode, double delta) {
  if (!d) return fail(nullptr, SAPB_EINVAL, "null device");
  if (mode < 0 || mode > 2 || !(delta >= 0.0) || delta > 1e-4)
    return fail(d, SAPB_EINVAL, "spatial mode %d, delta %g (mode 0..2, delta 0..1e-4)", mode, delta);
  d->sp.mode = mode;
  d->sp.far_c = (float)(0x1p-23 / (delta > 0.0 ? delta : kSpatialDelta));
  return SAPB_OK;
}

int sapb_set_near(sapb_dev *d, double factor) {
  if (!d) return fail(nullptr, SAPB_EINVAL, "null device");
  if (!(factor >= 0.0) || factor > 1e6)
    return fail(d, SAPB_EINVAL, "near-pair factor %g (0..1e6)", factor);
  d->near_k = factor;
  return SAPB_OK;
}

int sapb_spatial_stats(sapb_dev *d, unsigned long long *far_tiles,
                       unsigned long long *warp_tiles, int reset) {
  if (!d) return fail(nullptr, SAPB_EINVAL, "null device");
  CK(d, cudaSetDevice(d->device));
  unsigned long long h[2] = {0, 0};
  if (d->sp.stats) {
    CK(d, cudaMemcpyAsync(h, d->sp.stats, sizeof h, cudaMemcpyDeviceToHost, d->stream));
    if (reset) CK(d, cudaMemsetAsync(d->sp.stats, 0, sizeof h, d->stream));
    CK(d, cudaStreamSynchronize(d->stream));
  }
  if (far_tiles) *far_tiles = h[0];
  if (warp_tiles) *warp_tiles = h[1];
  return SAPB_OK;
}

int sapb_set_launch(sapb_dev *d, int tpi, int ip, int nslices) {
  if (!d) return fail(nullptr, SAPB_EINVAL, "null device");
  const bool ok_tpi = tpi == 0 || ((tpi == 1 || tpi == 2 || tpi == 4 || tpi == 8) && ip <= 2) ||
                      ((tpi == 16 || tpi == 32) && ip == 1) ||
                      ((tpi == 1 || tpi == 2) && ip == 4 && d->prec != DOUBLE);
  if (!ok_tpi || (ip != 0 && ip != 1 && ip != 2 && ip != 4) || nslices < 0 || (tpi && !ip))
    return fail(d, SAPB_EINVAL, "unsupported launch shape tpi=%d ip=%d slices=%d", tpi, ip, nslices);
  d->tpi = tpi;
  d->ip = ip;
  d->nslices = nslices;
  return SAPB_OK;
}

int sapb_get_plan(sapb_dev *d, int ni, int nj, int *tpi, int *ip, int *nslices) {
  if (!d || ni <= 0 || nj <= 0) return fail(d, SAPB_EINVAL, "bad sizes");
  const Plan P = make_plan(d, ni, nj, Call::device, false);
  if (tpi) *tpi = P.tpi;
  if (ip) *ip = P.ip;
  if (nslices) *nslices = P.ns;
  return SAPB_OK;
}

int sapb_read_j(sapb_dev *d, int first, int n, double ti, int predict, double *out) {
  if (!d || first < 0 || n < 0 || first + n > d->cap || (n > 0 && !out))
    return fail(d, SAPB_EINVAL, "read of j[%d, %d) (capacity %d)", first, first + n, d ? d->cap : 0);
  if (n == 0) return SAPB_OK;
  CK(d, cudaSetDevice(d->device));
  const size_t need = (size_t)n * 24;
  double *room = nullptr;
  int rc = ensure_part(d, need, &room);
  if (rc) return rc;
  CK(d, launch_readj(d->order, first, n, ti, predict, d->js, room, d->stream));
  CK(d, cudaMemcpyAsync(out, room, sizeof(double) * need, cudaMemcpyDeviceToHost, d->stream));
  CK(d, cudaStreamSynchronize(d->stream));
  return SAPB_OK;
}

}  // extern "C"
