// hpr_resident.cu — whole batches of HPR iterations for problems that fit
// the shared memory of one thread-block cluster.
//
// A small problem's half-step is a chain of dependent memory round trips (tile
// record, columns, gathers, epilogue inputs, stores) and of instructions, not
// bytes.  Measured on B200, us per iteration of a 150-iteration batch on the
// faster of the other schedules (single-CTA kernel through L2 up to n = 401,
// else the multi-CTA engine) and here: n = 61 5.3 / 3.2, n = 401 10.0 / 5.7, n =
// 803 18.2 / 10.5, with a diagonal Q 23.8 / 15.4, n = 2000 25.6 / 11.7, n = 3000
// with a general CSR Q 26.3 / 16.0.  What is left is the instruction chain of a
// tile: row sums, cone norms, projections.
// Here every CTA of one cluster copies its share of the matrices (columns as
// 16 bits, values in FP64, in the engine's run layout) and the tile records
// into shared memory once per batch and keeps a full copy of each gathered
// vector (x_hat and y; w, w_bar, tempv and y_bar with Q) there, so the chain
// of a half-step is shared-memory latency: the rows' epilogue inputs are
// requested from L2 before the row sums and arrive behind them.  A row's new
// value is stored into every CTA's copy (distributed shared memory), and one
// cluster barrier ends the half-step.
//
// Tile t belongs to CTA t mod C and within it to warp (t / C) mod kResWarps.
// Sums, projections and their order are the engine's (hpr_engine.cuh), so the
// iterates are the engine's to the bit.
#include <algorithm>
#include <map>
#include <mutex>
#include <set>
#include <tuple>
#include <vector>

#include "hpr_epilogues.cuh"

namespace hpr {

namespace {

constexpr int kResWarps = 16;
constexpr int kResThreads = kResWarps * 32;
constexpr int kResMaxCtas = 16;
constexpr int kResSmemMax = 226 * 1024;  // with the static reduction arrays within 227 KB
constexpr int kResUnroll = 4;  // nonzeros per lane per step

__host__ __device__ inline int pad_steps(int n) { return (n + kResUnroll - 1) / kResUnroll * kResUnroll; }

struct ResTile {
  int32_t rb, nrows, nnz, soff;  // soff: first slot in this CTA's arrays
  uint64_t nonempty;
  int16_t kind, ncones;
  int32_t cone, group, part;
};
static_assert(sizeof(ResTile) == 40, "ResTile layout");

// cone layout of a tile of whole cones: row of each row's cone head, first
// row of each cone (+ end)
struct ResCones {
  uint8_t head[kRowCap];
  uint8_t start[kRowCap + 4];
};

struct ResSide {
  const Task* tasks;
  const TileRun* runs;
  const uint64_t* desc;
  const int32_t* tcol;
  const double* tval;
  const int32_t* cone_start;
  const BigCone* big;
  double *raw, *cpart;
  int32_t ntasks, nwork, nbig;  // tasks, tasks before the apply tiles, split cones
  int32_t o_val, o_desc, o_tile, o_cone, o_col;  // byte offsets in shared memory
};

// One half-step: epilogue, matrix side, gathered vector and the vector the
// next half-steps gather (shared-memory copies at byte offsets gin / gout;
// the global vector is kept too).
template <class E>
struct RStage {
  E e;
  int side, gin, gout;
  double* gglob;
  int on;
  double* slots;  // reduction slots of the side's tiles (epilogues with reductions)
};

struct NoStage {};  // a half-step that the problem does not have
template <>
struct RStage<NoStage> {};

// The residual check after a batch (compute_residuals!): the half-steps of
// launch_residuals and where their lanes go.
struct ResCheck {
  RStage<EpiPlain> qx;
  RStage<EpiRd> rd;
  RStage<EpiRp> rp;
  const double *x_bar, *y_bar;
  int n, m, on;
  int slots_x, slots_y;
  double* partial;  // chunk sums of a two-level reduction
  double* out;      // Rd lanes at 0, Rp lanes at 8
};

struct ResArgs {
  ResSide side[3];  // A', A, Q
  int nsides;
  const double* g0;  // vector gathered by the first half-step
  int g0_off, g0_len;
  int o_state, o_ws;
  DevState* st;
  int iters, full_last;
};

struct ResWs {
  double acc[kRowCap + 32];  // as WarpSmem
  double sq[kRowCap];        // squares of the raw cone values; a cone's norm at its first row
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

// All CTAs of the cluster (a CTA barrier when the cluster is one CTA); the
// writes before it, local, remote and global, are visible after it.
__device__ __forceinline__ void res_sync(uint32_t C) {
  if (C == 1) {
    __syncthreads();
  } else {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

__device__ __forceinline__ void st_remote(uint32_t local_addr, uint32_t rank, double v) {
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(local_addr), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
}

// ||tail||_2 of the cone in rows [c0, c1) of a tile from the squares at sq, in
// ascending order as the reference adds them (eight loaded ahead of their
// additions).
__device__ __forceinline__ double cone_norm(uint32_t sq, int c0, int c1) {
  double ss = 0.0;
  int r = c0 + 1;
  for (; r + 8 <= c1; r += 8) {
    double q[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) q[u] = lds_f64(sq + 8 * (r + u));
#pragma unroll
    for (int u = 0; u < 8; ++u) ss = ss + q[u];
  }
  for (; r < c1; ++r) ss = ss + lds_f64(sq + 8 * r);
  return sqrt(ss);
}

__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}
// the epilogue output that later half-steps gather goes to the CTA's copy
__device__ __forceinline__ void gather_out(EpiX& e, double* p) { e.x_hat = p; }
__device__ __forceinline__ void gather_out(EpiQX& e, double* p) { e.w_bar = p; }
__device__ __forceinline__ void gather_out(EpiQT& e, double* p) { e.tempv = p; }
__device__ __forceinline__ void gather_out(EpiW2& e, double* p) { e.w = p; }
__device__ __forceinline__ void gather_out(EpiY& e, double* p) {
  if (e.ybar_always) e.y_bar = p;  // with Q the w2 half-step gathers y_bar
  else e.y = p;
}
__device__ __forceinline__ void gather_out(EpiPlain& e, double* p) { e.out = p; }
__device__ __forceinline__ void gather_out(EpiScale& e, double* p) { e.out = p; }
__device__ __forceinline__ void gather_out(EpiPow& e, double* p) { e.out = p; }
__device__ __forceinline__ void gather_out(EpiRd&, double*) {}
__device__ __forceinline__ void gather_out(EpiRp&, double*) {}
__device__ __forceinline__ void set_full(EpiPlain&, int) {}
__device__ __forceinline__ void set_full(EpiScale&, int) {}
__device__ __forceinline__ void set_full(EpiPow&, int) {}
__device__ __forceinline__ void set_full(EpiRd&, int) {}
__device__ __forceinline__ void set_full(EpiRp&, int) {}
__device__ __forceinline__ void set_full(EpiX& e, int f) { e.full = f; }
__device__ __forceinline__ void set_full(EpiY& e, int f) { e.full = f; }
__device__ __forceinline__ void set_full(EpiQX& e, int f) { e.full = f; }
__device__ __forceinline__ void set_full(EpiQT&, int) {}
__device__ __forceinline__ void set_full(EpiW2& e, int f) { e.full = f; }

// epilogue inputs through L2: another CTA may have written them
template <class Epi, int N = Epi::kSlots>
__device__ __forceinline__ void load_vals_l2(Vals<Epi::kSlots>& o, const Epi& epi, bool cone, int64_t i) {
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double* p = cone ? epi.cone_src[k] : epi.lin_src[k];
    o.v[k] = p ? __ldcg(p + i) : 0.0;
  }
}

// The reduction lanes of a tile to its slot.
template <class E>
__device__ __forceinline__ void put_red(double* slots, int slot, Red& red) {
  if constexpr (E::kNRed > 0) {
    warp_reduce<E::kNRed, E::kMaxMask>(red);
    if ((threadIdx.x & 31) == 0)
      for (int k = 0; k < E::kNRed; ++k) slots[(int64_t)slot * kMaxRed + k] = red.v[k];
  }
}

// Copies this CTA's tiles of one side into shared memory.
__device__ void load_side(const ResSide& s, unsigned char* sm, uint32_t rank, uint32_t C) {
  const int lane = threadIdx.x & 31;
  double* val = reinterpret_cast<double*>(sm + s.o_val);
  uint16_t* col = reinterpret_cast<uint16_t*>(sm + s.o_col);
  uint64_t* desc = reinterpret_cast<uint64_t*>(sm + s.o_desc);
  ResTile* tiles = reinterpret_cast<ResTile*>(sm + s.o_tile);
  ResCones* cones = reinterpret_cast<ResCones*>(sm + s.o_cone);
  for (int j = threadIdx.x >> 5; (int)rank + (int)C * j < s.nwork; j += kResWarps) {
    const int t = (int)rank + (int)C * j;
    const Task tk = s.tasks[t];
    const TileRun tr = s.runs[t];
    if (lane == 0) {
      ResTile x;
      x.rb = tk.rb;
      x.nrows = tk.re - tk.rb;
      x.nnz = tk.nze - tk.nzb;
      x.soff = tr.soff;
      x.nonempty = tr.nonempty;
      x.kind = tk.kind;
      x.ncones = tk.ncones;
      x.cone = tk.cone;
      x.group = tk.group;
      x.part = tk.part;
      tiles[j] = x;
    }
    desc[32 * j + lane] = s.desc[(int64_t)t * 32 + lane];
    for (int k = lane; k < tk.ncones; k += 32) {
      const int c0 = s.cone_start[tk.cone + k] - tk.rb, c1 = s.cone_start[tk.cone + k + 1] - tk.rb;
      cones[j].start[k] = (uint8_t)c0;
      if (k == tk.ncones - 1) cones[j].start[k + 1] = (uint8_t)c1;
      for (int r = c0; r < c1; ++r) cones[j].head[r] = (uint8_t)c0;
    }
    // the tile's steps, the last group padded with zeros
    const int steps = (tk.nze - tk.nzb + 31) >> 5, all = pad_steps(steps);
#pragma unroll 4
    for (int k = 0; k < all; ++k) {
      val[tr.soff + 32 * k + lane] = k < steps ? __ldcs(s.tval + tr.sbase + 32 * k + lane) : 0.0;
      col[tr.soff + 32 * k + lane] = k < steps ? (uint16_t)__ldcs(s.tcol + tr.sbase + 32 * k + lane) : (uint16_t)0;
    }
  }
}

// The value rows lane (and lane + 32) wrote to the gathered copy: to the
// global vector and to the other CTAs' copies.
__device__ __forceinline__ void publish_rows(double* gout, double* gglob, int rb, int nrows, uint32_t rank,
                                             uint32_t C) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 0; h < kRowCap / 32; ++h) {
    const int r = lane + 32 * h;
    if (r < nrows) {
      const double v = gout[rb + r];
      gglob[rb + r] = v;
      if (C > 1) {
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(gout + rb + r);
        for (uint32_t q = 1; q < C; ++q) st_remote(a, (rank + q) & (C - 1), v);
      }
    }
  }
}

// Row sums of a tile (process_warp_tile's steps 1 to 3).  The loads are not
// conditional (padding is value 0, column 0, and its product is not used) and
// go through 32-bit shared addresses (us per iteration with a branch around each
// load / through generic pointers / as here: n = 401 5.8 / 6.0 / 5.7, n = 2000
// 11.9 / 12.2 / 11.5).
__device__ __forceinline__ void run_sums(uint32_t val, uint32_t col, uint32_t xs, int nnz, uint64_t desc,
                                         uint64_t nonempty, uint32_t acc, double& acc0, double& acc1) {
  const int lane = threadIdx.x & 31;
  const int R = (nnz + 31) >> 5;
  int my = nnz - lane * R;
  my = my < 0 ? 0 : (my > R ? R : my);
  const uint32_t heads = (uint32_t)desc;
  const int j0 = (int)(desc >> kDescOrdShift);
  double sum = 0.0;
  uint32_t next = acc + 8 * j0;                    // slot of the next row to start
  uint32_t close = acc + 8 * (kRowCap + lane);     // where the segment being summed goes
  for (int k0 = 0; k0 < R; k0 += kResUnroll) {
    uint32_t c[kResUnroll];
    double v[kResUnroll], x[kResUnroll];
#pragma unroll
    for (int u = 0; u < kResUnroll; ++u) {
      c[u] = lds_u16(col + 64 * u);
      v[u] = lds_f64(val + 256 * u);
    }
#pragma unroll
    for (int u = 0; u < kResUnroll; ++u) x[u] = lds_f64(xs + 8 * c[u]);
    const uint32_t hb = heads >> k0;
#pragma unroll
    for (int u = 0; u < kResUnroll; ++u) {
      const double q = v[u] * x[u];
      const bool head = (hb >> u) & 1u;
      if (head) {
        sts_f64(close, sum);
        close = next;
        next += 8;
      }
      sum = (head ? 0.0 : sum) + (k0 + u < my ? q : 0.0);
    }
    col += 64 * kResUnroll;
    val += 256 * kResUnroll;
  }
  if (my > 0) sts_f64(close, sum);
  // rows that span runs: segmented scan of the continuations, then added to
  // the row's head segment (as the engine)
  {
    const bool has_cont = my > 0 && !(heads & 1u);
    if (__any_sync(0xffffffffu, has_cont)) {
      const int key = has_cont ? j0 - 1 : -2 - lane;
      double v = has_cont ? lds_f64(acc + 8 * (kRowCap + lane)) : 0.0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int ok = __shfl_up_sync(0xffffffffu, key, d);
        const bool add = lane >= d && ok == key;
        if (!__any_sync(0xffffffffu, add)) break;
        const double o = __shfl_up_sync(0xffffffffu, v, d);
        if (add) v = o + v;
      }
      const int nk = __shfl_down_sync(0xffffffffu, key, 1);
      __syncwarp();
      if (has_cont && (lane == 31 || nk != key)) sts_f64(acc + 8 * key, lds_f64(acc + 8 * key) + v);
    }
    __syncwarp();
  }
  {
    const unsigned lt = (1u << lane) - 1u;
    const uint64_t ne = nonempty;
    const unsigned b0 = (unsigned)(ne & 0xffffffffull), b1 = (unsigned)(ne >> 32);
    if ((b0 >> lane) & 1u) acc0 = lds_f64(acc + 8 * __popc(b0 & lt));
    if ((b1 >> lane) & 1u) acc1 = lds_f64(acc + 8 * (__popc(b0) + __popc(b1 & lt)));
    __syncwarp();
  }
}

// One tile with nonzeros: row sums, then the epilogue (whole rows and cones)
// or the raw values and norm share (a slice of a split cone).
template <class E>
__device__ __forceinline__ void res_tile(const ResSide& s, unsigned char* sm, E& epi, int j, uint32_t xs,
                                         ResWs& ws, double* gout, double* gglob, double* slots, uint32_t rank, uint32_t C) {
  const int lane = threadIdx.x & 31;
  const ResTile* tp = reinterpret_cast<const ResTile*>(sm + s.o_tile) + j;
  const int rb = tp->rb, nrows = tp->nrows;
  const uint64_t desc = reinterpret_cast<const uint64_t*>(sm + s.o_desc)[32 * j + lane];
  const bool part = tp->kind == TASK_CONE_PART;
  const bool cone = E::kCones && (part || tp->cone >= 0);
  Vals<E::kSlots> v0, v1;
  if (lane < nrows) load_vals_l2<E>(v0, epi, cone, rb + lane);
  if (lane + 32 < nrows) load_vals_l2<E>(v1, epi, cone, rb + lane + 32);
  const uint32_t smb = (uint32_t)__cvta_generic_to_shared(sm);
  const uint32_t val = smb + s.o_val + 8 * (tp->soff + lane), col = smb + s.o_col + 2 * (tp->soff + lane);
  double acc0 = 0.0, acc1 = 0.0;  // sums of rows rb + lane and rb + lane + 32
  run_sums(val, col, xs, tp->nnz, desc, tp->nonempty, (uint32_t)__cvta_generic_to_shared(ws.acc), acc0, acc1);
  Red red;
  red_init<E::kNRed, E::kMaxMask>(red);
  if (!cone) {
    if (lane < nrows) epi.linear(rb + lane, acc0, v0, red);
    if (lane + 32 < nrows) epi.linear(rb + lane + 32, acc1, v1, red);
  } else if (part) {
    // raw values and this slice's share of ||tail||^2 (big_norm_share)
    const int head = s.big[tp->group].rb;
    double sq = 0.0;
    if (lane < nrows) {
      const double r = epi.cone_raw(rb + lane, acc0, v0, red);
      s.raw[rb + lane] = r;
      if (rb + lane != head) sq = r * r;
    }
    if (lane + 32 < nrows) {
      const double r = epi.cone_raw(rb + lane + 32, acc1, v1, red);
      s.raw[rb + lane + 32] = r;
      if (rb + lane + 32 != head) sq = sq + r * r;
    }
    const double tot = warp_sum_bcast(sq);
    if (lane == 0) s.cpart[s.big[tp->group].part_base + tp->part] = tot;
    put_red<E>(slots, (int)rank + (int)C * j, red);
    return;
  } else {
    const ResCones& cn = reinterpret_cast<const ResCones*>(sm + s.o_cone)[j];
    const uint32_t raw = smem_addr(ws.acc), sqa = smem_addr(ws.sq);
    double w0 = 0.0, w1 = 0.0;
    if (lane < nrows) {
      w0 = epi.cone_raw(rb + lane, acc0, v0, red);
      sts_f64(raw + 8 * lane, w0);
      sts_f64(sqa + 8 * lane, w0 * w0);
    }
    if (lane + 32 < nrows) {
      w1 = epi.cone_raw(rb + lane + 32, acc1, v1, red);
      sts_f64(raw + 8 * (lane + 32), w1);
      sts_f64(sqa + 8 * (lane + 32), w1 * w1);
    }
    __syncwarp();
    // one lane per cone
    for (int k = lane; k < tp->ncones; k += 32) {
      const int c0 = cn.start[k], c1 = cn.start[k + 1];
      sts_f64(sqa + 8 * c0, cone_norm(sqa, c0, c1));
    }
    __syncwarp();
    if (lane < nrows) {
      const int h = cn.head[lane];
      epi.cone_apply(rb + lane, w0, lds_f64(raw + 8 * h), lds_f64(sqa + 8 * h), lane == h, v0, red);
    }
    if (lane + 32 < nrows) {
      const int r = lane + 32, h = cn.head[r];
      epi.cone_apply(rb + r, w1, lds_f64(raw + 8 * h), lds_f64(sqa + 8 * h), r == h, v1, red);
    }
    __syncwarp();
  }
  put_red<E>(slots, (int)rank + (int)C * j, red);
  if (gglob) publish_rows(gout, gglob, rb, nrows, rank, C);
}

// Projection of 64 rows of a split cone, after the barrier that follows its
// slices: every apply tile adds the shares itself, in publish_big_norm's
// order.
template <class E>
__device__ __forceinline__ void res_apply(const ResSide& s, E& epi, int t, double* gout, double* gglob, double* slots,
                                          uint32_t rank, uint32_t C) {
  const int lane = threadIdx.x & 31;
  const Task tk = s.tasks[t];
  const BigCone bc = s.big[tk.group];
  const int nrows = tk.re - tk.rb;
  Vals<E::kSlots> v0, v1;
  double rv0 = 0.0, rv1 = 0.0;
  constexpr int kN = ApplySlots<E>::value;
  if (lane < nrows) {
    load_vals_l2<E, kN>(v0, epi, true, tk.rb + lane);
    rv0 = __ldcg(s.raw + tk.rb + lane);
  }
  if (lane + 32 < nrows) {
    load_vals_l2<E, kN>(v1, epi, true, tk.rb + lane + 32);
    rv1 = __ldcg(s.raw + tk.rb + lane + 32);
  }
  double part = 0.0;
  for (int q = lane; q < bc.nparts; q += 32) part = part + __ldcg(s.cpart + bc.part_base + q);
  const double tv = __ldcg(s.raw + bc.rb);
  const double ns = sqrt(warp_sum_bcast(part));
  Red red;
  red_init<E::kNRed, E::kMaxMask>(red);
  if (lane < nrows) epi.cone_apply(tk.rb + lane, rv0, tv, ns, tk.rb + lane == bc.rb, v0, red);
  if (lane + 32 < nrows) epi.cone_apply(tk.rb + lane + 32, rv1, tv, ns, tk.rb + lane + 32 == bc.rb, v1, red);
  put_red<E>(slots, t, red);
  if (gglob) publish_rows(gout, gglob, tk.rb, nrows, rank, C);
}

__device__ __forceinline__ void res_stage(const RStage<NoStage>&, const ResArgs&, unsigned char*, const DevState*,
                                          bool, ResWs&, uint32_t, uint32_t) {}
template <class E>
__device__ __forceinline__ void res_stage(const RStage<E>& st, const ResArgs& a, unsigned char* sm,
                                          const DevState* cur, bool last, ResWs& ws, uint32_t rank, uint32_t C) {
  if (!st.on) return;
  const ResSide& s = a.side[st.side];
  E e = st.e;
  double* gout = reinterpret_cast<double*>(sm + st.gout);
  const uint32_t xs = (uint32_t)__cvta_generic_to_shared(sm + st.gin);
  set_full(e, last ? 1 : 0);
  gather_out(e, gout);
  e.setup(cur);
  for (int j = threadIdx.x >> 5; (int)rank + (int)C * j < s.nwork; j += kResWarps)
    res_tile<E>(s, sm, e, j, xs, ws, gout, st.gglob, st.slots, rank, C);
  if constexpr (E::kNRed > 0) {
    // the split cones' own slots carry nothing (their rows' terms are the tiles')
    if (rank == 0)
      for (int q = threadIdx.x; q < (E::kCones ? s.nbig : s.ntasks - s.nwork + s.nbig) * kMaxRed; q += kResThreads)
        st.slots[(int64_t)(E::kCones ? s.ntasks : s.nwork) * kMaxRed + q] = 0.0;
  }
  if constexpr (E::kCones) {
    if (s.nbig > 0) {
      res_sync(C);
      for (int j = threadIdx.x >> 5; s.nwork + (int)rank + (int)C * j < s.ntasks; j += kResWarps)
        res_apply<E>(s, e, s.nwork + (int)rank + (int)C * j, gout, st.gglob, st.slots, rank, C);
    }
  }
  res_sync(C);
}

// Slots b to e in final_reduce_kernel's order (kThreads strides, then the
// block's warps), by the first kThreads threads of one CTA; every thread calls it.
template <class E>
__device__ void res_combine(const double* slots, int b, int e, double* out, double (*s_red)[kThreads / 32]) {
  Red r;
  red_init<E::kNRed, E::kMaxMask>(r);
  if (threadIdx.x < kThreads) {
    for (int q = b + threadIdx.x; q < e; q += kThreads) {
      Red o;
#pragma unroll
      for (int k = 0; k < E::kNRed; ++k) o.v[k] = __ldcg(slots + (int64_t)q * kMaxRed + k);
      red_combine<E::kNRed, E::kMaxMask>(r, o);
    }
    warp_reduce<E::kNRed, E::kMaxMask>(r);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int k = 0; k < E::kNRed; ++k) s_red[k][threadIdx.x >> 5] = r.v[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < E::kNRed; ++k) r.v[k] = s_red[k][0];
    for (int w = 1; w < kThreads / 32; ++w) {
      Red o;
#pragma unroll
      for (int k = 0; k < E::kNRed; ++k) o.v[k] = s_red[k][w];
      red_combine<E::kNRed, E::kMaxMask>(r, o);
    }
#pragma unroll
    for (int k = 0; k < E::kNRed; ++k) out[k] = r.v[k];
  }
  __syncthreads();
}

// All slots of a side, in one level or, where engine_launch takes two, in its
// chunks: the host decides on residuals that must not depend on the schedule.
template <class E>
__device__ void res_final(const double* slots, int nslots, double* partial, double* out,
                          double (*s_red)[kThreads / 32]) {
  const int g = wide_chunks(nslots);
  if (g > 0) {
    const int per = (nslots + g - 1) / g;
    for (int b = 0; b < g; ++b)
      res_combine<E>(slots, b * per, min(b * per + per, nslots), partial + (int64_t)b * kMaxRed, s_red);
    slots = partial;
    nslots = g;
  }
  res_combine<E>(slots, 0, nslots, out, s_red);
}

// The residual lanes of the batch's last (full) iterate: x_bar and y_bar
// replace the gathered copies, and the passes of launch_residuals run over
// the tiles that are already in shared memory.  (ms per solve of 150 iterations
// and 16 checks, check as separate launches / here: n = 61 1.46 / 1.31, n = 401
// 2.01 / 1.85, n = 2000 3.17 / 2.84, n = 3000 with a CSR Q 3.91 / 3.72.)
__device__ void res_check(const ResCheck& k, const ResArgs& a, unsigned char* sm, const DevState* cur, ResWs& ws,
                          uint32_t rank, uint32_t C) {
  __shared__ double s_red[kMaxRed][kThreads / 32];
  double* gx = reinterpret_cast<double*>(sm + k.rp.gin);
  double* gy = reinterpret_cast<double*>(sm + k.rd.gin);
  for (int i = threadIdx.x; i < k.n; i += kResThreads) gx[i] = __ldcg(k.x_bar + i);
  for (int i = threadIdx.x; i < k.m; i += kResThreads) gy[i] = __ldcg(k.y_bar + i);
  __syncthreads();
  res_stage(k.qx, a, sm, cur, false, ws, rank, C);
  res_stage(k.rd, a, sm, cur, false, ws, rank, C);
  res_stage(k.rp, a, sm, cur, false, ws, rank, C);
  if (rank == 0) {
    res_final<EpiRd>(k.rd.slots, k.slots_x, k.partial, k.out, s_red);
    if (k.rp.on) res_final<EpiRp>(k.rp.slots, k.slots_y, k.partial, k.out + 8, s_red);
  }
}

template <class E0, class E1, class E2, class E3>
__global__ void __launch_bounds__(kResThreads, 1)
    resident_kernel(const __grid_constant__ ResArgs a, const __grid_constant__ RStage<E0> s0,
                    const __grid_constant__ RStage<E1> s1, const __grid_constant__ RStage<E2> s2,
                    const __grid_constant__ RStage<E3> s3, const __grid_constant__ ResCheck chk) {
  extern __shared__ __align__(16) unsigned char sm[];
  const uint32_t rank = cluster_rank(), C = cluster_size();
  ResWs& ws = reinterpret_cast<ResWs*>(sm + a.o_ws)[threadIdx.x >> 5];
  DevState* st = reinterpret_cast<DevState*>(sm + a.o_state);
  for (int i = 0; i < a.nsides; ++i) load_side(a.side[i], sm, rank, C);
  {
    double* g = reinterpret_cast<double*>(sm + a.g0_off);
    for (int i = threadIdx.x; i < a.g0_len; i += kResThreads) g[i] = a.g0[i];
  }
  if (threadIdx.x == 0) st[0] = st[1] = *a.st;
  res_sync(C);
  const long long inner = st[0].inner;
  for (int it = 0; it < a.iters; ++it) {
    const bool last = a.full_last && it + 1 == a.iters;
    // the next iteration's scalars, in the copy that no warp reads now
    if (threadIdx.x == 0) st[(it + 1) & 1].inner = inner + it + 1;
    const DevState* cur = st + (it & 1);
    res_stage(s0, a, sm, cur, last, ws, rank, C);
    res_stage(s1, a, sm, cur, last, ws, rank, C);
    res_stage(s2, a, sm, cur, last, ws, rank, C);
    res_stage(s3, a, sm, cur, last, ws, rank, C);
  }
  if (chk.on) res_check(chk, a, sm, st + (a.iters & 1), ws, rank, C);
  if (rank == 0 && threadIdx.x == 0) a.st->inner = inner + a.iters;
}

// Sums of NV lanes over i < n of f(i, lane sums), in the order of a block of
// kThreads threads (block_reduce), the same bits in every thread of every CTA.
template <int NV, class F>
__device__ __forceinline__ void res_sum(int n, F f, double (*s_red)[kThreads / 32], double* out) {
  if (threadIdx.x < kThreads) {
    Red r;
    red_init<NV, 0>(r);
    for (int i = threadIdx.x; i < n; i += kThreads) f(i, r);
    warp_reduce<NV, 0>(r);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) s_red[k][threadIdx.x >> 5] = r.v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double t = s_red[k][0];
    for (int w = 1; w < kThreads / 32; ++w) t = t + s_red[k][w];
    out[k] = t;
  }
  __syncthreads();
}

// The power iteration on lambda_max(AA') with A, A' and the vectors in the
// cluster's shared memory, in the arithmetic of the kernels it stands for, to
// the bit: fused_power_kernel (kTwoPass false: q = z/|z|, z = A (A' q), lambda
// = <q, z>, err = |z - lambda q| / (|z| + lambda); every CTA holds z and q in
// full and takes the sums itself, so only the products need the cluster) and
// power_two_pass_A (kTwoPass: the norm folded into the first product and the
// sums taken by the second product's tiles).  out[0] = lambda, out[1] =
// iterations run.  (B200, ms per estimate in those kernels / here: n = 61 0.76 /
// 0.53, n = 401 1.93 / 1.04, n = 803 11.1 / 2.8, n = 2000 7.3 / 2.8, n = 3000
// 14.0 / 5.8.)
struct ResPower {
  double *z, *z2;         // iterates in global memory (z: the start vector)
  const double* nz2;      // kTwoPass: |z|^2 of the start vector
  double *lanes, *out;
  int m, maxit, slots;
  double tol;
};
template <bool kTwoPass>
__global__ void __launch_bounds__(kResThreads, 1)
    resident_power_kernel(const __grid_constant__ ResArgs a, const __grid_constant__ RStage<EpiPlain> sat,
                          const __grid_constant__ RStage<EpiPlain> sa, const __grid_constant__ RStage<EpiScale> ss,
                          const __grid_constant__ RStage<EpiPow> sp, const __grid_constant__ ResPower p) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ double s_red[kMaxRed][kThreads / 32];
  __shared__ double s_nz2;
  const uint32_t rank = cluster_rank(), C = cluster_size();
  ResWs& ws = reinterpret_cast<ResWs*>(sm + a.o_ws)[threadIdx.x >> 5];
  const DevState* st = reinterpret_cast<const DevState*>(sm + a.o_state);
  for (int i = 0; i < 2; ++i) load_side(a.side[i], sm, rank, C);
  const int m = p.m;
  double* z = reinterpret_cast<double*>(sm + sa.gout);
  for (int i = threadIdx.x; i < m; i += kResThreads) z[i] = p.z[i];
  if (kTwoPass && threadIdx.x == 0) s_nz2 = *p.nz2;
  res_sync(C);
  double lambda = 1.0;
  int it = 0;
  if constexpr (kTwoPass) {
    double nz2 = s_nz2;
    while (it < p.maxit) {
      RStage<EpiScale> s1 = ss;
      s1.e.nz2 = &s_nz2;
      res_stage(s1, a, sm, st, false, ws, rank, C);
      RStage<EpiPow> s2 = sp;
      s2.e.lin_src[0] = (it & 1) ? p.z2 : p.z;
      s2.gglob = (it & 1) ? p.z : p.z2;
      res_stage(s2, a, sm, st, false, ws, rank, C);
      if (rank == 0) res_combine<EpiPow>(sp.slots, 0, p.slots, p.lanes, s_red);
      res_sync(C);
      const double nn2 = __ldcg(p.lanes), dot = __ldcg(p.lanes + 1);
      lambda = dot / sqrt(nz2);
      const double r2 = cmax(nn2 - lambda * lambda, 0.0);
      const double err = sqrt(r2) / (sqrt(nn2) + lambda);
      nz2 = nn2;
      ++it;
      if (err < p.tol) break;
      if (threadIdx.x == 0) s_nz2 = nn2;
      res_sync(C);
    }
  } else {
    double* q = reinterpret_cast<double*>(sm + sat.gin);
    double zz = 0.0;
    res_sum<1>(m, [&](int i, Red& r) { r.v[0] = r.v[0] + z[i] * z[i]; }, s_red, &zz);
    for (; it < p.maxit; ++it) {
      const double nz = sqrt(zz);
      for (int i = threadIdx.x; i < m; i += kResThreads) q[i] = z[i] / nz;
      __syncthreads();
      res_stage(sat, a, sm, st, false, ws, rank, C);
      res_stage(sa, a, sm, st, false, ws, rank, C);
      res_sum<1>(m, [&](int i, Red& r) { r.v[0] = r.v[0] + q[i] * z[i]; }, s_red, &lambda);
      double d[2];
      res_sum<2>(m, [&](int i, Red& r) {
        const double e = z[i] - lambda * q[i];
        r.v[0] = r.v[0] + e * e;
        r.v[1] = r.v[1] + z[i] * z[i];
      }, s_red, d);
      zz = d[1];
      if (sqrt(d[0]) / (sqrt(zz) + lambda) < p.tol) break;
    }
  }
  if (rank == 0 && threadIdx.x == 0) {
    p.out[0] = lambda;
    p.out[1] = (double)it;
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
int align16(int64_t b) { return (int)((b + 15) & ~(int64_t)15); }

// Shared-memory bytes of a batch on C CTAs, with the largest CTA's slots and
// tiles per side, and the offsets (when given).
int64_t resident_layout(const Ctx* c, const ResidentShape& r, ResArgs* a, int* goff, bool with_q) {
  int64_t o = 0;
  auto take = [&](int64_t bytes) {
    const int64_t at = o;
    o = align16(o + bytes);
    return (int)at;
  };
  const int o_state = take(2 * sizeof(DevState)), o_ws = take(kResWarps * sizeof(ResWs));
  if (a) {
    a->o_state = o_state;
    a->o_ws = o_ws;
  }
  // gathered vectors: y, x_hat; with Q y_bar, w (tempv in the same place: w is
  // gathered by the first half-step only), w_bar
  const int64_t len[3] = {c->m, c->n, c->n};
  for (int k = 0; k < (with_q ? 3 : 2); ++k) {
    const int at = take(8 * std::max<int64_t>(len[k], 1));
    if (goff) goff[k] = at;
  }
  for (int i = 0; i < (with_q ? 3 : 2); ++i) {
    const int ov = take(8LL * r.slots[i]), od = take(256LL * r.tiles[i]);
    const int ot = take((int64_t)sizeof(ResTile) * r.tiles[i]), oc = take((int64_t)sizeof(ResCones) * r.tiles[i]);
    const int ocol = take(2LL * r.slots[i]);
    if (a) {
      a->side[i].o_val = ov;
      a->side[i].o_desc = od;
      a->side[i].o_tile = ot;
      a->side[i].o_cone = oc;
      a->side[i].o_col = ocol;
    }
  }
  return o;
}

int nwork_of(const Plan& p) {
  int n = (int)p.tasks.size();
  while (n > 0 && p.tasks[n - 1].kind == TASK_CONE_APPLY) --n;
  return n;
}

cudaLaunchConfig_t resident_config(int C, int64_t smem, cudaStream_t stream, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)C);
  cfg.blockDim = dim3(kResThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// The kernel's attributes are set once per device; true if a cluster of C
// CTAs with the full shared memory can run on it.
template <class K>
bool cluster_fits(int device, K kernel, int C) {
  static std::mutex mu;
  static std::set<std::pair<int, const void*>> ready;              // (device, kernel) whose attributes are set
  static std::map<std::tuple<int, const void*, int>, bool> known;  // (device, kernel, CTAs)
  std::lock_guard<std::mutex> lk(mu);
  const void* id = (const void*)kernel;
  const auto it = known.find({device, id, C});
  if (it != known.end()) return it->second;
  if (!ready.count({device, id})) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmemMax) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    ready.insert({device, id});
  }
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = resident_config(C, kResSmemMax, nullptr, attr);
  int n = 0;
  const bool ok = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
  if (!ok) (void)cudaGetLastError();
  known[{device, id, C}] = ok;
  return ok;
}

}  // namespace

// The cluster size for the context's problem and the slot offsets of its plans'
// tiles in their CTA's shared memory (TileRun.soff).  c->res.ctas is 0 when the
// problem does not fit the largest cluster or a side has a row longer than a
// tile (full copies of the gathered vectors alone limit n + m to about 25,000).
// The smallest cluster is taken that holds it with at most one tile of a side
// per warp (or 16 CTAs).  More CTAs only add barriers to the same chains, and the
// other SMs serve other contexts (measured on B200, us per iteration on 1 / 2 /
// 4 / 8 / 16 CTAs: n = 61 3.2 / 4.3 / 4.2 / 4.4 / 4.2, n = 401 5.7 / 6.1 / 6.4 /
// 6.7 / 7.1).  With more tiles than warps a warp works on one after another, and
// a problem of few nonzeros per row has many tiles in little memory (us per
// iteration in the smallest cluster that holds it / with this rule / on the
// engine: n = 3000, 2 nonzeros per row, cones of 33 13.7 / 6.3 / 10.4; n = 6000,
// cones of 3 11.1 / 6.8 / 10.6; n = 3000, diagonal Q, cones of 33 27.0 / 14.5 /
// 18.6; the other way n = 1000 in cones of 65, 22 tiles with a barrier for their
// split cones, 7.6 / 9.0 / 21.1).
void resident_plan(Ctx* c) {
  c->res = ResidentShape();
  ResidentShape r;
  if (c->n > 65536 || c->m > 65536 || (c->q_kind != HPR_Q_NONE && c->q_kind != HPR_Q_CSR)) return;
  Plan* plans[3] = {&c->planX, &c->planY, &c->planQ};
  const int ns = c->has_q ? 3 : 2;
  for (int i = 0; i < ns; ++i)
    if (!plans[i]->lng.empty()) return;
  // 10 bytes per nonzero; A is kept by rows and by columns (early out)
  if (plans[0]->tasks.empty() || (20 * c->A.nnz + 10 * c->Q.nnz) / kResMaxCtas > kResSmemMax) return;
  int most = 0;  // tiles of the largest side
  for (int i = 0; i < ns; ++i) most = std::max(most, nwork_of(*plans[i]));
  r.ctas = 1;
  while (r.ctas < kResMaxCtas && most > kResWarps * r.ctas) r.ctas *= 2;
  for (; r.ctas <= kResMaxCtas; r.ctas *= 2) {
    const int C = r.ctas;
    for (int i = 0; i < ns; ++i) {
      Plan& p = *plans[i];
      int64_t used[kResMaxCtas] = {0};
      const int nw = nwork_of(p);
      for (int t = 0; t < nw; ++t) {
        p.runs[t].soff = (int32_t)used[t % C];
        used[t % C] += 32 * (int64_t)pad_steps((p.tasks[t].nze - p.tasks[t].nzb + 31) / 32);
      }
      r.slots[i] = (int)*std::max_element(used, used + C);
      r.tiles[i] = (nw + C - 1) / C;
    }
    if (resident_layout(c, r, nullptr, nullptr, c->has_q) <= kResSmemMax) {
      c->res = r;
      return;
    }
  }
}

bool resident_eligible(const Ctx* c) {
  if (c->schedule != HPR_SCHEDULE_AUTO || c->res.ctas == 0 || c->precision != HPR_PREC_FP64) return false;
  if (c->q_kind != HPR_Q_NONE && c->q_kind != HPR_Q_CSR) return false;
  return c->has_q ? cluster_fits(c->device, resident_kernel<EpiQX, EpiQT, EpiY, EpiW2>, c->res.ctas)
                  : cluster_fits(c->device, resident_kernel<EpiX, EpiY, NoStage, NoStage>, c->res.ctas);
}

namespace {
struct ResDotF {
  const double* a;
  __device__ void operator()(int64_t i, Red& r) const { r.v[0] = r.v[0] + a[i] * a[i]; }
};

// The matrices and tiles of the first `ns` sides.
void resident_sides(const Ctx* c, int ns, ResArgs& a) {
  const Plan* plans[3] = {&c->planX, &c->planY, &c->planQ};
  const int32_t* cs[3] = {c->d_var_start, c->d_con_start, c->d_var_start};
  a.nsides = ns;
  for (int i = 0; i < ns; ++i) {
    const PlanView v = view_of(*plans[i], cs[i]);
    ResSide& s = a.side[i];
    s.tasks = v.tasks;
    s.runs = v.runs;
    s.desc = v.desc;
    s.tcol = v.tcol;
    s.tval = v.tval;
    s.cone_start = v.cone_start;
    s.big = v.big;
    s.raw = v.raw;
    s.cpart = v.cpart;
    s.ntasks = v.ntasks;
    s.nwork = nwork_of(*plans[i]);
    s.nbig = v.nbig;
  }
}
}  // namespace

int launch_resident_power(Ctx* c, int maxit, double tol, double* lam, bool* done) {
  *done = false;
  if (c->schedule != HPR_SCHEDULE_AUTO || c->res.ctas == 0 || c->m == 0) return HPR_OK;
  const bool two = !(one_cta_plan(c->planX) && one_cta_plan(c->planY));
  const int slots = c->planY.nslots();
  if (two && wide_chunks(slots) > 0) return HPR_OK;  // its sums are two-level there
  HPR_TRY(prepare_engine(c));
  ResArgs a = ResArgs();
  int g[3] = {0, 0, 0};
  // q behind the batch's layout without Q
  const int64_t base = resident_layout(c, c->res, &a, g, false);
  const int64_t smem = base + (two ? 0 : 8 * c->m);
  if (smem > kResSmemMax ||
      !(two ? cluster_fits(c->device, resident_power_kernel<true>, c->res.ctas)
            : cluster_fits(c->device, resident_power_kernel<false>, c->res.ctas)))
    return HPR_OK;
  resident_sides(c, 2, a);
  a.st = c->d_state;
  std::vector<double> hz(c->m);
  power_start_vector(hz, 1);
  HPR_CUDA(c, cudaMemcpyAsync(c->pz, hz.data(), c->m * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  constexpr int kOut = 40;  // result lanes: lambda and iterations, then |z|^2, |z_new|^2, <z_old, z_new>
  if (two) HPR_TRY(vec_reduce<1, 0>(c, c->m, ResDotF{c->pz}, kOut + 2));
  const ResPower p{c->pz, c->pq, c->d_red_out + kOut + 2, c->d_red_out + kOut + 3, c->d_red_out + kOut,
                   (int)c->m, maxit, slots, tol};
  EpiScale es{};
  es.out = c->ptq;
  EpiPow ep{};
  ep.lin_src[0] = ep.cone_src[0] = c->pz;
  const RStage<EpiPlain> sat{plain(c->ptq), 0, (int)base, g[1], c->ptq, 1, nullptr};
  const RStage<EpiPlain> sa{plain(c->pz), 1, g[1], g[0], c->pq, 1, nullptr};
  const RStage<EpiScale> ss{es, 0, g[0], g[1], c->ptq, 1, nullptr};
  const RStage<EpiPow> sp{ep, 1, g[1], g[0], c->pq, 1, c->d_red};
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = resident_config(c->res.ctas, smem, c->stream, attr);
  if (two) HPR_CUDA(c, cudaLaunchKernelEx(&cfg, resident_power_kernel<true>, a, sat, sa, ss, sp, p));
  else HPR_CUDA(c, cudaLaunchKernelEx(&cfg, resident_power_kernel<false>, a, sat, sa, ss, sp, p));
  c->launches++;
  HPR_CUDA(c, cudaMemcpyAsync(c->h_red_out + kOut, c->d_red_out + kOut, 2 * sizeof(double), cudaMemcpyDeviceToHost,
                              c->stream));
  HPR_CUDA(c, cudaStreamSynchronize(c->stream));
  *lam = c->h_red_out[kOut];
  *done = true;
  return HPR_OK;
}

// k iterations (the last one full when full_last) in one launch; with `check`
// (full_last only) the residual lanes of launch_residuals too, in d_red_out.
int launch_resident(Ctx* c, int64_t k, bool full_last, bool check) {
  HPR_TRY(prepare_engine(c));
  IterEpis E;
  make_iter_epis(c, false, E);
  ResArgs a = ResArgs();
  int g[3] = {0, 0, 0};
  const int64_t smem = resident_layout(c, c->res, &a, g, c->has_q);
  resident_sides(c, c->has_q ? 3 : 2, a);
  a.st = c->d_state;
  a.g0 = c->has_q ? c->w : c->y;
  a.g0_off = c->has_q ? g[1] : g[0];
  a.g0_len = (int)(c->has_q ? c->n : c->m);
  const int hy = c->m > 0 ? 1 : 0;
  ResCheck chk = ResCheck();
  if (check) {
    ResidualEpis R;
    make_residual_epis(c, R);
    const int gx = g[1], gy = g[0];  // x_bar in x_hat's (w's) place, y_bar in y's
    chk.qx = {plain(c->Qx), 2, gx, g[2], c->Qx, c->has_q ? 1 : 0, nullptr};
    chk.rd = {R.rd, 0, gy, gy, nullptr, 1, c->d_red};
    chk.rp = {R.rp, 1, gx, gx, nullptr, hy, c->d_red + (int64_t)c->planX.nslots() * kMaxRed};
    chk.x_bar = c->x_bar;
    chk.y_bar = c->y_bar;
    chk.n = (int)c->n;
    chk.m = (int)c->m;
    chk.slots_x = c->planX.nslots();
    chk.slots_y = c->planY.nslots();
    chk.partial = c->d_red2;
    chk.out = c->d_red_out + kCheckLanes;
  }
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = resident_config(c->res.ctas, smem, c->stream, attr);
  for (int64_t done = 0; done < k;) {
    a.iters = (int)std::min<int64_t>(k - done, 1 << 20);
    a.full_last = (full_last && done + a.iters == k) ? 1 : 0;
    chk.on = check && done + a.iters == k ? 1 : 0;
    if (!c->has_q) {
      const RStage<EpiX> sx{E.ex, 0, g[0], g[1], c->x_hat, 1, nullptr};
      const RStage<EpiY> sy{E.ey, 1, g[1], g[0], c->y, hy, nullptr};
      const RStage<NoStage> off;
      HPR_CUDA(c, cudaLaunchKernelEx(&cfg, resident_kernel<EpiX, EpiY, NoStage, NoStage>, a, sx, sy, off, off, chk));
    } else {
      const RStage<EpiQX> sq{E.eq, 2, g[1], g[2], c->w_bar, 1, nullptr};
      const RStage<EpiQT> st{E.et, 2, g[2], g[1], c->tempv, hy, nullptr};
      const RStage<EpiY> sy{E.ey, 1, g[1], g[0], c->y_bar, hy, nullptr};
      const RStage<EpiW2> sw{E.e2, 0, g[0], g[1], c->w, 1, nullptr};
      HPR_CUDA(c, cudaLaunchKernelEx(&cfg, resident_kernel<EpiQX, EpiQT, EpiY, EpiW2>, a, sq, st, sy, sw, chk));
    }
    c->launches++;
    done += a.iters;
  }
  return HPR_OK;
}

}  // namespace hpr
