// Several iterations of a 2D lattice per pass over HBM.
//
// A plain iteration is bound by HBM (d2q9 FP32: 74 bytes per update): the
// state is read and written once per iteration. Here a launch advances every
// node by T iterations and moves the state once. Each warp owns a strip of
// columns (one or two per lane) and marches along y: it pulls one row of the
// source snapshot, updates it, and feeds the result to the next iteration's
// update of the row below, T stages deep. What stage k+1 needs of stage k is
// held in registers -- of the populations with e_y = 0 the last row, of those
// with e_y = +1 the last two, those with e_y = -1 are used at once -- and moves
// in x by warp shuffles. Only the source rows ahead pass through shared memory,
// each warp's own (cp.async, one __syncwarp a row). Nothing is
// exchanged between warps: every stage loses one column at each edge of the
// strip, so strips overlap, and a segment of H output rows runs 2(T-1) rows
// more through its first stage.
//
// The node updates are those of the other kernels (Model::run, pair_update)
// on the same values, and 16-bit storage rounds between the stages as a
// store and a load would, so one launch of T gives the bits of T launches.
#pragma once
#include "launch_rules.h"
#include "lbm_kernels.cuh"

namespace tclb {

constexpr int ROWS_WARPS = 4;   // warps per block, each on its own
constexpr int ROWS_AHEAD = 2;   // rows staged ahead of the one updated
// Output rows per warp. Few rows give more warps (a lattice of 4096 x 1024
// has 8832 for the 3552 the GPU holds at once) and keep those that run
// together on fewer rows of HBM; the 2 rows in 10 run twice cost less (FP32
// 4096 x 1024: 8 rows 33.3 us an iteration, 16 36.3, 32 47.4; 4096 x 4096:
// 115, 120, 132).
constexpr int ROWS_HEIGHT = 8;

// A lane's one or two nodes of a population as stored.
template <class St>
struct RowPair {  // 16-bit storage: two values in a word
  typedef unsigned Raw;
  __device__ __forceinline__ static void store(typename St::T* p, Raw w) { __stcs(reinterpret_cast<unsigned*>(p), w); }
  __device__ __forceinline__ static Raw from_left(Raw w) {  // values of the nodes one to the left
    return __byte_perm(__shfl_up_sync(0xffffffffu, w, 1), w, 0x5432);
  }
  __device__ __forceinline__ static Raw from_right(Raw w) {
    return __byte_perm(w, __shfl_down_sync(0xffffffffu, w, 1), 0x5432);
  }
  __device__ __forceinline__ static F2 get(Raw w) { return F2(Pack16<St>::unpack(w)); }
  __device__ __forceinline__ static Raw put(F2 v) { return Pack16<St>::pack(v.v.x, v.v.y); }
};
template <>
struct RowPair<StoreF32> {
  typedef float2 Raw;
  __device__ __forceinline__ static void store(float* p, Raw w) { __stcs(reinterpret_cast<float2*>(p), w); }
  __device__ __forceinline__ static Raw from_left(Raw w) {
    return make_float2(__shfl_up_sync(0xffffffffu, w.y, 1), w.x);
  }
  __device__ __forceinline__ static Raw from_right(Raw w) {
    return make_float2(w.y, __shfl_down_sync(0xffffffffu, w.x, 1));
  }
  __device__ __forceinline__ static F2 get(Raw w) { return F2(w); }
  __device__ __forceinline__ static Raw put(F2 v) { return v.v; }
};
template <class St>
struct RowOne {
  typedef typename St::T Raw;
  __device__ __forceinline__ static void store(Raw* p, Raw w) { __stcs(p, w); }
  __device__ __forceinline__ static Raw from_left(Raw w) { return __shfl_up_sync(0xffffffffu, w, 1); }
  __device__ __forceinline__ static Raw from_right(Raw w) { return __shfl_down_sync(0xffffffffu, w, 1); }
};

template <int BYTES>
__device__ __forceinline__ void copy_ahead(unsigned smem, const void* p) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem), "l"(p), "n"(BYTES) : "memory");
}

// The staged rows of a warp: population i of row y from row y - e_y, and the
// node types (the word that holds them).
template <class St, int Q, bool PAIR>
struct RowRing {
  typename std::conditional_t<PAIR, RowPair<St>, RowOne<St>>::Raw f[ROWS_AHEAD + 1][Q][32];
  unsigned types[ROWS_AHEAD + 1][32];
};

template <class M, class R, class St, bool PAIR, class Raw, class AR>
__device__ __forceinline__ void rows_update(Raw (&f)[M::Q], unsigned fl, const AR& a) {
  if constexpr (PAIR) {
    using Row = RowPair<St>;
    F2 v[M::Q];
#pragma unroll
    for (int i = 0; i < M::Q; i++) v[i] = Row::get(f[i]);
    pair_update<M, St::shifted, false>(v, (flag_t)(fl & 0xffffu), (flag_t)(fl >> 16), a);
#pragma unroll
    for (int i = 0; i < M::Q; i++) f[i] = Row::put(v[i]);
  } else {
    M::template run<R, false>(f, (flag_t)fl, a, (R*)nullptr);
  }
}

// One warp's work: output rows y0 .. of one strip, T iterations from the
// source planes of P to its destination planes.
template <class M, class R, class St, int T, bool PAIR, class A, class AR>
__device__ __forceinline__ void rows_walk(const AR& a, const A& P, int strip, int y0, RowRing<St, M::Q, PAIR>& ring) {
  static_assert(M::DIM == 2 && T >= 2, "2D models, two iterations or more");
  static_assert(PAIR || !St::shifted, "one node per lane: 32- and 64-bit storage");
  using Row = std::conditional_t<PAIR, RowPair<St>, RowOne<St>>;
  using Raw = typename Row::Raw;
  constexpr int Q = M::Q, LOST = rows_lost(PAIR, T), PER = PAIR ? 2 : 1;
  const int lane = threadIdx.x & 31;
  const int nx = a.nx, ny = a.ny;
  const int x0 = strip * rows_columns(PAIR, T) - LOST + PER * lane;  // not wrapped
  const bool mine = PER * lane >= LOST && PER * lane < 32 * PER - LOST && x0 < nx;
  int x = x0 % nx;
  if (x < 0) x += nx;
  const int xm = x == 0 ? nx - 1 : x - 1, xp = x + 1 == nx ? 0 : x + 1;  // one node per lane
  const int rows = min(ROWS_HEIGHT, ny - y0) + 2 * (T - 1);
  int y = (y0 - (T - 1)) % ny;
  if (y < 0) y += ny;
  unsigned o = (unsigned)nx * (unsigned)y0 + (unsigned)x;  // node of the first output row

  // Copies ahead that pass by the registers leave the warp free to run on its
  // other values.
  auto pull = [&](int slot, int y) {
    const unsigned r0 = (unsigned)nx * (unsigned)y;
    const unsigned rm = (unsigned)nx * (unsigned)(y == 0 ? ny - 1 : y - 1);
    const unsigned rp = (unsigned)nx * (unsigned)(y + 1 == ny ? 0 : y + 1);
#pragma unroll
    for (int i = 0; i < Q; i++) {
      const unsigned r = M::ey(i) == 0 ? r0 : (M::ey(i) > 0 ? rm : rp);
      const int c = PAIR || M::ex(i) == 0 ? x : (M::ex(i) > 0 ? xm : xp);
      copy_ahead<sizeof(Raw)>((unsigned)__cvta_generic_to_shared(&ring.f[slot][i][lane]), P.src(i) + (r + (unsigned)c));
    }
    copy_ahead<4>((unsigned)__cvta_generic_to_shared(&ring.types[slot][lane]),
                  a.flags + ((r0 + (unsigned)x) & ~1u));
  };
  auto shift = [&](int i, Raw v) -> Raw {
    return M::ex(i) == 0 ? v : (M::ex(i) > 0 ? Row::from_left(v) : Row::from_right(v));
  };
  Raw e0[T - 1][Q], e1[T - 1][Q], e2[T - 1][Q];  // rows kept between the stages (entries not used vanish)
  unsigned fl[T];  // node types of the rows in flight, the lane's one or two
#pragma unroll
  for (int k = 0; k < T - 1; k++) {
#pragma unroll
    for (int i = 0; i < Q; i++) e0[k][i] = e1[k][i] = e2[k][i] = Raw();
    fl[k] = 0;
  }
  fl[T - 1] = 0;
  int ahead = 0, yr = y;  // rows staged; the row updated
  auto stage = [&]() {
    if (ahead < rows) {
      pull(ahead % (ROWS_AHEAD + 1), y);
      y = y + 1 == ny ? 0 : y + 1;
      ahead++;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");  // an empty group past the last row
  };
#pragma unroll
  for (int k = 0; k < ROWS_AHEAD; k++) stage();
  int slot = 0;
  for (int j = 0; j < rows; j++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(ROWS_AHEAD - 1) : "memory");
    __syncwarp();  // every lane's copies of this row; and all have read the row that is overwritten next
    Raw f[Q];
#pragma unroll
    for (int i = 0; i < Q; i++) f[i] = PAIR ? shift(i, ring.f[slot][i][lane]) : ring.f[slot][i][lane];
#pragma unroll
    for (int k = T - 1; k > 0; k--) fl[k] = fl[k - 1];
    if constexpr (PAIR) fl[0] = ring.types[slot][lane];
    else fl[0] = (flag_t)(ring.types[slot][lane] >> (((unsigned)nx * (unsigned)yr + (unsigned)x) & 1u ? 16 : 0));
    yr = yr + 1 == ny ? 0 : yr + 1;
    slot = slot == ROWS_AHEAD ? 0 : slot + 1;
    stage();
    rows_update<M, R, St, PAIR>(f, fl[0], a);
#pragma unroll
    for (int k = 0; k < T - 1; k++) {
      // f: row r after stage k+1; pull for stage k+2 at row r-1
      Raw g[Q];
#pragma unroll
      for (int i = 0; i < Q; i++) {
        const Raw v = shift(i, f[i]);
        if (M::ey(i) < 0) {
          g[i] = v;
        } else if (M::ey(i) == 0) {
          g[i] = e0[k][i];
          e0[k][i] = v;
        } else {
          g[i] = e2[k][i];
          e2[k][i] = e1[k][i];
          e1[k][i] = v;
        }
      }
      // rows before the stage's first are not complete: not updated, not stored
      if (j >= 2 * (k + 1)) rows_update<M, R, St, PAIR>(g, fl[k + 1], a);
#pragma unroll
      for (int i = 0; i < Q; i++) f[i] = g[i];
    }
    if (j >= 2 * (T - 1)) {
      if (mine) {
#pragma unroll
        for (int i = 0; i < Q; i++) Row::store(P.dst(i) + o, f[i]);
      }
      o += (unsigned)nx;
    }
  }
}

template <class M, class R, class St, int T, bool PAIR>
__global__ void __launch_bounds__(ROWS_WARPS * 32, sizeof(R) == 8 ? 4 : 6)
    k_iterate_rows(const Args<R, M::NSET> a, const PlaneAddr<typename St::T, M::Q> P, int strips, int nwarps) {
  __shared__ RowRing<St, M::Q, PAIR> ring[ROWS_WARPS];
  const int wid = threadIdx.x >> 5, w = blockIdx.x * ROWS_WARPS + wid;
  pdl_wait_and_release();
  if (w >= nwarps) return;
  const int seg = w / strips;
  rows_walk<M, R, St, T, PAIR>(a, P, w - seg * strips, seg * ROWS_HEIGHT, ring[wid]);
}

}  // namespace tclb
