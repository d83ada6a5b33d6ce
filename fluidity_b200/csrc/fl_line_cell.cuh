// fl_line_cell.cuh -- one 1-D cell update per lane.
//
// One sweep of SplitSolver::invoke (solver/split_solver.hpp:138-162) with the
// arithmetic of sweep_kernel (fl_sweep.cuh) on a line in shared memory: a warp
// takes 32 consecutive cells, of which its middle 24 are its own (the stencil
// reaches 4 cells); neighbours' derived values come from warp shuffles.
#pragma once

#include <cstdint>

#include "fl_internal.cuh"
#include "fl_numerics.cuh"

namespace fl {

constexpr int kLineOwn = 24;  // cells a warp updates

template <typename T>
__device__ __forceinline__ T line_up(T v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
template <typename T>
__device__ __forceinline__ T line_dn(T v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }

// New state of this lane's cell (valid on lanes 4..27), x its index in the
// planes of `src` (plane stride ld).  SCREEN: skip the flattening where no
// lane can be flattened; where all the warps of a problem meet at a barrier
// every step, the slowest of them (one that holds a shock) sets the pace and
// the screen's vote only adds to its chain.
template <typename T, int FLUX, int LIM, bool MUSCL, bool FLAT, bool SCREEN>
__device__ __forceinline__ Cons<T, 1> line_cell(const T* src, int ld, int x, T gamma, T gm1, T adi,
                                                T dtdh, T dhdt, T pinf) {
  constexpr int NC = 3;
  Cons<T, 1> u, er, el;
#pragma unroll
  for (int c = 0; c < NC; ++c) u.v[c] = src[c * ld + x];
  if constexpr (MUSCL) {
    T ch = T(0.5);
    if constexpr (FLAT) {
      const Derived<T, 1> q = derive(u, gm1);
      bool steep = true;
      if constexpr (SCREEN) {
        const uint32_t key = press_key(q.p);
        steep = __any_sync(0xffffffffu, may_flatten<T>(line_dn(key, 1), line_up(key, 1)));
      }
      if (steep) {
        const T pr = line_dn(q.p, 1), pl = line_up(q.p, 1);
        const T base = (T)chi_base<T>(pr, pl, line_dn(q.p, 2), line_up(q.p, 2),
                                      line_up(q.v[0], 1), line_dn(q.v[0], 1));
        const T br = line_dn(base, 1), bl = line_up(base, 1);
        const T dx = pr - pl;
        ch *= std_min(base, dx > T(0) ? br : (dx < T(0) ? bl : base));
      }
    }
    const int xm = x > 0 ? x - 1 : 0, xp = x + 1 < ld ? x + 1 : x;  // edge lanes: unused
    Cons<T, 1> a, b, fa, fb;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const T d = ch * limited_slope<T>(LIM, u.v[c] - src[c * ld + xm], src[c * ld + xp] - u.v[c]);
      a.v[c] = u.v[c] - d;
      b.v[c] = u.v[c] + d;
    }
    flux_q(a, derive(a, gm1), 0, fa);
    flux_q(b, derive(b, gm1), 0, fb);
    const T hd = T(0.5) * dtdh;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const T df = fa.v[c] - fb.v[c];
      er.v[c] = b.v[c] + hd * df;
      el.v[c] = a.v[c] + hd * df;
    }
  } else {
    er = u;
    el = u;
  }
  Cons<T, 1> ul, f;
#pragma unroll
  for (int c = 0; c < NC; ++c) ul.v[c] = line_up(er.v[c], 1);
  riemann_qh<FLUX>(ul, derive(ul, gm1), el, derive(el, gm1), 0, gamma, gm1, adi, dtdh, dhdt, f,
                   pinf);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const T fr = line_dn(f.v[c], 1);
    u.v[c] = u.v[c] + dtdh * (f.v[c] - fr);
  }
  return u;
}

}  // namespace fl
