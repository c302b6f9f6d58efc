// Shared-memory staged step of the 8- and 4-byte formats: the standard cavity
// (FP64 FAST; FP32 with nx even) and the sphere channel (FP64; FP32 with nx
// even), from some size on (line_supported).
//
// What bounded the register kernels here is the time a warp waits for its 27
// loads with nothing else to do: 16 warps an SM, and the cavity's wall rules
// or the sphere's mask in front of the loads.  Here a plane is one line of
// elements, rows end to end, and a tile a run of 2 KB of it (256 FP64 or 512
// FP32 cells); bulk copies bring a tile's 27 shifted runs into a stage while
// the tiles before are collided, one cell (x-pair) a thread.  A block holds
// two stages, an SM two blocks.  The last warp to have read a stage refills
// it at once, so that copies are in flight all through the collision, and
// tiles go out by tickets (take_tile): in equal shares the same kernels took
// 165 us a step against 148 (128^3 FP64 FAST cavity) and 142 against 124
// (384x96x96 FP32 sphere), since the SMs do not get equal bandwidth.
//
// us a step, start of the register kernels | here | the two buffers once
// through HBM: FP64 FAST cavity 128^3 158 | 148 | 138, 151x133x117 222 | 186
// | 155; FP32 cavity 160x144x150 169 | 122 | 114; FP32 sphere 384x96x96 199 |
// 124 | 117; FP64 EXACT sphere 384x96x96 314 | 275 | 234.  What is left is
// the last wave of tiles, and in EXACT arithmetic the FP64 pipe.
//
// Boundaries: a run that leaves the plane is wrapped (sphere) or, beyond a
// cavity wall, replaced by the tile's own elements of the opposite
// population, which the halfway bounce-back returns.  The x walls' values
// are the cell's own, nine a wall cell, loaded from global memory before the
// wait for the stage.  The sphere's mask and links are read only in the box
// around the body.
//
// Every wait on a stage gives up after StepArgs::wait_ns (a second, or the
// bound that imexlb_set_wait_limit sets), records it and lets the copies in
// flight land, as the 2-byte staged kernels do.
#include "line.h"

#include "launch.cuh"
#include "stage_core.cuh"
#include "step_core.cuh"

namespace imx {
namespace {

using namespace core;

// Which lattices step here (line_supported).  us a step, registers | staged:
//   sphere channel: FP64 EXACT 128x40x40 15.7 | 22.2, 160x44x44 29.8 | 27.8,
//     128x60x60 42.7 | 39.7, 300x70x70 130.7 | 107.2; FP32 128x40x40 10.1 |
//     10.2, 160x44x44 14.2 | 16.6, 128x60x60 23.8 | 20.0, 300x70x70 84.9 | 64.5
//   FP32 cavity: 64^3 8.8 | 10.9, 80x72x72 18.7 | 19.2, 76^3 29.5 | 27.2,
//     96x90x90 36.6 | 28.6
//   FP64 FAST cavity: 80^3 40.3 | 40.7, 96^3 66.1 | 67.6, 112x112x80 75.5 |
//     74.3, 128^3 151.7 | 148.8, 144^3 216.8 | 205.2, 160^3 288.8 | 279.0
//   FP64 EXACT cavity, whose arithmetic sets the pace: 100x70x70 40.0 | 46.5,
//     144^3 204.9 | 209.8, 192^3 476.5 | 488.4, 240^3 908.7 | 927.3: never
// 450,000 cells are seven FP64 or four FP32 tiles a block.  A plane that leaves
// its last tile mostly empty wastes the copies in flight: FP32 cavity 96x6x850
// (56 % filled) 21.0 | 25.7, 64x12x640 (75 %) 20.5 | 21.6, 112x7x640 (87 %)
// 26.4 | 20.8; FP64 FAST 16x8x4000 (50 %) 39.9 | 52.8.  The sphere, whose mask
// and links hold the registers up, gains even so (FP64 EXACT 96x6x850 48.2 |
// 47.2, FP32 64x12x640 26.0 | 23.3).
constexpr int64_t LINE_MIN_CELLS = 450000, LINE_MIN_CELLS_F64_CAVITY = 950000;
constexpr int LINE_THREADS = 256;
constexpr int LINE_STAGES = 2;
constexpr int LINE_BYTES = 2048;  // a tile's run of one population
constexpr int GUARD_BYTES = 16;   // staged on either side of it
constexpr int SLOT_BYTES = LINE_BYTES + 2 * GUARD_BYTES;

template <class T> constexpr int LINE_C = LINE_BYTES / static_cast<int>(sizeof(T));
template <class T> constexpr int LINE_G = GUARD_BYTES / static_cast<int>(sizeof(T));
template <class T> constexpr int LINE_SLOT = SLOT_BYTES / static_cast<int>(sizeof(T));
constexpr size_t LINE_SMEM = static_cast<size_t>(LINE_STAGES) * Q * SLOT_BYTES + 8 * LINE_STAGES;

struct LineGeo {
  int P, np, nty, ntiles;
  uint32_t m_P, m_nty;
  int s_P, s_nty;
};

// The copies of population q for tile [e0, e0 + n) of plane k: at most two
// runs (element offsets in their population's plane, and in the slot).
struct LineRun {
  int32_t src, dst, len, pop;
};

template <bool WRAP, int C, int G>
__host__ __device__ __forceinline__ void line_runs(const StepArgs& a, const LineGeo& g, int q, int e0, int k,
                                                   LineRun& main, LineRun& edge) {
  main.len = edge.len = 0;
  main.pop = edge.pop = q;
  const int np = g.np;
  const int n = np - e0 < C ? np - e0 : C;
  const int ey = stage::ey_of(q);
  int kk = k - stage::ez_of(q);
  if (kk < 0 || kk >= a.nz) {
    if (!WRAP) {
      main.pop = stage::bb_of(q);
      main.src = a.base32 + k * a.sz32 + e0;
      main.dst = G;
      main.len = n;
      return;
    }
    kk = kk < 0 ? kk + a.nz : kk - a.nz;
  }
  const int32_t plane = a.base32 + kk * a.sz32;
  const int32_t s0 = e0 - ey * g.P - G, s1 = e0 + n - ey * g.P + G;
  if (WRAP && (s1 <= 0 || s0 >= np)) {
    main.src = plane + (s1 <= 0 ? s0 + np : s0 - np);
    main.dst = 0;
    main.len = s1 - s0;
    return;
  }
  const int32_t lo = s0 < 0 ? 0 : s0, hi = s1 > np ? np : s1;
  if (hi > lo) {
    main.src = plane + lo;
    main.dst = lo - s0;
    main.len = hi - lo;
  }
  if (WRAP) {
    if (s0 < 0) {
      edge.src = plane + s0 + np;
      edge.dst = 0;
      edge.len = -s0;
    } else if (s1 > np) {
      edge.src = plane;
      edge.dst = np - s0;
      edge.len = s1 - np;
    }
  } else if (ey != 0) {
    // cells of the row at the wall: their own elements of bb(q)
    const int32_t c0 = ey > 0 ? e0 : (e0 > np - g.P ? e0 : np - g.P);
    const int32_t c1 = ey > 0 ? (e0 + n < g.P ? e0 + n : g.P) : e0 + n;
    if (c1 > c0) {
      edge.pop = stage::bb_of(q);
      edge.src = a.base32 + k * a.sz32 + c0;
      edge.dst = G + c0 - e0;
      edge.len = c1 - c0;
    }
  }
}

// m-th population with e_x = +1
constexpr int wall_pos(int m) {
  int n = 0;
  for (int q = 0; q < Q; ++q)
    if (D3Q27::ex[q] == 1) {
      if (n == m) return q;
      ++n;
    }
  return -1;
}
constexpr int wall_index(int q) {  // of q (e_x = +1) or bb(q) (e_x = -1)
  int n = 0;
  const int p = D3Q27::ex[q] == 1 ? q : D3Q27::bb[q];
  for (int r = 0; r < p; ++r)
    if (D3Q27::ex[r] == 1) ++n;
  return n;
}

// Adds v to a counter in shared memory, ordered with the block's other
// accesses before and after it; returns the value before.
__device__ __forceinline__ int atom_add_cta(int* p, int v) {
  int old;
  asm volatile("atom.acq_rel.cta.shared::cta.add.s32 %0, [%1], %2;"
               : "=r"(old)
               : "r"(stage::smem_addr(p)), "r"(v)
               : "memory");
  return old;
}

// Two x-neighbours of the FP32 sphere channel with the arithmetic the
// one-cell kernel gives each: cells it updates in pairs of rows (pair0 /
// pair1) in paired instructions, the others (beside a solid cell, or in an
// odd last row) alone.
template <class P>
__device__ __forceinline__ void compute_line_pair(const StepArgs& a, const P& pl, const int x, const int k,
                                                  const int32_t b, const int64_t cell, float (&f0)[Q], float (&f1)[Q],
                                                  const bool live0, const bool live1, const bool pair0,
                                                  const bool pair1) {
  const bool store = a.store != 0;
  const bool p0 = live0 && pair0, p1 = live1 && pair1;
  if (p0 || p1)
    compute_two<Store::F32, CaseRule::SphereStd, true>(a, pl, x, x + 1, k, b, b + 1, cell, cell + 1, store, f0, f1, p0,
                                                       p1);
  if (live0 && !pair0) compute_cell_at<Store::F32, CaseRule::SphereStd, false>(a, pl, x, k, b, cell, store, f0);
  if (live1 && !pair1)
    compute_cell_at<Store::F32, CaseRule::SphereStd, false>(a, pl, x + 1, k, b + 1, cell + 1, store, f1);
  if (store && !(live0 && live1)) {
    for (int c = 0; c < 2; ++c) {
      if (c == 0 ? live0 : live1) continue;
      a.mu[cell + c] = 0;
      a.mv[cell + c] = 0;
      a.mw[cell + c] = 0;
      a.mp[cell + c] = a.p_shift;
    }
  }
}

template <Store S, CaseRule RULE, bool EXACT>
__global__ void __launch_bounds__(LINE_THREADS, 2) line_kernel(const StepArgs a, const LineGeo g) {
  using T = typename StoreT<S>::T;
  using namespace stage;
  constexpr bool WRAP = RULE == CaseRule::SphereStd;
  constexpr bool PAIR = S == Store::F32;
  constexpr int C = LINE_C<T>, G = LINE_G<T>, SLOT = LINE_SLOT<T>;
  constexpr int NS = LINE_STAGES;
  extern __shared__ __align__(128) unsigned char smem[];
  T* stages = reinterpret_cast<T*>(smem);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + static_cast<size_t>(NS) * Q * SLOT_BYTES);
  __shared__ int abort_flag, issued;
  __shared__ int readers[NS];  // warps that have read the stage's tile
  __shared__ int tile_of[NS];  // the stage's tile, -1: no more
  __shared__ int tile_next[NS];  // the tile that refills the stage
  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; ++s) {
      bar_init(&full[s], 1);
      readers[s] = 0;
      tile_of[s] = -1;
    }
    abort_flag = 0;
    issued = 0;
    bar_init_fence();
  }
  pdl_wait();
  __syncthreads();
  volatile int* abort_v = &abort_flag;
  const int grid = gridDim.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Planes<T> pl{reinterpret_cast<const T* const*>(a.srcq), reinterpret_cast<T* const*>(a.dstq)};

  // A stage's phases begun, skipped ones too: those complete as well.  The warps
  // that issue follow one another through `readers`, so a plain count behind the
  // copies will do; an atomic ahead of them cost 1 to 7 % (FP32 sphere 160x60x60
  // 22.1 us a step | 22.8, FP64 cavity 16x8x4000 52.4 | 56.6).
  auto count_issue = [&] {
    volatile int* n = &issued;
    if (lane == 0) *n = *n + 1;
  };
  // (one warp) start the copies of tile t into stage sn
  auto issue = [&](int t, int sn) {
    if (lane == 0) tile_of[sn] = t < g.ntiles ? t : -1;
    __syncwarp();
    if (t >= g.ntiles) {
      issue_skip(&full[sn]);
      count_issue();
      return;
    }
    const int k = item_quotient(t, g.m_nty, g.s_nty);
    const int e0 = (t - k * g.nty) * C;
    LineRun m{0, 0, 0, 0}, w{0, 0, 0, 0};
    if (lane < Q) line_runs<WRAP, C, G>(a, g, lane, e0, k, m, w);
    uint32_t total = (m.len + w.len) * static_cast<uint32_t>(sizeof(T));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (lane == 0) bar_arrive_expect(&full[sn], total);
    __syncwarp();
    T* st = stages + sn * (Q * SLOT) + lane * SLOT;
    const T* src = static_cast<const T*>(a.src);
    if (m.len) bulk_g2s(st + m.dst, src + m.pop * a.sq + m.src, m.len * sizeof(T), &full[sn]);
    if (w.len) bulk_g2s(st + w.dst, src + w.pop * a.sq + w.src, w.len * sizeof(T), &full[sn]);
    count_issue();
  };

  if (warp == 0) {
    for (int n = 0; n < NS; ++n) issue(blockIdx.x + n * grid, n);
    if (lane == 0) {
      const int next = NS * grid + take_tiles(a.tickets, NS);
      for (int n = 0; n < NS; ++n) tile_next[n] = next + n;
    }
  }
  // this warp has read its part of stage s; the last of the block's warps to
  // say so refills the stage, and fetches the number of the tile after that
  int ticket = 0, ticket_stage = -1;
  auto release = [&](int s) {
    __syncwarp();
    int before = 0;
    if (lane == 0) before = atom_add_cta(&readers[s], 1);
    before = __shfl_sync(0xffffffffu, before, 0);
    if (before == LINE_THREADS / 32 - 1) {
      const int t = *reinterpret_cast<volatile int*>(&tile_next[s]);
      if (lane == 0) readers[s] = 0;
      __syncwarp();
      issue(t, s);
      if (t < g.ntiles) {
        if (lane == 0) ticket = NS * grid + take_tile(a.tickets);
        ticket_stage = s;
      }
    }
  };

  // the cell (the x-pair) of tile t that is this thread's
  struct Place {
    int k, e, j, x;
    bool act, lo, hi;
    int32_t b;
  };
  const int p = (PAIR ? 2 : 1) * threadIdx.x;
  auto place = [&](int t) {
    Place c;
    c.k = item_quotient(t, g.m_nty, g.s_nty);
    c.e = (t - c.k * g.nty) * C + p;
    c.j = item_quotient(c.e, g.m_P, g.s_P);
    c.x = c.e - c.j * g.P;
    c.act = c.e < g.np && c.x < a.nx;
    c.lo = c.x == 0;
    c.hi = c.x + (PAIR ? 2 : 1) >= a.nx;
    c.b = a.base32 + c.k * a.sz32 + c.e;
    return c;
  };
  // the cavity's x walls: the nine values that the halfway bounce-back
  // returns to a wall cell, from the cell's own column
  [[maybe_unused]] T wv[9];
  auto wall_values = [&](const Place& c) {
    if (c.act && (c.lo || c.hi)) {
      const int32_t bw = PAIR && c.hi ? c.b + 1 : c.b;
      static_for<0, 9>([&](auto mc) {
        constexpr int m = decltype(mc)::value;
        constexpr int qp = wall_pos(m), qm = D3Q27::bb[qp];
        wv[m] = pl.load(c.lo ? qm : qp, bw);
      });
    }
  };

  int i = 0, before1 = -1, before2 = -1;  // the tiles of the last two turns
  for (;; ++i) {
    const int s = i % NS;
    // the next tile's number is mostly there before its copies are: start
    // its wall values on their way
    [[maybe_unused]] int early = -1;
    if constexpr (RULE == CaseRule::CavityStd) {
      early = *reinterpret_cast<volatile int*>(&tile_of[s]);
      if (early == before2) early = -1;
      early = __shfl_sync(0xffffffffu, early, 0);
      if (early >= 0) wall_values(place(early));
    }
    if (!__all_sync(0xffffffffu, bar_wait_for(&full[s], (i / NS) & 1u, a.wait_ns))) {
      *abort_v = 1;
      break;
    }
    const int t = tile_of[s];
    if (t < 0) break;
    before2 = before1;
    before1 = t;
    const Place c = place(t);
    const int k = c.k, j = c.j, x = c.x;
    const bool act = c.act, lo = c.lo, hi = c.hi;
    const int32_t b = c.b;
    const int64_t cell = x + static_cast<int64_t>(a.nx) * (j + static_cast<int64_t>(a.ny) * k);
    [[maybe_unused]] uint32_t links0 = 0, links1 = 0;
    [[maybe_unused]] bool live0 = true, live1 = true;
    if constexpr (RULE == CaseRule::CavityStd) {
      if (early < 0) wall_values(c);
    } else {
      const bool near = act && in_body(a, x, PAIR ? 2 : 1, j, k);
      if (near) {
        links0 = a.links[cell];
        live0 = a.usr[cell] != 0;
        if constexpr (PAIR) {
          links1 = a.links[cell + 1];
          live1 = a.usr[cell + 1] != 0;
        }
      }
    }

    const T* st = stages + s * (Q * SLOT) + G + p;

    if constexpr (!PAIR) {
      typename StoreT<S>::R f[Q];
      if constexpr (RULE == CaseRule::CavityStd) {
        const bool y0 = j == 0, y1 = j == a.ny - 1, z0 = k == 0, z1 = k == a.nz - 1;
        if (__any_sync(0xffffffffu, act && (y0 || y1 || z0 || z1))) {
          static_for<0, Q>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int ex = D3Q27::ex[q], ey = D3Q27::ey[q], ez = D3Q27::ez[q];
            const bool out = (ey > 0 && y0) || (ey < 0 && y1) || (ez > 0 && z0) || (ez < 0 && z1);
            f[q] = st[q * SLOT - (ex != 0 && !out ? ex : 0)];
          });
        } else {
          static_for<0, Q>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int ex = D3Q27::ex[q];
            f[q] = st[q * SLOT - ex];
          });
        }
      } else {
        static_for<0, Q>([&](auto qc) {
          constexpr int q = decltype(qc)::value;
          constexpr int ex = D3Q27::ex[q];
          f[q] = ex < 0 ? st[q * SLOT + (hi ? 0 : 1)] : st[q * SLOT - ex];
        });
      }
      release(s);
      if constexpr (RULE == CaseRule::CavityStd) {
        static_for<0, Q>([&](auto qc) {
          constexpr int q = decltype(qc)::value;
          constexpr int ex = D3Q27::ex[q];
          if constexpr (ex > 0) {
            if (lo) f[q] = wv[wall_index(q)];
          } else if constexpr (ex < 0) {
            if (hi) f[q] = wv[wall_index(q)];
          }
          if constexpr (ex != 0 && D3Q27::ez[q] < 0) {
            using R = typename StoreT<S>::R;
            using A = Ar<R, EXACT>;
            constexpr int cls = D3Q27::wclass[q];
            if (k == a.nz - 1) f[q] = A::add(f[q], A::mul(A::mul(R(6.0 * a.rho_w * a.lid_u), wgt<R>(cls)), R(ex)));
          }
        });
        if (act) compute_cell_at<S, RULE, EXACT>(a, pl, x, k, b, cell, a.store != 0, f);
      } else {
        if (__any_sync(0xffffffffu, links0 != 0)) {
          static_for<0, Q>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int qb = D3Q27::bb[q];
            if ((links0 >> q) & 1u) f[q] = pl.load(qb, b);
          });
        }
        if (lo) {
          static_for<0, Q>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            if constexpr (D3Q27::ex[q] > 0) f[q] = typename StoreT<S>::R(a.feq_in[q]);
          });
        }
        if (act && live0) compute_cell_at<S, RULE, EXACT>(a, pl, x, k, b, cell, a.store != 0, f);
        if (act && !live0 && a.store) {
          a.mu[cell] = 0;
          a.mv[cell] = 0;
          a.mw[cell] = 0;
          a.mp[cell] = a.p_shift;
        }
      }
    } else if constexpr (RULE == CaseRule::CavityStd) {
      uint2 raw[Q];
      const bool y0 = j == 0, y1 = j == a.ny - 1, z0 = k == 0, z1 = k == a.nz - 1;
      auto word = [&](int q, int d) { return __float_as_uint(st[q * SLOT + d]); };
      if (__any_sync(0xffffffffu, act && (y0 || y1 || z0 || z1))) {
        static_for<0, Q>([&](auto qc) {
          constexpr int q = decltype(qc)::value;
          constexpr int ex = D3Q27::ex[q], ey = D3Q27::ey[q], ez = D3Q27::ez[q];
          const bool out = (ey > 0 && y0) || (ey < 0 && y1) || (ez > 0 && z0) || (ez < 0 && z1);
          const int d = ex != 0 && !out ? -ex : 0;
          raw[q] = make_uint2(word(q, d), word(q, d + 1));
        });
      } else {
        static_for<0, Q>([&](auto qc) {
          constexpr int q = decltype(qc)::value;
          constexpr int ex = D3Q27::ex[q];
          if constexpr (ex == 0) {
            raw[q] = *reinterpret_cast<const uint2*>(st + q * SLOT);
          } else {
            raw[q] = make_uint2(word(q, -ex), word(q, 1 - ex));
          }
        });
      }
      release(s);
      static_for<0, Q>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        constexpr int ex = D3Q27::ex[q];
        if constexpr (ex > 0) {
          if (lo) raw[q].x = __float_as_uint(wv[wall_index(q)]);
        } else if constexpr (ex < 0) {
          if (hi) raw[q].y = __float_as_uint(wv[wall_index(q)]);
        }
      });
      if (act)
        finish_pair_at<S, RULE, false, false>(a, pl, raw, x, k, b, cell, k == a.nz - 1, lo, true, true, a.store != 0,
                                              0u);
    } else {
      // FP32 sphere: the one-cell kernel's arithmetic, two cells along x
      float f0[Q], f1[Q];
      static_for<0, Q>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        constexpr int ex = D3Q27::ex[q];
        f0[q] = st[q * SLOT - ex];
        f1[q] = ex < 0 ? st[q * SLOT + (hi ? 1 : 2)] : st[q * SLOT + 1 - ex];
      });
      release(s);
      // the rows the one-cell kernel pairs: (j0, j0 + 1), j0 even
      bool pair0 = true, pair1 = true;
      if ((j ^ 1) >= a.ny) {
        pair0 = pair1 = false;
      } else if (act && in_body(a, x, 2, j ^ 1, k)) {
        const int64_t other = cell + ((j & 1) ? -a.nx : a.nx);
        pair0 = a.usr[other] != 0;
        pair1 = a.usr[other + 1] != 0;
      }
      if (__any_sync(0xffffffffu, (links0 | links1) != 0)) {
        static_for<0, Q>([&](auto qc) {
          constexpr int q = decltype(qc)::value;
          constexpr int qb = D3Q27::bb[q];
          if ((links0 >> q) & 1u) f0[q] = pl.load(qb, b);
          if ((links1 >> q) & 1u) f1[q] = pl.load(qb, b + 1);
        });
      }
      if (lo) {
        static_for<0, Q>([&](auto qc) {
          constexpr int q = decltype(qc)::value;
          if constexpr (D3Q27::ex[q] > 0) f0[q] = static_cast<float>(a.feq_in[q]);
        });
      }
      if (act) {
        compute_line_pair(a, pl, x, k, b, cell, f0, f1, live0, live1, pair0, pair1);
      }
    }

    if (ticket_stage >= 0) {
      if (lane == 0) tile_next[ticket_stage] = ticket;
      ticket_stage = -1;
    }
    if (__any_sync(0xffffffffu, *abort_v != 0)) break;
  }
  pdl_release();
  __syncthreads();
  if (abort_flag && warp == 0 && lane == 0) {
    // let copies still in flight land before the block exits: each stage's
    // last phase (bounded by the full second whatever a.wait_ns is)
    for (int m = issued > NS ? issued - NS : 0; m < issued; ++m) (void)bar_wait(&full[m % NS], (m / NS) & 1u);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (abort_flag) atomicOr(a.err, 1);
    finish_tiles(a.tickets);
  }
}

template <class T>
bool line_geo(bool wrap, int nx, int ny, int nz, int64_t pitch, LineGeo* g) {
  constexpr int C = LINE_C<T>, G = LINE_G<T>;
  const int64_t np = pitch * ny;
  if (nx < 4 || np > (int64_t(1) << 30)) return false;
  if (wrap && np < C + 2 * pitch + 2 * G) return false;
  g->P = static_cast<int>(pitch);
  g->np = static_cast<int>(np);
  g->nty = static_cast<int>((np + C - 1) / C);
  if (static_cast<int64_t>(g->nty) * nz > (int64_t(1) << 30)) return false;
  g->ntiles = g->nty * nz;
  item_magic(g->P, &g->m_P, &g->s_P);
  item_magic(g->nty, &g->m_nty, &g->s_nty);
  return true;
}

template <Store S, CaseRule RULE, bool EXACT>
cudaError_t launch_line_impl(const StepArgs& a, cudaStream_t s) {
  using T = typename StoreT<S>::T;
  LineGeo g;
  if (!line_geo<T>(RULE == CaseRule::SphereStd, a.nx, a.ny, a.nz, a.pitch, &g)) return cudaErrorInvalidValue;
  static PerDevice known;
  int resident = 0;
  if (const cudaError_t e = resident_blocks(known, line_kernel<S, RULE, EXACT>, LINE_THREADS, LINE_SMEM, &resident))
    return e;
  const int blocks = g.ntiles < resident ? g.ntiles : resident;
  return launch_pdl(line_kernel<S, RULE, EXACT>, dim3(blocks), dim3(LINE_THREADS), LINE_SMEM, s, a, g);
}

}  // namespace

template <class T>
static int64_t line_plan_impl(bool wrap, int nx, int ny, int nz, int32_t* geo, int32_t* runs, int64_t max_runs) {
  constexpr int C = LINE_C<T>, G = LINE_G<T>;
  const Layout L = make_layout(nx, ny, nz, 0, static_cast<int>(sizeof(T)));
  LineGeo g;
  if (!line_geo<T>(wrap, nx, ny, nz, L.pitch, &g)) return -1;
  StepArgs a;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.base32 = static_cast<int32_t>(L.idx(0, 0, 0, 0));
  a.sz32 = static_cast<int32_t>(L.sz);
  const int32_t v[8] = {g.P, g.nty, C, G, LINE_SLOT<T>, a.base32, a.sz32, static_cast<int32_t>(L.sq)};
  for (int i = 0; i < 8; ++i) geo[i] = v[i];
  int64_t n = 0;
  for (int t = 0; t < g.ntiles; ++t) {
    const int k = item_quotient(t, g.m_nty, g.s_nty), e0 = (t - k * g.nty) * C;
    for (int q = 0; q < Q; ++q) {
      LineRun m, w;
      if (wrap)
        line_runs<true, C, G>(a, g, q, e0, k, m, w);
      else
        line_runs<false, C, G>(a, g, q, e0, k, m, w);
      for (const LineRun* r : {&m, &w}) {
        if (!r->len) continue;
        if (n < max_runs) {
          const int32_t o[6] = {t, q, r->pop, r->src, r->dst, r->len};
          for (int i = 0; i < 6; ++i) runs[6 * n + i] = o[i];
        }
        ++n;
      }
    }
  }
  return n;
}

int64_t line_plan(int nx, int ny, int nz, bool wrap, int elem, int32_t* geo, int32_t* runs, int64_t max_runs) {
  return elem == 8 ? line_plan_impl<double>(wrap, nx, ny, nz, geo, runs, max_runs)
                   : line_plan_impl<float>(wrap, nx, ny, nz, geo, runs, max_runs);
}

bool line_supported(const LaunchCfg& c, int nx, int ny, int nz, int64_t pitch) {
  if (c.bc != Bc::Standard || (c.rule != CaseRule::CavityStd && c.rule != CaseRule::SphereStd)) return false;
  LineGeo g;
  const bool wrap = c.rule == CaseRule::SphereStd;
  if (c.store == Store::F64) {
    if (!line_geo<double>(wrap, nx, ny, nz, pitch, &g)) return false;
  } else if (c.store != Store::F32 || nx % 2 != 0 || !line_geo<float>(wrap, nx, ny, nz, pitch, &g)) {
    return false;
  }
  const int64_t cells = static_cast<int64_t>(nx) * ny * nz;
  if (!wrap) {
    const int64_t tile = c.store == Store::F64 ? LINE_C<double> : LINE_C<float>;
    if (c.exact || 5 * static_cast<int64_t>(g.np) < 4 * g.nty * tile) return false;
    if (c.store == Store::F64 && cells < LINE_MIN_CELLS_F64_CAVITY) return false;
  }
  // (the padding at the row ends is copied too: 100x120x140 FP32, padded by
  // 28 %, is still 84.3 against 85.7)
  return cells >= LINE_MIN_CELLS && pitch * ny * nz <= cells + cells / 3;
}

cudaError_t launch_line(const LaunchCfg& c, const StepArgs& a, cudaStream_t s) {
  const bool cavity = c.rule == CaseRule::CavityStd;
  if (c.store == Store::F32)
    return cavity ? launch_line_impl<Store::F32, CaseRule::CavityStd, false>(a, s)
                  : launch_line_impl<Store::F32, CaseRule::SphereStd, false>(a, s);
  if (c.exact) return cavity ? cudaErrorInvalidValue : launch_line_impl<Store::F64, CaseRule::SphereStd, true>(a, s);
  return cavity ? launch_line_impl<Store::F64, CaseRule::CavityStd, false>(a, s)
                : launch_line_impl<Store::F64, CaseRule::SphereStd, false>(a, s);
}

}  // namespace imx
