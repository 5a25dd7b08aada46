// sweep_march.cuh -- the eta and zeta sweeps of the explicit schemes as a march along the lines
// (throughput build; included by kernels.cuh inside its namespace).
//
// Same phases as sweep_kernel (split fluxes, faces, cells: src/physicsModel.cpp:420-760,
// src/euler3d.cpp:305-366, :143-241, :368-427, src/TVD-RK3.cpp:16-137), but a thread owns a
// line, not a cell: lane l of a warp walks one line of 32 neighbouring ones (consecutive in
// memory, so every load and store is coalesced) from the first to the last cell of a segment.
// Per step it splits one new cell, evaluates one face from the split fluxes it keeps in
// registers, and finishes the cell behind it.  What that buys over the tiles:
//   * no shared-memory round trip of the split and face fluxes, and no barrier at all;
//   * each cell is loaded and split once per segment (the tiles redo 6 of every 32 or 64);
//   * the face index is the same in every lane, so the physical-face schemes, the neighbour
//     ghosts and the weno5z quirk are uniform branches.
// The FP64 pipe takes a warp instruction every 2 cycles per scheduler with 8 cycles of
// latency, so two warps per scheduler with two independent chains each fill it; two it is
// (255 registers: 10 windows of 2R-1 split fluxes, 50 doubles for WENO5).  Global latency is
// hidden by cp.async: the next cell's state, Jacobian and metric, and the right-hand side and
// u_n of the cell to finish, are copied one step (>= 1200 cycles) ahead into shared memory
// that only the same thread reads.
// Measured, us per launch at 256^3, tiles / march: eta 1212 / 875, zeta 1232 / 930,
// Navier-Stokes eta 1600 / 934, zeta 2174 / 1052 (1290 with the update's kind a branch at run
// time); the FP64 pipe is busy 62-65% (eta) and 54-58% (zeta), Navier-Stokes 55% and 42-46%
// (48% in the tiles), and a register-only loop of the same arithmetic takes 1274
// cycles a cell and warp where the march takes 1690.  Tried and dropped: three warps per
// scheduler in 168 registers (spills, and the rings leave little L1 for them: eta 0.90, zeta
// 2.3 ms); the ten reconstructions interleaved step by step in the source (no change).
#pragma once

constexpr int kMarchThreads = 128;  // 4 warps, each on its own; two CTAs per SM
constexpr int kMarchWarps = kMarchThreads / 32;
constexpr int kMarchRes = 8;        // cells per partial sum of the residual

template <int DIR, int SCH, bool NSV> struct MarchGeo {
  static constexpr int R = Halo<SCH>::R, NW = 2 * R - 1;
  // ring slots: the state back to the cell being finished (zeta), else two
  static constexpr int QS = DIR == 2 ? 8 : 2;
  static constexpr int OFF_Q = 0;                                  // [6][QS] q, jac
  static constexpr int OFF_M = OFF_Q + 6 * QS;                     // [3][2] metric
  static constexpr int OFF_R = OFF_M + 3 * 2;                      // [5][2] right-hand side
  static constexpr int OFF_N = OFF_R + 5 * 2;                      // [5][2] u_n (zeta)
  static constexpr int OFF_V = OFF_N + (DIR == 2 ? 5 * 2 : 0);     // [4][8] viscous fluxes
  static constexpr int WORDS = OFF_V + (NSV ? 4 * 8 : 0);          // doubles per thread
  static constexpr size_t BYTES = (size_t)WORDS * kMarchThreads * sizeof(double);
};

// The share of a launch: lines line0 .. line1-1 and cells c0 .. c1-1 of each block (a z-slab
// of one block), segments of len cells.
struct MarchPart {
  int line0, line1, c0, c1, len;
};

// F+ + F- of a face k faces from a physical one (k < ts), from the line's windows: the stencils
// of recon_pos / recon_neg there sit at the same places of the windows at both ends.
template <int R, int NW>
__device__ __forceinline__ double march_edge(int k, const double (&p)[NW], const double (&n)[NW]) {
  if (k == 0) return p[R - 1] + n[R - 1];
  if constexpr (R >= 2) {
    if (k == 1) return rb_second(p[R - 1], p[R]) + rb_second(n[R - 1], n[R - 2]);
  }
  if constexpr (R >= 3) {
    if (k == 2) return rb_third(p[R - 2], p[R - 1], p[R]) + rb_third(n[R], n[R - 1], n[R - 2]);
  }
  if constexpr (R >= 4) return weno5js(p[1], p[2], p[3], p[4], p[5]) + weno5js(n[5], n[4], n[3], n[2], n[1]);
  return 0.0;
}

// RKM: 0 the right-hand side alone, 1 the RK update of stage 0, 2 of stages 1 and 2 (zeta).
template <int DIR, int SCH, bool NSV, int RIE, int RKM>
__global__ void __launch_bounds__(kMarchThreads, 2)
march_kernel(const BlockDev *__restrict__ blocks, TileMap tm, SolverParams P, StepState *S, int stage,
             int flags, MarchPart part) {
  using M = MarchGeo<DIR, SCH, NSV>;
  constexpr int R = M::R, NW = M::NW, QS = M::QS;
  extern __shared__ double smem[];
  double *const mine = smem + threadIdx.x;
  auto word = [mine](int i) -> double & { return mine[i * kMarchThreads]; };

  const int t = tm.base + (int)blockIdx.x, b = find_block(tm, t);
  const BlockDev &B = blocks[b];
  const int nx = B.n[0], ny = B.n[1], L = B.n[DIR];
  const long long N = B.N;
  const int lines = DIR == 1 ? nx * B.n[2] : nx * ny;
  const int line0 = part.line0, line1 = min(part.line1, lines);
  const int c0 = part.c0, c1 = min(part.c1, L);
  const int nlw = (line1 - line0 + 31) / 32;
  const int item = (t - tm.tile_start[b]) * kMarchWarps + (int)(threadIdx.x >> 5);
  const int seg = item / nlw, lw = item - seg * nlw;
  const int s0 = c0 + seg * part.len, s1 = min(c1, s0 + part.len);
  if (s0 >= c1) return;
  const int lane = threadIdx.x & 31;
  const bool live = line0 + lw * 32 + lane < line1;
  const int line = min(line0 + lw * 32 + lane, line1 - 1);  // spare lanes repeat the last line
  int w = line, o = 0;
  if (DIR == 1) { o = line / nx; w = line - o * nx; }
  else { o = line / nx; w = line - o * nx; }
  const long long sL = DIR == 1 ? nx : (long long)nx * ny;
  const long long cell0 = DIR == 1 ? w + (long long)o * nx * ny : line;  // the line's cell 0
  const int sa = DIR == 1 ? o : w, sb = DIR == 1 ? w : o;                // slab coordinates
  const bool physL = B.face[2 * DIR].type < 0, physR = B.face[2 * DIR + 1].type < 0;
  const int ts = P.ts[DIR];
  const bool compat = P.weno5z_compat != 0;
  constexpr bool rk = RKM > 0, need_n = RKM == 2;
  const bool res = (flags & SW_RES) != 0;
  double dt = 0.0;
  if (rk) {
    dt = stage == 0 ? 1.0 / __longlong_as_double((long long)S->max_eig_bits) * P.cfl : S->dt;
    if (t == tm.base && threadIdx.x == 0 && b == 0 && s0 == 0 && line0 == 0) {
      if (stage == 0) S->dt = dt;
      if (stage == 2) S->time = S->time + dt;
    }
  }
  const double *__restrict__ q = B.q[stage], *__restrict__ qn = B.q[0], *__restrict__ jac = B.jac,
               *__restrict__ met = B.met[DIR];
  double *__restrict__ rhs = B.rhs;
  double *__restrict__ qo = B.q[(stage + 1) % 3];

  // copies x: the state, Jacobian and metric of cell x, and what step x - 1 needs to finish
  // its cell x - 1 - R: the right-hand side, u_n and the viscous flux of the cell 3 further
  auto copy_cell = [&](int x) {
    const long long idx = cell0 + x * sL;
    const int s = x & (QS - 1), h = x & 1;
#pragma unroll
    for (int v = 0; v < 5; ++v) cp_async8(&word(M::OFF_Q + v * QS + s), q + v * N + idx);
    cp_async8(&word(M::OFF_Q + 5 * QS + s), jac + idx);
#pragma unroll
    for (int k = 0; k < 3; ++k) cp_async8(&word(M::OFF_M + k * 2 + h), met + k * N + idx);
  };
  auto copy_rhs = [&](int c, int p) {
    const long long idx = cell0 + c * sL;
#pragma unroll
    for (int v = 0; v < 5; ++v) cp_async8(&word(M::OFF_R + v * 2 + p), rhs + v * N + idx);
  };
  auto copy_un = [&](int c, int p) {
    const long long idx = cell0 + c * sL;
#pragma unroll
    for (int v = 0; v < 5; ++v) cp_async8(&word(M::OFF_N + v * 2 + p), qn + v * N + idx);
  };
  auto copy_vis = [&](int y) {
    const long long idx = cell0 + y * sL;
#pragma unroll
    for (int v = 0; v < 4; ++v) cp_async8(&word(M::OFF_V + v * 8 + (y & 7)), B.vis + (DIR * 4 + v) * N + idx);
  };
  auto commit = [] { asm volatile("cp.async.commit_group;\n" ::: "memory"); };
  auto issue = [&](int x) {
    if (x >= 0 && x < L) copy_cell(x);
    const int c = x - 1 - R, p = (x - 1) & 1;
    if (c >= s0 && c < s1) {
      copy_rhs(c, p);
      if (need_n) copy_un(c, p);
    }
    if constexpr (NSV) {
      // ghosts come from the neighbour (a physical face's one-sided differences read none)
      const int y = c + 3;
      if (y >= s0 - 3 && y < s1 + 3) {
        if (y >= 0 && y < L) {
          copy_vis(y);
        } else {
          long long nidx;
          const int nb = ghost_cell(blocks, B, DIR, y, sa, sb, P.bfs, nidx);
#pragma unroll
          for (int v = 0; v < 4; ++v)
            word(M::OFF_V + v * 8 + (y & 7)) =
                nb >= 0 ? __ldg(blocks[nb].vis + (DIR * 4 + v) * blocks[nb].N + nidx) : 0.0;
        }
      }
    }
    commit();
  };

  unsigned st = 0;
  double racc = 0.0;
  // split fluxes of any cell x of the line, its ghosts included; an energy that con2prim reset
  // goes into the ring, where the RK update takes u_i from
  auto split = [&](int x, double (&fp)[5], double (&fn)[5]) {
    double u[5], j = 0.0, m0 = 0.0, m1 = 0.0, m2 = 0.0;
#pragma unroll
    for (int v = 0; v < 5; ++v) fp[v] = fn[v] = 0.0;
    if (x >= 0 && x < L) {
      const int s = x & (QS - 1), h = x & 1;
#pragma unroll
      for (int v = 0; v < 5; ++v) u[v] = word(M::OFF_Q + v * QS + s);
      j = word(M::OFF_Q + 5 * QS + s);
      m0 = word(M::OFF_M + h);
      m1 = word(M::OFF_M + 2 + h);
      m2 = word(M::OFF_M + 4 + h);
    } else {
      long long nidx;
      const int nb = ghost_cell(blocks, B, DIR, x, sa, sb, P.bfs, nidx);
      if (nb < 0) {
        if (x == -1 || x == L) {  // the ghost flux bc_ghost_kernel left
          const double *gh = B.ghost + B.goff[2 * DIR + (x < 0 ? 0 : 1)] +
                             (sa + (long long)(DIR == 1 ? B.n[2] : nx) * sb);
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            const double y = __ldg(gh + (long long)v * lines);
            if (x < 0) fp[v] = y; else fn[v] = y;
          }
        }
        return;
      }
      const BlockDev &C = blocks[nb];
      load_q(C.q[stage], C.N, nidx, u);
      j = __ldg(C.jac + nidx);
      const double *m = C.met[DIR];
      m0 = __ldg(m + nidx);
      m1 = __ldg(m + C.N + nidx);
      m2 = __ldg(m + 2 * C.N + nidx);
    }
    CellPrim s;
    cell_prim(u, j, P.gamma, P.mach, s, st);
    u[4] = s.q4;
    if (DIR == 2 && s.reset && x >= 0 && x < L) word(M::OFF_Q + 4 * QS + (x & (QS - 1))) = s.q4;
    cell_fluxes(RIE, u, s, m0, m1, m2, j, fp, fn);
  };

  // right-hand side and RK3 stage of cell c, whose step is g = c + R, from its flux difference
  auto finish = [&](int c, const double (&d)[5]) {
    const long long idx = cell0 + c * sL;
    const int p = (c + R) & 1, s = c & (QS - 1);
    double r[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) r[v] = word(M::OFF_R + v * 2 + p) + d[v];
    if constexpr (!rk) {
      if (live) {
#pragma unroll
        for (int v = 0; v < 5; ++v) rhs[v * N + idx] = r[v];
      }
    } else {
      double un[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
      if constexpr (need_n) {  // u_n with stage 0's energy reset
#pragma unroll
        for (int v = 0; v < 5; ++v) un[v] = word(M::OFF_N + v * 2 + p);
        CellPrim sn;
        unsigned stn = 0;
        cell_prim(un, word(M::OFF_Q + 5 * QS + s), P.gamma, P.mach, sn, stn);
        un[4] = sn.q4;
      }
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const double x = rk3_update(stage, r[v], word(M::OFF_Q + v * QS + s), un[v], dt);
        if (!isfinite(x)) st |= ST_NONFINITE;
        if (live) qo[v * N + idx] = x;
        if (res && live) res_value(B, v, idx, x, un[v], racc);
      }
      if (res && ((c & (kMarchRes - 1)) == kMarchRes - 1 || c == L - 1)) {
        // one partial sum per warp of lines and kMarchRes cells, whatever the segments
        double a = racc;
#pragma unroll
        for (int x = 16; x > 0; x >>= 1) a += __shfl_xor_sync(0xffffffffu, a, x);
        if (lane == 0) P.res_part[B.res_off + (long long)(c / kMarchRes) * nlw + lw] = a;
        racc = 0.0;
      }
    }
  };

  // kAhead: the split of the next cell runs beside the reconstructions (zeta, whose RK update
  // wants the registers, gains nothing from it); kInline: the copies and the finished cell's
  // update are part of the common step's block (Navier-Stokes: eta 256^3 1.08 -> 0.96 ms, the
  // 128^3 vortex's step 2.02 -> 1.95 ms by zeta's; Euler eta 0.87 -> 0.90, so not there)
  constexpr bool kAhead = DIR == 1, kInline = NSV;
  const bool vis6 = P.vis[DIR] == VIS_CD6;
  // Step g: wn holds F- of the cells g-2R+2 .. g, wp F+ of g-2R+1 .. g-1 and fp F+ of g; the
  // step evaluates face f = g-R+1, finishes cell f-1 and splits cell g+1.
  double wp[5][NW], wn[5][NW], fp[5], fnn[5], fpn[5], hprev[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    hprev[v] = 0.0;
#pragma unroll
    for (int k = 0; k < NW; ++k) wp[v][k] = wn[v][k] = 0.0;
  }
  issue(s0 - R);
  issue(s0 - R + 1);
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
  split(s0 - R, fp, fnn);
#pragma unroll
  for (int v = 0; v < 5; ++v) wn[v][NW - 1] = fnn[v];
#pragma unroll 1
  for (int g = s0 - R; g < s1 + R; ++g) {
    const int f = g - R + 1;
    const int k = min(physL ? f : ts, physR ? L - f : ts);  // faces to a physical one (ts: none near)
    const bool cz = compat && f >= ts && f <= L - ts;
    double h[5];
    auto faces = [&](bool quirk) {
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const double(&a)[NW] = wp[v];
        const double(&c)[NW] = wn[v];
        auto Pacc = [&a](int i) { return a[i + R]; };
        auto Nacc = [&c](int i) { return c[i + R - 1]; };
        h[v] = recon_pos_in<SCH>(0, quirk, Pacc) + recon_neg_in<SCH>(0, Nacc);
      }
    };
    auto shift = [&](double (&d)[5]) {
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        d[v] = h[v] - hprev[v];
        hprev[v] = h[v];
#pragma unroll
        for (int i = 0; i < NW - 1; ++i) wp[v][i] = wp[v][i + 1];
        wp[v][NW - 1] = fp[v];
#pragma unroll
        for (int i = 0; i < NW - 1; ++i) wn[v][i] = wn[v][i + 1];
        if (kAhead) {
          fp[v] = fpn[v];
          wn[v][NW - 1] = fnn[v];
        }
      }
    };
    double d[5];
    const bool common = kInline ? f > s0 && g + 2 < s1 + R - 1 && g + 2 < L && vis6 && f - 1 >= ts && f - 1 < L - ts
                            : f >= s0 && g + 1 >= 0 && g + 1 < L;
    if ((kAhead || kInline) && k >= ts && common) {
      // the common step in one block with as few branches as can be, so that its chains of
      // dependent operations overlap the reconstructions
      if constexpr (kInline) {
        copy_cell(g + 2);
        copy_rhs(f, (g + 1) & 1);
        if (need_n) copy_un(f, (g + 1) & 1);
        copy_vis(f + 3);
        commit();
      } else {
        issue(g + 2);
      }
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
      if constexpr (kAhead) {
        double u[5];
        const int s = (g + 1) & (QS - 1), p = (g + 1) & 1;
#pragma unroll
        for (int v = 0; v < 5; ++v) u[v] = word(M::OFF_Q + v * QS + s);
        const double j = word(M::OFF_Q + 5 * QS + s);
        CellPrim c;
        double rinv, ek;
        const bool low = cell_plain(u, j, P.gamma, c, rinv, ek);
        cell_fluxes(RIE, u, c, word(M::OFF_M + p), word(M::OFF_M + 2 + p), word(M::OFF_M + 4 + p), j, fpn, fnn);
        faces(cz);
        if (low) split(g + 1, fpn, fnn);
      } else {
        faces(cz);
      }
      shift(d);
      if constexpr (kInline) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          auto V = [&](int x) { return word(M::OFF_V + v * 8 + ((f - 1 + x) & 7)); };
          d[v + 1] -= cd6(V(-3), V(-2), V(-1), V(1), V(2), V(3));
        }
        finish(f - 1, d);
        if constexpr (!kAhead) {
          split(g + 1, fp, fnn);
#pragma unroll
          for (int v = 0; v < 5; ++v) wn[v][NW - 1] = fnn[v];
        }
        continue;
      }
    } else {
      issue(g + 2);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
      if (kAhead && g + 1 < s1 + R) split(g + 1, fpn, fnn);
      if (f >= s0) {
        if (k < ts) {
#pragma unroll
          for (int v = 0; v < 5; ++v) h[v] = march_edge<R>(k, wp[v], wn[v]);
        } else {
          faces(cz);
        }
      } else {
#pragma unroll
        for (int v = 0; v < 5; ++v) h[v] = 0.0;
      }
      shift(d);
    }
    // ---- cell c = f - 1: difference, right-hand side, RK3 stage ----
    const int c = f - 1;
    if (c >= s0 && c < s1) {
      if constexpr (NSV) {
        double dv[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          auto V = [&](int x) { return word(M::OFF_V + v * 8 + (x & 7)); };
          dv[v] = diff_at(c, L, ts, physL, physR, P.vis[DIR], V);
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) d[v + 1] -= dv[v];
      }
      finish(c, d);
    }
    if (!kAhead && g + 1 < s1 + R) {
      split(g + 1, fp, fnn);
#pragma unroll
      for (int v = 0; v < 5; ++v) wn[v][NW - 1] = fnn[v];
    }
  }
  if (st) atomicOr(&S->status, st);
}

// ---- host side ----
// Segment length of a march over blocks of the given line warps and cells per line: the one
// with the smallest estimated time, (rounds of the resident warps) x (cells + start-up), the
// start-up being the 2R - 1 cells split before the first face (about a third of a full step
// each) and the first copies.  Multiples of kMarchRes cells.
template <int R>
inline int march_length(const BlockDev *h, int b0, int b1, int dir, const MarchPart &part) {
  constexpr int kSlots = 148 * 2 * kMarchWarps;  // resident warps of a B200
  constexpr double kStart = 0.35 * (2 * R - 1) + 2.0;
  int longest = 0;
  for (int b = b0; b < b1; ++b)
    longest = std::max(longest, std::min(part.c1, h[b].n[dir]) - part.c0);
  double best = 1e300;
  int len = kMarchRes;
  for (int l = kMarchRes; l < longest + kMarchRes; l += kMarchRes) {
    long long items = 0;
    for (int b = b0; b < b1; ++b) {
      const int cells = std::min(part.c1, h[b].n[dir]) - part.c0;
      const int lines = std::min<long long>(part.line1, h[b].N / h[b].n[dir]) - part.line0;
      items += (long long)((lines + 31) / 32) * ((cells + l - 1) / l);
    }
    const double cost = (double)((items + kSlots - 1) / kSlots) * (std::min(l, longest) + kStart);
    if (cost < best * 0.999) { best = cost; len = l; }
  }
  return len;
}

// Cells of a launch.
template <int DIR> inline long long march_cells(const Launch &L) {
  const BlockDev *h = L.h_blocks;
  if (L.k1 > 0) return (long long)h[0].n[0] * h[0].n[1] * (L.k1 - L.k0);
  long long n = 0;
  for (int b = L.b0; b < (L.b1 > 0 ? L.b1 : L.tm_dir[DIR].nblocks); ++b) n += h[b].N;
  return n;
}

template <int DIR, int SCH, bool NSV, int RIE>
inline cudaError_t launch_march_r(const Launch &L, int stage, int flags) {
  using M = MarchGeo<DIR, SCH, NSV>;
  const BlockDev *h = L.h_blocks;
  const int nb = L.tm_dir[DIR].nblocks, b1 = L.b1 > 0 ? L.b1 : nb;
  MarchPart part{0, 0x7fffffff, 0, 0x7fffffff, 0};
  if (L.k1 > 0) {  // a z-slab of the one block
    if (DIR == 1) { part.line0 = L.k0 * h[0].n[0]; part.line1 = L.k1 * h[0].n[0]; }
    else { part.c0 = L.k0; part.c1 = L.k1; }
  }
  part.len = march_length<M::R>(h, L.b0, b1, DIR, part);
  TileMap tm;
  tm.nblocks = nb;
  tm.tile_start[0] = 0;
  for (int b = 0; b < nb; ++b) {
    const int cells = std::min(part.c1, h[b].n[DIR]) - part.c0;
    const long long lines = std::min<long long>(part.line1, h[b].N / h[b].n[DIR]) - part.line0;
    const long long items = ((lines + 31) / 32) * ((cells + part.len - 1) / part.len);
    tm.tile_start[b + 1] = tm.tile_start[b] + (int)((items + kMarchWarps - 1) / kMarchWarps);
  }
  tm.base = tm.tile_start[L.b0];
  tm.end = tm.tile_start[b1];
  const int grid = tm.end - tm.base;
  if (grid <= 0) return cudaSuccess;
  auto run = [&](auto kernel) {
    kernel<<<grid, kMarchThreads, M::BYTES, L.stream>>>(L.d_blocks, tm, L.P, L.d_state, stage, flags, part);
    return cudaGetLastError();
  };
  if constexpr (DIR == 2) {
    if (flags & SW_RK)
      return stage == 0 ? run(march_kernel<DIR, SCH, NSV, RIE, 1>) : run(march_kernel<DIR, SCH, NSV, RIE, 2>);
  }
  return run(march_kernel<DIR, SCH, NSV, RIE, 0>);
}

template <int DIR, int SCH, bool NSV>
inline cudaError_t launch_march(const Launch &L, int stage, int flags) {
  switch (L.P.riemann) {
    case RIE_LF: return launch_march_r<DIR, SCH, NSV, RIE_LF>(L, stage, flags);
    case RIE_AUSM: return launch_march_r<DIR, SCH, NSV, RIE_AUSM>(L, stage, flags);
    default: return launch_march_r<DIR, SCH, NSV, RIE_AUSMP>(L, stage, flags);
  }
}

// Whether direction dir of a launch marches: WENO5 lines (the windows of WENO7 do not fit the
// registers), no face sensor, and viscous stencils of at most three cells.
inline bool march_dir(const SolverParams &P, int dir) {
  if (dir == 0 || (P.scheme[dir] != SCH_WENO5JS && P.scheme[dir] != SCH_WENO5Z)) return false;
  if (P.sensor && P.scheme[dir] == SCH_WENO5Z) return false;
  return P.model != MODEL_NS || P.vis[dir] != VIS_CD8;
}
template <int DIR, int SCH, bool NSV, int RIE> inline cudaError_t configure_march_r() {
  static_assert(2 * (MarchGeo<DIR, SCH, NSV>::BYTES + 1024) <= 228 * 1024, "two CTAs per SM");
  auto set = [](auto kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)MarchGeo<DIR, SCH, NSV>::BYTES);
  };
  if constexpr (DIR == 2) {
    cudaError_t e;
    if ((e = set(march_kernel<DIR, SCH, NSV, RIE, 1>)) != cudaSuccess) return e;
    if ((e = set(march_kernel<DIR, SCH, NSV, RIE, 2>)) != cudaSuccess) return e;
  }
  return set(march_kernel<DIR, SCH, NSV, RIE, 0>);
}
template <int DIR, int SCH> inline cudaError_t configure_march() {
  cudaError_t e;
  if ((e = configure_march_r<DIR, SCH, false, RIE_LF>()) != cudaSuccess) return e;
  if ((e = configure_march_r<DIR, SCH, false, RIE_AUSM>()) != cudaSuccess) return e;
  if ((e = configure_march_r<DIR, SCH, false, RIE_AUSMP>()) != cudaSuccess) return e;
  if ((e = configure_march_r<DIR, SCH, true, RIE_LF>()) != cudaSuccess) return e;
  if ((e = configure_march_r<DIR, SCH, true, RIE_AUSM>()) != cudaSuccess) return e;
  return configure_march_r<DIR, SCH, true, RIE_AUSMP>();
}
