// compact_march.cuh -- the eta and zeta sweeps of crweno5 as a march along the lines
// (throughput build, Euler; included by kernels.cuh inside its namespace).
//
// compact_line_kernel gives a line's ten tridiagonal systems a warp each and solves them by
// partition and cyclic reduction: every lane walks chains of dependent divisions, and the two
// lines a CTA holds leave the FP64 pipe a tenth busy.  Here a lane owns a line and walks it
// twice, as the reference's Thomas solve does (src/crweno5.cpp:207-218): forward it splits the
// cells, builds each face's row from the split fluxes it keeps in registers and eliminates it,
// backward it substitutes, adds the two splits and finishes the cells.  A warp takes one of the
// five variables of 32 neighbouring lines (every access is coalesced); the five warps of a CTA
// share their cells' loads through L1 and repeat the split, which costs half again the FP64
// work but gives five times the warps.  The eliminated rows (c', d' of both splits: 32 bytes a
// face and variable) go through B.rows.
// Measured, us per launch, compact_line_kernel / march: 96^3 eta 291 / 205, zeta 294 / 237;
// 128^3 582 / 356, 582 / 386; 256^3 4244 / 2282, 4298 / 2737.  Four CTAs per SM (96 registers,
// a few spills) against three (128): 256^3 2282 / 2584, and 128^3's 512 CTAs are one round.
#pragma once

constexpr int kCmThreads = 160;  // five warps: one variable each
// The rule: lines enough to fill the GPU (a third of its 592 CTAs), else a launch takes as long
// as one line's walk and compact_line_kernel is the faster one: 80x64x90 zeta (5120 lines) 155 /
// 214 us, eta (7200 lines) 194 / 142.
constexpr int kCmLines = 6144;

template <int DIR>
__global__ void __launch_bounds__(kCmThreads, 4)
compact_march_kernel(const BlockDev *__restrict__ blocks, TileMap tm, SolverParams P, StepState *S, int stage,
                     int flags) {
  constexpr int R = 3, NW = 5;
  const int t = (int)blockIdx.x, b = find_block(tm, t);
  const BlockDev &B = blocks[b];
  const int nx = B.n[0], ny = B.n[1], L = B.n[DIR], lw = t - tm.tile_start[b];
  const long long N = B.N;
  const int lines = DIR == 1 ? nx * B.n[2] : nx * ny;
  const int lane = threadIdx.x & 31, v = threadIdx.x >> 5;
  const bool live = lw * 32 + lane < lines;
  const int line = min(lw * 32 + lane, lines - 1);
  const int o = line / nx, w = line - o * nx;
  const long long sL = DIR == 1 ? nx : (long long)nx * ny;
  const long long cell0 = DIR == 1 ? w + (long long)o * nx * ny : line;
  const int sa = DIR == 1 ? o : w, sb = DIR == 1 ? w : o;
  const bool physL = B.face[2 * DIR].type < 0, physR = B.face[2 * DIR + 1].type < 0;
  const bool rk = DIR == 2 && (flags & SW_RK) != 0, res = (flags & SW_RES) != 0;
  double dt = 0.0;
  if (rk) {
    dt = stage == 0 ? 1.0 / __longlong_as_double((long long)S->max_eig_bits) * P.cfl : S->dt;
    if (t == 0 && threadIdx.x == 0) {
      if (stage == 0) S->dt = dt;
      if (stage == 2) S->time = S->time + dt;
    }
  }
  const bool un_read = rk && stage != 0;
  const double *__restrict__ q = B.q[stage];
  double *q0 = B.q[0];  // u_n; stage 2 writes the new state over it
  // rows [face][c', d' of F+, c', d' of F-][variable][line]
  const long long S5 = 5ll * lines;
  double *__restrict__ row = B.rows + (long long)v * lines + line;
  unsigned st = 0;

  struct Cell {
    double u[5], j, m[3];
  };
  // cell x of the line (its own or a neighbour block's); false: beyond a physical face
  auto load = [&](int x, Cell &c) -> bool {
    const BlockDev *C = &B;
    long long idx = cell0 + x * sL;
    if (x < 0 || x >= L) {
      const int nb = ghost_cell(blocks, B, DIR, x, sa, sb, P.bfs, idx);
      if (nb < 0) return false;
      C = &blocks[nb];
    }
    load_q(C->q[stage], C->N, idx, c.u);
    c.j = __ldg(C->jac + idx);
#pragma unroll
    for (int k = 0; k < 3; ++k) c.m[k] = __ldg(C->met[DIR] + k * C->N + idx);
    return true;
  };
  auto pick = [v](const double (&f)[5]) { return v == 0 ? f[0] : v == 1 ? f[1] : v == 2 ? f[2] : v == 3 ? f[3] : f[4]; };

  // ---- forward: split, rows, elimination ----
  double wp[NW], wn[NW], cp[2] = {0.0, 0.0}, dp[2] = {0.0, 0.0};
#pragma unroll
  for (int k = 0; k < NW; ++k) wp[k] = wn[k] = 0.0;
  Cell cur, nxt;
  bool have = load(-R, cur), more = false;
#pragma unroll 1
  for (int g = -R; g < L + R; ++g) {
    if (g + 1 < L + R) more = load(g + 1, nxt);  // a step ahead
    double fp = 0.0, fn = 0.0;
    if (have) {
      CellPrim s;
      double p5[5], n5[5];
      con2prim(cur.u, cur.j, P.gamma, P.mach, s, st);
      cur.u[4] = s.q4;
      split_cell(P.riemann, cur.u, s, cur.m[0], cur.m[1], cur.m[2], cur.j, p5, n5);
      fp = pick(p5);
      fn = pick(n5);
    } else if (g == -1 || g == L) {  // the ghost flux bc_ghost_kernel left
      const double *gh = B.ghost + B.goff[2 * DIR + (g < 0 ? 0 : 1)] +
                         (sa + (long long)(DIR == 1 ? B.n[2] : nx) * sb) + (long long)v * lines;
      if (g < 0) fp = __ldg(gh); else fn = __ldg(gh);
    }
    if (un_read && v == 4 && live && g >= 0 && g < L) {
      // u_n's energy after stage 0's reset, in place: the other variables' warps may overwrite
      // u_n in the backward walk, so its last use as a whole is here
      const long long idx = cell0 + g * sL;
      double e[5];
      CellPrim s;
      unsigned none = 0;
#pragma unroll
      for (int k = 0; k < 5; ++k) e[k] = q0[k * N + idx];
      con2prim(e, __ldg(B.jac + idx), P.gamma, P.mach, s, none);
      if (s.reset) q0[4 * N + idx] = s.q4;
    }
#pragma unroll
    for (int k = 0; k < NW - 1; ++k) wn[k] = wn[k + 1];
    wn[NW - 1] = fn;
    const int f = g - R + 1;  // wp: F+ of f-3 .. f+1, wn: F- of f-2 .. f+2
    if (f >= 0) {
      const int k = min(physL ? f : R, physR ? L - f : R);  // faces to a physical one (R: none near)
      if (f <= R || f >= L - R) {
        // faces next to the ends and the system's end rows are explicit: rows 0 1 0 | h
        double h[2];
        if (k < R) {
          h[0] = k == 0 ? wp[2] : (k == 1 ? rb_second(wp[2], wp[3]) : rb_third(wp[1], wp[2], wp[3]));
          h[1] = k == 0 ? wn[2] : (k == 1 ? rb_second(wn[2], wn[1]) : rb_third(wn[3], wn[2], wn[1]));
        } else {
          h[0] = weno5js(wp[0], wp[1], wp[2], wp[3], wp[4]);
          h[1] = weno5js(wn[4], wn[3], wn[2], wn[1], wn[0]);
        }
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          // (the system's last row: a NaN of the rows before reaches it, as by the elimination)
          dp[z] = f == L - R ? h[z] - 0.0 * (dp[z] + cp[z]) : h[z];
          cp[z] = 0.0;
        }
      } else {
        const double s0[5] = {wp[0], wp[1], wp[2], wp[3], wp[4]}, s1[5] = {wn[4], wn[3], wn[2], wn[1], wn[0]};
        double lo[2], di[2], up[2], d[2];
        crweno5_row(s0, lo[0], di[0], up[0], d[0]);
        crweno5_row(s1, up[1], di[1], lo[1], d[1]);  // F-: upwind is the next face
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const double r = qdiv(1.0, di[z] - cp[z] * lo[z]);
          dp[z] = (d[z] - dp[z] * lo[z]) * r;
          cp[z] = up[z] * r;
        }
      }
      if (live) {
        double *x = row + (long long)f * 4 * S5;
        x[0] = cp[0];
        x[S5] = dp[0];
        x[2 * S5] = cp[1];
        x[3 * S5] = dp[1];
      }
    }
#pragma unroll
    for (int k = 0; k < NW - 1; ++k) wp[k] = wp[k + 1];
    wp[NW - 1] = fp;
    cur = nxt;
    have = more;
  }

  __syncthreads();
  // ---- backward: substitution, difference, right-hand side, RK3 stage ----
  double *__restrict__ rhs = B.rhs + v * N;
  double *__restrict__ qo = B.q[(stage + 1) % 3] + v * N;
  double racc = 0.0, hn = 0.0, xp = 0.0, xm = 0.0;
  double a[4], na[4], nr = 0.0, nu = 0.0, nn = 0.0;  // rows of face f; those and the cell's values a step ahead
#pragma unroll
  for (int k = 0; k < 4; ++k) na[k] = row[(long long)L * 4 * S5 + k * S5];
#pragma unroll 1
  for (int f = L; f >= 0; --f) {
    const double r0 = nr, u0 = nu, n0 = nn;
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = na[k];
    if (f > 0) {
      const long long idx = cell0 + (f - 1) * sL;
#pragma unroll
      for (int k = 0; k < 4; ++k) na[k] = row[(long long)(f - 1) * 4 * S5 + k * S5];
      nr = rhs[idx];
      if (rk) nu = __ldg(q + v * N + idx);
      if (un_read) nn = q0[v * N + idx];
    }
    // (the faces outside the system, f < R and f > L - R, and its last row have no next face: times
    // a zero, a NaN or Inf of that face would reach them)
    if (f < R || f >= L - R) xp = xm = 0.0;
    xp = a[1] - a[0] * xp;
    xm = a[3] - a[2] * xm;
    const double h = xp + xm;
    if (f < L && live) {
      const long long idx = cell0 + f * sL;
      const double r = r0 + (hn - h);
      if (!rk) {
        rhs[idx] = r;
      } else {
        double ui = u0;
        const double un = n0;
        if (v == 4) {  // u_i's energy after con2prim's reset (u_n's: above)
          CellPrim s;
          double e[5];
          unsigned none = 0;
          load_q(q, N, idx, e);
          con2prim(e, __ldg(B.jac + idx), P.gamma, P.mach, s, none);
          ui = s.q4;
        }
        const double x = rk3_update(stage, r, ui, un, dt);
        if (!isfinite(x)) st |= ST_NONFINITE;
        qo[idx] = x;
        if (res) racc = fma(x - un, x - un, racc);
      }
    }
    hn = h;
  }
  if (res) {  // one partial sum per variable of a warp of lines
#pragma unroll
    for (int x = 16; x > 0; x >>= 1) racc += __shfl_xor_sync(0xffffffffu, racc, x);
    if (lane == 0) P.res_part[B.cres_off + (long long)lw * 5 + v] = racc;
  }
  if (st) atomicOr(&S->status, st);
}

// Whether direction dir of a launch marches: crweno5, Euler, fused solves on (line_dirs), and
// lines enough.
inline bool compact_march_dir(const Launch &L, int dir) {
  if (dir == 0 || L.P.scheme[dir] != SCH_CRWENO5 || L.P.model == MODEL_NS || !((L.line_dirs >> dir) & 1)) return false;
  long long lines = 0;
  for (int b = 0; b < L.tm_cells.nblocks; ++b) lines += L.h_blocks[b].N / L.h_blocks[b].n[dir];
  return lines >= kCmLines;
}
template <int DIR> inline cudaError_t launch_compact_march(const Launch &L, int stage, int flags) {
  TileMap tm;
  tm.nblocks = L.tm_cells.nblocks;
  tm.base = tm.end = 0;
  tm.tile_start[0] = 0;
  for (int b = 0; b < tm.nblocks; ++b)
    tm.tile_start[b + 1] = tm.tile_start[b] + (int)((L.h_blocks[b].N / L.h_blocks[b].n[DIR] + 31) / 32);
  compact_march_kernel<DIR><<<tm.tile_start[tm.nblocks], kCmThreads, 0, L.stream>>>(L.d_blocks, tm, L.P, L.d_state,
                                                                                   stage, flags);
  return cudaGetLastError();
}
