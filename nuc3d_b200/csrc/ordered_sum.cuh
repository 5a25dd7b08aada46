// ordered_sum.cuh -- the left-to-right floating-point sum of squares, in parallel and bit for
// bit (included by kernels.cuh inside its namespace, reference-order build).
//
// The residual of the reference adds (u - u_n)^2 value after value (src/PDEData3d.cpp:103-116);
// the rounding of each addition depends on every one before it, so one thread per block did
// it: 8 cycles per value, 77 ms of an 81 ms step at 128^3.  The terms are not negative, and
// that makes the sum parallel.  While the running sum S stays in one binade [2^e, 2^(e+1)) it
// is an integer multiple of u = 2^(e-52), and adding x rounds x to such a multiple:
// S + x -> S + rn(x / u) u, whatever S is, except when x / u lies halfway between two
// integers, where the even result is taken and the increment depends on the parity of S / u.
// A run of values is then a function of that parity with two integer values (Incr), and such
// functions compose associatively.  The kernel therefore
//   * gives each CTA a segment of kOsSeg values, in ticket order; it sums chunks of kOsChunk
//     values in any order and finds the approximate sum before each chunk by looking back
//     over its predecessors (decoupled look-back; predecessors hold earlier tickets, so they
//     never wait for this CTA), which predicts the chunk's binade;
//   * evaluates each chunk's function for the predicted binade, and the segment's;
//   * the last CTA of a block walks the segments from S = 0: where S is in the predicted
//     binade before and after a function, S / u moves by its increment; where not (S = 0, S
//     crosses into the next binade, a value too large) it goes down to the segment's chunks
//     and there adds value after value.
// The prediction only decides which runs take the short way: the walk checks each one, so the
// result does not depend on it.  A look-back that gives up (kOsSpins) predicts nothing.
// Sums that are not finite have no functions and need none: a NaN among the values makes the
// sum NaN wherever it stands, so the CTA that meets one says so in the block's count and there
// is no walk; and without a NaN, a sum that reaches Inf stays Inf, so the walk ends there.
// (Walked value by value, a block that is NaN throughout took twice the plain loop's time:
// 64^3 19.0 ms where a finite one takes 0.07.  Finite sums that the walk has to add value by
// value over long stretches still do: S below 2^-1022, or so close below a power of two that
// only the approximate sum passes it.)
// One launch, each value read once.  Measured: 24^3 0.51 -> 0.07 ms, 64^3 9.0 -> 0.11 ms,
// 128^3 78 -> 0.45 ms.  What is left is the walk: 1.5-3 us for each binade S grows through (a
// chunk's 128 dependent additions and the loads before them; chunks of 256 and one function
// after the other in place of incr_run's scan: 0.10 / 0.22 / 0.74 ms).
#pragma once

constexpr int kOsThreads = 256;
constexpr int kOsChunk = 128;              // values added one by one where S changes its binade
constexpr int kOsChunks = 32;              // chunks per segment: one lane each in the walk
constexpr int kOsSeg = kOsChunk * kOsChunks;
constexpr int kOsLane = kOsChunk / 32;       // a chunk's values per lane
constexpr int kOsPer = kOsSeg / kOsThreads;  // values per thread: 4 chunks per warp
constexpr int kOsSpins = 1 << 20;
constexpr int kOsNone = 0x7fffffff;        // no function: add the values one by one
constexpr int kOsAny = 0x7ffffffe;         // the identity in every binade (all values zero)
constexpr unsigned long long kOsTop = 1ull << 53;
constexpr unsigned long long kOsInf = 0x7ffull << 52;       // bits of +Inf
constexpr unsigned kOsNanBit = 1u << 31;   // in a block's done count: a NaN among its values

// The increment of S / u over a run of values for S / u even (a) and odd (b); e: the binade.
struct Incr {
  unsigned long long a, b;
  int e;
};
__device__ __forceinline__ Incr incr_then(const Incr &x, const Incr &y) {
  Incr r;
  r.a = x.a + ((x.a & 1) ? y.b : y.a);
  r.b = x.b + ((x.b & 1) ? y.a : y.b);
  r.e = x.e == kOsAny ? y.e : (y.e == kOsAny || y.e == x.e ? x.e : kOsNone);
  if (r.a > kOsTop || r.b > kOsTop) r.e = kOsNone;  // more than a binade holds
  if (r.e == kOsNone) r.a = r.b = 0;
  return r;
}
// The functions of the warp's 32 lanes in lane order; lane 0 gets the composition.
__device__ __forceinline__ Incr incr_warp(Incr x) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    Incr y;
    y.a = __shfl_down_sync(0xffffffffu, x.a, o);
    y.b = __shfl_down_sync(0xffffffffu, x.b, o);
    y.e = __shfl_down_sync(0xffffffffu, x.e, o);
    const Incr c = incr_then(x, y);
    // only lanes whose 2o positions are a whole run compose (the others are not read again)
    if ((threadIdx.x & (2 * o - 1)) == 0) x = c;
  }
  return x;
}
// S (not negative, as bits) after the run f; false where f does not apply.
__device__ __forceinline__ bool incr_apply(const Incr &f, unsigned long long &s) {
  if (f.e == kOsAny) return true;
  if (f.e == kOsNone || (int)(s >> 52) != f.e + 1023) return false;
  const unsigned long long t = s + ((s & 1) ? f.b : f.a);
  if ((t >> 52) != (s >> 52)) return false;
  s = t;
  return true;
}

// The longest run of the lanes' functions from lane `start` on that applies to S, in lane
// order: S moves over it; returns the first lane whose function does not apply, or 32.
__device__ __forceinline__ int incr_run(Incr x, int start, unsigned long long &s) {
  const int lane = threadIdx.x & 31;
  if (lane < start) x = Incr{0, 0, kOsAny};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    Incr y;
    y.a = __shfl_up_sync(0xffffffffu, x.a, o);
    y.b = __shfl_up_sync(0xffffffffu, x.b, o);
    y.e = __shfl_up_sync(0xffffffffu, x.e, o);
    if (lane >= o) x = incr_then(y, x);
  }
  unsigned long long t = s;
  const unsigned stop = ~__ballot_sync(0xffffffffu, incr_apply(x, t));
  const int c = stop ? __ffs(stop) - 1 : 32;
  if (c > 0) s = __shfl_sync(0xffffffffu, t, c - 1);
  return c;
}

// Function of the warp's chunk of kOsLane x 32 values (x[r] of lane l is value 32 r + l) in the
// binade of the approximate sum before it.
__device__ __forceinline__ Incr chunk_incr(const double *x, double before) {
  const unsigned bits = (unsigned)((unsigned long long)__double_as_longlong(before) >> 52);
  const int e = (int)bits - 1023;
  double most = 0.0;
#pragma unroll
  for (int r = 0; r < kOsLane; ++r) most = x[r] > most || x[r] != x[r] ? x[r] : most;
  if (__all_sync(0xffffffffu, most == 0.0)) return Incr{0, 0, kOsAny};
  // a normal number whose binade has 2^(52 - e) as a normal scale (Inf, NaN: 0x7ff)
  const bool ok = bits >= 1 && bits <= 2046 && 52 - e <= 1023;
  const double scale = ok ? __longlong_as_double((long long)(52 - e + 1023) << 52) : 0.0;
  if (!__all_sync(0xffffffffu, ok && most * scale < (double)kOsTop)) return Incr{0, 0, kOsNone};
  unsigned long long sum = 0;
  bool tie = false;
#pragma unroll
  for (int r = 0; r < kOsLane; ++r) {
    const double y = x[r] * scale, k = rint(y);
    tie |= fabs(y - k) == 0.5;
    sum += (unsigned long long)(long long)k;
  }
  Incr f{0, 0, e};
  if (!__any_sync(0xffffffffu, tie)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    f.a = f.b = sum;
  } else {
#pragma unroll 1
    for (int r = 0; r < kOsLane; ++r) {
      const double y = x[r] * scale, k = rint(y), lo = floor(y);
      const unsigned long long n = (unsigned long long)(long long)k, l = (unsigned long long)(long long)lo;
      Incr g{n, n, e};
      if (fabs(y - k) == 0.5) {
        g.a = (l & 1) ? l + 1 : l;
        g.b = (l & 1) ? l : l + 1;
      }
      g = incr_warp(g);
      f = incr_then(f, g);  // lane 0's is the chunk's
    }
    f.a = __shfl_sync(0xffffffffu, f.a, 0);
    f.b = __shfl_sync(0xffffffffu, f.b, 0);
    f.e = __shfl_sync(0xffffffffu, f.e, 0);
  }
  if (f.a > kOsTop || f.b > kOsTop) f = Incr{0, 0, kOsNone};
  return f;
}

// Look-back cells: the bits of an approximate sum with its two lowest replaced by a flag
// (0 nothing yet, 1 this segment's sum, 2 the sum up to and including it).
__device__ __forceinline__ void look_put(unsigned long long *p, double v, unsigned flag) {
  *(volatile unsigned long long *)p = ((unsigned long long)__double_as_longlong(v) & ~3ull) | flag;
}
// Approximate sum of the block's values before segment `seg` (the block's first is `first`),
// by one warp.
__device__ __forceinline__ double look_back(const unsigned long long *look, int first, int seg) {
  const int lane = threadIdx.x & 31;
  double before = 0.0;
  int pos = seg - 1;
  for (int spin = 0; spin < kOsSpins; ++spin) {
    const int i = pos - lane;
    const unsigned long long c = i >= first ? *(const volatile unsigned long long *)(look + i) : 2ull;
    const unsigned flag = (unsigned)(c & 3u);
    const unsigned whole = __ballot_sync(0xffffffffu, flag == 2u), none = __ballot_sync(0xffffffffu, flag == 0u);
    const int stop = whole ? __ffs(whole) - 1 : 32;           // the nearest inclusive sum
    if (none & (stop < 32 ? (2u << stop) - 1u : 0xffffffffu)) continue;  // one before it is missing
    double v = i >= first && lane <= stop ? __longlong_as_double((long long)(c & ~3ull)) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    before += v;
    if (stop < 32) return before;
    pos -= 32;
  }
  return __longlong_as_double(0x7ff8000000000000ll);
}

// d_res_ord workspace of the launch: the ticket, one done count per block, one look-back cell
// per segment (all zero between launches), the segments' and the chunks' functions.
struct OrdWork {
  unsigned *ticket, *done;
  unsigned long long *look;
  Incr *seg, *chunk;
};
__device__ __forceinline__ OrdWork ord_work(unsigned char *w, int nblocks, int nseg) {
  OrdWork o;
  o.ticket = reinterpret_cast<unsigned *>(w);
  o.done = o.ticket + 1;
  o.look = reinterpret_cast<unsigned long long *>(w + ((size_t)(nblocks + 1) * 4 + 7) / 8 * 8);
  o.seg = reinterpret_cast<Incr *>(o.look + nseg);
  o.chunk = o.seg + nseg;
  return o;
}

__global__ void __launch_bounds__(kOsThreads)
residual_ordered_kernel(const BlockDev *__restrict__ blocks, TileMap tm, unsigned char *work,
                        double *__restrict__ res_last, StepState *S) {
  __shared__ int s_ticket, s_last, s_nan;
  __shared__ double s_sum[kOsChunks];
  __shared__ Incr s_f[kOsThreads], s_g[kOsThreads / 32];
  __shared__ double s_x[kOsChunk];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nseg = tm.tile_start[tm.nblocks];
  const OrdWork W = ord_work(work, tm.nblocks, nseg);
  if (tid == 0) {
    const int t = (int)atomicAdd(W.ticket, 1u);
    if (t == nseg - 1) *W.ticket = 0;  // the last ticket: ready for the next launch
    s_ticket = t;
  }
  __syncthreads();
  const int seg = s_ticket, b = find_block(tm, seg), first = tm.tile_start[b], end = tm.tile_start[b + 1];
  const double *__restrict__ d = blocks[b].dres;
  const long long n = 5 * blocks[b].N, base = (long long)(seg - first) * kOsSeg;

  // warp w holds the chunks 4 w .. 4 w + 3
  double x[kOsPer];
#pragma unroll
  for (int r = 0; r < kOsPer; ++r) {
    const long long i = base + (long long)(warp * 4 + r / kOsLane) * kOsChunk + r % kOsLane * 32 + lane;
    const double v = i < n ? d[i] : 0.0;
    x[r] = v * v;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    double s = 0.0;
#pragma unroll
    for (int r = 0; r < kOsLane; ++r) s += x[kOsLane * c + r];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) s_sum[warp * 4 + c] = s;
  }
  __syncthreads();
  if (warp == 0) {
    const double own = s_sum[lane];
    double incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const double all = __shfl_sync(0xffffffffu, incl, 31);
    double before = 0.0;
    if (seg > first) {
      if (lane == 0) look_put(W.look + seg, all, 1u);
      before = look_back(W.look, first, seg);
    }
    if (lane == 0) {
      look_put(W.look + seg, before + all, 2u);
      if (all != all) atomicOr(W.done + b, kOsNanBit);  // (no term is negative: Inf alone gives no NaN)
    }
    s_sum[lane] = before + (incl - own);
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const Incr f = chunk_incr(x + kOsLane * c, s_sum[warp * 4 + c]);
    if (lane == 0) s_f[warp * 4 + c] = f;
  }
  __syncthreads();
  if (warp == 0) {
    const Incr f = s_f[lane];
    W.chunk[(size_t)seg * kOsChunks + lane] = f;
    const Incr g = incr_warp(f);
    if (lane == 0) W.seg[seg] = g;
    __threadfence();
    __syncwarp();
    if (lane == 0) {
      const unsigned c = atomicAdd(W.done + b, 1u);
      s_last = (c & ~kOsNanBit) == (unsigned)(end - first - 1);
      s_nan = (c & kOsNanBit) != 0;
      __threadfence();
    }
  }
  __syncthreads();
  if (!s_last) return;

  // the block's last CTA: from S = 0 over all its segments, as long as S is finite
  unsigned long long s = s_nan ? 0x7ff8ull << 48 : 0;
  for (int p = first; p < end; p += kOsThreads) {
    const int i = p + tid;
    Incr f{0, 0, kOsAny};
    if (i < end) {
      const volatile Incr *v = W.seg + i;
      f.a = v->a;
      f.b = v->b;
      f.e = v->e;
      W.look[i] = 0;  // every CTA of the block has looked back
    }
    s_f[tid] = f;
    f = incr_warp(f);
    if (lane == 0) s_g[warp] = f;
    __syncthreads();
    if (warp == 0) {
      for (int g = 0; g < kOsThreads / 32 && s < kOsInf; ++g) {
        if (incr_apply(s_g[g], s)) continue;
        // segments p + 32 g + c (those past the block's last are identities)
        for (int c = 0; c < 32 && s < kOsInf; ++c) {
          if ((c = incr_run(s_f[32 * g + lane], c, s)) == 32) break;
          const int k = p + 32 * g + c;
          const volatile Incr *v = W.chunk + (size_t)k * kOsChunks + lane;
          Incr h;
          h.a = v->a;
          h.b = v->b;
          h.e = v->e;
          for (int m = 0; m < kOsChunks && s < kOsInf; ++m) {
            if ((m = incr_run(h, m, s)) == kOsChunks) break;
            const long long at = (long long)(k - first) * kOsSeg + (long long)m * kOsChunk;
#pragma unroll
            for (int r = 0; r < kOsLane; ++r) {
              const long long j = at + 32 * r + lane;
              const double y = j < n ? d[j] : 0.0;
              s_x[32 * r + lane] = y * y;
            }
            __syncwarp();
            double t = __longlong_as_double((long long)s);
#pragma unroll 32
            for (int r = 0; r < kOsChunk; ++r) t = t + s_x[r];
            s = (unsigned long long)__double_as_longlong(t);
            __syncwarp();
          }
        }
      }
    }
    __syncthreads();
  }
  if (tid == 0) {
    W.done[b] = 0;
    residual_finish(blocks[b], b, __longlong_as_double((long long)s), res_last, S);
  }
}
