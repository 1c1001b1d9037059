// Reduced FP32 inner BiCGStab with a tile's system resident on its SM.
//
// The single-reduction iteration of cms_schur.cuh (schur_body_sr: the same
// recurrences and the same arithmetic per row), for systems whose tiles fit
// one SM each.  In the streaming form an iteration takes 14-16 us on small
// systems and 28 us on the 1M-cell one although its 100 MB stay in L2: gather
// phases of dependent L1/L2 loads (each acquire empties L1) and fences,
// progress flags, an arrival counter and partial sums.  Here
//
//  * Chat's coefficients and columns stay in the block's shared memory for
//    the whole launch (sliced ELL over 32-row slices, column = 16-bit index
//    into the block's own and halo rows), and a thread keeps the vectors of
//    its rows in registers; a gather reads shared memory only;
//  * tiles are as square as the numbering allows (resident_partition), and
//    only rows that another tile gathers are written to global memory, each
//    as one word that holds the value and the iteration's tag (8 bytes for
//    nu, 16 for s and t); a reader polls the word itself until the tag is the
//    one it needs.  No fence, no progress flag and no L1 invalidation: an
//    exchange takes 550 cycles within a die and 950 across (measured; with
//    release and acquire 1000 and 1600);
//  * the nine sums travel the same way through one collecting tile, which is
//    the grid barrier as well;
//  * one warp forms the scalars of the recurrence while the others gather.
//
// Measured (one B200, kernel time per iteration, start and end of the launch
// included, form of cms_schur.cuh / this form): 1k cells 14.7 / 4.4 us, 30k
// 16.4 / 4.8, 250k 16.9 / 6.5, 1M 28.9 / 15.2.  What bounds it: at 1M cells the
// shared-memory wavefronts of the two gathers (about 3000 cycles of 4400
// each); at 30k cells the three exchanges through L2 (about 5300 of 9000
// cycles).
//
// Why a word is never overwritten too early.  nu of iteration i is replaced
// in iteration i+1 after the sums of i, which a reader contributes to after
// it has read nu.  s, t of iteration i are replaced after the block has read
// nu of iteration i+1 of every tile it shares an edge with (the pattern is
// symmetric), which such a tile stores after it has read s, t of i.  A sum's
// word has two copies by parity: copy i is replaced by i+2, after the sums of
// i+1, which every block contributes to after it has read those of i.
// Tags grow over the launches of a handle, so no word needs clearing.
//
// Every poll is bounded by A.spin_limit and sets the barrier's error flag.
#pragma once
#include "cms_schur.cuh"

namespace cms {

constexpr int RES_BS = 512;   // threads per block, one block per SM (128 registers: nine vectors of 8 rows)
constexpr int RES_NW = RES_BS / 32;
constexpr int RES_TOT = 16;    // words between the two copies of the totals
constexpr int RES_NRMAX = 8;  // rows per thread: at most 4096 B rows per tile

// A value and its tag in one 16-byte word, stored and loaded as one access.
__device__ __forceinline__ void st_word16(void* p, unsigned long long v, unsigned long long tag) {
  asm volatile(
      "{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p), "l"(v),
      "l"(tag)
      : "memory");
}
__device__ __forceinline__ void ld_word16(const void* p, unsigned long long& v, unsigned long long& tag) {
  asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
               : "=l"(v), "=l"(tag)
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void st_word8(unsigned long long* p, unsigned int v, unsigned int tag) {
  const unsigned long long w = (unsigned long long)tag << 32 | v;
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long ld_word8(const unsigned long long* p) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}

// One more poll of a wait: true when the wait gives up.
__device__ __forceinline__ bool poll_failed(GridBar* bar, unsigned int& spins, unsigned int limit) {
  if (++spins > limit) {
    atomicExch(&bar->err, 1);
    return true;
  }
  return (spins & 255u) == 0 && bar_failed(bar);
}

// Warp sums of eight values at once: each of three exchange steps halves the
// values a lane carries (4 + 2 + 1 exchanges, then two on one value, instead
// of 8 x 5).  Lane l ends with value l >> 2.
__device__ __forceinline__ double warp_sum8(const double* v) {
  const int lane = threadIdx.x & 31;
  double a[4], b[2];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const bool up = lane & 16;
    const double send = up ? v[j] : v[j + 4];
    a[j] = (up ? v[j + 4] : v[j]) + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const bool up = lane & 8;
    const double send = up ? a[j] : a[j + 2];
    b[j] = (up ? a[j + 2] : a[j]) + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  const bool up = lane & 4;
  double c = (up ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}

// This block's sums of v[q] over its threads, stored with the tag as the
// tile's words of copy buf.  act: the warp has rows (others add zero).  Ends
// with every thread past the block barrier inside.
template <int NS, int NW>
__device__ __forceinline__ void publish_sums(double (&v)[NS], bool act, double (*sm)[NW], ulonglong2* slots, int nt,
                                             int tile, int buf, unsigned int tag) {
  constexpr int N8 = NS >= 8 ? 8 : 0;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (act) {
    if constexpr (N8 == 8) {
      const double x = warp_sum8(v);
      if ((lane & 3) == 0) sm[lane >> 2][wid] = x;
    }
#pragma unroll
    for (int q = N8; q < NS; ++q) {
      const double x = warp_sum(v[q]);
      if (lane == 0) sm[q][wid] = x;
    }
  } else if (lane < NS) {
    sm[lane][wid] = 0.0;
  }
  __syncthreads();
  for (int q = wid; q < NS; q += NW) {
    double x = sm[q][lane & (NW - 1)];
#pragma unroll
    for (int o = NW / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0)
      st_word16(slots + ((size_t)buf * NSMAX + q) * nt + tile, (unsigned long long)__double_as_longlong(x), tag);
  }
}

// The sums of all tiles of copy buf into bc.  One tile collects: its warp q
// polls the tiles' words of value q (lane l adds tiles l, l + 32, ... in that
// order, then a butterfly) and stores the total, tagged, in tot; every tile
// polls the totals.  (Every tile polling every tile's words is one hop
// shorter, but at 148 tiles a round of it moves 3 MB: 5000 cycles against
// 3000 for the two hops, measured.)  A lane's words of up to 160 tiles are
// polled together.  Returns true when a poll gave up.  The caller
// synchronises the block.
template <int NS, int NW>
__device__ __forceinline__ bool collect_sums(double* bc, const ulonglong2* slots, ulonglong2* tot, int nt, int tile,
                                             int buf, unsigned int tag, GridBar* bar, unsigned int limit) {
  constexpr int U = 5;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  bool fail = false;
  if (tile == nt / 2) {
    for (int q = wid; q < NS; q += NW) {
      const ulonglong2* src = slots + ((size_t)buf * NSMAX + q) * nt;
      double acc = 0.0;
      for (int b = lane; b < nt; b += 32 * U) {
        unsigned long long v[U], t[U];
        unsigned int spins = 0;
        for (;;) {
          bool all = true;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            v[u] = 0ull;
            t[u] = tag;
            if (b + 32 * u < nt) ld_word16(src + b + 32 * u, v[u], t[u]);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) all = all && t[u] == tag;
          if (all) break;
          if (poll_failed(bar, spins, limit)) { fail = true; break; }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) acc += __longlong_as_double((long long)v[u]);
      }
      acc = warp_sum(acc);
      if (lane == 0) st_word16(tot + buf * RES_TOT + q, (unsigned long long)__double_as_longlong(acc), tag);
    }
  }
  if (threadIdx.x < NS) {
    unsigned long long v, t;
    unsigned int spins = 0;
    for (;;) {
      ld_word16(tot + buf * RES_TOT + threadIdx.x, v, t);
      if (t == tag) break;
      if (poll_failed(bar, spins, limit)) { fail = true; break; }
    }
    bc[threadIdx.x] = __longlong_as_double((long long)v);
  }
  return fail;
}

// Scalars of one iteration, formed by one warp and read by the block, and the
// recurrence's state, touched by that warp only (in shared memory: in
// registers every thread would hold it).
struct ResScal {
  float ax, be, ay;  // alf of the finished iteration, bet, alf of the next
  int stop, keep;    // 1: the loop ends, 2: non-finite, 4: a y update is pending; the iterate is the best so far
};
struct ResState {
  double rho, alf, tol2, rr_last, best2, res0;
  int it_best, converged, nonfinite;
};

// The start, from r0.r0 and f0.r0.
__device__ __forceinline__ void resident_first(double rr, double fr, double tol, ResState& st, ResScal& sc) {
  const double res0 = sqrt(rr);
  st.res0 = res0;
  st.rho = st.rr_last = st.best2 = rr;
  st.tol2 = (tol * res0) * (tol * res0);
  st.it_best = 0;
  st.converged = res0 == 0.0 ? 1 : 0;
  st.nonfinite = res0 != 0.0 && (!isfinite(fr) || !isfinite(res0)) ? 1 : 0;
  st.alf = res0 != 0.0 && !st.nonfinite && fr != 0.0 ? rr / fr : 0.0;
  sc.ay = (float)st.alf;
  // a breakdown before the first step (f0.r0 = 0) stops with x = 0
  sc.stop = (st.converged || st.nonfinite || fr == 0.0 ? 1 : 0) | (st.nonfinite ? 2 : 0);
}

// The solve's record: last: the result is the last iterate, not the best one.
__device__ __forceinline__ void resident_report(DevState* d, const ResState& st, int it, int nonfinite, bool last) {
  const double rr = !nonfinite && !last ? st.best2 : st.rr_last;
  d->iter = it;
  d->s[S_RELRES] = nonfinite ? rr : st.res0 > 0.0 ? sqrt(rr) / st.res0 : 0.0;
  d->s[S_RES0] = st.res0;
  d->converged = st.converged;
  d->nonfinite = nonfinite;
  d->done = 1;
}

// omg of an iteration, by every thread.
__device__ __forceinline__ double resident_omega(const double* t) {
  return t[0] / fmax(t[1], SMALL);
}

// The other scalars, from the sums of iteration it (as schur_body_sr).
__device__ __forceinline__ void resident_scalars(const double* t, double omg, ResState& st, ResScal& sc, int it,
                                                 int maxit) {
  const double alf = st.alf, rho = st.rho;
  const double rr = fmax(t[2] - 2.0 * omg * t[0] + omg * omg * t[1], 0.0);
  const double rho1 = t[3] - omg * t[4];
  const double bet = (rho1 / rho) * (alf / omg);
  const double tau = (t[5] - omg * t[6]) + bet * (t[8] - omg * t[7]);
  const double alf_n = rho1 / tau;
  const bool finite = isfinite(rr) && isfinite(omg) && isfinite(rho1);
  const bool save = finite && rr < st.best2;  // y += alf p + omg s is valid even at a breakdown below
  const double best2 = save ? rr : st.best2;
  const int it_best = save ? it : st.it_best;
  const bool conv = finite && rr < st.tol2;
  // breakdown of the next step, divergence or stagnation: the best iterate is the result
  bool end = !finite || conv || omg == 0.0 || rho1 == 0.0 || rr > (kDiverge * kDiverge) * best2 ||
             it - it_best >= kStall;
  bool bad = !finite;
  if (!end) {
    bad = !isfinite(tau) || !isfinite(bet);
    end = bad || tau == 0.0;
  }
  if (it >= maxit) end = true;
  if ((threadIdx.x & 31) == 0) {
    sc.ax = (float)alf;
    sc.be = (float)bet;
    sc.ay = (float)alf_n;
    sc.keep = save ? 1 : 0;
    sc.stop = (end ? 1 : 0) | (bad ? 2 : 0) | (finite ? 4 : 0);
    st.rho = rho1;
    st.alf = alf_n;
    st.rr_last = rr;
    st.best2 = best2;
    st.it_best = it_best;
    st.converged = conv ? 1 : 0;
    st.nonfinite = bad ? 1 : 0;
  }
}

template <int NR>
__device__ __forceinline__ void schur_body_resident(const SchurArgs& A) {
  extern __shared__ __align__(16) unsigned char res_smem[];
  __shared__ double s_sum[NSMAX][RES_NW], s_bc[NSMAX];
  __shared__ ResScal s_sc;
  __shared__ ResState s_st;
  const int n = A.n, g1 = A.g1, nB = A.nB, nt = A.ntiles, tile = A.tile;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  PhaseState ph{0u, 0u, true, true};
  const int t0 = __ldg(A.tptr + tile), nb = __ldg(A.tptr + tile + 1) - t0, ns = (nb + 31) >> 5;
  const int h0 = __ldg(A.hptr + tile), nh = __ldg(A.hptr + tile + 1) - h0;
  const int* hrow = A.hrow + h0;
  const int* soff_g = A.sloff + __ldg(A.slptr + tile);
  // shared memory: slice offsets (pairs of slots x 32 lanes), coefficient
  // pairs, column pairs, and the gathered vectors over own then halo rows
  const int npair = ns > 0 ? __ldg(soff_g + ns) : 0;
  float2* cf = reinterpret_cast<float2*>(res_smem);
  ushort2* lc = reinterpret_cast<ushort2*>(cf + (size_t)npair * 32);
  float* rb = reinterpret_cast<float*>(lc + (size_t)npair * 32);
  const int hb = ns * 32;  // halo rows follow the own rows' slices
  float* nub = rb + hb + nh;
  int* soff = reinterpret_cast<int*>(nub + hb + nh);
  for (int j = threadIdx.x; j <= ns; j += RES_BS) soff[j] = ns > 0 ? __ldg(soff_g + j) : 0;
  __syncthreads();
  // this thread's rows: local k = slice * 32 + lane, slices wid, wid + 32, ...
  int row[NR], xw[NR];  // device row and its exchanged word (-1 for none)
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    const int j = wid + RES_NW * q, k = j * 32 + lane;
    row[q] = -1;
    xw[q] = -1;
    if (k < nb) {
      row[q] = g1 + __ldg(A.trow + t0 + k);
      xw[q] = __ldg(A.rexp + (row[q] - g1));
    }
    if (j < ns) {
      const int i = row[q] - g1;
      for (int s = soff[j]; s < soff[j + 1]; ++s) {
        const int c = 2 * (s - soff[j]);
        float2 a = make_float2(0.0f, 0.0f);
        ushort2 l = make_ushort2(0, 0);
        if (k < nb) {
          a.x = __ldg(A.coff + (size_t)c * nB + i);
          l.x = __ldg(A.lcol + (size_t)c * nB + i);
          l.y = l.x;
          if (c + 1 < A.KC) {
            a.y = __ldg(A.coff + (size_t)(c + 1) * nB + i);
            l.y = __ldg(A.lcol + (size_t)(c + 1) * nB + i);
          }
        }
        cf[s * 32 + lane] = a;
        lc[s * 32 + lane] = l;
      }
    }
  }
  const bool act = wid < ns;
  ulonglong2* tot = A.slots + (size_t)2 * NSMAX * nt;
  // out[k] = v[k] - sum of Chat's row k over the vector v (slots in order), own
  // rows of this thread; a loop over its slices, not unrolled over the rows it
  // holds (the unrolled form's instruction fetches cost more than its loads)
  auto gather = [&](const float* v, float* out) {
    for (int j = wid; j < ns; j += RES_NW) {
      float acc = v[j * 32 + lane];
      const int e = soff[j + 1];
#pragma unroll 4
      for (int s = soff[j]; s < e; ++s) {
        const float2 a = cf[s * 32 + lane];
        const ushort2 l = lc[s * 32 + lane];
        acc = acc - a.x * v[l.x];
        acc = acc - a.y * v[l.y];
      }
      out[j * 32 + lane] = acc;
    }
  };
  // the halo rows' words of tag: s and t into rb and nub, or nu into nub; a
  // thread's HU words are polled together (one round trip, not HU)
  constexpr int HU = 4;
  auto halo_st = [&](unsigned int tag) -> bool {
    bool fail = false;
    for (int h = threadIdx.x; h < nh; h += HU * RES_BS) {
      unsigned long long v[HU], t[HU];
      unsigned int spins = 0;
      int i[HU];
#pragma unroll
      for (int u = 0; u < HU; ++u) i[u] = __ldg(hrow + (h + u * RES_BS < nh ? h + u * RES_BS : h));
      for (;;) {
        bool all = true;
#pragma unroll
        for (int u = 0; u < HU; ++u) {
          v[u] = 0ull;
          t[u] = tag;
          if (h + u * RES_BS < nh) ld_word16(A.xst + i[u], v[u], t[u]);
        }
#pragma unroll
        for (int u = 0; u < HU; ++u) all = all && t[u] == tag;
        if (all) break;
        if (poll_failed(A.bar, spins, A.spin_limit)) { fail = true; break; }
      }
#pragma unroll
      for (int u = 0; u < HU; ++u) {
        if (h + u * RES_BS < nh) {
          rb[hb + h + u * RES_BS] = __uint_as_float((unsigned int)v[u]);
          nub[hb + h + u * RES_BS] = __uint_as_float((unsigned int)(v[u] >> 32));
        }
      }
    }
    return fail;
  };
  auto halo_nu = [&](unsigned int tag) -> bool {
    bool fail = false;
    for (int h = threadIdx.x; h < nh; h += HU * RES_BS) {
      unsigned long long w[HU];
      unsigned int spins = 0;
      int i[HU];
#pragma unroll
      for (int u = 0; u < HU; ++u) i[u] = __ldg(hrow + (h + u * RES_BS < nh ? h + u * RES_BS : h));
      for (;;) {
        bool all = true;
#pragma unroll
        for (int u = 0; u < HU; ++u) {
          w[u] = (unsigned long long)tag << 32;
          if (h + u * RES_BS < nh) w[u] = ld_word8(A.xnu + i[u]);
        }
#pragma unroll
        for (int u = 0; u < HU; ++u) all = all && (unsigned int)(w[u] >> 32) == tag;
        if (all) break;
        if (poll_failed(A.bar, spins, A.spin_limit)) { fail = true; break; }
      }
#pragma unroll
      for (int u = 0; u < HU; ++u)
        if (h + u * RES_BS < nh) nub[hb + h + u * RES_BS] = __uint_as_float((unsigned int)w[u]);
    }
    return fail;
  };
  auto put_st = [&](int q, float s, float t, unsigned int tag) {
    if (xw[q] >= 0)
      st_word16(A.xst + xw[q], (unsigned long long)__float_as_uint(t) << 32 | __float_as_uint(s), tag);
  };
  auto put_nu = [&](int q, float v, unsigned int tag) {
    if (xw[q] >= 0) st_word8(A.xnu + xw[q], __float_as_uint(v), tag);
  };
  const unsigned int base = A.tag0;
  float sv[NR], tv[NR], yv[NR], pv[NR], nv[NR], qv[NR], uv[NR], rv[NR], r0v[NR], f0v[NR];
  // start, first phase: r0 = b_B - AB0 D0^-1 b_0, y = 0
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    float acc = 0.0f;
    if (row[q] >= 0) {
      const int r = row[q];
      acc = __ldg(&A.b[r]);
      const int kl = __ldg(&A.nlo[r]);
      for (int s = 0; s < kl; ++s) {
        const size_t e = (size_t)s * n + r;
        const int j = __ldg(&A.col[e]);
        if (j < g1) acc = acc + __ldg(&A.aoff[e]) * (__ldg(&A.b[j]) * __ldg(&A.sinv[j]));
      }
      rb[(wid + RES_NW * q) * 32 + lane] = acc;
      put_st(q, acc, 0.0f, base);
    }
    r0v[q] = rv[q] = sv[q] = acc;
    tv[q] = yv[q] = qv[q] = 0.0f;
  }
  // second phase: f0 = op^T r0, u = nu = op r0, p = r0; r0.r0, f0.r0
  ph.ok = !__syncthreads_or(halo_st(base));
  double s2[2] = {0.0, 0.0};
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    uv[q] = f0v[q] = r0v[q];
    if (row[q] >= 0) {
      const int i = row[q] - g1, kc = __ldg(&A.ccnt[i]);
      for (int s = 0; s < kc; ++s) {
        const size_t e = (size_t)s * nB + i;
        const float rk = rb[__ldg(&A.lcol[e])];
        uv[q] = uv[q] - __ldg(&A.coff[e]) * rk;
        f0v[q] = f0v[q] - __ldg(&A.coff[__ldg(&A.ctr[e])]) * rk;
      }
      s2[0] += (double)r0v[q] * (double)r0v[q];
      s2[1] += (double)f0v[q] * (double)r0v[q];
      nub[(wid + RES_NW * q) * 32 + lane] = uv[q];
      put_nu(q, uv[q], base + 1u);
    }
    nv[q] = uv[q];
    pv[q] = r0v[q];
  }
  publish_sums<2, RES_NW>(s2, act, s_sum, A.slots, nt, tile, 0, base);
  ph.ok = !__syncthreads_or(!ph.ok | collect_sums<2, RES_NW>(s_bc, A.slots, tot, nt, tile, 0, base, A.bar, A.spin_limit));
  if (threadIdx.x == 0) {
    resident_first(s_bc[0], s_bc[1], A.tol, s_st, s_sc);
  }
  __syncthreads();
  int it = 0, nonfinite = (s_sc.stop & 2) ? 1 : 0;
  bool stop = (s_sc.stop & 1) != 0, pending = false, save = false;
  bool y_best = true;  // y (without a pending update) is the best iterate so far
  float ay = s_sc.ay, ax = ay, w = 0.0f;
  while (ph.ok && !stop && it < A.maxit) {
    ++it;
    const unsigned int tag = base + (unsigned int)it;
    // Y: q = op nu, s = r - alf nu, t = u - alf q, nine sums
    if (__syncthreads_or(halo_nu(tag))) { ph.ok = false; break; }
    double s9[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    gather(nub, rb);
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (row[q] < 0) continue;
      qv[q] = rb[(wid + RES_NW * q) * 32 + lane];
      sv[q] = rv[q] - ay * nv[q];
      tv[q] = uv[q] - ay * qv[q];
      put_st(q, sv[q], tv[q], tag);
      const double sd = sv[q], td = tv[q], od = r0v[q], fd = f0v[q];
      s9[0] += td * sd;
      s9[1] += td * td;
      s9[2] += sd * sd;
      s9[3] += od * sd;
      s9[4] += od * td;
      s9[5] += fd * sd;
      s9[6] += fd * td;
      s9[7] += od * (double)qv[q];
      s9[8] += od * (double)nv[q];
    }
    publish_sums<9, RES_NW>(s9, act, s_sum, A.slots, nt, tile, it & 1, tag);
    bool fail = halo_st(tag);  // the neighbours' s and t arrive while the sums are collected
    fail |= collect_sums<9, RES_NW>(s_bc, A.slots, tot, nt, tile, it & 1, tag, A.bar, A.spin_limit);
    if (__syncthreads_or(fail)) { ph.ok = false; break; }
    // X: r = s - omg t (own rows and halo), u = op r, the y update (the best
    // iterate so far is kept in yb when it is not the last), p and nu.  The last warp forms
    // the other scalars while the others gather
    const double omg = resident_omega(s_bc);
    w = (float)omg;
    for (int h = threadIdx.x; h < nh; h += RES_BS) rb[hb + h] = rb[hb + h] - w * nub[hb + h];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (row[q] < 0) continue;
      rv[q] = sv[q] - w * tv[q];
      rb[(wid + RES_NW * q) * 32 + lane] = rv[q];
    }
    __syncthreads();
    if (wid == RES_NW - 1) resident_scalars(s_bc, omg, s_st, s_sc, it, A.maxit);
    gather(rb, nub);
    __syncthreads();
    ax = s_sc.ax;
    save = s_sc.keep != 0;
    nonfinite = (s_sc.stop & 2) ? 1 : 0;
    pending = (s_sc.stop & 4) != 0;
    if (s_sc.stop & 1) {
      stop = true;
      break;
    }
    const float be = s_sc.be;
    const bool park = y_best && !save;  // y is the best iterate and this update is not: keep it in yb
    y_best = save;
    ay = s_sc.ay;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (row[q] < 0) continue;
      uv[q] = nub[(wid + RES_NW * q) * 32 + lane];
      if (park) A.yb[row[q]] = yv[q];
      yv[q] = yv[q] + ax * pv[q] + w * sv[q];
      pv[q] = rv[q] + be * (pv[q] - w * nv[q]);
      nv[q] = uv[q] + be * (nv[q] - w * qv[q]);
      nub[(wid + RES_NW * q) * 32 + lane] = nv[q];
      put_nu(q, nv[q], tag + 1u);
    }
    pending = false;
  }
  // the best iterate: the last one (its y update still pending), y or yb;
  // x_B = S^-1 y, then x_0 = D0^-1 (b_0 + sum aoff x_B)
  const bool last = !pending || save;
  if (ph.ok && !nonfinite) {
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (row[q] < 0) continue;
      float y;
      if (last || y_best) {
        y = yv[q];
        if (last && pending) y = y + ax * pv[q] + w * sv[q];
      } else {
        y = A.yb[row[q]];
      }
      A.x[row[q]] = y * __ldg(&A.sinv[row[q]]);
    }
    grid_barrier(A, ph);
    if (ph.ok) {
      const int r1 = (int)((long long)g1 * (tile + 1) / nt);
      for (int r = (int)((long long)g1 * tile / nt) + (int)threadIdx.x; r < r1; r += RES_BS) {
        float acc = __ldg(&A.b[r]);
        const int ku = __ldg(&A.nup[r]);
        for (int t2 = 0; t2 < ku; ++t2) {
          const size_t e = (size_t)(A.KL + t2) * n + r;
          acc = acc + __ldg(&A.aoff[e]) * ldm(&A.x[__ldg(&A.col[e])]);
        }
        A.x[r] = acc * __ldg(&A.sinv[r]);
      }
    }
  }
  if (tile == 0 && threadIdx.x == 0) resident_report(A.st, s_st, it, nonfinite, last);
}

// One system: block b works on tile b.
template <int NR>
__global__ void __launch_bounds__(RES_BS, 1) k_schur_resident(SchurArgs A) {
  __shared__ SchurArgs sA;
  if (threadIdx.x == 0) {
    sA = A;
    sA.ntiles = gridDim.x;
    sA.tile = blockIdx.x;
  }
  __syncthreads();
  schur_body_resident<NR>(sA);
}

// Several independent systems (an ensemble): bmap[b] = (member, tile) of block b.
template <int NR>
__global__ void __launch_bounds__(RES_BS, 1) k_schur_resident_batched(const SchurArgs* __restrict__ members,
                                                                      const int2* __restrict__ bmap) {
  __shared__ SchurArgs sA;
  if (threadIdx.x == 0) {
    const int2 mt = bmap[blockIdx.x];
    sA = members[mt.x];
    sA.tile = mt.y;
  }
  __syncthreads();
  schur_body_resident<NR>(sA);
}

inline const void* resident_kernel(int nr, bool batched) {
  if (nr <= 1) return batched ? (const void*)k_schur_resident_batched<1> : (const void*)k_schur_resident<1>;
  if (nr <= 2) return batched ? (const void*)k_schur_resident_batched<2> : (const void*)k_schur_resident<2>;
  if (nr <= 4) return batched ? (const void*)k_schur_resident_batched<4> : (const void*)k_schur_resident<4>;
  return batched ? (const void*)k_schur_resident_batched<8> : (const void*)k_schur_resident<8>;
}

// Shared memory of a tile with npair slot pairs of 32 rows, nb own and nh halo rows.
inline size_t resident_smem(size_t npair, int nb, int nh) {
  return npair * 32 * (sizeof(float2) + sizeof(ushort2)) + 2 * sizeof(float) * (((size_t)nb + 31) / 32 * 32 + nh) +
         sizeof(int) * ((size_t)(nb + 31) / 32 + 1);
}

}  // namespace cms
