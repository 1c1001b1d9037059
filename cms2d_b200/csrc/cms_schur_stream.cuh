// The reduced FP32 inner BiCGStab for systems too large for cms_resident.cuh:
// the same iteration, tiles, words and sums, with Chat's packed slices and the
// vectors streamed from memory and only the gathered vectors in shared memory.
//
// The 4M-cell system's matrix and vectors (150 MB) do not fit in L2.  The
// form of cms_schur.cuh read 420 MB per iteration (8 bytes per entry, separate
// own-row and gather reads) at 2.7 TB/s: its gathers are dependent loads that
// an L1 of 1024 threads' footprints does not hold.  Here a tile's r and nu
// (own and halo rows) lie in shared memory, columns are 16-bit indices into
// them, and each slice's coefficients, columns and row values are loaded
// together in one coalesced round trip per slice; the row updates of X and Y
// are done in the gather's loop.  About 310 MB per iteration, less what the
// vectors kept in shared memory save (the first ones of SV_* that fit).
//
// Why a word is never overwritten too early.  The halo is the reduced Krylov
// solves' one, extended along the special rows: a tile may read another's words
// while that one reads none of its (an inlet of 2.0M cells has such a pair), so
// the argument of cms_resident.cuh for s and t, which needs every edge both ways, does not hold.
// s and t have STR_ST_COPIES = 2 copies by the tag's parity: those of iteration
// i are replaced by those of i+2, after the sums of i+1, which a reader
// contributes to after it has read s, t of i.  nu and the sums are as in
// cms_resident.cuh, whose argument for them needs no symmetry.
//
// Measured: at its rule, stream_choose in cms_reduced_host.cuh.
#pragma once
#include "cms_reduced.cuh"

namespace cms {

constexpr int STR_BS = 1024;
constexpr int STR_NW = STR_BS / 32;
constexpr int STR_ST_COPIES = 2;  // of the words of s and t
// vectors in the order in which they are kept in shared memory
enum StreamVec : int { SV_S = 0, SV_T, SV_Y, SV_P, SV_U, SV_Q, SV_R0, SV_F0, SV_N };

struct StreamArgs {
  SchurArgs S;               // system, ELL form of Chat (for f0), result, state, limits
  const int *tptr, *trow, *tpad, *rexp, *hptr, *hword, *slptr, *sloff, *mbase;  // as RedArgs
  const float2* pcoef;
  const ushort2* plcol;
  float* gvec;
  size_t npad;
  int nvs;
  float keep;                // share of the slices that L2 is to keep
  ulonglong2* xst;           // [STR_ST_COPIES][words]
  size_t words;
  unsigned long long* xnu;
  ulonglong2* slots;
};

__global__ void __launch_bounds__(STR_BS, 1) k_schur_stream(StreamArgs Ain) {
  extern __shared__ __align__(16) unsigned char str_smem[];
  __shared__ StreamArgs B;
  __shared__ double s_sum[NSMAX][STR_NW], s_bc[NSMAX];
  __shared__ ResScal s_sc;
  __shared__ ResState s_st;
  if (threadIdx.x == 0) {
    B = Ain;
    B.S.ntiles = gridDim.x;
    B.S.tile = blockIdx.x;
  }
  __syncthreads();
  const SchurArgs& A = B.S;
  const int n = A.n, g1 = A.g1, nB = A.nB, nt = A.ntiles, tile = A.tile;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int t0 = __ldg(B.tptr + tile), nb = __ldg(B.tptr + tile + 1) - t0, ns = (nb + 31) >> 5, hb = ns * 32;
  const int h0 = __ldg(B.hptr + tile), nh = __ldg(B.hptr + tile + 1) - h0;
  const int* hw = B.hword + h0;
  const int* rexp = B.rexp + t0;
  const int* sog = B.sloff + __ldg(B.slptr + tile);
  const float2* cf = B.pcoef + (size_t)__ldg(B.mbase + tile) * 32;
  const ushort2* lc = B.plcol + (size_t)__ldg(B.mbase + tile) * 32;
  float* rb = reinterpret_cast<float*>(str_smem);
  float* nub = rb + hb + nh;
  int* soff = reinterpret_cast<int*>(nub + hb + nh);
  float* vec[SV_N];
  {
    float* next = reinterpret_cast<float*>(soff + ns + 1);
    const int pad = __ldg(B.tpad + tile);
#pragma unroll
    for (int v = 0; v < SV_N; ++v) {
      vec[v] = v < B.nvs ? next : B.gvec + (size_t)v * B.npad + pad;
      if (v < B.nvs) next += hb;
    }
  }
  float *sv = vec[SV_S], *tv = vec[SV_T], *yv = vec[SV_Y], *pv = vec[SV_P], *uv = vec[SV_U], *qv = vec[SV_Q],
        *r0v = vec[SV_R0], *f0v = vec[SV_F0];
  for (int j = threadIdx.x; j <= ns; j += STR_BS) soff[j] = ns > 0 ? __ldg(sog + j) : 0;
  __syncthreads();
  PhaseState ph{0u, 0u, true, true};
  const bool act = wid < ns;
  ulonglong2* tot = B.slots + (size_t)2 * NSMAX * nt;
  const unsigned int base = A.tag0;
  // f(k) for this thread's own rows
  auto rows = [&](auto&& f) {
    for (int j = wid; j < ns; j += STR_NW)
      if (j * 32 + lane < nb) f(j * 32 + lane);
  };
  // acc - sum of Chat's row (slice j) over v, slots in order; slices from jkeep
  // on are read with the evict-first policy, so that the others and the
  // vectors stay in L2 from one gather to the next
  const int jkeep = (int)(B.keep * (float)ns);
  auto gather = [&](int j, const float* v, float acc) {
    const int e = soff[j + 1];
    if (j < jkeep) {
#pragma unroll 4
      for (int s = soff[j]; s < e; ++s) {
        const float2 a = __ldg(cf + (size_t)s * 32 + lane);
        const ushort2 l = __ldg(lc + (size_t)s * 32 + lane);
        acc = acc - a.x * v[l.x];
        acc = acc - a.y * v[l.y];
      }
    } else {
#pragma unroll 4
      for (int s = soff[j]; s < e; ++s) {
        const float2 a = __ldcs(cf + (size_t)s * 32 + lane);
        const ushort2 l = __ldcs(lc + (size_t)s * 32 + lane);
        acc = acc - a.x * v[l.x];
        acc = acc - a.y * v[l.y];
      }
    }
    return acc;
  };
  constexpr int HU = 2;
  auto halo_st = [&](unsigned int tag) -> bool {
    bool fail = false;
    const ulonglong2* xst = B.xst + tag % STR_ST_COPIES * B.words;
    for (int h = threadIdx.x; h < nh; h += HU * STR_BS) {
      unsigned long long v[HU], t[HU];
      unsigned int spins = 0;
      int i[HU];
#pragma unroll
      for (int u = 0; u < HU; ++u) i[u] = __ldg(hw + (h + u * STR_BS < nh ? h + u * STR_BS : h));
      for (;;) {
        bool all = true;
#pragma unroll
        for (int u = 0; u < HU; ++u) {
          v[u] = 0ull;
          t[u] = tag;
          if (h + u * STR_BS < nh) ld_word16(xst + i[u], v[u], t[u]);
          all = all && t[u] == tag;
        }
        if (all) break;
        if (poll_failed(A.bar, spins, A.spin_limit)) { fail = true; break; }
      }
#pragma unroll
      for (int u = 0; u < HU; ++u) {
        if (h + u * STR_BS < nh) {
          rb[hb + h + u * STR_BS] = __uint_as_float((unsigned int)v[u]);
          nub[hb + h + u * STR_BS] = __uint_as_float((unsigned int)(v[u] >> 32));
        }
      }
    }
    return fail;
  };
  auto halo_nu = [&](unsigned int tag) -> bool {
    bool fail = false;
    for (int h = threadIdx.x; h < nh; h += HU * STR_BS) {
      unsigned long long w[HU];
      unsigned int spins = 0;
      int i[HU];
#pragma unroll
      for (int u = 0; u < HU; ++u) i[u] = __ldg(hw + (h + u * STR_BS < nh ? h + u * STR_BS : h));
      for (;;) {
        bool all = true;
#pragma unroll
        for (int u = 0; u < HU; ++u) {
          w[u] = (unsigned long long)tag << 32;
          if (h + u * STR_BS < nh) w[u] = ld_word8(B.xnu + i[u]);
          all = all && (unsigned int)(w[u] >> 32) == tag;
        }
        if (all) break;
        if (poll_failed(A.bar, spins, A.spin_limit)) { fail = true; break; }
      }
#pragma unroll
      for (int u = 0; u < HU; ++u)
        if (h + u * STR_BS < nh) nub[hb + h + u * STR_BS] = __uint_as_float((unsigned int)w[u]);
    }
    return fail;
  };
  auto put_st = [&](int k, float s, float t, unsigned int tag) {
    const int w = __ldg(rexp + k);
    if (w >= 0)
      st_word16(B.xst + tag % STR_ST_COPIES * B.words + w, (unsigned long long)__float_as_uint(t) << 32 | __float_as_uint(s), tag);
  };
  auto put_nu = [&](int k, float v, unsigned int tag) {
    const int w = __ldg(rexp + k);
    if (w >= 0) st_word8(B.xnu + w, __float_as_uint(v), tag);
  };
  // start, first phase: r0 = b_B - AB0 D0^-1 b_0, y = 0
  rows([&](int k) {
    const int r = g1 + __ldg(B.trow + t0 + k);
    float acc = __ldg(&A.b[r]);
    const int kl = __ldg(&A.nlo[r]);
    for (int s = 0; s < kl; ++s) {
      const size_t e = (size_t)s * n + r;
      const int j = __ldg(&A.col[e]);
      if (j < g1) acc = acc + __ldg(&A.aoff[e]) * (__ldg(&A.b[j]) * __ldg(&A.sinv[j]));
    }
    rb[k] = r0v[k] = acc;
    yv[k] = 0.0f;
    qv[k] = 0.0f;
    put_st(k, acc, 0.0f, base);
  });
  ph.ok = !__syncthreads_or(halo_st(base));
  // second phase: f0 = op^T r0, u = nu = op r0, p = r0; r0.r0, f0.r0
  double s2[2] = {0.0, 0.0};
  rows([&](int k) {
    const int i = __ldg(B.trow + t0 + k), kc = __ldg(&A.ccnt[i]), o = soff[k >> 5];
    const float r0 = rb[k];
    float u = r0, f = r0;
    for (int s = 0; s < kc; ++s) {
      const size_t e = (size_t)s * nB + i;
      const ushort2 l = __ldg(lc + (size_t)(o + (s >> 1)) * 32 + (k & 31));
      const float rk = rb[s & 1 ? l.y : l.x];
      u = u - __ldg(&A.coff[e]) * rk;
      f = f - __ldg(&A.coff[__ldg(&A.ctr[e])]) * rk;
    }
    uv[k] = u;
    f0v[k] = f;
    pv[k] = r0;
    nub[k] = u;
    put_nu(k, u, base + 1u);
    s2[0] += (double)r0 * (double)r0;
    s2[1] += (double)f * (double)r0;
  });
  publish_sums<2, STR_NW>(s2, act, s_sum, B.slots, nt, tile, 0, base);
  ph.ok = !__syncthreads_or(!ph.ok | collect_sums<2, STR_NW>(s_bc, B.slots, tot, nt, tile, 0, base, A.bar, A.spin_limit));
  if (threadIdx.x == 0) resident_first(s_bc[0], s_bc[1], A.tol, s_st, s_sc);
  __syncthreads();
  int it = 0, nonfinite = (s_sc.stop & 2) ? 1 : 0;
  bool stop = (s_sc.stop & 1) != 0, pending = false, save = false;
  bool y_best = true;  // y (without a pending update) is the best iterate so far
  float ay = s_sc.ay, ax = ay, w = 0.0f;
  while (ph.ok && !stop && it < A.maxit) {
    ++it;
    const unsigned int tag = base + (unsigned int)it;
    // Y: q = op nu, s = r - alf nu, t = u - alf q, nine sums (r in rb)
    if (__syncthreads_or(halo_nu(tag))) { ph.ok = false; break; }
    double s9[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int j = wid; j < ns; j += STR_NW) {
      const int k = j * 32 + lane;
      const bool ok = k < nb;
      float u = 0.0f, r0 = 0.0f, f0 = 0.0f;
      if (ok) {
        u = uv[k];
        r0 = r0v[k];
        f0 = f0v[k];
      }
      const float nu = nub[k], q = gather(j, nub, nu);
      if (!ok) continue;
      const float s = rb[k] - ay * nu, t = u - ay * q;
      qv[k] = q;
      sv[k] = s;
      tv[k] = t;
      put_st(k, s, t, tag);
      const double sd = s, td = t, od = r0, fd = f0;
      s9[0] += td * sd;
      s9[1] += td * td;
      s9[2] += sd * sd;
      s9[3] += od * sd;
      s9[4] += od * td;
      s9[5] += fd * sd;
      s9[6] += fd * td;
      s9[7] += od * (double)q;
      s9[8] += od * (double)nu;
    }
    publish_sums<9, STR_NW>(s9, act, s_sum, B.slots, nt, tile, it & 1, tag);
    bool fail = halo_st(tag);
    fail |= collect_sums<9, STR_NW>(s_bc, B.slots, tot, nt, tile, it & 1, tag, A.bar, A.spin_limit);
    if (__syncthreads_or(fail)) { ph.ok = false; break; }
    const double omg = resident_omega(s_bc);
    w = (float)omg;
    if (wid == STR_NW - 1) resident_scalars(s_bc, omg, s_st, s_sc, it, A.maxit);
    for (int h = threadIdx.x; h < nh; h += STR_BS) rb[hb + h] = rb[hb + h] - w * nub[hb + h];
    rows([&](int k) { rb[k] = sv[k] - w * tv[k]; });
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
    // X: u = op r, the y update, p and nu
    for (int j = wid; j < ns; j += STR_NW) {
      const int k = j * 32 + lane;
      const bool ok = k < nb;
      float y = 0.0f, p = 0.0f, s = 0.0f, q = 0.0f;
      if (ok) {
        y = yv[k];
        p = pv[k];
        s = sv[k];
        q = qv[k];
      }
      const float r = rb[k], u = gather(j, rb, r), nu = nub[k];
      if (!ok) continue;
      if (park) A.yb[g1 + __ldg(B.trow + t0 + k)] = y;
      yv[k] = y + ax * p + w * s;
      uv[k] = u;
      pv[k] = r + be * (p - w * nu);
      const float nn = u + be * (nu - w * q);
      nub[k] = nn;
      put_nu(k, nn, tag + 1u);
    }
    pending = false;
  }
  // the best iterate: the last one (its y update still pending), y or yb;
  // x_B = S^-1 y, then x_0 = D0^-1 (b_0 + sum aoff x_B)
  const bool last = !pending || save;
  if (ph.ok && !nonfinite) {
    rows([&](int k) {
      const int r = g1 + __ldg(B.trow + t0 + k);
      float y;
      if (last || y_best) {
        y = yv[k];
        if (last && pending) y = y + ax * pv[k] + w * sv[k];
      } else {
        y = A.yb[r];
      }
      A.x[r] = y * __ldg(&A.sinv[r]);
    });
    grid_barrier(A, ph);
    if (ph.ok) {
      const int r1 = (int)((long long)g1 * (tile + 1) / nt);
      for (int r = (int)((long long)g1 * tile / nt) + (int)threadIdx.x; r < r1; r += STR_BS) {
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

// Shared memory of a tile with nb own and nh halo rows and nvs vectors.
inline size_t stream_smem(int nb, int nh, int nvs) {
  const size_t hb = ((size_t)nb + 31) / 32 * 32;
  return sizeof(float) * (2 * (hb + nh) + nvs * hb) + sizeof(int) * (hb / 32 + 1);
}

}  // namespace cms
