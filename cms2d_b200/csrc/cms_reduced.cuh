// ILU(0)-BiCGStab and GMRES(3) on the rows of groups >= 1 of a multicolour
// ordering, one cooperative launch per solve (BiCGStab in FP64, GMRES in FP64 and FP32).
//
// Group 0 is an independent set placed first, so with A = [D0 A0B; AB0 ABB]
// the multicolour ILU(0) factor is
//
//   M = [I 0; AB0/D0 I] diag(D0, M_S) [I D0^-1 A0B; 0 I],
//
// M_S the factor's part among the rows of the later groups (set B), and with
// the exact Schur complement C = ABB - AB0 D0^-1 A0B
//
//   A M^-1 (v_0, v_B) = (v_0, C M_S^-1 (v_B - g) + g),   g = AB0 D0^-1 v_0.
//
// The operator of the right-preconditioned Krylov methods keeps the group-0
// part of a vector as it is.  So every vector of the iteration is (c rho, v_B)
// with one scalar c per vector and rho the group-0 part of the first residual:
// the methods of pbicgstab.f90:20-96 and pgmres.f90:129-241 run here on v_B
// and c, with the inner products of the full vectors (c c' rho.rho +
// v_B.v'_B).  They are the same iterates as with triangular sweeps over the
// whole matrix, up to rounding, on half the rows and with one gather per
// operator application (GMRES looks at b - A x again where rounding has come
// between it and the recurrence, see GmState).  x_B collects M_S^-1 (v_B - c g); x_0 follows at the
// end from A's group-0 rows and the group-0 residual c rho.
//
// M_S is diagonal except at rows coupled to other B rows (telescoping
// interfaces, "special" rows, about 1 %).  Their small sweeps are done by
// every tile for the rows it needs, on an extended halo, group by group in
// shared memory, with no further exchange.
//
// Blocks, tiles, exchanged words and sums are those of cms_resident.cuh; the
// safety of reusing a word follows from the sums between any two operator
// applications: a tile contributes to them after it has read its halo, and a
// word is written again after the sums are known.  A sum's word has two
// copies by parity.  The vectors (own rows, tile order) and C's packed slices
// lie in shared memory as far as they fit, else in global memory (read once
// per application, coalesced); the gathered vector always in shared memory.
//
// Measured, bound and chosen range: at run_reduced's rule in
// cms_reduced_host.cuh.
#pragma once
#include "cms_resident.cuh"

namespace cms {

constexpr unsigned short RED_SIMPLE = 0xffff;
constexpr int RED_NV_BICG = 8;   // x, invd, g, r0, v, u, p, r
constexpr int RED_NV_GMRES = 7;  // x, invd, g, v1..v4

template <typename T>
struct RedArgs {
  int n, g1, nB, KL, nt, tile;
  const int *tptr, *trow;    // [nt+1] rows of a tile (reduced rows)
  const int* tpad;           // [nt] first padded row of a tile (slices of 32)
  const int* rexp;           // [nB, tile order] word of a row that other tiles gather, -1 none
  const unsigned short* kind;  // [nB, tile order] own special row's ordinal, RED_SIMPLE
  const int *hptr, *hword;   // [nt+1] halo words
  const int *slptr, *sloff;  // slot-pair offsets of a tile's slices
  const int* mbase;          // [nt] first slot-pair row (of 32) of the tile in the packed arrays
  const void* pcoef;         // packed pairs of T
  const ushort2* plcol;
  int nphase;                // phases of the special rows' sweeps: groups 2.., then G-1 .. 1
  const int* spp;            // [nt][nphase+1] special rows per phase (offsets into sprow)
  const int2* sprow;         // local row, device row
  const int* spe;            // [rows+1] entries of a special row
  const int* spoff;          // entry: offset into luoff
  const unsigned short* spcol;  // entry: local column
  const int *osptr, *osrow;  // [nt+1] own special rows (local), in order of their ordinals
  int nfwd;                  // the first nfwd phases are the forward ones
  const T *luoff, *invd, *aoff, *diag, *b, *cdiag;  // cdiag [nB]: C's diagonal
  T* x;
  T* rho;                    // [n]: the first residual (group-0 rows are read back)
  const int* col;
  const signed char *nlo, *nup;
  T* gvec;                   // [vectors][padded rows] vectors not in shared memory
  size_t npad;
  int nvs, mat_smem;         // vectors in shared memory (the last ones), packed C in shared memory
  ulonglong2 *xw, *slots;
  unsigned int tag0;
  GridBar* bar;
  DevState* st;
  int maxit, norm, xzero;
  double tol;
  unsigned int spin_limit;
  unsigned int* progress;  // (grid_barrier's argument fields)
  int ntiles;
};

__device__ __forceinline__ unsigned long long to_bits(double v) { return (unsigned long long)__double_as_longlong(v); }
__device__ __forceinline__ unsigned long long to_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ void from_bits(unsigned long long b, double& v) { v = __longlong_as_double((long long)b); }
__device__ __forceinline__ void from_bits(unsigned long long b, float& v) { v = __uint_as_float((unsigned int)b); }
template <typename T> struct Pair;
template <> struct Pair<double> { using type = double2; };
template <> struct Pair<float> { using type = float2; };

// C's coefficients in the packed slices and its diagonal, from A
// (coff = -C_ik, sums in FP64), and the part of the ILU(0) factor that the
// solve needs: 1/C_rr for the rows without couplings among B rows, whose
// factor row that is; for the special rows C's values at A's couplings among B
// rows, which are the final upper entries of a group-1 row and the start of the
// others' elimination (k_red_special).  (This and k_red_special replace a
// factorisation of all rows, one launch per group: at 1M cells FP64 117 us and
// 71 us for the coefficients; now 55 us together.)
template <typename T, int KS>
__global__ void __launch_bounds__(TPB, 4) k_red_pack(int n, int g1, int nB, int KL, const int* __restrict__ col,
                                                     const signed char* __restrict__ nlo,
                                                     const signed char* __restrict__ nup, const T* __restrict__ aoff,
                                                     const T* __restrict__ diag, SchurMap M,
                                                     const signed char* __restrict__ ccnt,
                                                     const int2* __restrict__ ppos,
                                                     typename Pair<T>::type* __restrict__ pcoef,
                                                     T* __restrict__ cdiag, T* __restrict__ luoff,
                                                     T* __restrict__ invd) {
  __shared__ double s_acc[KSC][TPB];
  double* acc = &s_acc[0][threadIdx.x];
  for (int i = blockIdx.x * TPB + threadIdx.x; i < nB; i += gridDim.x * TPB) {
    const int r = g1 + i, kc = ccnt[i], kl = nlo[r], kt = kl + nup[r];
    for (int q = 0; q < kc; ++q) acc[q * TPB] = 0.0;
    double d = diag[r];
    schur_row<T, KS>(n, g1, nB, KL, i, kl, kt, col, aoff, diag, M.smap, acc, d);
    cdiag[i] = (T)d;
    invd[r] = (T)(1.0 / d);
    for (int c = 0; c < kt; ++c) {
      const size_t e = (size_t)(c < kl ? c : KL + (c - kl)) * n + r;
      if (__ldg(col + e) >= g1) luoff[e] = (T)-acc[(int)(__ldg(M.smap + (size_t)c * nB + i) & 0xff) * TPB];
    }
    const int2 pp = ppos[i];
    for (int q = 0; q < pp.y; ++q) {
      typename Pair<T>::type v;
      v.x = 2 * q < kc ? (T)acc[2 * q * TPB] : T(0);
      v.y = 2 * q + 1 < kc ? (T)acc[(2 * q + 1) * TPB] : T(0);
      pcoef[(size_t)pp.x + (size_t)q * 32] = v;
    }
  }
}

// ILU(0) elimination among B rows for the special rows of group g >= 2 (rows
// in list): k_ilu0's steps on the couplings to B rows, the couplings to group
// 0 already eliminated.
template <typename T>
__global__ void __launch_bounds__(TPB) k_red_special(int n, int g1, int KL, int count, const int* __restrict__ list,
                                                     const int* __restrict__ col, const signed char* __restrict__ nlo,
                                                     const signed char* __restrict__ nup, const T* __restrict__ cdiag,
                                                     T* luoff, T* invd) {
  for (int p = blockIdx.x * TPB + threadIdx.x; p < count; p += gridDim.x * TPB) {
    const int r = list[p], kl = nlo[r], ku = nup[r];
    T al[KMAX], au[KMAX];
    int cl[KMAX], cu[KMAX];
#pragma unroll
    for (int s = 0; s < KMAX; ++s) {
      cl[s] = cu[s] = -1;
      al[s] = au[s] = T(0);
      if (s < kl) {
        const int c = col[(size_t)s * n + r];
        if (c >= g1) {
          cl[s] = c;
          al[s] = luoff[(size_t)s * n + r];
        }
      }
      if (s < ku) {
        cu[s] = col[(size_t)(KL + s) * n + r];
        au[s] = luoff[(size_t)(KL + s) * n + r];
      }
    }
    T d = cdiag[r - g1];
#pragma unroll
    for (int s = 0; s < KMAX; ++s) {
      const int j = cl[s];
      if (j < 0) continue;
      const T lij = al[s] * invd[j];
      al[s] = lij;
      const int nuj = nup[j];
#pragma unroll 1
      for (int t2 = 0; t2 < nuj; ++t2) {
        const int k = col[(size_t)(KL + t2) * n + j];
        const T ujk = luoff[(size_t)(KL + t2) * n + j];
        if (k == r) {
          d = d - lij * ujk;
        } else {
#pragma unroll
          for (int s2 = s + 1; s2 < KMAX; ++s2)
            if (cl[s2] == k) al[s2] = al[s2] - lij * ujk;
#pragma unroll
          for (int t = 0; t < KMAX; ++t)
            if (cu[t] == k) au[t] = au[t] - lij * ujk;
        }
      }
    }
    invd[r] = T(1) / d;
#pragma unroll
    for (int s = 0; s < KMAX; ++s) {
      if (s < kl && cl[s] >= 0) luoff[(size_t)s * n + r] = al[s];
      if (s < ku) luoff[(size_t)(KL + s) * n + r] = au[s];
    }
  }
}

// What a block works with: its tile's sizes and arrays.
template <typename T>
struct RedTile {
  using P2 = typename Pair<T>::type;
  int nb, ns, hb, nh, t0, nsp, nosp;
  const int* spp;
  int* soff;
  unsigned short* kind;
  T* zb;
  int2* sp_row;         // local row, first entry
  T *sp_inv, *sp_val;
  unsigned short* sp_col;
  unsigned short* os_row;  // own special rows
  T *os_cd, *os_z;      // C's diagonal; z of GMRES's three applications
  const P2* cf;
  const ushort2* lc;
  T* vec[RED_NV_BICG];
};

__device__ __forceinline__ size_t red_up16(size_t b) { return (b + 15) & ~(size_t)15; }

// Lays the tile out in shared memory and loads its tables.
template <typename T, int BS>
__device__ __forceinline__ void red_setup(const RedArgs<T>& A, RedTile<T>& L, unsigned char* smem, int nvec) {
  using P2 = typename Pair<T>::type;
  const int tile = A.tile;
  L.t0 = __ldg(A.tptr + tile);
  L.nb = __ldg(A.tptr + tile + 1) - L.t0;
  L.ns = (L.nb + 31) >> 5;
  L.hb = L.ns * 32;
  const int h0 = __ldg(A.hptr + tile);
  L.nh = __ldg(A.hptr + tile + 1) - h0;
  L.spp = A.spp + (size_t)tile * (A.nphase + 1);
  const int s0 = __ldg(L.spp), o0 = __ldg(A.osptr + tile);
  L.nsp = __ldg(L.spp + A.nphase) - s0;
  L.nosp = __ldg(A.osptr + tile + 1) - o0;
  const int e0 = __ldg(A.spe + s0), ne = __ldg(A.spe + s0 + L.nsp) - e0;
  const int* sog = A.sloff + __ldg(A.slptr + tile);
  const int npair = L.ns > 0 ? __ldg(sog + L.ns) : 0;
  unsigned char* p = smem;
  auto take = [&](size_t bytes) {
    unsigned char* q = p;
    p += red_up16(bytes);
    return q;
  };
  L.zb = (T*)take(sizeof(T) * ((size_t)L.hb + L.nh));
  L.soff = (int*)take(sizeof(int) * (L.ns + 1));
  L.kind = (unsigned short*)take(sizeof(unsigned short) * L.hb);
  L.sp_row = (int2*)take(sizeof(int2) * (L.nsp + 1));
  L.sp_inv = (T*)take(sizeof(T) * L.nsp);
  L.sp_val = (T*)take(sizeof(T) * ne);
  L.sp_col = (unsigned short*)take(sizeof(unsigned short) * ne);
  L.os_row = (unsigned short*)take(sizeof(unsigned short) * L.nosp);
  L.os_cd = (T*)take(sizeof(T) * L.nosp);
  L.os_z = (T*)take(sizeof(T) * 3 * L.nosp);
  const P2* gcf = (const P2*)A.pcoef + (size_t)__ldg(A.mbase + tile) * 32;
  const ushort2* glc = A.plcol + (size_t)__ldg(A.mbase + tile) * 32;
  L.cf = gcf;
  L.lc = glc;
  const int tid = threadIdx.x;
  for (int v = 0; v < nvec; ++v)
    L.vec[v] = v >= nvec - A.nvs ? (T*)take(sizeof(T) * L.hb) : A.gvec + (size_t)v * A.npad + __ldg(A.tpad + tile);
  if (A.mat_smem) {
    P2* cf = (P2*)take(sizeof(P2) * 32 * npair);
    ushort2* lc = (ushort2*)take(sizeof(ushort2) * 32 * npair);
    for (int e = tid; e < npair * 32; e += BS) {
      cf[e] = __ldg(gcf + e);
      lc[e] = __ldg(glc + e);
    }
    L.cf = cf;
    L.lc = lc;
  }
  for (int j = tid; j <= L.ns; j += BS) L.soff[j] = L.ns > 0 ? __ldg(sog + j) : 0;
  for (int k = tid; k < L.hb; k += BS) L.kind[k] = k < L.nb ? __ldg(A.kind + L.t0 + k) : RED_SIMPLE;
  for (int s = tid; s <= L.nsp; s += BS) {
    int2 v = make_int2(0, __ldg(A.spe + s0 + s) - e0);
    if (s < L.nsp) {
      const int2 rr = __ldg(A.sprow + s0 + s);
      v.x = rr.x;
      L.sp_inv[s] = __ldg(A.invd + rr.y);
    }
    L.sp_row[s] = v;
  }
  for (int e = tid; e < ne; e += BS) {
    L.sp_val[e] = __ldg(A.luoff + __ldg(A.spoff + e0 + e));
    L.sp_col[e] = __ldg(A.spcol + e0 + e);
  }
  for (int o = tid; o < L.nosp; o += BS) {
    const int k = __ldg(A.osrow + o0 + o);
    L.os_row[o] = (unsigned short)k;
    L.os_cd[o] = __ldg(A.cdiag + __ldg(A.trow + L.t0 + k));
  }
  __syncthreads();
}

// out = B part of A M^-1 (c rho, src); zb = M_S^-1 (src - c g) on own rows.
// False when a wait gave up.
template <typename T, int BS>
__device__ __forceinline__ bool red_apply(const RedArgs<T>& A, const RedTile<T>& L, const T* src, const T* g,
                                          const T* invd, double c, T* out, unsigned int tag, int zslot) {
  constexpr int NW = (BS / 32), HU = 4;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const T ct = (T)c;
  for (int j = wid; j < L.ns; j += NW) {
    const int k = j * 32 + lane;
    if (k < L.nb) {
      const T v = src[k] - ct * g[k];
      const T e = L.kind[k] == RED_SIMPLE ? invd[k] * v : v;
      L.zb[k] = e;
      const int w = __ldg(A.rexp + L.t0 + k);
      if (w >= 0) st_word16(A.xw + w, to_bits(e), tag);
    }
  }
  bool fail = false;
  const int* hw = A.hword + __ldg(A.hptr + A.tile);
  for (int h = threadIdx.x; h < L.nh; h += HU * BS) {
    unsigned long long v[HU], t[HU];
    unsigned int spins = 0;
    int i[HU];
#pragma unroll
    for (int u = 0; u < HU; ++u) i[u] = __ldg(hw + (h + u * BS < L.nh ? h + u * BS : h));
    for (;;) {
      bool all = true;
#pragma unroll
      for (int u = 0; u < HU; ++u) {
        v[u] = 0ull;
        t[u] = tag;
        if (h + u * BS < L.nh) ld_word16(A.xw + i[u], v[u], t[u]);
      }
#pragma unroll
      for (int u = 0; u < HU; ++u) all = all && t[u] == tag;
      if (all) break;
      if (poll_failed(A.bar, spins, A.spin_limit)) { fail = true; break; }
    }
#pragma unroll
    for (int u = 0; u < HU; ++u)
      if (h + u * BS < L.nh) from_bits(v[u], L.zb[L.hb + h + u * BS]);
  }
  if (__syncthreads_or(fail)) return false;
  if (L.nsp > 0) {  // the special rows' sweeps, group by group
    const int s0 = __ldg(L.spp);
    for (int ph = 0; ph < A.nphase; ++ph) {
      const int a = __ldg(L.spp + ph) - s0, b = __ldg(L.spp + ph + 1) - s0;
      for (int s = a + (int)threadIdx.x; s < b; s += BS) {
        const int2 r = L.sp_row[s];
        const int e1 = L.sp_row[s + 1].y;
        T acc = L.zb[r.x];
        for (int e = r.y; e < e1; ++e) acc = acc - L.sp_val[e] * L.zb[L.sp_col[e]];
        L.zb[r.x] = ph < A.nfwd ? acc : L.sp_inv[s] * acc;
      }
      __syncthreads();
    }
    if (zslot >= 0)
      for (int o = threadIdx.x; o < L.nosp; o += BS) L.os_z[zslot * L.nosp + o] = L.zb[L.os_row[o]];
  }
  for (int j = wid; j < L.ns; j += NW) {
    const int k = j * 32 + lane;
    const unsigned short kd = L.kind[k];
    T acc = T(0);
    if (k < L.nb) acc = kd == RED_SIMPLE ? src[k] : L.os_cd[kd] * L.zb[k] + ct * g[k];
    const int e = L.soff[j + 1];
#pragma unroll 4
    for (int s = L.soff[j]; s < e; ++s) {
      const typename Pair<T>::type a = L.cf[s * 32 + lane];
      const ushort2 l = L.lc[s * 32 + lane];
      acc = acc - a.x * L.zb[l.x];
      acc = acc - a.y * L.zb[l.y];
    }
    if (k < L.nb) out[k] = acc;
  }
  return true;
}

// Block sums, exchanged; the totals in bc for every thread.  False on a wait
// that gave up.  all: values of every warp (the group-0 rows are dealt to all
// threads), else of the warps that have slices of own rows.
template <typename T, int BS, int NS>
__device__ __forceinline__ bool red_sums(const RedArgs<T>& A, const RedTile<T>& L, double (&v)[NS],
                                         double (*sm)[(BS / 32)], double* bc, int buf, unsigned int tag, bool fail,
                                         bool all = false) {
  ulonglong2* tot = A.slots + (size_t)2 * NSMAX * A.nt;
  publish_sums<NS, (BS / 32)>(v, all || (int)(threadIdx.x >> 5) < L.ns, sm, A.slots, A.nt, A.tile, buf, tag);
  fail |= collect_sums<NS, (BS / 32)>(bc, A.slots, tot, A.nt, A.tile, buf, tag, A.bar, A.spin_limit);
  return !__syncthreads_or(fail);
}

// r = b - A x (+ add) of the own rows and this block's share of the group-0
// rows (stored in A.rho), g; sums |r_B|, r_B^2, |rho|, rho^2 and, with NS = 5,
// (d x)^2 over the rows of both.  first: the start of a solve, which also loads x and invd;
// else A.x is what red_finish has stored.
template <typename T, int BS, int NS>
__device__ __forceinline__ bool red_start(const RedArgs<T>& A, const RedTile<T>& L, T* x, T* invd, T* g, T* r, T add,
                                          double (&sum)[NS], PhaseState& ph, bool first = true) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, n = A.n, g1 = A.g1;
  const bool zero = first && A.xzero;
  auto resid = [&](int row, T xr) {
    T acc = T(0);
    if (!zero) {
      const int kl = __ldg(A.nlo + row), ku = __ldg(A.nup + row);
      for (int s = 0; s < kl + ku; ++s) {
        const size_t e = (size_t)(s < kl ? s : A.KL + (s - kl)) * n + row;
        acc = acc + __ldg(A.aoff + e) * ldm(A.x + __ldg(A.col + e));
      }
      const T dx = __ldg(A.diag + row) * xr;
      if constexpr (NS == 5) sum[4] += (double)dx * (double)dx;
      acc = acc + __ldg(A.b + row) - dx;
    } else {
      acc = __ldg(A.b + row);
    }
    return acc + add;
  };
#pragma unroll
  for (int q = 0; q < NS; ++q) sum[q] = 0.0;
  const int r1 = (int)((long long)g1 * (A.tile + 1) / A.nt);
  for (int row = (int)((long long)g1 * A.tile / A.nt) + (int)threadIdx.x; row < r1; row += BS) {
    const T v = resid(row, zero ? T(0) : ldm(A.x + row));
    A.rho[row] = v;
    sum[2] += fabs((double)v);
    sum[3] += (double)v * (double)v;
  }
  for (int j = wid; j < L.ns; j += (BS / 32)) {
    const int k = j * 32 + lane;
    if (k >= L.nb) continue;
    const int row = g1 + __ldg(A.trow + L.t0 + k);
    const T xr = first ? (zero ? T(0) : A.x[row]) : x[k];
    const T v = resid(row, xr);
    r[k] = v;
    if (first) {
      x[k] = xr;
      invd[k] = __ldg(A.invd + row);
    }
    sum[0] += fabs((double)v);
    sum[1] += (double)v * (double)v;
  }
  grid_barrier(A, ph);  // A.rho written, A.x no longer read
  if (!ph.ok) return false;
  for (int j = wid; j < L.ns; j += (BS / 32)) {
    const int k = j * 32 + lane;
    if (k >= L.nb) continue;
    const int row = g1 + __ldg(A.trow + L.t0 + k);
    T acc = T(0);
    const int kl = __ldg(A.nlo + row);
    for (int s = 0; s < kl; ++s) {
      const size_t e = (size_t)s * n + row;
      const int c = __ldg(A.col + e);
      if (c < g1) acc = acc - __ldg(A.aoff + e) * (ldm(A.rho + c) / __ldg(A.diag + c));
    }
    g[k] = acc;
  }
  return true;
}

// End: x_B, then x_0 = (b_0 - c rho + sub + sum aoff x_B) / d_0.
template <typename T, int BS>
__device__ __forceinline__ void red_finish(const RedArgs<T>& A, const RedTile<T>& L, const T* x, double c, T sub,
                                           PhaseState& ph) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int j = wid; j < L.ns; j += (BS / 32)) {
    const int k = j * 32 + lane;
    if (k < L.nb) A.x[A.g1 + __ldg(A.trow + L.t0 + k)] = x[k];
  }
  grid_barrier(A, ph);
  if (!ph.ok) return;
  const T ct = (T)c;
  const int r1 = (int)((long long)A.g1 * (A.tile + 1) / A.nt);
  for (int row = (int)((long long)A.g1 * A.tile / A.nt) + (int)threadIdx.x; row < r1; row += BS) {
    T acc = __ldg(A.b + row) - (ct * ldm(A.rho + row) - sub);
    const int ku = __ldg(A.nup + row);
    for (int t2 = 0; t2 < ku; ++t2) {
      const size_t e = (size_t)(A.KL + t2) * A.n + row;
      acc = acc + __ldg(A.aoff + e) * ldm(A.x + __ldg(A.col + e));
    }
    A.x[row] = acc / __ldg(A.diag + row);
  }
}

// BiCGStab (pbicgstab.f90:20-96).
template <typename T, int BS>
__global__ void __launch_bounds__(BS, 1) k_red_bicg(RedArgs<T> Ain) {
  extern __shared__ __align__(16) unsigned char red_smem[];
  __shared__ RedArgs<T> A;
  __shared__ RedTile<T> L;
  __shared__ double s_sum[NSMAX][(BS / 32)], s_bc[NSMAX];
  if (threadIdx.x == 0) {
    A = Ain;
    A.nt = A.ntiles = gridDim.x;
    A.tile = blockIdx.x;
  }
  __syncthreads();
  {
    RedTile<T> l;
    red_setup<T, BS>(A, l, red_smem, RED_NV_BICG);
    if (threadIdx.x == 0) L = l;
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nb = L.nb, ns = L.ns;
  T *x = L.vec[0], *invd = L.vec[1], *g = L.vec[2], *r0 = L.vec[3], *v = L.vec[4], *u = L.vec[5], *p = L.vec[6],
    *r = L.vec[7];
  PhaseState ph{0u, 0u, true, true};
  auto rows = [&](auto&& f) {
    for (int j = wid; j < ns; j += (BS / 32))
      if (j * 32 + lane < nb) f(j * 32 + lane);
  };
  unsigned int tag = A.tag0;
  int buf = 0;
  double s4[4];
  red_start<T, BS>(A, L, x, invd, g, r, (T)SMALL, s4, ph);
  rows([&](int k) {
    r0[k] = r[k];
    p[k] = T(0);
    u[k] = T(0);
  });
  bool ok = red_sums<T, BS, 4>(A, L, s4, s_sum, s_bc, buf, tag++, !ph.ok, true);
  buf ^= 1;
  const double rho1 = s_bc[2], rho2 = s_bc[3];
  double bet = s_bc[1] + rho2;
  const double res0 = A.norm == 1 ? s_bc[0] + rho1 : sqrt(bet);
  double alf = 1.0, bet0 = 1.0, gam = 1.0, rel = 1.0;
  double cp = 0.0, cu = 0.0, cr = 1.0;  // group-0 multiples of p, u, r (r0's is 1)
  int it = 0, converged = 0, nonfinite = 0;
  while (ok && it < A.maxit) {
    ++it;
    const double omg = bet * gam / (alf * bet0 + SMALL);
    const T om = (T)omg, al = (T)alf;
    cp = cr + omg * (cp - alf * cu);
    rows([&](int k) { p[k] = r[k] + om * (p[k] - al * u[k]); });
    ok = red_apply<T, BS>(A, L, p, g, invd, cp, u, tag++, -1);
    cu = cp;
    double s1[1] = {0.0};
    rows([&](int k) { s1[0] += (double)u[k] * (double)r0[k]; });
    ok = red_sums<T, BS, 1>(A, L, s1, s_sum, s_bc, buf, tag++, !ok);
    buf ^= 1;
    if (!ok) break;
    const double ukr0 = s_bc[0] + cu * rho2;
    gam = bet / ukr0;
    bet0 = bet;
    const T ga = (T)gam;
    cr = cr - gam * cu;
    rows([&](int k) {
      x[k] = x[k] + ga * L.zb[k];
      r[k] = r[k] - ga * u[k];
    });
    ok = red_apply<T, BS>(A, L, r, g, invd, cr, v, tag++, -1);
    double s2[2] = {0.0, 0.0};
    rows([&](int k) {
      const double vv = v[k];
      s2[0] += vv * (double)r[k];
      s2[1] += vv * vv;
    });
    ok = red_sums<T, BS, 2>(A, L, s2, s_sum, s_bc, buf, tag++, !ok);
    buf ^= 1;
    if (!ok) break;
    const double vr = s_bc[0] + cr * cr * rho2, vv = fmax(s_bc[1] + cr * cr * rho2, SMALL);
    alf = vr / vv;
    const T a2 = (T)alf;
    cr = cr - alf * cr;
    double s3[3] = {0.0, 0.0, 0.0};
    rows([&](int k) {
      x[k] = x[k] + a2 * L.zb[k];
      const T rn = r[k] - a2 * v[k];
      r[k] = rn;
      s3[0] += fabs((double)rn);
      s3[1] += (double)rn * (double)rn;
      s3[2] += (double)rn * (double)r0[k];
    });
    ok = red_sums<T, BS, 3>(A, L, s3, s_sum, s_bc, buf, tag++, false);
    buf ^= 1;
    if (!ok) break;
    const double res = A.norm == 1 ? s_bc[0] + fabs(cr) * rho1 : sqrt(s_bc[1] + cr * cr * rho2);
    rel = res / res0;
    bet = s_bc[2] + cr * rho2;
    if (!isfinite(rel)) { nonfinite = 1; break; }
    if (rel < A.tol) { converged = 1; break; }
  }
  if (ok) {
    ph.ok = true;
    red_finish<T, BS>(A, L, x, cr, (T)SMALL, ph);
  }
  if (A.tile == 0 && threadIdx.x == 0) {
    A.st->iter = it;
    A.st->s[S_RELRES] = rel;
    A.st->s[S_RES0] = res0;
    A.st->converged = converged;
    A.st->nonfinite = nonfinite;
    A.st->done = 1;
    A.st->s[S_BET] = bet;
  }
}

// GMRES(3) (pgmres.f90:129-241) with the basis vectors scaled only in the
// scalars: vh_1 is the residual, vh_{i+1} what is left of A M^-1 v_i after the
// orthogonalisation, v_i = a_i vh_i with a_i known after the next sums, so a
// step takes one reduction (vh_i.vh_i, vh_j.w, and vh_j.vh_i, which turn the
// products with w into those of the modified Gram-Schmidt steps) instead of
// 1 + i.  The norm that ends a step arrives with the next step's sums; a step
// begun although the last one met the tolerance is dropped.  The next cycle
// starts from the combination of the vh_i that the Hessenberg relation gives,
// until rounding may have taken that away from b - A x: then from b - A x
// itself, as pgmres does at every restart.  A cycle adds about u |A||x| of
// rounding to the difference (u the type's half unit, |A||x| taken as RED_DEV
// |D x|, or of the first residual where that is larger); once the sum passes
// RED_ETA of the residual it is computed anew and the sum starts over, the
// rule of van der Vorst and Ye's residual replacement (SIAM J. Sci. Comput. 22,
// 2000).  Near the attainable accuracy that is every cycle, so the stopping
// test sees what it saw with a residual per restart; in FP64 down to about
// 1e-11 of |D x| never.
constexpr double RED_ETA = 1e-3, RED_DEV = 10.0;
template <typename T> __device__ __forceinline__ constexpr double half_unit() { return sizeof(T) == 8 ? 1.1102230246251565e-16 : 5.9604644775390625e-08; }

struct GmState {
  double h[4][3];         // h[j][i]: coefficients of step i, h[i+1][i] the norm
  double rt[4][3];        // the same, rotated
  double a[4], c[4];      // scale of vh_i, its group-0 multiple
  double rs[4], gc[3], gs[3], y[3], e[4];
  double ro, ro0, eps;
  double dev, dx2;        // rounding since b - A x was formed, |D x|^2
  int i, inner, cyc, end, stop, nonfinite, converged;  // end: steps of the finished cycle
  int renew;              // the next cycle starts from b - A x
};

// Closes step i (0-based) with the norm^2 of vh_{i+1}: scale, rotations, the
// residual estimate; true when the cycle ends here.
__device__ __forceinline__ bool gm_close(GmState& G, int i, double nrm2) {
  const double t = sqrt(nrm2 + SMALL);
  G.h[i + 1][i] = t;
  G.a[i + 1] = 1.0 / fmax(t, SMALL);
  for (int k = 0; k <= i; ++k) G.rt[k][i] = G.h[k][i];
  for (int k = 0; k < i; ++k) {
    const double tt = G.rt[k][i], ck = G.gc[k], sk = G.gs[k];
    G.rt[k][i] = ck * tt + sk * G.rt[k + 1][i];
    G.rt[k + 1][i] = -sk * tt + ck * G.rt[k + 1][i];
  }
  double gam = sqrt(G.rt[i][i] * G.rt[i][i] + t * t);
  if (gam == 0.0) gam = SMALL;
  G.gc[i] = G.rt[i][i] / gam;
  G.gs[i] = t / gam;
  G.rs[i + 1] = -G.gs[i] * G.rs[i];
  G.rs[i] = G.gc[i] * G.rs[i];
  G.rt[i][i] = G.gc[i] * G.rt[i][i] + G.gs[i] * t;
  G.ro = fabs(G.rs[i + 1]);
  G.inner += 1;
  if (i < 2 && G.ro > G.eps) return false;
  // the cycle's coefficients y, and those of the next residual on vh_1..vh_{m+1}
  const int m = i + 1;
  double y[3];
  for (int k = 0; k < m; ++k) y[k] = G.rs[k];
  for (int k = m - 1; k >= 0; --k) {
    double tt = y[k];
    for (int j = k + 1; j < m; ++j) tt -= G.rt[k][j] * y[j];
    y[k] = tt / G.rt[k][k];
  }
  for (int l = 0; l <= m; ++l) {
    double e = l == 0 ? 1.0 : 0.0;
    for (int j = l; j < m; ++j) e -= y[j] * G.h[l][j] * G.a[l];
    if (l > 0) e -= y[l - 1];
    G.e[l] = e;
  }
  for (int k = 0; k < m; ++k) G.y[k] = y[k] * G.a[k];
  G.end = m;
  if (!isfinite(G.ro)) {
    G.nonfinite = 1;
    G.stop = 1;
  }
  if (G.ro <= G.eps) G.stop = 1;
  return true;
}

template <typename T, int BS>
__global__ void __launch_bounds__(BS, 1) k_red_gmres(RedArgs<T> Ain) {
  extern __shared__ __align__(16) unsigned char red_smem[];
  __shared__ RedArgs<T> A;
  __shared__ RedTile<T> L;
  __shared__ double s_sum[NSMAX][(BS / 32)], s_bc[NSMAX];
  __shared__ GmState G;
  if (threadIdx.x == 0) {
    A = Ain;
    A.nt = A.ntiles = gridDim.x;
    A.tile = blockIdx.x;
    G.inner = G.cyc = G.stop = G.nonfinite = G.converged = 0;
    G.ro = G.ro0 = G.eps = G.dev = 0.0;
    G.renew = 0;
    G.c[0] = 1.0;
  }
  __syncthreads();
  {
    RedTile<T> l;
    red_setup<T, BS>(A, l, red_smem, RED_NV_GMRES);
    if (threadIdx.x == 0) L = l;
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nb = L.nb, ns = L.ns;
  T *x = L.vec[0], *invd = L.vec[1], *g = L.vec[2];
  T *v0 = L.vec[3], *v1 = L.vec[4], *v2 = L.vec[5], *v3 = L.vec[6];
  PhaseState ph{0u, 0u, true, true};
  auto rows = [&](auto&& f) {
    for (int j = wid; j < ns; j += (BS / 32))
      if (j * 32 + lane < nb) f(j * 32 + lane);
  };
  unsigned int tag = A.tag0;
  int buf = 0, cyc = 0;
  double s5[5];
  red_start<T, BS>(A, L, x, invd, g, v0, T(0), s5, ph);
  bool ok = red_sums<T, BS, 5>(A, L, s5, s_sum, s_bc, buf, tag++, !ph.ok, true);
  buf ^= 1;
  double rho2 = s_bc[3];
  if (threadIdx.x == 0) G.dx2 = s_bc[4];
  double dx2 = 0.0;  // of this thread's rows
  bool stored = false;  // the result is in A.x
  while (ok && cyc < A.maxit) {
    // step 1: w = A M^-1 vh_1 (into v1); vh_1.vh_1, vh_1.w, and |D x|^2 after the last cycle
    ok = red_apply<T, BS>(A, L, v0, g, invd, G.c[0], v1, tag++, 0);
    double a3[3] = {0.0, 0.0, dx2};
    rows([&](int k) {
      const double p = v0[k];
      a3[0] += p * p;
      a3[1] += p * (double)v1[k];
    });
    ok = red_sums<T, BS, 3>(A, L, a3, s_sum, s_bc, buf, tag++, !ok);
    buf ^= 1;
    if (!ok) break;
    if (threadIdx.x == 0) {
      const double cc = G.c[0] * G.c[0] * rho2, ro = sqrt(s_bc[0] + cc + SMALL);
      if (cyc == 0) {
        G.eps = A.tol * ro;
        G.ro0 = ro;
      }
      G.ro = G.rs[0] = ro;
      G.a[0] = 1.0 / (ro + SMALL);
      G.end = 0;
      G.dx2 = fmax(G.dx2, 2.0 * s_bc[2]);  // (B rows: about half of them)
      const double h = G.a[0] * G.a[0] * (s_bc[1] + cc);
      G.h[0][0] = h;
      G.c[1] = G.a[0] * G.c[0] - h * G.a[0] * G.c[0];
    }
    __syncthreads();
    {
      const T p = (T)G.a[0], q = (T)(G.h[0][0] * G.a[0]);
      rows([&](int k) { v1[k] = p * v1[k] - q * v0[k]; });
    }
    // step 2: w = A M^-1 vh_2 (into v2)
    ok = red_apply<T, BS>(A, L, v1, g, invd, G.c[1], v2, tag++, 1);
    double b4[4] = {0.0, 0.0, 0.0, 0.0};
    rows([&](int k) {
      const double p = v0[k], q = v1[k], w = v2[k];
      b4[0] += q * q;
      b4[1] += p * q;
      b4[2] += p * w;
      b4[3] += q * w;
    });
    ok = red_sums<T, BS, 4>(A, L, b4, s_sum, s_bc, buf, tag++, !ok);
    buf ^= 1;
    if (!ok) break;
    if (threadIdx.x == 0) {
      const double c0 = G.c[0], c1 = G.c[1];
      if (!gm_close(G, 0, s_bc[0] + c1 * c1 * rho2)) {
        const double a0 = G.a[0], a1 = G.a[1];
        const double v01 = a0 * a1 * (s_bc[1] + c0 * c1 * rho2);
        const double h0 = a0 * a1 * (s_bc[2] + c0 * c1 * rho2);
        const double h1 = a1 * a1 * (s_bc[3] + c1 * c1 * rho2) - h0 * v01;
        G.h[0][1] = h0;
        G.h[1][1] = h1;
        G.c[2] = a1 * c1 - h0 * a0 * c0 - h1 * a1 * c1;
      }
    }
    __syncthreads();
    if (G.end == 0) {
      {
        const T p = (T)G.a[1], q = (T)(G.h[0][1] * G.a[0]), s = (T)(G.h[1][1] * G.a[1]);
        rows([&](int k) { v2[k] = p * v2[k] - q * v0[k] - s * v1[k]; });
      }
      // step 3: w = A M^-1 vh_3 (into v3)
      ok = red_apply<T, BS>(A, L, v2, g, invd, G.c[2], v3, tag++, 2);
      double c6[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      rows([&](int k) {
        const double p = v0[k], q = v1[k], s = v2[k], w = v3[k];
        c6[0] += s * s;
        c6[1] += p * s;
        c6[2] += q * s;
        c6[3] += p * w;
        c6[4] += q * w;
        c6[5] += s * w;
      });
      // (vh_2.vh_1 is needed again: kept in G.y until the cycle's end)
      if (threadIdx.x == 0) G.y[0] = s_bc[1];
      ok = red_sums<T, BS, 6>(A, L, c6, s_sum, s_bc, buf, tag++, !ok);
      buf ^= 1;
      if (!ok) break;
      if (threadIdx.x == 0) {
        const double c0 = G.c[0], c1 = G.c[1], c2 = G.c[2], p01 = G.y[0];
        if (!gm_close(G, 1, s_bc[0] + c2 * c2 * rho2)) {
          const double a0 = G.a[0], a1 = G.a[1], a2s = G.a[2];
          const double v01 = a0 * a1 * (p01 + c0 * c1 * rho2);
          const double v02 = a0 * a2s * (s_bc[1] + c0 * c2 * rho2), v12 = a1 * a2s * (s_bc[2] + c1 * c2 * rho2);
          const double h0 = a0 * a2s * (s_bc[3] + c0 * c2 * rho2);
          const double h1 = a1 * a2s * (s_bc[4] + c1 * c2 * rho2) - h0 * v01;
          const double h2 = a2s * a2s * (s_bc[5] + c2 * c2 * rho2) - h0 * v02 - h1 * v12;
          G.h[0][2] = h0;
          G.h[1][2] = h1;
          G.h[2][2] = h2;
          G.c[3] = a2s * c2 - h0 * a0 * c0 - h1 * a1 * c1 - h2 * a2s * c2;
        }
      }
      __syncthreads();
      if (G.end == 0) {
        const T p = (T)G.a[2], q = (T)(G.h[0][2] * G.a[0]), s = (T)(G.h[1][2] * G.a[1]),
                t = (T)(G.h[2][2] * G.a[2]);
        double d1[1] = {0.0};
        rows([&](int k) {
          const T w = p * v3[k] - q * v0[k] - s * v1[k] - t * v2[k];
          v3[k] = w;
          d1[0] += (double)w * (double)w;
        });
        ok = red_sums<T, BS, 1>(A, L, d1, s_sum, s_bc, buf, tag++, false);
        buf ^= 1;
        if (!ok) break;
        if (threadIdx.x == 0) gm_close(G, 2, s_bc[0] + G.c[3] * G.c[3] * rho2);
        __syncthreads();
      }
    }
    // x_B += M_S^-1 (sum y_j v_j - c g); the next residual
    const int m = G.end;
    const double cy = G.y[0] * G.c[0] + (m > 1 ? G.y[1] * G.c[1] : 0.0) + (m > 2 ? G.y[2] * G.c[2] : 0.0);
    const double cn = G.e[0] * G.c[0] + G.e[1] * G.c[1] + (m > 1 ? G.e[2] * G.c[2] : 0.0) +
                      (m > 2 ? G.e[3] * G.c[3] : 0.0);
    const T y0 = (T)G.y[0], y1 = m > 1 ? (T)G.y[1] : T(0), y2 = m > 2 ? (T)G.y[2] : T(0), ct = (T)cy;
    const T e0 = (T)G.e[0], e1 = (T)G.e[1], e2 = m > 1 ? (T)G.e[2] : T(0), e3 = m > 2 ? (T)G.e[3] : T(0);
    dx2 = 0.0;
    rows([&](int k) {
      const T p = v0[k], q = v1[k];
      T yv = y0 * p, rn = e0 * p + e1 * q;
      if (m > 1) {
        const T s = v2[k];
        yv = yv + y1 * q;
        rn = rn + e2 * s;
        if (m > 2) {
          yv = yv + y2 * s;
          rn = rn + e3 * v3[k];
        }
      }
      const unsigned short kd = L.kind[k];
      if (kd == RED_SIMPLE) {
        const T xk = x[k], di = invd[k];
        const T xn = xk + di * (yv - ct * g[k]);
        x[k] = xn;
        const double dx = (double)xn / (double)di;
        dx2 += dx * dx;
      } else {
        T z = y0 * L.os_z[kd];
        if (m > 1) z = z + y1 * L.os_z[L.nosp + kd];
        if (m > 2) z = z + y2 * L.os_z[2 * L.nosp + kd];
        x[k] = x[k] + z;
      }
      v0[k] = rn;
    });
    ++cyc;
    __syncthreads();  // G.c, G.y read
    if (threadIdx.x == 0) {
      G.c[0] = cn;
      const bool fresh = G.dev == 0.0;
      G.dev += half_unit<T>() * RED_DEV * fmax(sqrt(G.dx2), G.ro0);
      G.renew = G.dev > RED_ETA * G.ro && !(G.stop && fresh) ? 1 : 0;
    }
    __syncthreads();
    if (!G.renew) {
      if (G.stop) break;
      continue;
    }
    if (cyc >= A.maxit && !G.stop) break;
    red_finish<T, BS>(A, L, x, G.c[0], T(0), ph);
    grid_barrier(A, ph);
    if (ph.ok) red_start<T, BS>(A, L, x, invd, g, v0, T(0), s5, ph, false);
    ok = red_sums<T, BS, 5>(A, L, s5, s_sum, s_bc, buf, tag++, !ph.ok, true);
    buf ^= 1;
    if (!ok) break;
    rho2 = s_bc[3];
    if (threadIdx.x == 0) {
      G.c[0] = 1.0;
      G.dev = 0.0;
      G.dx2 = fmax(G.dx2, s_bc[4]);
      if (G.stop) {  // met by the cycle's estimate: by the residual too?
        G.ro = sqrt(s_bc[1] + rho2 + SMALL);
        if (!(G.ro <= G.eps)) G.stop = 0;
      }
    }
    __syncthreads();
    if (G.stop) {
      stored = true;
      break;
    }
  }
  if (ok && !stored) {
    ph.ok = true;
    red_finish<T, BS>(A, L, x, G.c[0], T(0), ph);
  }
  if (A.tile == 0 && threadIdx.x == 0) {
    A.st->iter = cyc;
    A.st->inner = G.inner;
    A.st->s[S_RELRES] = cyc > 0 ? G.ro / G.ro0 : 1.0;
    A.st->s[S_RO] = G.ro;
    A.st->converged = G.stop && !G.nonfinite ? 1 : 0;
    A.st->nonfinite = G.nonfinite;
    A.st->done = 1;
  }
}

// The kernel for a method (3 BiCGStab, FP64 only; 4 GMRES) and block size.
template <typename T>
inline const void* red_kernel(int nsolv, int bs) {
  if constexpr (sizeof(T) == 8) {
    if (nsolv == 3) return bs == 512 ? (const void*)k_red_bicg<T, 512> : (const void*)k_red_bicg<T, 1024>;
  }
  return bs == 512 ? (const void*)k_red_gmres<T, 512> : (const void*)k_red_gmres<T, 1024>;
}

}  // namespace cms
