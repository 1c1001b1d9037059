// GMRES(3) on the multicolour ILU(0) factor for small systems: the per-phase
// kernels of cms_krylov.cuh as one launch of a single thread-block cluster,
// with the same rounding.
//
// The flow step's GMRES has to keep its rounding (see solve_core64), so the
// reduced form of cms_reduced.cuh is not open to it.  The per-phase kernels
// take 25-31 launches per cycle, 2-6 us each on a 20k-cell system for less
// than 0.5 us of work.  Here 1 to 16 blocks of 1024 threads form one cluster:
// a phase ends at the cluster's hardware barrier (about 0.3 us against 1.7 us
// of a grid barrier through L2, and against a launch), the dot products'
// partial sums go to every block's shared memory, and every block forms the
// scalars.  The matrix and factor rows of a block stay in its shared memory
// when they fit.
//
// Same rounding: a row's sums run over its slots in the same order, and a dot
// product is added as grid_sum adds it: partial sums of the same 256-row
// blocks ("virtual blocks", four per block of this kernel at a time; by
// groups for the products formed with the matrix, over all rows for the
// Gram-Schmidt steps), each by the same warp and block tree, then the same
// tree over the partial sums.  What is fused (the scaling and the forward
// sweep of groups 0 and 1, the last group's backward step, group 0's backward
// step with its rows of the product) evaluates the same expressions.
//
// Measured (one B200, GMRES cycle of the default flow step on the 20k-cell
// basin): 130 us with the per-phase kernels, 53 us here; two steps of a flow
// model 171 -> 70 ms (20k cells, Cartesian), 209 -> 167 ms (62k), 215 -> 96
// ms (10k, telescoping), 293 -> 264 ms (51k).  Bound by the latency of a phase, about
// 20 phases per cycle: 1200-1500 cycles of the fence and the barrier, dependent
// loads through L2, and the trees of the sums.
#pragma once
#include <cooperative_groups.h>

#include "cms_krylov.cuh"

namespace cms {

constexpr int GMC_BS = 1024;           // threads per block: four virtual blocks of TPB rows
constexpr int GMC_SLOTS = GMC_BS / TPB;
constexpr int GMC_ROWS = 65536;        // largest system (4 rows per thread at 16 blocks)
constexpr int GMC_PART = 272;          // virtual blocks of a launch (256 + a partial one per group)

// product and sum rounded one by one (never contracted)
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }

template <typename T>
struct GmcArgs {
  int n, KL, maxit, stage;  // stage: couplings from global memory (0), A's (1), A's and the factor's (2) in shared memory
  double tol;
  GroupTab tab;
  int gku_last;
  const int* col;
  const signed char *nlo, *nup;
  const T *aoff, *diag, *luoff, *invd, *b;
  T *x, *z;
  T* vh[4];  // unscaled basis vectors
  T* vs[3];  // scaled ones
  DevState* st;
};

struct GmcState {
  double hh[4][3], c[4], s[4], rs[5], y[4], scale[5];
  double ro, ro0, eps, relres;
  int iter, inner, ifinal, stop, nonfinite, active, done, converged;
};

// The scalars that follow Gram-Schmidt step j of Arnoldi step i (both from 1)
// and its sum v (as the last block of k_mgs).
__device__ __forceinline__ void gmc_scalars(GmcState& G, int j, int i, double v) {
  auto HH = [&G](int jj, int ii) -> double& { return G.hh[jj - 1][ii - 1]; };
  if (j < i) {
    HH(j + 1, i) = v;
    return;
  }
  const int i1 = i + 1;
  double t = sqrt(v + SMALL);
  HH(i1, i) = t;
  G.scale[i] = 1.0 / fmax(t, SMALL);
  for (int k = 2; k <= i; ++k) {
    const int k1 = k - 1;
    const double tt = HH(k1, i);
    const double ck = G.c[k1], sk = G.s[k1];
    HH(k1, i) = ck * tt + sk * HH(k, i);
    HH(k, i) = -sk * tt + ck * HH(k, i);
  }
  double gam = sqrt(HH(i, i) * HH(i, i) + HH(i1, i) * HH(i1, i));
  if (gam == 0.0) gam = SMALL;
  const double ci = HH(i, i) / gam, si = HH(i1, i) / gam;
  G.c[i] = ci;
  G.s[i] = si;
  G.rs[i1] = -si * G.rs[i];
  G.rs[i] = ci * G.rs[i];
  HH(i, i) = ci * HH(i, i) + si * HH(i1, i);
  const double ro = fabs(G.rs[i1]);
  G.ro = ro;
  G.inner += 1;
  if (i < 3 && ro > G.eps) return;
  G.active = 0;
  G.ifinal = i;
  double rs[4];
  for (int k = 1; k <= i; ++k) rs[k] = G.rs[k];
  rs[i] = rs[i] / HH(i, i);
  for (int ii = 2; ii <= i; ++ii) {
    const int k = i - ii + 1, k1 = k + 1;
    double tt = rs[k];
    for (int jj = k1; jj <= i; ++jj) tt = tt - HH(k, jj) * rs[jj];
    rs[k] = tt / HH(k, k);
  }
  for (int k = 1; k <= i; ++k) G.y[k] = rs[k];
  G.relres = (double)ro / G.ro0;
  if (!isfinite((double)ro)) { G.nonfinite = 1; G.stop = 1; }
  if (ro <= G.eps) G.stop = 1;
}

// Barrier of the cluster that orders all its threads' accesses: the block
// barrier, one thread's fence, then the hardware barrier without a fence of
// its own (every warp's fence took most of a phase).  The .aligned forms want a
// converged warp, which the fence's branch leaves open.
__device__ __forceinline__ void gmc_sync() {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("fence.acq_rel.cluster;" ::: "memory");
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// NS: most couplings of a row (4 on Cartesian grids, 6 on telescoping ones), so that a row's gathers
// are all in flight before its sum starts.
template <typename T, int NS>
__global__ void __launch_bounds__(GMC_BS, 1) k_gmres_cluster(GmcArgs<T> Ain) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char gmc_smem[];
  __shared__ GmcArgs<T> A;
  __shared__ GmcState G;
  __shared__ double s_part[2][GMC_PART];
  __shared__ double s_w[GMC_SLOTS][8], s_tot;
  cg::cluster_group cl = cg::this_cluster();
  const int cta = (int)cl.block_rank(), nc = (int)cl.num_blocks();
  const int slot = threadIdx.x >> 8, t = threadIdx.x & 255, lane = threadIdx.x & 31, w8 = t >> 5;
  if (threadIdx.x == 0) {
    A = Ain;
    G.iter = G.inner = G.ifinal = G.stop = G.nonfinite = G.active = G.converged = 0;
    G.done = Ain.maxit <= 0 ? 1 : 0;
    G.relres = 1.0;
    G.ro = G.ro0 = G.eps = 0.0;
  }
  __syncthreads();
  const int n = A.n, ng = A.tab.ng, nbg = A.tab.blk[ng], nbr = (n + TPB - 1) / TPB;
  const int nlv = (nbg + nc - 1) / nc;  // virtual blocks (by groups) of this block, at most
  // a virtual block's row, by groups: -1 past its group
  auto row_of = [&](int vb, int& g) {
    g = tab_group(A.tab, vb);
    const int r = A.tab.start[g] + (vb - A.tab.blk[g]) * TPB + t;
    return r < A.tab.start[g + 1] ? r : -1;
  };
  // rows of this block in shared memory: diagonal, 1/u_rr, counts, and (stage)
  // the couplings' columns and values, lower slots then upper
  const int LR = nlv * TPB;
  T* sD = reinterpret_cast<T*>(gmc_smem);
  T* sI = sD + LR;
  T* sA = sI + LR;
  T* sL = sA + (A.stage >= 1 ? (size_t)NS * LR : 0);
  int* sC = reinterpret_cast<int*>(sL + (A.stage >= 2 ? (size_t)NS * LR : 0));
  unsigned char* sN = reinterpret_cast<unsigned char*>(sC + (A.stage >= 1 ? (size_t)NS * LR : 0));
  for (int lv = slot; lv < nlv; lv += GMC_SLOTS) {
    const int vb = cta + lv * nc, li = lv * TPB + t;
    int g;
    const int r = vb < nbg ? row_of(vb, g) : -1;
    sN[li] = 0;
    if (r < 0) continue;
    const int kl = A.nlo[r], ku = A.nup[r];
    sN[li] = (unsigned char)(kl | ku << 4);
    sD[li] = A.diag[r];
    sI[li] = A.invd[r];
    if (A.stage >= 1) {
      for (int q = 0; q < kl + ku; ++q) {
        const size_t e = (size_t)(q < kl ? q : A.KL + (q - kl)) * n + r;
        const size_t o = (size_t)q * LR + li;
        sA[o] = A.aoff[e];
        sC[o] = A.col[e];
        if (A.stage >= 2) sL[o] = A.luoff[e];
      }
    }
  }
  // the gathered values v(column) of entries [q0, q1) of a row (kl lower
  // entries first), and the entries' values in A or the factor
  auto gather = [&](T (&out)[NS], const T* v, int q0, int q1, int kl, int r, int li) {
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      out[q] = T(0);
      if (q >= q0 && q < q1) {
        const int c = A.stage >= 1 ? sC[(size_t)q * LR + li] : __ldg(A.col + (size_t)(q < kl ? q : A.KL + (q - kl)) * n + r);
        out[q] = __ldcg(v + c);
      }
    }
  };
  auto ent_a = [&](int q, int kl, int r, int li) {
    return A.stage >= 1 ? sA[(size_t)q * LR + li] : __ldg(A.aoff + (size_t)(q < kl ? q : A.KL + (q - kl)) * n + r);
  };
  auto ent_l = [&](int q, int kl, int r, int li) {
    return A.stage >= 2 ? sL[(size_t)q * LR + li] : __ldg(A.luoff + (size_t)(q < kl ? q : A.KL + (q - kl)) * n + r);
  };
  // f(row, group, local index) for the rows of groups ga..gb
  auto for_group = [&](int ga, int gb, auto&& f) {
    for (int lv = slot; lv < nlv; lv += GMC_SLOTS) {
      const int vb = cta + lv * nc;
      if (vb < A.tab.blk[ga] || vb >= A.tab.blk[gb + 1]) continue;
      int g;
      const int r = row_of(vb, g);
      if (r >= 0) f(r, g, lv * TPB + t);
    }
  };
  // partial sum of virtual block vb: grid_sum's block tree (its last steps add
  // zeros), then to every block
  auto put_part = [&](double v, int vb, int buf) {
    v = warp_sum(v);
    if (lane == 0) s_w[slot][w8] = v;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(TPB) : "memory");
    if (w8 == 0) {
      double x = s_w[slot][lane & 7];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane < nc) *cl.map_shared_rank(&s_part[buf][vb], lane) = x;
    }
    asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(TPB) : "memory");
  };
  // the total over nb partial sums, for thread 0 (grid_sum's last block)
  auto total = [&](int nb, int buf) {
    if (threadIdx.x < TPB) {
      double acc = 0.0;
      for (int b = threadIdx.x; b < nb; b += TPB) acc += s_part[buf][b];
      acc = warp_sum(acc);
      if (lane == 0) s_w[0][w8] = acc;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      double x = s_w[0][lane & 7];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (threadIdx.x == 0) s_tot = x;
    }
  };
  int buf = 0;
  auto fwd_row = [&](int r, int li) {  // y (in z) - sum of the lower entries
    const int kl = sN[li] & 15;
    T zv[NS];
    gather(zv, A.z, 0, kl, kl, r, li);
    T acc = __ldcg(A.z + r);
#pragma unroll
    for (int q = 0; q < NS; ++q)
      if (q < kl) acc = acc - ent_l(q, kl, r, li) * zv[q];
    return acc;
  };
  auto bwd_row = [&](int r, int li) {  // z - sum of the upper entries, without the factor 1/u_rr
    const int kl = sN[li] & 15, k = kl + (sN[li] >> 4);
    T zv[NS];
    gather(zv, A.z, kl, k, kl, r, li);
    T acc = __ldcg(A.z + r);
#pragma unroll
    for (int q = 0; q < NS; ++q)
      if (q >= kl && q < k) acc = acc - ent_l(q, kl, r, li) * zv[q];
    return acc;
  };
  const bool fuse = A.gku_last == 0;  // the last group's backward step needs no other row
  // z = (LU)^-1 y after groups 0 and 1 of the forward sweep (z holds it), up
  // to and without group 0's backward step; fin(row, invd, acc), z = invd acc,
  // for each finished row
  auto sweep_rest = [&](auto&& fin) {
    for (int g = 2; g < ng; ++g) {
      gmc_sync();
      for_group(g, g, [&](int r, int, int li) {
        T v = fwd_row(r, li);
        if (fuse && g == ng - 1) {
          fin(r, sI[li], v);
          v = sI[li] * v;
        }
        A.z[r] = v;
      });
    }
    for (int g = fuse ? ng - 2 : ng - 1; g >= 1; --g) {
      gmc_sync();
      for_group(g, g, [&](int r, int, int li) {
        const T v = bwd_row(r, li);
        fin(r, sI[li], v);
        A.z[r] = sI[li] * v;
      });
    }
    gmc_sync();
  };
  // every block of the cluster has started before the first store to its shared memory (put_part)
  gmc_sync();
  while (!G.done) {
    // restart residual v_1 = b - A x
    for (int lv = slot; lv < nlv; lv += GMC_SLOTS) {
      const int vb = cta + lv * nc;
      if (vb >= nbg) continue;
      int g;
      const int r = row_of(vb, g), li = lv * TPB + t;
      double v = 0.0;
      if (r >= 0) {
        const int kl = sN[li] & 15, k = kl + (sN[li] >> 4);
        T xv[NS];
        gather(xv, A.x, 0, k, kl, r, li);
        const T xr = __ldcg(A.x + r), br = __ldg(A.b + r);
        T sum = T(0);
#pragma unroll
        for (int q = 0; q < NS; ++q)
          if (q < k) sum = sum + ent_a(q, kl, r, li) * xv[q];
        const T vr = sum + br - sD[li] * xr;
        A.vh[0][r] = vr;
        v += (double)vr * (double)vr;
      }
      put_part(v, vb, buf);
    }
    gmc_sync();
    total(nbg, buf);
    buf ^= 1;
    if (threadIdx.x == 0) {
      const double ro = sqrt(s_tot + SMALL);
      if (G.iter == 0) {
        G.eps = A.tol * ro;
        G.ro0 = ro;
      }
      G.ro = ro;
      G.scale[0] = 1.0 / (ro + SMALL);
      G.rs[1] = ro;
      G.active = 1;
      G.ifinal = 0;
      G.stop = 0;
    }
    __syncthreads();
    for (int i = 1; i <= 3 && G.active; ++i) {
      // v_i scaled; forward sweep of groups 0 and 1 (a group-0 neighbour's z is
      // its scaled v), the last group's backward step when that is group 1
      const T sc = (T)G.scale[i - 1];
      const T* vi = A.vh[i - 1];
      for_group(0, ng > 1 ? 1 : 0, [&](int r, int g, int li) {
        const int kl = sN[li] & 15;
        T zv[NS];
        if (g == 1) gather(zv, vi, 0, kl, kl, r, li);
        const T y = sc * __ldcg(vi + r);
        A.vs[i - 1][r] = y;
        T acc = y;
        if (g == 1) {
#pragma unroll
          for (int q = 0; q < NS; ++q)
            if (q < kl) acc = acc - ent_l(q, kl, r, li) * mul_rn(sc, zv[q]);
          if (fuse && ng == 2) acc = sI[li] * acc;
        }
        A.z[r] = acc;
      });
      for (int g = 2; g < ng; ++g)
        for_group(g, g, [&](int r, int, int) {
          const T y = sc * __ldcg(vi + r);
          A.vs[i - 1][r] = y;
          A.z[r] = y;
        });
      sweep_rest([](int, T, T) {});
      // group 0's backward step and its rows of w = A z, then the other rows'
      T* w = A.vh[i];
      for_group(0, 0, [&](int r, int, int li) {
        const int kl = sN[li] & 15, k = kl + (sN[li] >> 4);
        T zv[NS];
        gather(zv, A.z, kl, k, kl, r, li);
        T acc = __ldcg(A.z + r), sum = T(0);
#pragma unroll
        for (int q = 0; q < NS; ++q)
          if (q >= kl && q < k) {
            acc = acc - ent_l(q, kl, r, li) * zv[q];
            sum = sum + ent_a(q, kl, r, li) * zv[q];
          }
        const T zr = sI[li] * acc;
        A.z[r] = zr;
        w[r] = sD[li] * zr - sum;
      });
      gmc_sync();
      for (int lv = slot; lv < nlv; lv += GMC_SLOTS) {
        const int vb = cta + lv * nc;
        if (vb >= nbg) continue;
        int g;
        const int r = row_of(vb, g), li = lv * TPB + t;
        double v = 0.0;
        if (r >= 0) {
          const T v1 = __ldcg(A.vs[0] + r);
          T yr;
          if (g == 0) {
            yr = w[r];  // (this thread's own store)
          } else {
            const int kl = sN[li] & 15, k = kl + (sN[li] >> 4);
            T zv[NS];
            gather(zv, A.z, 0, k, kl, r, li);
            const T zr = __ldcg(A.z + r);
            T sum = T(0);
#pragma unroll
            for (int q = 0; q < NS; ++q)
              if (q < k) sum = sum + ent_a(q, kl, r, li) * zv[q];
            yr = sD[li] * zr - sum;
            w[r] = yr;
          }
          v += (double)v1 * (double)yr;
        }
        put_part(v, vb, buf);
      }
      gmc_sync();
      total(nbg, buf);
      buf ^= 1;
      if (threadIdx.x == 0) G.hh[0][i - 1] = s_tot;
      __syncthreads();
      // modified Gram-Schmidt, over all rows in order; a thread's rows of w stay
      // in registers from step to step
      constexpr int RW = GMC_ROWS / (16 * GMC_BS);
      T wq[RW];
      for (int j = 1; j <= i; ++j) {
        const T h = (T)G.hh[j - 1][i - 1];
        T vj[RW], vn[RW];
#pragma unroll
        for (int m = 0; m < RW; ++m) {
          const int q = ((cta + m * nc) * GMC_SLOTS + slot) * TPB + t;
          if (q < n) {
            if (j == 1) wq[m] = __ldcg(w + q);
            vj[m] = __ldcg(A.vs[j - 1] + q);
            if (j < i) vn[m] = __ldcg(A.vs[j] + q);
          }
        }
#pragma unroll
        for (int m = 0; m < RW; ++m) {
          const int vb = (cta + m * nc) * GMC_SLOTS + slot, q = vb * TPB + t;
          if (vb >= nbr) continue;
          double v = 0.0;
          if (q < n) {
            if (h != T(0)) wq[m] = wq[m] + (-h) * vj[m];
            if (j == i) w[q] = wq[m];
            if (j < i) v += (double)vn[m] * (double)wq[m];
            else v += (double)wq[m] * (double)wq[m];
          }
          put_part(v, vb, buf);
        }
        gmc_sync();
        total(nbr, buf);
        buf ^= 1;
        if (threadIdx.x == 0) gmc_scalars(G, j, i, s_tot);
        __syncthreads();
      }
    }
    // x += (LU)^-1 sum y_j v_j
    const int ni = G.ifinal;
    for_group(0, ng - 1, [&](int r, int, int) {
      T y = T(0);
#pragma unroll
      for (int j = 1; j <= 3; ++j)
        if (j <= ni) y = y + __ldcg(A.vs[j - 1] + r) * (T)G.y[j];
      A.z[r] = y;
    });
    gmc_sync();
    auto add_x = [&](int r, T iv, T acc) { A.x[r] = add_rn(__ldcg(A.x + r), mul_rn(iv, acc)); };
    if (ng > 1)
      for_group(1, 1, [&](int r, int, int li) {
        T v = fwd_row(r, li);
        if (fuse && ng == 2) {
          add_x(r, sI[li], v);
          v = sI[li] * v;
        }
        A.z[r] = v;
      });
    sweep_rest(add_x);
    for_group(0, 0, [&](int r, int, int li) { add_x(r, sI[li], bwd_row(r, li)); });
    if (threadIdx.x == 0) {  // k_gm_cycle_end
      G.iter += 1;
      if (G.stop) {
        G.done = 1;
        G.converged = G.nonfinite ? 0 : 1;
      } else if (G.iter >= A.maxit) {
        G.done = 1;
      }
    }
    gmc_sync();
  }
  if (cta == 0 && threadIdx.x == 0) {
    DevState* st = A.st;
    st->iter = G.iter;
    st->inner = G.inner;
    st->maxit = A.maxit;
    st->s[S_TOL] = A.tol;
    st->s[S_RELRES] = G.relres;
    st->s[S_RO] = G.ro;
    st->s[S_RO0] = G.ro0;
    st->converged = G.converged;
    st->nonfinite = G.nonfinite;
    st->done = 1;
  }
}

template <typename T>
inline const void* gmc_kernel(int nslot) {
  return nslot <= 4 ? (const void*)k_gmres_cluster<T, 4>
                    : nslot <= 6 ? (const void*)k_gmres_cluster<T, 6> : (const void*)k_gmres_cluster<T, 8>;
}

}  // namespace cms
