// Host side of the reduced Krylov solves (cms_reduced.cuh): tables per handle,
// C's values per solve, the launches.  Included by cms_solver.cu after the
// reduced system's pattern (schur_pattern) and the tiles (resident_partition).
#pragma once

namespace cms {

constexpr int RED_WIDE = 1024;  // rows per tile above which a block has 1024 threads

// Shared memory of a tile besides its vectors and packed coefficients.
template <typename T>
static size_t red_smem_base(const RedTables& R, int t) {
  const size_t hb = R.hb[t], ns = hb / 32, nsp = R.h_nsp[t], ne = R.h_ne[t], nos = R.h_nos[t];
  auto up = [](size_t b) { return (b + 15) & ~(size_t)15; };
  return up(sizeof(T) * (hb + R.h_nh[t])) + up(4 * (ns + 1)) + up(2 * hb) + up(8 * (nsp + 1)) + up(sizeof(T) * nsp) +
         up(sizeof(T) * ne) + up(2 * ne) + up(2 * nos) + up(sizeof(T) * nos) + up(sizeof(T) * 3 * nos);
}

// How a launch with nvec vectors lays out its shared memory: the number of
// vectors kept there (the last ones, the most used), then C's packed slices if
// they fit too.  False when not even the gathered vector fits.
template <typename T>
static bool red_plan(const RedTables& R, int nvec, size_t limit, int* nvs, int* mat, size_t* smem) {
  auto up = [](size_t b) { return (b + 15) & ~(size_t)15; };
  auto need = [&](int v, int m) {
    size_t most = 0;
    for (int t = 0; t < R.tiles; ++t)
      most = std::max(most, red_smem_base<T>(R, t) + v * up(sizeof(T) * R.hb[t]) +
                                (m ? up(sizeof(T) * 64 * (size_t)R.h_npair[t]) + up(128 * (size_t)R.h_npair[t]) : 0));
    return most;
  };
  int v = nvec;
  while (v > 0 && need(v, 0) > limit) --v;
  if (need(v, 0) > limit) return false;
  *nvs = v;
  *mat = v == nvec && need(v, 1) <= limit ? 1 : 0;
  *smem = need(v, *mat);
  return true;
}

// Vectors of the streamed reduced solve (cms_schur_stream.cuh) that fit in
// shared memory beside the gathered ones, -1 when those do not; the launch's
// shared memory.
static int stream_vectors(const RedTables& R, size_t limit, size_t* smem) {
  for (int v = SV_N; v >= 0; --v) {
    size_t most = 0;
    for (int t = 0; t < R.tiles; ++t) most = std::max(most, stream_smem(R.hb[t], R.h_nh[t], v));
    *smem = most;
    if (most <= limit) return v;
  }
  return -1;
}

// Dynamic shared memory the kernels may use, set as their attribute.
static int red_limit(Solver* S, size_t* limit) {
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, S->dev) != cudaSuccess) return CMS_DEVICE_ERROR;
  const void* k[7] = {red_kernel<double>(3, 512), red_kernel<double>(3, 1024), red_kernel<double>(4, 512),
                      red_kernel<double>(4, 1024), red_kernel<float>(4, 512), red_kernel<float>(4, 1024),
                      (const void*)k_schur_stream};
  size_t most = (size_t)optin;
  for (const void* f : k) {
    cudaFuncAttributes fa;
    CMS_CUDA(cudaFuncGetAttributes(&fa, f));
    if (fa.sharedSizeBytes >= (size_t)optin) return CMS_UNSUPPORTED;
    most = std::min(most, (size_t)optin - fa.sharedSizeBytes);
  }
  for (const void* f : k) CMS_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
  *limit = most;
  return CMS_OK;
}

// What a tile of the reduced forms needs of shared memory at the least, as an
// average over the tiles (own rows and own special rows only), so that a system
// whose tiles cannot fit is left to the other forms without building the
// tables first (9M cells: 1.7 s; the count takes 30 ms).
static const RedRoom& red_room(Solver* S) {
  RedRoom& M = S->rroom;
  if (M.state != 0) return M;
  M.state = -1;
  const HostPattern& P = S->hp;
  size_t rs_limit = 0;
  const int blocks = resident_blocks(S->dev, &rs_limit);
  if (!P.symmetric || P.G < 2 || P.G > GFLAT || blocks <= 0 || red_limit(S, &M.limit) != CMS_OK) return M;
  const int n = P.n, g1 = P.gstart[1];
  M.tiles = resident_count(S, blocks);
  long long rows = 0, phases = 0, entries = 0;  // special rows, with their phases and the entries swept in these
  for (int g = 1; g < P.G; ++g) {
    for (int r = P.gstart[g]; r < P.gstart[g + 1]; ++r) {
      int lo = 0;
      for (int s = 0; s < P.nlo[r]; ++s) lo += P.col[(size_t)s * n + r] >= g1;
      if (lo + P.nup[r] == 0) continue;
      ++rows;
      phases += g >= 2 ? 2 : 1;
      entries += lo + P.nup[r];
    }
  }
  auto krylov = [&](double T) {
    return ((T + 2.0) * (n - g1) + (8.0 + T) * phases + (T + 2.0) * entries + (2.0 + 4.0 * T) * rows) / M.tiles;
  };
  M.krylov64 = krylov(sizeof(double));
  M.krylov32 = krylov(sizeof(float));
  M.stream = 2.0 * sizeof(float) * (n - g1) / M.tiles;
  if (std::min(M.krylov64, M.stream) <= (double)M.limit) M.state = 1;  // (red_tables wants one of them to fit)
  return M;
}

// Tables of the reduced Krylov solves for the handle's pattern, built on first
// use.  S->rd.state: 1 built, -1 the pattern or its size does not take them.
static int red_tables(Solver* S) {
  if (S->rd.state != 0) return CMS_OK;
  S->rd.state = -1;
  RedTables R;
  const HostPattern& P = S->hp;
  if (P.G < 2 || P.G > GFLAT || schur_pattern(S) != CMS_OK || !S->sc_sym) return CMS_OK;
  size_t rs_limit = 0;
  const int blocks = resident_blocks(S->dev, &rs_limit);
  if (blocks <= 0) return CMS_OK;
  const int n = P.n, g1 = P.gstart[1], nB = n - g1, KC = S->sc_KC, G = P.G;
  const int nt = resident_count(S, blocks);
  if ((size_t)KC * nB > (size_t)INT32_MAX || (size_t)S->K * n > (size_t)INT32_MAX) return CMS_OK;
  std::vector<int> ccol, tile_of, loc(nB), nb(nt, 0), tptr(nt + 1, 0), trow(nB);
  std::vector<signed char> cnt;
  CHK(schur_host_pattern(S, ccol, cnt));
  resident_partition(P, nt, tile_of);
  for (int i = 0; i < nB; ++i) loc[i] = nb[tile_of[i]]++;
  for (int t = 0; t < nt; ++t) tptr[t + 1] = tptr[t] + nb[t];
  for (int i = 0; i < nB; ++i) trow[tptr[tile_of[i]] + loc[i]] = i;
  // couplings among B rows (special rows), by side
  auto lower = [&](int i, auto&& f) {
    const int r = g1 + i;
    for (int s = 0; s < P.nlo[r]; ++s) {
      const size_t e = (size_t)s * n + r;
      if (P.col[e] >= g1) f(P.col[e] - g1, (int)e);
    }
  };
  auto upper = [&](int i, auto&& f) {
    const int r = g1 + i;
    for (int s = 0; s < P.nup[r]; ++s) {
      const size_t e = (size_t)(P.KL + s) * n + r;
      f(P.col[e] - g1, (int)e);
    }
  };
  std::vector<char> special(nB, 0);
  for (int i = 0; i < nB; ++i) {
    bool sp = false;
    lower(i, [&](int, int) { sp = true; });
    upper(i, [&](int, int) { sp = true; });
    special[i] = sp;
  }
  std::vector<int> group(nB);
  for (int g = 1; g < G; ++g)
    for (int r = P.gstart[g]; r < P.gstart[g + 1]; ++r) group[r - g1] = g;
  std::vector<int> slist, sgroup;
  for (int g = 2; g < G; ++g) {
    sgroup.push_back((int)slist.size());
    for (int r = P.gstart[g]; r < P.gstart[g + 1]; ++r) slist.push_back(r);
  }
  sgroup.push_back((int)slist.size());
  // per tile: rows whose z (bit 2) or y (bit 1) it needs
  const int nphase = (G - 2) + (G - 1);
  std::vector<std::vector<int>> halo(nt);
  std::vector<int> word(nB, -1);
  std::vector<int> spp((size_t)nt * (nphase + 1)), spe, spoff, osptr(nt + 1, 0), osrow;
  std::vector<int2> sprow;
  std::vector<unsigned short> spcol, kind(nB, RED_SIMPLE);
  std::vector<int> hptr(nt + 1, 0), hrow, slptr(nt), sloff, mbase(nt), tpad(nt);
  std::vector<unsigned char> mark(nB, 0);
  std::vector<int> lidx(nB, -1);
  R.hb.assign(nt, 0);
  R.h_nh.assign(nt, 0);
  R.h_nsp.assign(nt, 0);
  R.h_ne.assign(nt, 0);
  R.h_nos.assign(nt, 0);
  R.h_npair.assign(nt, 0);
  std::vector<ushort2> plcol;
  std::vector<int2> ppos(nB);
  std::vector<int> touched, stack;
  int pairs = 0, pad = 0;
  for (int t = 0; t < nt; ++t) {
    const int hb = (nb[t] + 31) / 32 * 32;
    R.hb[t] = hb;
    tpad[t] = pad;
    pad += hb;
    touched.clear();
    auto need = [&](int i, int bits) {
      if ((mark[i] & bits) == bits) return;
      if (!mark[i]) touched.push_back(i);
      mark[i] |= bits;
      if (special[i]) stack.push_back(i);
    };
    auto drain = [&] {
      while (!stack.empty()) {
        const int i = stack.back();
        stack.pop_back();
        lower(i, [&](int j, int) { need(j, 1); });
        if (mark[i] & 2) upper(i, [&](int j, int) { need(j, 3); });
      }
    };
    for (int k = 0; k < nb[t]; ++k) need(trow[tptr[t] + k], 3);
    for (int k = 0; k < nb[t]; ++k) {
      const int i = trow[tptr[t] + k];
      for (int q = 0; q < cnt[i]; ++q) need(ccol[(size_t)q * nB + i] - g1, 3);
    }
    drain();
    for (int i : touched)
      if (tile_of[i] != t) halo[t].push_back(i);
    std::sort(halo[t].begin(), halo[t].end());
    for (int k = 0; k < nb[t]; ++k) lidx[trow[tptr[t] + k]] = k;
    for (size_t h = 0; h < halo[t].size(); ++h) {
      lidx[halo[t][h]] = hb + (int)h;
      word[halo[t][h]] = 0;
    }
    hrow.insert(hrow.end(), halo[t].begin(), halo[t].end());
    hptr[t + 1] = (int)hrow.size();
    R.h_nh[t] = (int)halo[t].size();
    if (hb + R.h_nh[t] > 65535) return CMS_OK;
    // special rows by phase
    std::vector<int> sp;
    for (int i : touched)
      if (special[i]) sp.push_back(i);
    std::sort(sp.begin(), sp.end());
    const int s_first = (int)sprow.size(), e_first = (int)spoff.size();
    int ph = 0;
    auto phase = [&](int g, bool fwd) {
      spp[(size_t)t * (nphase + 1) + ph++] = (int)sprow.size();
      for (int i : sp) {
        if (group[i] != g || (!fwd && !(mark[i] & 2))) continue;
        sprow.push_back(make_int2(lidx[i], g1 + i));
        spe.push_back((int)spoff.size());
        auto entry = [&](int j, int e) {
          spoff.push_back(e);
          spcol.push_back((unsigned short)lidx[j]);
        };
        if (fwd) lower(i, entry);
        else upper(i, entry);
      }
    };
    for (int g = 2; g < G; ++g) phase(g, true);
    for (int g = G - 1; g >= 1; --g) phase(g, false);
    spp[(size_t)t * (nphase + 1) + ph] = (int)sprow.size();
    R.h_nsp[t] = (int)sprow.size() - s_first;
    R.h_ne[t] = (int)spoff.size() - e_first;
    for (int k = 0; k < nb[t]; ++k) {
      const int i = trow[tptr[t] + k];
      if (!special[i]) continue;
      kind[tptr[t] + k] = (unsigned short)R.h_nos[t]++;
      osrow.push_back(k);
    }
    osptr[t + 1] = (int)osrow.size();
    if (R.h_nos[t] >= RED_SIMPLE) return CMS_OK;
    // slices: slot pairs per 32 rows, local columns in the packed order
    slptr[t] = (int)sloff.size();
    mbase[t] = pairs;
    int o = 0;
    for (int j = 0; j < hb / 32; ++j) {
      int w = 0;
      for (int k = j * 32; k < std::min(nb[t], j * 32 + 32); ++k) w = std::max(w, (cnt[trow[tptr[t] + k]] + 1) / 2);
      sloff.push_back(o);
      const size_t base = plcol.size();
      plcol.resize(base + (size_t)w * 32);
      for (int l = 0; l < 32; ++l) {
        const int k = j * 32 + l, i = k < nb[t] ? trow[tptr[t] + k] : -1;
        if (i >= 0) ppos[i] = make_int2((int)base + l, w);
        const unsigned short own = (unsigned short)std::min(k, nb[t] - 1);
        for (int q = 0; q < w; ++q) {
          auto lc = [&](int s) {
            return i >= 0 && s < cnt[i] ? (unsigned short)lidx[ccol[(size_t)s * nB + i] - g1] : own;
          };
          plcol[base + (size_t)q * 32 + l] = make_ushort2(lc(2 * q), lc(2 * q + 1));
        }
      }
      o += w;
    }
    sloff.push_back(o);
    pairs += o;
    R.h_npair[t] = o;
    for (int i : touched) mark[i] = 0;
  }
  spe.push_back((int)spoff.size());
  R.tiles = nt;
  size_t limit = 0, smem = 0;
  CHK(red_limit(S, &limit));
  int nvs, mat;
  if (!red_plan<double>(R, RED_NV_BICG, limit, &nvs, &mat, &smem) && stream_vectors(R, limit, &smem) < 0) return CMS_OK;
  // words: a tile's are consecutive, on lines of their own
  size_t words = 0;
  std::vector<int> rexp(nB, -1);
  for (int t = 0; t < nt; ++t) {
    words = (words + 15) / 16 * 16;
    for (int k = tptr[t]; k < tptr[t + 1]; ++k)
      if (word[trow[k]] >= 0) rexp[k] = word[trow[k]] = (int)words++;
  }
  std::vector<int> hword(hrow.size());
  for (size_t k = 0; k < hrow.size(); ++k) hword[k] = word[hrow[k]];
  cudaStream_t s = S->stream;
  AllocScope scope{S};
  auto put = [&](auto** d, const auto& h) -> int {
    CHK(S->alloc(d, h.size()));
    if (!h.empty()) CMS_CUDA(cudaMemcpyAsync(*d, h.data(), h.size() * sizeof(h[0]), cudaMemcpyHostToDevice, s));
    return CMS_OK;
  };
  CHK(put(&R.tptr, tptr));
  CHK(put(&R.trow, trow));
  CHK(put(&R.tpad, tpad));
  CHK(put(&R.rexp, rexp));
  CHK(put(&R.kind, kind));
  CHK(put(&R.hptr, hptr));
  CHK(put(&R.hword, hword));
  CHK(put(&R.slptr, slptr));
  CHK(put(&R.sloff, sloff));
  CHK(put(&R.mbase, mbase));
  CHK(put(&R.plcol, plcol));
  CHK(put(&R.ppos, ppos));
  CHK(put(&R.slist, slist));
  R.sgroup = sgroup;
  CHK(put(&R.spp, spp));
  CHK(put(&R.sprow, sprow));
  CHK(put(&R.spe, spe));
  CHK(put(&R.spoff, spoff));
  CHK(put(&R.spcol, spcol));
  CHK(put(&R.osptr, osptr));
  CHK(put(&R.osrow, osrow));
  CHK(S->alloc(&R.xw, STR_ST_COPIES * (words + 1)));  // (the streamed form's copies of s, t)
  CHK(S->alloc(&R.slots, (size_t)2 * (NSMAX * nt + RES_TOT)));
  CMS_CUDA(cudaStreamSynchronize(s));
  R.words = words;
  R.npad = pad;
  R.pairs = pairs;
  R.nphase = nphase;
  R.nfwd = G - 2;
  R.limit = limit;
  R.state = 1;
  S->rd = R;
  scope.kept = true;
  return CMS_OK;
}

// need tags for a launch; the words are cleared before the 32-bit tags run over.
static int red_tags(Solver* S, unsigned int need, unsigned int* tag0) {
  RedTables& R = S->rd;
  if (R.tag > 0xffffffffu - need) {
    CMS_CUDA(cudaMemsetAsync(R.xw, 0, STR_ST_COPIES * (R.words + 1) * sizeof(ulonglong2), S->stream));
    CMS_CUDA(cudaMemsetAsync(R.slots, 0, (size_t)2 * (NSMAX * R.tiles + RES_TOT) * sizeof(ulonglong2), S->stream));
    if (S->st_xnu) CMS_CUDA(cudaMemsetAsync(S->st_xnu, 0, (R.words + 1) * sizeof(unsigned long long), S->stream));
    R.tag = 1;
  }
  *tag0 = R.tag;
  R.tag += need;
  return CMS_OK;
}

template <typename T>
static RedBuf& red_buf(Solver* S) {
  return sizeof(T) == 8 ? S->rd64 : S->rd32;
}

// Whether the reduced inner solve of refinement streams (the automatic layout,
// too large for the resident form, the gathered vectors fit; up to about 8M
// cells); allocates its buffers.  Kernel time per iteration, one B200,
// telescoping systems, form of cms_schur.cuh / streamed: 1.3M cells 42.7 / 19.9
// us, 2.0M 87.3 / 27.4, 4.0M 156 / 66, 7.3M 280 / 150.  Bound by HBM at 4M and
// above (about 70 % of the measured copy rate).
static bool stream_choose(Solver* S) {
  const RedRoom& M = red_room(S);
  if (M.state != 1 || M.stream > (double)M.limit) return false;
  if (red_tables(S) != CMS_OK || S->rd.state != 1) return false;
  RedTables& R = S->rd;
  size_t smem = 0;
  if (stream_vectors(R, R.limit, &smem) < 0) return false;
  if (!S->st_coef) {
    float2* coef = nullptr;
    float* vec = nullptr;
    unsigned long long* xnu = nullptr;
    AllocScope scope{S};
    if (S->alloc(&coef, (size_t)R.pairs * 32) || S->alloc(&vec, (size_t)SV_N * R.npad) ||
        S->alloc(&xnu, R.words + 1))
      return false;
    scope.kept = true;
    S->st_coef = coef;
    S->st_vec = vec;
    S->st_xnu = xnu;
  }
  return true;
}

// Its arguments beyond the system's (tags from the tables' words).
static int stream_args(Solver* S, int maxit, StreamArgs* a, size_t* smem) {
  RedTables& R = S->rd;
  a->tptr = R.tptr; a->trow = R.trow; a->tpad = R.tpad; a->rexp = R.rexp; a->hptr = R.hptr; a->hword = R.hword;
  a->slptr = R.slptr; a->sloff = R.sloff; a->mbase = R.mbase;
  a->pcoef = S->st_coef; a->plcol = R.plcol; a->gvec = S->st_vec; a->npad = R.npad;
  a->nvs = stream_vectors(R, R.limit, smem);
  // what L2 keeps of the matrix beside the vectors of global memory: of 126 MB,
  // 75 (per iteration at 2.9M cells: 48.7 us with every slice evict-first, 44.7
  // with 60-80 MB kept, 54.2 with 100 MB; at 2.0M 35.7, 27.4, 27.4; at 4.0M
  // 66.4, 66.1-67.3, 75.0)
  const double mat = 32.0 * R.pairs * (sizeof(float2) + sizeof(ushort2)), vecs = (SV_N - a->nvs) * 4.0 * (double)R.npad;
  constexpr double kL2Keep = 75e6;
  a->keep = (float)std::min(1.0, std::max(0.0, (kL2Keep - vecs) / mat));
  a->xst = R.xw; a->words = R.words + 1; a->xnu = S->st_xnu; a->slots = R.slots;
  return red_tags(S, (unsigned int)maxit + 2u, &a->S.tag0);
}

// Whether a solve runs in reduced form: a multicolour ordering of a symmetric
// pattern (a cell that is not its neighbour's neighbour may share its group, and
// group 0 is then not independent) whose tiles'
// gathered vector fits an SM's shared memory (red_tables; about 8M cells in
// FP64), on the exact factor.  BiCGStab only in FP64: in FP32 its recurrence
// turns rounding into a different iteration count in one solve of seven
// (40 random systems to 1e-5), so FP32 keeps the arithmetic of
// k_bicg_persistent; so do refinement's inner solves with inner_relax 0 or 1.
// Solve times, one B200 (per-phase kernels for GMRES, k_bicg_persistent for
// BiCGStab / reduced form):
//   GMRES(3) to 1e-3     20k cells 1.29 / 0.21 ms, 1M 4.39 / 0.73, 4M 10.7 / 2.8
//   BiCGStab to 1e-6     100k cells 1.7 / 0.49 ms, 1M 4.9 / 1.11, 4M 14.0 / 5.4
// What bounds it: up to 250k cells the exchanges and sums (2 and 3 per
// BiCGStab iteration, 3 and 4 per GMRES cycle); at 4M HBM (160 MB per
// application and the vectors); at 1M not known: the coefficients come from L2
// (40 MB per application), but at 2.2 TB/s, below what L2 gives.
template <typename T>
static bool red_wanted(Solver* S, int nsolv, int maxit) {
  if (S->opts.multi_kernel || S->opts.ordering != CMS_ORDER_MULTICOLOR || S->cur_relax || S->cur_fuse || maxit < 1 ||
      maxit > (1 << 26) || (nsolv == 3 && sizeof(T) == 4))
    return false;
  const RedRoom& M = red_room(S);
  if (M.state != 1 || (sizeof(T) == 8 ? M.krylov64 : M.krylov32) > (double)M.limit) return false;
  return red_tables(S) == CMS_OK && S->rd.state == 1;
}

// The solve of A x = b (W.b, W.x) by BiCGStab (nsolv 3) or GMRES(3) (nsolv 4)
// on its own part of the factor.  Returns 1 when its buffers or the launch are
// refused; does not wait for the launch: the caller copies the state to the host and calls
// check_waits.
template <typename T>
static int run_reduced(Solver* S, Mat<T>& A, Work<T>& W, int nsolv, int maxit, int norm, double tol, int xzero) {
  const HostPattern& P = S->hp;
  RedTables& R = S->rd;
  RedBuf& B = red_buf<T>(S);
  const int n = P.n, g1 = P.gstart[1], nB = n - g1;
  using P2 = typename Pair<T>::type;
  const int nvec = nsolv == 3 ? RED_NV_BICG : RED_NV_GMRES;
  int nvs = 0, mat = 0;
  size_t smem = 0;
  if (!red_plan<T>(R, nvec, R.limit, &nvs, &mat, &smem)) return 1;
  if (!B.coef) {
    P2* c = nullptr;
    T *cd = nullptr, *gv = nullptr;
    AllocScope scope{S};
    if (S->alloc(&c, (size_t)R.pairs * 32) || S->alloc(&cd, (size_t)nB) ||
        S->alloc(&gv, (size_t)RED_NV_BICG * R.npad))
      return 1;
    scope.kept = true;
    B.coef = c;
    B.cdiag = cd;
    B.gvec = gv;
  }
  const double s = sizeof(T);
  int rc = CMS_OK;
  with_couplings(S->sc_KS, [&](auto ks) {
    rc = [&]() -> int {
      KLAUNCH(S, P_SCHUR_BUILD, (2 * s + 12) * (double)P.nnz_off + 10.0 * n + s * 32.0 * 2 * R.pairs,
              (k_red_pack<T, decltype(ks)::value><<<gsz(nB), TPB, 0, S->stream>>>(
                  n, g1, nB, P.KL, S->d_col, S->d_nlo, S->d_nup, A.aoff, A.diag, SchurMap{S->d_smap, S->d_dmap},
                  S->d_sccnt, R.ppos, (P2*)B.coef, (T*)B.cdiag, A.luoff, A.invd)));
      return CMS_OK;
    }();
  });
  CHK(rc);
  for (size_t g = 0; g + 1 < R.sgroup.size(); ++g) {
    const int cnt = R.sgroup[g + 1] - R.sgroup[g];
    if (cnt <= 0) continue;
    KLAUNCH(S, P_ILU0, (double)cnt * 20 * s,
            (k_red_special<T><<<gsz(cnt), TPB, 0, S->stream>>>(n, g1, P.KL, cnt, R.slist + R.sgroup[g], S->d_col,
                                                               S->d_nlo, S->d_nup, (const T*)B.cdiag, A.luoff,
                                                               A.invd)));
  }
  RedArgs<T> a;
  std::memset(&a, 0, sizeof(a));
  a.n = n; a.g1 = g1; a.nB = nB; a.KL = P.KL; a.nt = a.ntiles = R.tiles;
  a.tptr = R.tptr; a.trow = R.trow; a.tpad = R.tpad; a.rexp = R.rexp; a.kind = R.kind;
  a.hptr = R.hptr; a.hword = R.hword; a.slptr = R.slptr; a.sloff = R.sloff; a.mbase = R.mbase;
  a.pcoef = B.coef; a.plcol = R.plcol;
  a.nphase = R.nphase; a.nfwd = R.nfwd; a.spp = R.spp; a.sprow = R.sprow; a.spe = R.spe; a.spoff = R.spoff;
  a.spcol = R.spcol; a.osptr = R.osptr; a.osrow = R.osrow;
  a.luoff = A.luoff; a.invd = A.invd; a.aoff = A.aoff; a.diag = A.diag; a.b = W.b; a.cdiag = (T*)B.cdiag;
  a.x = W.x; a.rho = W.r;
  a.col = S->d_col; a.nlo = S->d_nlo; a.nup = S->d_nup;
  a.gvec = (T*)B.gvec; a.npad = R.npad; a.nvs = nvs; a.mat_smem = mat;
  a.xw = R.xw; a.slots = R.slots; a.bar = &S->d_st->bar; a.st = S->d_st;
  a.maxit = maxit; a.norm = norm; a.xzero = xzero; a.tol = tol; a.spin_limit = S->spin_limit;
  CHK(red_tags(S, 8u * (unsigned int)maxit + 8u, &a.tag0));  // at most 8 per cycle, 5 per iteration
  CMS_CUDA(cudaMemsetAsync(&S->d_st->bar, 0, sizeof(GridBar), S->stream));
  void* args[] = {&a};
  prof_begin(S);
  // 1024 threads where a tile has more rows than that, for the loads in flight
  // (BiCGStab at 1M cells, 3400 rows: 1330 us with 512, 1129 with 1024; GMRES at
  // 4M 4.46 and 2.81 ms); below, fewer warps make the sums shorter (gradient at
  // 100k cells, 340 rows: 1611 and 1815 us)
  const int bs = *std::max_element(R.hb.begin(), R.hb.end()) > RED_WIDE ? 1024 : 512;
  const void* kern = red_kernel<T>(nsolv, bs);
  const cudaError_t e = cudaLaunchCooperativeKernel(kern, dim3(R.tiles), dim3(bs), args, smem, S->stream);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    R.state = -1;
    return 1;
  }
  if (e != cudaSuccess) {
    std::snprintf(g_last_error, sizeof(g_last_error), "cooperative launch (reduced Krylov): %s", cudaGetErrorString(e));
    return CMS_DEVICE_ERROR;
  }
  S->launches++;
  const size_t nrec = S->prof_recs.size();
  prof_end(S, P_PERSIST, 0.0);
  S->wait_check = true;
  if (S->prof_recs.size() > nrec) {  // profiling: the iterations, for the byte count
    CMS_CUDA(cudaMemcpyAsync(S->h_st, S->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, S->stream));
    CMS_CUDA(cudaStreamSynchronize(S->stream));
    // C's entries once per operator application; vectors: BiCGStab 26 accesses
    // of a B row per iteration, GMRES 36 per cycle
    const double C = (s + 2) * (double)S->sc_nnz;
    S->prof_recs.back().bytes = nsolv == 3 ? S->h_st->iter * (2 * C + 26.0 * s * nB)
                                           : S->h_st->inner * C + S->h_st->iter * 36.0 * s * nB;
  }
  return CMS_OK;
}

}  // namespace cms
