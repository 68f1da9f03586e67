// sem_resident_run.cuh — host side of the resident kernels: tilings, waves, launches.
// Included by sem_kernels.cu after run_group.

namespace {

SolveIo solve_io(const sem_solve_t& s, const Workspace& ws, char* a);

typedef void (*ResFn)(const SolveDev*, const int*, ResLay, unsigned long long*, unsigned, int, int, int, int, int);

template <bool ADJ, bool STC>
ResFn res_fn(int N) {
  switch (N) {
    case 1: return sem_resident_kernel<1, ADJ, STC>;
    case 2: return sem_resident_kernel<2, ADJ, STC>;
    case 3: return sem_resident_kernel<3, ADJ, STC>;
    case 4: return sem_resident_kernel<4, ADJ, STC>;
    case 5: return sem_resident_kernel<5, ADJ, STC>;
    case 6: return sem_resident_kernel<6, ADJ, STC>;
    case 7: return sem_resident_kernel<7, ADJ, STC>;
  }
  return nullptr;
}
ResFn res_kernel_for(int N, bool adj, bool stc) {
  if (adj) return stc ? res_fn<true, true>(N) : res_fn<true, false>(N);
  return stc ? res_fn<false, true>(N) : res_fn<false, false>(N);
}

// Receiver lists of the balanced tiling ntx x ntz of a plan (tiles from res_start).
int get_res_lists(const sem_plan_s* p, int ntx, int ntz, sem_plan_s::ResLists* out) {
  std::lock_guard<std::mutex> lk(p->mu);
  auto key = std::make_pair(ntx, ntz);
  auto it = p->res_lists.find(key);
  if (it != p->res_lists.end()) { *out = it->second; return SEM_OK; }
  const int N = p->npol, NP = N + 1;
  auto owner = [](int e, int nel, int n) {  // tile of element e (the last one for the mesh's last node)
    return e >= nel ? n - 1 : (int)(((long long)e * n) / nel);
  };
  const int nt = ntx * ntz;
  std::vector<std::vector<int>> rec(nt), inj(nt);
  // per tile and quad (row << 16 | element): the receivers that reach it, with node masks and weights
  struct Term { int q, mask; std::vector<float> w; };
  std::vector<std::map<int, std::vector<Term>>> quads(nt);
  for (int r = 0; r < p->nrec; ++r) {
    const int bx = p->h_rec_base[2 * r], bz = p->h_rec_base[2 * r + 1];
    rec[owner(bz / N, p->nelz, ntz) * ntx + owner(bx / N, p->nelx, ntx)].push_back(r);
    for (int j = 0; j < NP; ++j)
      for (int i = 0; i < NP; ++i) {
        const int gx = bx + i, gz = bz + j;
        const int tx = owner(gx / N, p->nelx, ntx), tz = owner(gz / N, p->nelz, ntz);
        const int t = tz * ntx + tx;
        if (inj[t].empty() || inj[t].back() != r) inj[t].push_back(r);
        const int q = (int)inj[t].size() - 1;
        const int x0 = res_start(tx, p->nelx, ntx) * N, z0 = res_start(tz, p->nelz, ntz) * N;
        auto& terms = quads[t][((gz - z0) << 16) | ((gx - x0) / N)];
        if (terms.empty() || terms.back().q != q) terms.push_back(Term{q, 0, std::vector<float>(N, 0.f)});
        terms.back().mask |= 1 << ((gx - x0) % N);
        terms.back().w[(gx - x0) % N] = p->h_rec_w[(size_t)r * NP * NP + j * NP + i];
      }
  }
  sem_plan_s::ResLists L{};
  std::vector<int> ro(1, 0), ri, io(1, 0), ii, qo(1, 0), qp, eo, et;
  std::vector<float> ew;
  for (int t = 0; t < nt; ++t) {
    ri.insert(ri.end(), rec[t].begin(), rec[t].end());
    ro.push_back((int)ri.size());
    ii.insert(ii.end(), inj[t].begin(), inj[t].end());
    io.push_back((int)ii.size());
    const size_t e0 = et.size();
    for (auto& kv : quads[t]) {
      qp.push_back(kv.first);
      eo.push_back((int)et.size());
      for (auto& term : kv.second) {
        et.push_back(term.q << 8 | term.mask);
        ew.insert(ew.end(), term.w.begin(), term.w.end());
      }
    }
    qo.push_back((int)qp.size());
    L.nrec = std::max(L.nrec, (int)rec[t].size());
    L.ninj = std::max(L.ninj, (int)inj[t].size());
    L.nquad = std::max(L.nquad, (int)quads[t].size());
    L.nterm = std::max(L.nterm, (int)(et.size() - e0));
  }
  eo.push_back((int)et.size());
  int rc;
  if ((rc = upload(&L.l.rec_off, ro.data(), ro.size())) || (rc = upload(&L.l.rec_ids, ri.data(), ri.size())) ||
      (rc = upload(&L.l.inj_off, io.data(), io.size())) || (rc = upload(&L.l.inj_ids, ii.data(), ii.size())) ||
      (rc = upload(&L.iq_off, qo.data(), qo.size())) || (rc = upload(&L.iq_pos, qp.data(), qp.size())) ||
      (rc = upload(&L.iterm_off, eo.data(), eo.size())) || (rc = upload(&L.iterm, et.data(), et.size())) ||
      (rc = upload(&L.iterm_w, ew.data(), ew.size())))
    return rc;
  p->res_lists[key] = L;
  *out = L;
  return SEM_OK;
}

struct ResCounts { int nrec = 0, ninj = 0, nquad = 0, nterm = 0; };

ResLay res_layout(int N, bool adj, bool stc, int exm, int ezm, const ResCounts& c) {
  ResLay L{};
  const int NP = N + 1;
  auto odd4 = [](int v) { const int q = (v + 3) / 4; return 4 * (q | 1); };  // 128-bit rows of lanes spread over the banks
  L.Rm = ezm * N + 1;
  L.Cm = exm * N + 1;
  L.qx = exm + 1;
  L.Wp = odd4((N == 4 ? 0 : 4) + N + (exm + 1) * N);
  L.Cp = odd4((exm + 1) * N);
  const int rows = (ezm + 1) * N;  // one more element row: the mesh's last line of nodes starts it
  L.H = N + rows + 1;
  int o = 0;
  auto take = [&](long long n, int align = 4) { o = (int)round_up(o, align); const int at = o; o += (int)n; return at; };
  L.reg = L.Wp * L.H;
  L.wreg = (int)round_up(L.reg, 32);
  const int own = L.Cp * rows;
  if (adj) L.w = take(2LL * L.wreg, 32);
  L.b = take(2LL * L.reg); L.c = take(L.reg); L.v = take(own);
  if (adj) L.g = take(own);
  L.tz = take(8LL * rows);
  const long long words = (long long)(L.Rm + L.Cm) * NP + 1;
  L.wi = take(2 * words); L.wo = take(2 * words);
  if (adj) {
    L.nrm = std::max(1, c.ninj);
    L.niq = c.nquad;
    L.rs = take(4LL * L.nrm);
    L.ia = take(2LL * c.nquad * N);
    L.io = take((long long)c.nquad + 1);
    L.iq = take(c.nterm);
    L.ie = take((long long)c.nterm * N);
    L.im = take(((long long)rows * L.qx + 1) / 2);
  }
  if (stc) { const int bn = 2 * L.Rm + L.Cm; L.be = take(3LL * bn); L.bd = take(2LL * bn); }
  L.total = (int)round_up(o, 4);
  L.ll_t = L.Rm * N; L.ll_r = L.ll_t + L.Cm * N; L.ll_b = L.ll_r + L.Rm; L.ll_c = L.ll_b + L.Cm;
  L.llw = (int)round_up(L.ll_c + 1, 16);
  return L;
}

constexpr int kResSmem = 230400;  // dynamic shared bytes: one CTA per SM
// Threads of a launch whose largest tile is exm x ezm elements (the lowest ezl high): lanes per
// tile row, element rows per chunk, compute and receiver threads.
struct ResShape { int sw, ezc, nc, nio; };
bool res_shape(bool adj, int exm, int ezm, int ezl, int nrec, ResShape* h) {
  const int ezr = std::max(ezm, ezl + 1);  // element rows, the mesh's last line of nodes counted as one
  h->nio = (int)round_up(std::max(nrec, 1), 32);
  const int tmax = res_threads(adj) - h->nio;
  h->sw = 4;
  while (h->sw < exm + 2) h->sw *= 2;
  if (h->sw > 32 || tmax < 32) return false;
  h->ezc = (ezr + tmax / h->sw - 1) / (tmax / h->sw);
  h->nc = (int)round_up((long long)((ezr + h->ezc - 1) / h->ezc) * h->sw, 32);
  return true;
}
// Modelled cycles of one step: the exchange (send, 0.47 us between SMs, poll), then the warps'
// work: per element and chunk the fp32 operations, at 1.95 cycles each for a warp alone on its
// scheduler and 1.9 (adjoint 2.6: fewer warps) times the warps per scheduler beyond that.
// Fitted to 100x50 meshes, order 4: a forward step of 25x25 tiles 11.0k cycles measured (11.1k
// modelled), adjoint at 13x25 12.6k (12.3k), 4x2 tiles 3.7k / 4.5k (3.8k / 4.5k).  Two or three
// smaller CTAs per SM, which hide one another's exchange, measured the same or slower (16
// models, forward + adjoint: 18.1 us a step at best with one, 18.9 with two, 22.5 with three).
double res_step_cost(int N, bool adj, const ResShape& h) {
  const double NP = N + 1;
  const double el = adj ? 2 * N * (3 * NP * NP + 4 * NP) + 16 * N * N : 2 * N * (2 * NP * NP + 2 * NP) + 10 * N * N;
  const double carry = N * (NP * NP + 3 * NP) + (adj ? N * (NP + 2) : 0);
  const double work = h.ezc * el + carry, warps = h.nc / 32.0;
  return 2200.0 + work * std::max(1.95, (adj ? 2.6 : 1.9) * warps / 4.0);
}
bool res_fits(const ResLay& L) { return L.Wp <= 256 && L.H <= 256 && (long long)L.total * 4 <= kResSmem; }

// bounds of the receivers of one tile of a tiling
ResCounts res_counts(const sem_plan_s* p, int ntx, int ntz) {
  ResCounts c;
  const int N = p->npol;
  std::map<int, std::pair<int, std::vector<int>>> tiles;  // receivers and their elements
  for (int r = 0; r < p->nrec; ++r) {
    const int ex = p->h_rec_base[2 * r] / N, ez = p->h_rec_base[2 * r + 1] / N;
    int seen[4], ns = 0;
    for (int q = 0; q < 4; ++q) {  // an element's last nodes may belong to the next tiles
      const int x = std::min(ex + (q & 1), p->nelx - 1), z = std::min(ez + (q >> 1), p->nelz - 1);
      const int tx = std::min((int)(((long long)(x + 1) * ntx - 1) / p->nelx), ntx - 1);
      const int tz = std::min((int)(((long long)(z + 1) * ntz - 1) / p->nelz), ntz - 1);
      const int t = tz * ntx + tx;
      if (std::find(seen, seen + ns, t) != seen + ns) continue;
      seen[ns++] = t;
      auto& e = tiles[t];
      e.first++;
      if (std::find(e.second.begin(), e.second.end(), ez * p->nelx + ex) == e.second.end())
        e.second.push_back(ez * p->nelx + ex);
    }
  }
  for (auto& kv : tiles) {
    c.nrec = std::max(c.nrec, kv.second.first);
    c.nquad = std::max(c.nquad, (int)kv.second.second.size() * 2 * (N + 1));
  }
  c.ninj = c.nrec;
  c.nterm = c.ninj * 2 * (N + 1);
  return c;
}

// Tiling of a plan into tiles of at most E elements that fit a CTA: the one with the least work
// (tiles times modelled step); kept with the plan.  (0, 0): none.
std::pair<int, int> res_tiling(const sem_plan_s* p, bool adj, int E) {
  std::lock_guard<std::mutex> lk(p->mu);
  const auto key = std::make_pair(adj, E);
  auto it = p->res_tilings.find(key);
  if (it != p->res_tilings.end()) return it->second;
  std::pair<int, int> best(0, 0);
  double best_c = -1.0;
  const bool stc = p->bnd_n > 0;
  for (int tx = 1; tx <= p->nelx; ++tx) {
    const int ex = (p->nelx + tx - 1) / tx;
    if (tx > 1 && ex == (p->nelx + tx - 2) / (tx - 1)) continue;  // no narrower than with one tile less
    const int ezm = E / ex;
    if (ezm < 1 || ex > 30) continue;
    const int tz = (p->nelz + ezm - 1) / ezm, ez = (p->nelz + tz - 1) / tz;
    ResShape h;
    if (!res_shape(adj, ex, ez, p->nelz / tz, 1, &h)) continue;
    const double c = (double)tx * tz * res_step_cost(p->npol, adj, h);
    if (best_c >= 0.0 && c >= best_c) continue;
    const ResCounts cnt = res_counts(p, tx, tz);
    if (!res_shape(adj, ex, ez, p->nelz / tz, std::max(cnt.nrec, cnt.ninj), &h) ||
        !res_fits(res_layout(p->npol, adj, stc, ex, ez, cnt)))
      continue;
    best_c = c;
    best = std::make_pair(tx, tz);
  }
  p->res_tilings[key] = best;
  return best;
}

struct ResWave {
  std::vector<int> idx;                        // solves
  std::vector<std::pair<int, int>> tiles;      // their tilings
  std::vector<int> k;                          // their checkpoint intervals
};

int res_steps(const sem_solve_t& s, int k) {
  const int nt = s.plan->nt;
  if (!(s.flags & SEM_F_ADJOINT)) return nt;
  const int nseg = (nt + k - 1) / k;
  return nt + k * (nseg - 1);
}

// Waves of one class of solves (same order, boundary mode, forward-only or not): for each tile
// capacity, pack the solves (longest first) into waves whose CTAs are resident at once and
// whose workspaces fit the budget, and keep the capacity with the smallest modelled time.
// Empty when a solve fits no way.
std::vector<ResWave> res_plan(const sem_solve_t* sv, const std::vector<int>& cls, int sms, long long budget) {
  const sem_plan_s* p0 = sv[cls[0]].plan;
  const int N = p0->npol;
  const bool adj = sv[cls[0]].flags & SEM_F_ADJOINT;
  std::vector<int> ord(cls);
  std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) {
    return (long long)sv[a].plan->nt * 64 + sv[a].plan->npoints / 4096 > (long long)sv[b].plan->nt * 64 + sv[b].plan->npoints / 4096;
  });
  // checkpoint interval and bytes of each solve by itself
  std::vector<int> kk(ord.size());
  std::vector<long long> bytes(ord.size());
  for (size_t j = 0; j < ord.size(); ++j) {
    const sem_solve_t& s = sv[ord[j]];
    int ns, k = 2;
    if (adj) {
      k = std::max(2, std::min(s.ckpt_k > 0 ? (int)s.ckpt_k : s.plan->nt, s.plan->nt));
      if (s.ckpt_k <= 0 && layout(s.plan, s.flags, k, &ns).bytes > budget) {
        int lo = std::max(2, std::min(s.plan->nt, (int)std::sqrt(2.0 * s.plan->nt))), hi = k;
        while (lo < hi) {
          const int mid = lo + (hi - lo + 1) / 2;
          if (layout(s.plan, s.flags, mid, &ns).bytes <= budget) lo = mid; else hi = mid - 1;
        }
        k = lo;
      }
    }
    kk[j] = k;
    bytes[j] = layout(s.plan, s.flags, k, &ns).bytes;
  }
  std::vector<ResWave> best;
  double best_cost = -1.0;
  for (double Ed = 8.0; Ed < 1200.0; Ed *= 1.15) {
    const int E = (int)Ed;
    std::vector<ResWave> waves;
    double cost = 0.0;
    bool ok = true;
    long long used = 0, mem = 0;
    double wave_step = 0.0;
    int wave_nt = 0;
    auto close = [&]() { cost += wave_step * wave_nt; used = mem = 0; wave_step = 0.0; wave_nt = 0; };
    for (size_t j = 0; j < ord.size() && ok; ++j) {
      const sem_plan_s* p = sv[ord[j]].plan;
      const std::pair<int, int> tile = res_tiling(p, adj, E);
      const int tx = tile.first, tz = tile.second;
      if (!tx || (long long)tx * tz > sms) { ok = false; break; }
      if (waves.empty() || used + (long long)tx * tz > sms || mem + bytes[j] > budget) {
        if (!waves.empty()) close();
        waves.emplace_back();
      }
      ResWave& w = waves.back();
      w.idx.push_back(ord[j]);
      w.tiles.push_back(tile);
      w.k.push_back(kk[j]);
      used += (long long)tx * tz;
      mem += bytes[j];
      ResShape h;
      const int ex = (p->nelx + tx - 1) / tx, ez = (p->nelz + tz - 1) / tz;
      double c = 0.0;
      for (int a = 0; a <= (adj ? 1 : 0); ++a) {
        if (!res_shape(a, ex, ez, p->nelz / tz, 32, &h)) { ok = false; break; }
        c += res_step_cost(N, a, h);
      }
      wave_step = std::max(wave_step, c);
      wave_nt = std::max(wave_nt, res_steps(sv[ord[j]], kk[j]));
      if (best_cost >= 0.0 && cost > best_cost) ok = false;
    }
    if (!ok) continue;
    close();
    if (best_cost < 0.0 || cost < best_cost) { best_cost = cost; best = waves; }
  }
  return best;
}

// One wave: set-up, forward launch, (replay and) adjoint launches, outputs.
// SEM_ERR_UNSUPPORTED without a message when the wave cannot run this way (nothing launched).
int run_res_wave(sem_batch_t* b, const sem_solve_t* sv, const ResWave& w, int sms, cudaStream_t stream) {
  const int n = (int)w.idx.size();
  const sem_plan_s* p0 = sv[w.idx[0]].plan;
  const int N = p0->npol;
  const bool adj = sv[w.idx[0]].flags & SEM_F_ADJOINT, stc = p0->bnd_n > 0;
  int exm = 1, ezm = 1;
  ResCounts c;
  std::vector<sem_plan_s::ResLists> lists(n);
  long long ncta = 0;
  int ezl = 1;
  for (int j = 0; j < n; ++j) {
    const sem_plan_s* p = sv[w.idx[j]].plan;
    const int tx = w.tiles[j].first, tz = w.tiles[j].second;
    if (int rc = get_res_lists(p, tx, tz, &lists[j])) return rc;
    c.nrec = std::max(c.nrec, lists[j].nrec); c.ninj = std::max(c.ninj, lists[j].ninj);
    c.nquad = std::max(c.nquad, lists[j].nquad); c.nterm = std::max(c.nterm, lists[j].nterm);
    exm = std::max(exm, (p->nelx + tx - 1) / tx); ezm = std::max(ezm, (p->nelz + tz - 1) / tz);
    ezl = std::max(ezl, p->nelz / tz);
    ncta += (long long)tx * tz;
  }
  const ResLay Lf = res_layout(N, false, stc, exm, ezm, c), La = adj ? res_layout(N, true, stc, exm, ezm, c) : Lf;
  ResShape hf, ha;
  if (!res_shape(false, exm, ezm, ezl, c.nrec, &hf) || !res_shape(true, exm, ezm, ezl, c.ninj, &ha))
    return SEM_ERR_UNSUPPORTED;
  ResFn ff = res_kernel_for(N, false, stc), fa = adj ? res_kernel_for(N, true, stc) : nullptr;
  for (int q = 0; q < (adj ? 2 : 1); ++q) {
    ResFn fn = q ? fa : ff;
    const ResLay& L = q ? La : Lf;
    const int T = q ? ha.nc + ha.nio : hf.nc + hf.nio;
    int nb = 0;
    if (!res_fits(L) || raise_smem_limit((const void*)fn, (size_t)L.total * 4) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, T, (size_t)L.total * 4) != cudaSuccess ||
        (long long)nb * sms < ncta) {
      cudaGetLastError();
      return SEM_ERR_UNSUPPORTED;
    }
  }

  // ---- workspaces, descriptors
  std::vector<Workspace> ws(n);
  std::vector<int> nseg(n);
  long long total = 0;
  int max_prog = 0, max_seg = 1;
  for (int j = 0; j < n; ++j) {
    const sem_solve_t& s = sv[w.idx[j]];
    ws[j] = layout(s.plan, s.flags, w.k[j], &nseg[j]);
    total += ws[j].bytes;
    max_seg = std::max(max_seg, nseg[j]);
    const int nt = s.plan->nt;
    max_prog = std::max(max_prog, nt + ((s.flags & SEM_F_SHIFT) ? 1 : 0) + (adj ? 1 + nt + w.k[j] * (nseg[j] - 1) : 0));
  }
  if (total > b->arena_bytes) {
    cudaFree(b->arena);
    b->arena = nullptr;
    b->arena_bytes = 0;
    CUDA_TRY(cudaMalloc((void**)&b->arena, total));
    b->arena_bytes = total;
  }
  if (adj && n > b->tmaps_cap) {
    cudaFree(b->d_tmaps);
    b->d_tmaps = nullptr;
    b->tmaps_cap = 0;
    CUDA_TRY(cudaMalloc((void**)&b->d_tmaps, sizeof(CUtensorMap) * n));
    b->tmaps_cap = n;
  }
  b->h_tmaps.resize(n);
  b->h_solves.assign(n, SolveDev{});
  b->h_cta.clear();
  b->h_io.clear();
  long long off = 0, max_pts = 1;
  for (int j = 0; j < n; ++j) {
    const sem_solve_t& s = sv[w.idx[j]];
    const sem_plan_s* p = s.plan;
    char* a = b->arena + off;
    SolveDev& d = b->h_solves[j];
    d.nelx = p->nelx; d.nelz = p->nelz; d.nxg = p->nxg; d.nzg = p->nzg; d.pitch = p->pitch;
    d.tiles_x = w.tiles[j].first; d.tiles_z = w.tiles[j].second;
    d.zchunk = p->nelz;
    d.tile_base = (int)b->h_cta.size();
    d.nt = p->nt; d.k = w.k[j]; d.nseg = nseg[j]; d.flags = s.flags; d.start_tick = 0;
    d.it0 = s.it0; d.it1 = s.it1; d.decim = s.decim;
    d.src_gx = p->src_gx; d.src_gz = p->src_gz; d.nrec = p->nrec;
    d.fstride = p->fstride;
    d.c2 = (const float*)(a + ws[j].c2);
    d.W = (float*)(a + ws[j].W);
    d.V = (float*)(a + ws[j].V);
    if (adj) {
      d.ckpt = (float*)(a + ws[j].ckpt);
      d.ring = (float*)(a + ws[j].ring);
      d.L = (float*)(a + ws[j].L);
      d.Mu = (float*)(a + ws[j].Mu);
      d.grad = (float*)(a + ws[j].grad);
      d.grad64 = (double*)(a + ws[j].grad64);
      if (int rc = encode_band_map(&b->h_tmaps[j], a, p, field_slots(ws[j], p, true), La.Wp, La.H)) return rc;
      d.tmap = b->d_tmaps + j;
    }
    d.D = p->D; d.beta = p->beta; d.tx = p->tx; d.tz = p->tz; d.src_term = p->src_term;
    d.rec_base = p->rec_base; d.rec_w = p->rec_w;
    d.rec_tile_off = lists[j].l.rec_off; d.rec_tile_ids = lists[j].l.rec_ids;
    d.inj_tile_off = lists[j].l.inj_off; d.inj_tile_ids = lists[j].l.inj_ids;
    d.iq_off = lists[j].iq_off; d.iq_pos = lists[j].iq_pos; d.iterm_off = lists[j].iterm_off;
    d.iterm = lists[j].iterm; d.iterm_w = lists[j].iterm_w;
    d.rec_out = s.rec_out; d.yobs = s.y_obs;
    d.misfit = (double*)(a + ws[j].misfit);
    d.rmax = d.misfit + p->nrec;
    d.adj_scale = d.misfit + 2 * p->nrec;
    d.status = (int*)(a + ws[j].status);
    d.ws = (const float*)a;
    d.bnd_n = p->bnd_n; d.bnd_pitch = bnd_pitch_of(p);
    d.bnd_coef = p->bnd_n ? (const float*)(a + ws[j].bnd_coef) : nullptr;
    d.bnd_hist = ws[j].bnd_hist >= 0 ? (float*)(a + ws[j].bnd_hist) : nullptr;
    b->h_cta.insert(b->h_cta.end(), d.tiles_x * d.tiles_z, j);
    b->h_io.push_back(solve_io(s, ws[j], a));
    max_pts = std::max(max_pts, (long long)p->npoints);
    off += ws[j].bytes;
  }
  if (n > b->solves_cap) {
    cudaFree(b->d_solves);
    b->d_solves = nullptr;
    b->solves_cap = 0;
    CUDA_TRY(cudaMalloc((void**)&b->d_solves, sizeof(SolveDev) * n));
    b->solves_cap = n;
  }
  if ((long long)b->h_cta.size() > b->cta_cap) {
    cudaFree(b->d_cta);
    b->d_cta = nullptr;
    b->cta_cap = 0;
    CUDA_TRY(cudaMalloc((void**)&b->d_cta, sizeof(int) * b->h_cta.size()));
    b->cta_cap = b->h_cta.size();
  }
  if (n > b->io_cap) {
    cudaFree(b->d_io);
    b->d_io = nullptr;
    b->io_cap = 0;
    CUDA_TRY(cudaMalloc((void**)&b->d_io, sizeof(SolveIo) * n));
    b->io_cap = n;
  }
  const long long ll_bytes = ncta * kResSlots * (long long)std::max(Lf.llw, La.llw) * 8;
  if (ll_bytes > b->ll_cap) {
    cudaFree(b->d_ll);
    b->d_ll = nullptr;
    b->ll_cap = 0;
    CUDA_TRY(cudaMalloc((void**)&b->d_ll, ll_bytes));
    b->ll_cap = ll_bytes;
    CUDA_TRY(cudaMemsetAsync(b->d_ll, 0, ll_bytes, stream));
    b->ll_tag = 0;
  }
  CUDA_TRY(cudaMemcpyAsync(b->d_solves, b->h_solves.data(), sizeof(SolveDev) * n, cudaMemcpyHostToDevice, stream));
  if (adj)
    CUDA_TRY(cudaMemcpyAsync(b->d_tmaps, b->h_tmaps.data(), sizeof(CUtensorMap) * n, cudaMemcpyHostToDevice, stream));
  CUDA_TRY(cudaMemcpyAsync(b->d_cta, b->h_cta.data(), sizeof(int) * b->h_cta.size(), cudaMemcpyHostToDevice, stream));
  CUDA_TRY(cudaMemcpyAsync(b->d_io, b->h_io.data(), sizeof(SolveIo) * n, cudaMemcpyHostToDevice, stream));
  const unsigned io_bx = (unsigned)std::min<long long>(64, (max_pts + 2047) / 2048);
  for (int s0 = 0; s0 < n; s0 += 65535)
    batch_setup_kernel<<<dim3(io_bx, (unsigned)std::min(65535, n - s0)), 256, 0, stream>>>(b->d_io, s0);
  b->last_launches++;
  CUDA_TRY(cudaGetLastError());

  while ((int)b->tick_ev.size() < b->tick_ev_used + 2) {
    cudaEvent_t e;
    CUDA_TRY(cudaEventCreate(&e));
    b->tick_ev.push_back(e);
  }
  CUDA_TRY(cudaEventRecord(b->tick_ev[b->tick_ev_used], stream));
  auto launch = [&](int kind, int idx) -> int {
    int steps = 0;
    for (int j = 0; j < n; ++j) {
      const SolveDev& d = b->h_solves[j];
      int seg, t0, t1;
      if ((kind == RES_FWD || (d.flags & F_ADJ)) && res_range(kind, idx, d.nt, d.k, d.nseg, d.it0, d.it1, seg, t0, t1))
        steps = std::max(steps, t1 - t0);
    }
    if (steps == 0) return SEM_OK;
    if (b->ll_tag > 0xf0000000u - (unsigned)steps) {
      CUDA_TRY(cudaMemsetAsync(b->d_ll, 0, b->ll_cap, stream));
      b->ll_tag = 0;
    }
    const bool a = kind == RES_ADJ;
    const ResLay& L = a ? La : Lf;
    const ResShape& h = a ? ha : hf;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)ncta);
    lc.blockDim = dim3((unsigned)(h.nc + h.nio));
    lc.dynamicSmemBytes = (size_t)L.total * 4;
    lc.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    CUDA_TRY(cudaLaunchKernelEx(&lc, a ? fa : ff, (const SolveDev*)b->d_solves, (const int*)b->d_cta, L, b->d_ll,
                                b->ll_tag, kind, idx, h.nc, h.sw, h.ezc));
    b->ll_tag += (unsigned)steps + 2;
    b->last_launches++;
    return SEM_OK;
  };
  int rc = launch(RES_FWD, 0);
  for (int i = 0; i < (adj ? max_seg : 0) && !rc; ++i) {
    if (i > 0) rc = launch(RES_REPLAY, i);
    if (!rc) rc = launch(RES_ADJ, i);
  }
  if (rc) return rc;
  CUDA_TRY(cudaEventRecord(b->tick_ev[b->tick_ev_used + 1], stream));
  b->tick_ev_used += 2;
  b->last_ticks += max_prog;
  for (int s0 = 0; s0 < n; s0 += 65535)
    batch_output_kernel<<<dim3(io_bx, (unsigned)std::min(65535, n - s0)), 256, 0, stream>>>(b->d_io, s0);
  b->last_launches++;
  CUDA_TRY(cudaGetLastError());
  b->last_kernel = 5;
  b->last_tile_ex = exm; b->last_tile_ez = ezm; b->last_zchunk = 0;
  b->last_groups++;
  return SEM_OK;
}

// Runs what can run resident and returns the solves that cannot in `rest`.
int run_resident(sem_batch_t* b, const sem_solve_t* sv, int n, long long budget, cudaStream_t stream,
                 std::vector<int>* rest) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
  std::map<std::tuple<int, bool, bool>, std::vector<int>> classes;
  for (int i = 0; i < n; ++i)
    classes[std::make_tuple(sv[i].plan->npol, sv[i].plan->bnd_n > 0, (sv[i].flags & SEM_F_ADJOINT) != 0)].push_back(i);
  for (auto& kv : classes) {
    const std::vector<ResWave> waves = res_plan(sv, kv.second, sms, budget);
    if (waves.empty()) { rest->insert(rest->end(), kv.second.begin(), kv.second.end()); continue; }
    for (const ResWave& w : waves) {
      const int rc = run_res_wave(b, sv, w, sms, stream);
      if (rc == SEM_ERR_UNSUPPORTED) rest->insert(rest->end(), w.idx.begin(), w.idx.end());
      else if (rc) return rc;
    }
  }
  std::sort(rest->begin(), rest->end());
  return SEM_OK;
}

}  // namespace
