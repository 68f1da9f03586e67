// sem_resident_run.cuh — host side of the resident kernels: tilings, waves, launches.
// Included by sem_kernels.cu after run_group.

namespace {

SolveIo solve_io(const sem_solve_t& s, const Workspace& ws, char* a);

constexpr int kResSmem = 231424;  // dynamic shared bytes: one CTA per SM, 1 KB left for its static ones
typedef void (*ResFn)(const SolveDev*, const int*, ResLay, unsigned long long*, unsigned, int, int, int, int, int);

// variants: one lane per element, two (order 4), one with the increment and the partial gradient in
// memory (adjoint, for meshes whose tiles fit in no other way: 400x200 alone, forward + adjoint, 15.7 us
// a step, 27.7 by strips; not above order 4, where its registers spill: order 5, 240x150, 26.0 us, 24.2
// by strips); and the first two with each solve's tiles in one cluster
enum : int { RES_ONE = 1, RES_TWO = 2, RES_MEM = 3, RES_CONE = 4, RES_CTWO = 5, RES_LAST = 5 };
bool res_clus(int vr) { return vr >= RES_CONE; }
bool res_two(int vr) { return vr == RES_TWO || vr == RES_CTWO; }
int res_lanes(int vr) { return res_two(vr) ? 2 : 1; }
bool res_has(int N, int vr, bool adj) { return vr == RES_MEM ? adj && N <= 4 : !res_two(vr) || N == 4; }
// Clusters of `size` CTAs that fill an SM each which the device holds at once (a cluster stays within a
// GPC); size 1, 2, 4, 8 or 16
int res_clusters(int device, int size);

template <int N, bool ADJ, bool STC>
ResFn res_fn(int vr) {
  if constexpr (N == 4) {
    if (vr == RES_TWO) return sem_resident_kernel<N, 2, ADJ, STC, false, false>;
    if (vr == RES_CTWO) return sem_resident_kernel<N, 2, ADJ, STC, false, true>;
  }
  if constexpr (ADJ && N <= 4) {
    if (vr == RES_MEM) return sem_resident_kernel<N, 1, ADJ, STC, true, false>;
  }
  if (vr == RES_CONE) return sem_resident_kernel<N, 1, ADJ, STC, false, true>;
  return sem_resident_kernel<N, 1, ADJ, STC, false, false>;
}
template <bool ADJ, bool STC>
ResFn res_fn(int N, int vr) {
  switch (N) {
    case 1: return res_fn<1, ADJ, STC>(vr);
    case 2: return res_fn<2, ADJ, STC>(vr);
    case 3: return res_fn<3, ADJ, STC>(vr);
    case 4: return res_fn<4, ADJ, STC>(vr);
    case 5: return res_fn<5, ADJ, STC>(vr);
    case 6: return res_fn<6, ADJ, STC>(vr);
    case 7: return res_fn<7, ADJ, STC>(vr);
  }
  return nullptr;
}
ResFn res_kernel_for(int N, int vr, bool adj, bool stc) {
  if (adj) return stc ? res_fn<true, true>(N, vr) : res_fn<true, false>(N, vr);
  return stc ? res_fn<false, true>(N, vr) : res_fn<false, false>(N, vr);
}

int res_clusters(int device, int size) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, int> have;
  std::lock_guard<std::mutex> lk(mu);
  const auto it = have.find(std::make_pair(device, size));
  if (it != have.end()) return it->second;
  const ResFn fn = res_kernel_for(4, RES_CTWO, true, false);
  int n = 0;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)size);
  lc.blockDim = dim3(512);
  lc.dynamicSmemBytes = kResSmem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)size;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  if (raise_smem_limit((const void*)fn, kResSmem) != cudaSuccess ||
      cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, fn, &lc) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  return have[std::make_pair(device, size)] = n;
}

typedef sem_plan_s::ResCounts ResCounts;
typedef sem_plan_s::ResTiling ResTiling;
typedef sem_plan_s::ResSites ResSites;
// Tile of element e among n tiles of nel elements: the inverse of res_start (the last one for the
// mesh's last node).
int res_owner(int e, int nel, int n) { return e >= nel ? n - 1 : (int)(((long long)e * n) / nel); }

// Receiver lists of the balanced tiling ntx x ntz of a mesh.
struct ResListsHost {
  std::vector<int> ro{0}, ri, io{0}, ii, qo{0}, qp, eo, et;
  std::vector<float> ew;
  ResCounts n;
};
void build_res_lists(int N, int nelx, int nelz, int nrec, const int* base, const float* wts, int ntx, int ntz,
                     ResListsHost* out) {
  const int NP = N + 1, nt = ntx * ntz;
  ResListsHost& L = *out;
  std::vector<std::vector<int>> rec(nt), inj(nt);
  // per tile and quad (row << 16 | element): the receivers that reach it, with node masks and weights
  struct Term { int q, mask; std::vector<float> w; };
  std::vector<std::map<int, std::vector<Term>>> quads(nt);
  for (int r = 0; r < nrec; ++r) {
    const int bx = base[2 * r], bz = base[2 * r + 1];
    rec[res_owner(bz / N, nelz, ntz) * ntx + res_owner(bx / N, nelx, ntx)].push_back(r);
    for (int j = 0; j < NP; ++j)
      for (int i = 0; i < NP; ++i) {
        const int gx = bx + i, gz = bz + j;
        const int tx = res_owner(gx / N, nelx, ntx), tz = res_owner(gz / N, nelz, ntz);
        const int t = tz * ntx + tx;
        if (inj[t].empty() || inj[t].back() != r) inj[t].push_back(r);
        const int q = (int)inj[t].size() - 1;
        const int x0 = res_start(tx, nelx, ntx) * N, z0 = res_start(tz, nelz, ntz) * N;
        auto& terms = quads[t][((gz - z0) << 16) | ((gx - x0) / N)];
        if (terms.empty() || terms.back().q != q) terms.push_back(Term{q, 0, std::vector<float>(N, 0.f)});
        terms.back().mask |= 1 << ((gx - x0) % N);
        terms.back().w[(gx - x0) % N] = wts ? wts[(size_t)r * NP * NP + j * NP + i] : 0.f;
      }
  }
  for (int t = 0; t < nt; ++t) {
    L.ri.insert(L.ri.end(), rec[t].begin(), rec[t].end());
    L.ro.push_back((int)L.ri.size());
    L.ii.insert(L.ii.end(), inj[t].begin(), inj[t].end());
    L.io.push_back((int)L.ii.size());
    const size_t e0 = L.et.size();
    for (auto& kv : quads[t]) {
      L.qp.push_back(kv.first);
      L.eo.push_back((int)L.et.size());
      for (auto& term : kv.second) {
        L.et.push_back(term.q << 8 | term.mask);
        L.ew.insert(L.ew.end(), term.w.begin(), term.w.end());
      }
    }
    L.qo.push_back((int)L.qp.size());
    L.n.nrec = std::max(L.n.nrec, (int)rec[t].size());
    L.n.ninj = std::max(L.n.ninj, (int)inj[t].size());
    L.n.nquad = std::max(L.n.nquad, (int)quads[t].size());
    L.n.nterm = std::max(L.n.nterm, (int)(L.et.size() - e0));
  }
  L.eo.push_back((int)L.et.size());
}
// the same on the device, kept with the plan
int get_res_lists(const sem_plan_s* p, int ntx, int ntz, sem_plan_s::ResLists* out) {
  std::lock_guard<std::mutex> lk(p->mu);
  auto key = std::make_pair(ntx, ntz);
  auto it = p->res_lists.find(key);
  if (it != p->res_lists.end()) { *out = it->second; return SEM_OK; }
  ResListsHost h;
  build_res_lists(p->npol, p->nelx, p->nelz, p->nrec, p->h_rec_base.data(), p->h_rec_w.data(), ntx, ntz, &h);
  sem_plan_s::ResLists L{};
  L.nrec = h.n.nrec; L.ninj = h.n.ninj; L.nquad = h.n.nquad; L.nterm = h.n.nterm;
  int rc;
  if ((rc = upload(&L.l.rec_off, h.ro.data(), h.ro.size())) || (rc = upload(&L.l.rec_ids, h.ri.data(), h.ri.size())) ||
      (rc = upload(&L.l.inj_off, h.io.data(), h.io.size())) || (rc = upload(&L.l.inj_ids, h.ii.data(), h.ii.size())) ||
      (rc = upload(&L.iq_off, h.qo.data(), h.qo.size())) || (rc = upload(&L.iq_pos, h.qp.data(), h.qp.size())) ||
      (rc = upload(&L.iterm_off, h.eo.data(), h.eo.size())) || (rc = upload(&L.iterm, h.et.data(), h.et.size())) ||
      (rc = upload(&L.iterm_w, h.ew.data(), h.ew.size())))
    return rc;
  p->res_lists[key] = L;
  *out = L;
  return SEM_OK;
}

void take_max(ResCounts& a, const ResCounts& b) {
  a.nrec = std::max(a.nrec, b.nrec); a.ninj = std::max(a.ninj, b.ninj);
  a.nquad = std::max(a.nquad, b.nquad); a.nterm = std::max(a.nterm, b.nterm);
}

ResLay res_layout(int N, int vr, bool adj, bool stc, int exm, int ezm, int ezl, const ResCounts& c) {
  ResLay L{};
  const int NP = N + 1;
  // rows of lanes spread over the banks: two lanes per element read rows two apart at once
  auto pitch = [&](int v) { return res_two(vr) ? (v + 7) / 16 * 16 + 8 : 4 * ((v + 3) / 4 | 1); };
  L.Rm = ezm * N + 1;
  L.Cm = exm * N + 1;
  L.qx = exm + 1;
  L.Wp = pitch((N == 4 ? 0 : 4) + N + (exm + 1) * N);
  L.Cp = pitch((exm + 1) * N);
  const int rows = std::max(ezm, ezl + 1) * N;  // in the last tiles the mesh's last line of nodes starts an element row
  L.H = N + rows + 1;
  int o = 0;
  auto take = [&](long long n, int align = 4) { o = (int)round_up(o, align); const int at = o; o += (int)n; return at; };
  L.reg = L.Wp * L.H;
  L.wreg = (int)round_up(L.reg, 32);
  const int own = L.Cp * rows;
  if (adj) L.w = take(2LL * L.wreg, 32);
  L.b = take(2LL * L.reg); L.c = take(L.reg);
  if (vr != RES_MEM) L.v = take(own);
  if (adj && vr != RES_MEM) L.g = take(own);
  L.tz = take(8LL * rows);
  const long long words = (long long)(L.Rm + L.Cm) * NP + 1;
  L.wi = take(vr == RES_MEM ? words : 2 * words); L.wo = take(vr == RES_MEM ? words : 2 * words);
  if (adj) {
    L.nrm = std::max(1, c.ninj);
    L.niq = c.nquad;
    L.rs = take(4LL * L.nrm);
    L.ia = take(2LL * c.nquad * N);
    L.io = take((long long)c.nquad + 1);
    if (vr != RES_MEM) {
      L.iq = take(c.nterm);
      L.ie = take((long long)c.nterm * N);
    }
    L.im = take(((long long)rows * L.qx + 1) / 2);
  }
  if (stc) { const int bn = 2 * L.Rm + L.Cm; L.be = take(3LL * bn); L.bd = take(2LL * bn); }
  L.ll_t = L.Rm * N; L.ll_r = L.ll_t + L.Cm * N; L.ll_b = L.ll_r + L.Rm; L.ll_c = L.ll_b + L.Cm;
  L.llw = (int)round_up(L.ll_c + 1, 16);
  L.sl = res_clus(vr) ? take(2LL * kResSlots * L.llw) : -1;
  L.total = (int)round_up(o, 4);
  return L;
}

// Threads of a launch whose largest tile is exm x ezm elements (the lowest ezl high): lanes per
// tile row, element rows per chunk, compute and receiver threads; exchange words.
struct ResShape { int sw, ezc, nc, nio, edge; };
bool res_shape(int N, int vr, bool adj, int exm, int ezm, int ezl, int nrec, ResShape* h) {
  const int ezr = std::max(ezm, ezl + 1);  // element rows, the mesh's last line of nodes counted as one
  h->nio = (int)round_up(std::max(nrec, 1), 32);
  h->edge = (exm + ezm) * N * (N + 1);
  const int tmax = res_threads(N, res_lanes(vr), adj) - h->nio;
  h->sw = 4;
  while (h->sw < (exm + 2) * res_lanes(vr)) h->sw *= 2;
  if (h->sw > 32 || tmax < 32) return false;
  h->ezc = (ezr + tmax / h->sw - 1) / (tmax / h->sw);
  h->nc = (int)round_up((long long)((ezr + h->ezc - 1) / h->ezc) * h->sw, 32);
  return true;
}
// Modelled cycles of one step: the exchange (0.47 us between SMs, poll, send, barrier; 1.2 a word),
// then the warps' work: the fp32 operations of a lane, chunk by chunk, at 1.6 cycles (adjoint 1.7
// with two lanes per element, 1.9 with one: fewer warps hide less) times the warps per scheduler.
// Fitted to meshes of 20x10 to 200x100, order 4, to within 8 % (adjoint with two lanes: 14 %).
// Two lanes per element halve a step's serial work, which decides small tiles (100x50 alone:
// 1.84 us forward and 4.35 with the adjoint, 2.16 and 4.79 with one lane); one lane has no
// swaps between them, which decides full SMs (128 of 100x50: 133 us a step, 142 with two).
// Two or three smaller CTAs per SM, which hide one another's exchange, measured the same or
// slower (16 of 100x50 with one lane: 18.1 us a step with one, 18.9 with two, 22.5 with three).
// A cluster's exchange is shorter, but a solve then has 16 SMs at most (a B200 holds 7 clusters of 16, 15
// of 8): us a step forward / adjoint, all SMs -> one cluster: 20x10 1.62 / 1.88 -> 1.18 / 1.70, 48x28 forward
// 1.68 -> 1.51, order 3, 40x20 1.80 / 2.02 -> 1.27 / 1.58, order 5, 37x31 2.95 / 4.85 -> 2.43 / 4.23; with too
// much work per SM, order 3, 80x40: 1.73 / 2.01 -> 2.20 / 2.08 (before the cluster kernels were compiled apart).
double res_step_cost(int N, int vr, bool adj, const ResShape& h) {
  const double NP = N + 1;
  const double el = adj ? 2 * N * (3 * NP * NP + 4 * NP) + 16 * N * N : 2 * N * (2 * NP * NP + 2 * NP) + 10 * N * N;
  const double carry = N * (NP * NP + 3 * NP) + (adj ? N * (NP + 2) : 0);
  const double fixed = (res_two(vr) ? 2600.0 : adj ? 2300.0 : 2500.0) - (!res_clus(vr) ? 0.0 : res_two(vr) ? (adj ? 380.0 : 900.0) : adj ? 900.0 : 1050.0);
  const double rate = !adj ? 1.6 : res_two(vr) ? 1.7 : vr == RES_MEM ? 2.1 : 1.9;
  return fixed + 1.2 * h.edge + rate * std::max(1.0, h.nc / 128.0) * (h.ezc * el + carry) / res_lanes(vr);
}
bool res_fits(const ResLay& L) {  // (256: the history box; 4096: the place of a packed exchange word)
  return L.Wp <= 256 && L.H <= 256 && L.llw <= 4096 && (long long)L.total * 4 <= kResSmem;
}

// Where a mesh's receivers are, whatever the tiling: elements with receivers, and the cells (one
// element's own columns of nodes times one element row's own rows) that they reach, with their quads
// (rows of N nodes) and the receivers' terms in them.  The last row and column of an element's nodes
// are the next cells'.
ResSites res_sites(int N, int nrec, const int* base) {
  std::map<std::pair<int, int>, int> el;                     // receivers by element (z, x)
  std::map<std::pair<int, int>, std::pair<int, int>> cells;  // quads and terms by cell (z, x)
  for (int r = 0; r < nrec; ++r) ++el[std::make_pair(base[2 * r + 1] / N, base[2 * r] / N)];
  for (auto& kv : el)
    for (int q = 0; q < 4; ++q) {
      const int rows = q < 2 ? N : 1;
      auto& c = cells[std::make_pair(kv.first.first + (q >> 1), kv.first.second + (q & 1))];
      c.first = std::max(c.first, rows);
      c.second += rows * kv.second;
    }
  ResSites s;
  for (auto& kv : el) s.el.push_back({kv.first.second, kv.first.first, kv.second});
  for (auto& kv : cells) s.cells.push_back({kv.first.second, kv.first.first, kv.second.first, kv.second.second});
  return s;
}
// The largest counts that build_res_lists finds in any tile of a tiling, without the lists: a search
// meets many tilings, and a mesh may have thousands of receivers (first forward call of a plan, 100x50
// with 8000: 40 ms when each tiling went through all receivers, 11 now; 60x30 with 5000: 25 and 6.5).
ResCounts res_counts(const ResSites& s, int nelx, int nelz, int ntx, int ntz) {
  std::vector<int> ox(nelx + 1), oz(nelz + 1);
  for (int e = 0; e <= nelx; ++e) ox[e] = res_owner(e, nelx, ntx);
  for (int e = 0; e <= nelz; ++e) oz[e] = res_owner(e, nelz, ntz) * ntx;
  std::vector<ResCounts> t((size_t)ntx * ntz);
  ResCounts c;
  for (const auto& e : s.el) {
    t[oz[e.ez] + ox[e.ex]].nrec += e.n;
    for (int z = 0; z < (oz[e.ez + 1] != oz[e.ez] ? 2 : 1); ++z)
      for (int x = 0; x < (ox[e.ex + 1] != ox[e.ex] ? 2 : 1); ++x) t[oz[e.ez + z] + ox[e.ex + x]].ninj += e.n;
  }
  for (const auto& e : s.cells) {
    ResCounts& q = t[oz[e.ez] + ox[e.ex]];
    q.nquad += e.quads;
    q.nterm += e.terms;
  }
  for (const ResCounts& q : t) take_max(c, q);
  return c;
}

// Tiling of a plan into at most sms tiles of at most E elements that fit a CTA: the one with the
// least work (tiles times modelled step); kept with the plan.  0 x 0: none.
ResTiling res_tiling(const sem_plan_s* p, int vr, bool adj, int E, int sms) {
  std::lock_guard<std::mutex> lk(p->mu);
  const auto key = std::make_tuple(vr, adj, E);
  auto it = p->res_tilings.find(key);
  if (it != p->res_tilings.end()) return it->second;
  if (p->nrec > 0 && p->res_sites.el.empty()) p->res_sites = res_sites(p->npol, p->nrec, p->h_rec_base.data());
  ResTiling best;
  double best_c = -1.0;
  const bool stc = p->bnd_n > 0;
  for (int tx = 1; tx <= p->nelx; ++tx) {
    const int ex = (p->nelx + tx - 1) / tx;
    if (tx > 1 && ex == (p->nelx + tx - 2) / (tx - 1)) continue;  // no narrower than with one tile less
    const int ezm = E / ex;
    if (ezm < 1 || (ex + 2) * res_lanes(vr) > 32) continue;
    const int tz = (p->nelz + ezm - 1) / ezm, ez = (p->nelz + tz - 1) / tz;
    const int nt = tx * tz;
    if ((long long)tx * tz > sms) continue;
    if (res_clus(vr) && (nt > 16 || (nt & (nt - 1)) || !res_clusters(p->device, nt))) continue;
    ResShape h;
    if (!res_shape(p->npol, vr, adj, ex, ez, p->nelz / tz, 1, &h)) continue;
    const double c = res_step_cost(p->npol, vr, adj, h);
    if (best_c >= 0.0 && tx * tz * c >= best_c) continue;
    // (counted once per tiling: the search meets each many times, and a plan may serve one call only)
    const auto at = p->res_tile_counts.find(std::make_pair(tx, tz));
    const ResCounts cnt = at != p->res_tile_counts.end()
                              ? at->second
                              : (p->res_tile_counts[std::make_pair(tx, tz)] = res_counts(p->res_sites, p->nelx, p->nelz, tx, tz));
    if (!res_shape(p->npol, vr, adj, ex, ez, p->nelz / tz, adj ? cnt.ninj : cnt.nrec, &h) ||
        !res_fits(res_layout(p->npol, vr, adj, stc, ex, ez, p->nelz / tz, cnt)))
      continue;
    best.tx = tx; best.tz = tz;
    best.n = cnt;
    best_c = tx * tz * c;
  }
  p->res_tilings[key] = best;
  return best;
}

// Tile capacities that are tried: 8 to 1200 elements
template <class F>
void res_capacities(F&& f) {
  for (double E = 8.0; E < 1200.0; E *= 1.15) f((int)E);
}
// The variants a plan's solve needs by itself: RES_ONE (or RES_TWO), RES_MEM (its adjoint tiles fit
// in no other way) or 0 (too large).
int res_need(const sem_plan_s* p, bool adj, int sms) {
  {
    std::lock_guard<std::mutex> lk(p->mu);
    if (p->res_need[adj] >= 0) return p->res_need[adj];
  }
  auto any = [&](int vr, bool a) {
    bool fit = false;
    if (res_has(p->npol, vr, a)) res_capacities([&](int E) { fit = fit || res_tiling(p, vr, a, E, sms).tx > 0; });
    return fit;
  };
  int need = any(RES_ONE, false) || any(RES_TWO, false) ? RES_ONE : 0;
  if (need && adj) need = any(RES_ONE, true) || any(RES_TWO, true) ? RES_ONE : any(RES_MEM, true) ? RES_MEM : 0;
  std::lock_guard<std::mutex> lk(p->mu);
  return p->res_need[adj] = need;
}

// Waves of one kernel over a group of solves: each solve's tiling, and the solves (places in the
// group) whose CTAs are resident at once.  A wave's launch shape is its largest tile's.
struct ResPack {
  int vr = 0;          // variant
  double cost = -1.0;  // modelled cycles; < 0: a solve does not fit
  std::vector<ResTiling> tiles;
  std::vector<std::vector<int>> waves;
};
struct ResGroup {
  std::vector<int> idx, k;  // solves and their checkpoint intervals
  ResPack fwd, adj;
};

// For each tile capacity, pack the solves (in order) into waves and keep the capacity, and the
// lanes per element, with the smallest modelled time.  steps: time steps of each solve's launches.
ResPack res_pack(const sem_solve_t* sv, const std::vector<int>& idx, const std::vector<int>& steps, bool adj, int sms) {
  const int n = (int)idx.size(), N = sv[idx[0]].plan->npol;
  std::vector<const sem_plan_s*> plans;
  std::vector<int> pl(n);
  for (int j = 0; j < n; ++j) {
    const auto f = std::find(plans.begin(), plans.end(), sv[idx[j]].plan);
    pl[j] = (int)(f - plans.begin());
    if (f == plans.end()) plans.push_back(sv[idx[j]].plan);
  }
  const bool stc = plans[0]->bnd_n > 0;
  ResPack best;
  auto rounds = [&](int size, int count) {  // of a wave of clusters
    const int at_once = size > 0 ? std::max(1, res_clusters(plans[0]->device, size)) : 1;
    return (double)((count + at_once - 1) / at_once);
  };
  std::vector<ResTiling> tl(plans.size()), last;
  std::vector<int> first;
  for (int vr = RES_ONE; vr <= RES_LAST; ++vr) {
    if (!res_has(N, vr, adj)) continue;
    last.clear();
    res_capacities([&](int E) {
      bool ok = true, same = !last.empty();
      for (size_t q = 0; q < plans.size() && ok; ++q) {
        tl[q] = res_tiling(plans[q], vr, adj, E, sms);
        ok = tl[q].tx > 0;
        same = same && tl[q].tx == last[q].tx && tl[q].tz == last[q].tz;
      }
      if (!ok || same) return;
      last = tl;
      first.clear();
      double cost = 0.0, step = 0.0;
      int used = 0, nt = 0, exm = 0, ezm = 0, ezl = 0, in_wave = 0;
      ResCounts cnt;
      for (int j = 0; j < n; ++j) {
        const ResTiling& t = tl[pl[j]];
        const sem_plan_s* p = plans[pl[j]];
        const int ex = (p->nelx + t.tx - 1) / t.tx, ez = (p->nelz + t.tz - 1) / t.tz, el = p->nelz / t.tz;
        ResCounts c = cnt;
        take_max(c, t.n);
        ResShape h;
        // a wave of clusters has one size of cluster and needs not be resident at once
        bool fits = j > 0 && (res_clus(vr) ? t.tx * t.tz == used : used + t.tx * t.tz <= sms);
        if (fits) {
          const int x = std::max(ex, exm), z = std::max(ez, ezm);
          fits = res_shape(N, vr, adj, x, z, std::max(el, ezl), adj ? c.ninj : c.nrec, &h) &&
                 res_fits(res_layout(N, vr, adj, stc, x, z, std::max(el, ezl), c));
        }
        if (!fits) {  // the next wave
          cost += step * (res_clus(vr) ? rounds(used, in_wave) * nt : nt);
          in_wave = 0;
          first.push_back(j);
          used = nt = exm = ezm = ezl = 0;
          c = t.n;
          res_shape(N, vr, adj, ex, ez, el, adj ? c.ninj : c.nrec, &h);
        }
        cnt = c;
        used = res_clus(vr) ? t.tx * t.tz : used + t.tx * t.tz;
        ++in_wave;
        exm = std::max(exm, ex); ezm = std::max(ezm, ez); ezl = std::max(ezl, el);
        step = res_step_cost(N, vr, adj, h);
        nt = std::max(nt, steps[j]);
      }
      cost += step * (res_clus(vr) ? rounds(used, in_wave) * nt : nt);
      if (best.cost >= 0.0 && cost >= best.cost) return;
      best.cost = cost;
      best.vr = vr;
      best.tiles.resize(n);
      for (int j = 0; j < n; ++j) best.tiles[j] = tl[pl[j]];
      best.waves.clear();
      for (size_t w = 0; w < first.size(); ++w) {
        best.waves.emplace_back();
        for (int j = first[w]; j < (w + 1 < first.size() ? first[w + 1] : n); ++j) best.waves.back().push_back(j);
      }
    });
  }
  return best;
}

// Groups of one class of solves (same order, boundary mode, forward-only or not), longest first:
// each group's workspaces fit the budget.  Forward and adjoint launches have waves of their own:
// the forward kernel needs less room per element, so its waves hold more solves (128 models of
// 100x50, forward and adjoint: 146 us a step when both had the adjoint's tiles, 132 now).
// Empty when a solve fits no way.
std::vector<ResGroup> res_plan(const sem_solve_t* sv, const std::vector<int>& cls, int sms, long long budget) {
  const bool adj = sv[cls[0]].flags & SEM_F_ADJOINT;
  std::vector<int> ord(cls);
  std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) {
    return (long long)sv[a].plan->nt * 64 + sv[a].plan->npoints / 4096 > (long long)sv[b].plan->nt * 64 + sv[b].plan->npoints / 4096;
  });
  std::vector<ResGroup> groups;
  long long mem = 0;
  for (int i : ord) {
    // checkpoint interval and bytes of the solve by itself
    const sem_solve_t& s = sv[i];
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
    const long long bytes = layout(s.plan, s.flags, k, &ns).bytes;
    if (groups.empty() || mem + bytes > budget) {
      groups.emplace_back();
      mem = 0;
    }
    groups.back().idx.push_back(i);
    groups.back().k.push_back(k);
    mem += bytes;
  }
  for (ResGroup& g : groups) {
    std::vector<int> nf, na;
    for (size_t j = 0; j < g.idx.size(); ++j) {
      const int nt = sv[g.idx[j]].plan->nt, k = g.k[j];
      nf.push_back(nt + (adj ? k * ((nt + k - 1) / k - 1) : 0));
      na.push_back(nt);
    }
    g.fwd = res_pack(sv, g.idx, nf, false, sms);
    if (g.fwd.cost < 0.0) return {};
    if (!adj) continue;
    g.adj = res_pack(sv, g.idx, na, true, sms);
    if (g.adj.cost < 0.0) return {};
  }
  return groups;
}

// One launch shape: a wave of one kernel.
struct ResWave {
  ResFn fn;
  ResLay L;
  ResShape h;
  int ncta, cta0;           // CTAs, and where their list starts
  int cluster;              // CTAs per cluster, or 0: a cooperative launch
  const std::vector<int>* solves;
};

// One group: set-up, forward launches, (replay and) adjoint launches, outputs.  at: the solves'
// workspaces, or null (the batch's arena).  SEM_ERR_UNSUPPORTED without a message when the group cannot run this way (nothing launched).
int run_res_group(sem_batch_t* b, const sem_solve_t* sv, char* const* at, const ResGroup& w, int sms, cudaStream_t stream) {
  if (b->fail_groups > 0 && b->fail_skip-- <= 0) {
    b->fail_skip = 0;
    --b->fail_groups;
    return fail(SEM_ERR_OOM, "resident group refused by sem_selftest_fail_marches");
  }
  const int n = (int)w.idx.size();
  const sem_plan_s* p0 = sv[w.idx[0]].plan;
  const int N = p0->npol;
  const bool adj = sv[w.idx[0]].flags & SEM_F_ADJOINT, stc = p0->bnd_n > 0;
  // ---- launch shapes of the forward and adjoint waves
  std::vector<sem_plan_s::ResLists> lists[2];
  std::vector<ResWave> waves[2];
  std::vector<int> wave_of(n), base[2];
  long long ll_words = 0;
  int cta0 = 0;
  for (int q = 0; q < (adj ? 2 : 1); ++q) {
    const ResPack& pk = q ? w.adj : w.fwd;
    lists[q].resize(n);
    base[q].resize(n);
    for (const std::vector<int>& wv : pk.waves) {
      ResWave v{};
      ResCounts c;
      int exm = 1, ezm = 1, ezl = 1;
      for (int j : wv) {
        const sem_plan_s* p = sv[w.idx[j]].plan;
        const int tx = pk.tiles[j].tx, tz = pk.tiles[j].tz;
        sem_plan_s::ResLists& l = lists[q][j];
        if (int rc = get_res_lists(p, tx, tz, &l)) return rc;
        c.nrec = std::max(c.nrec, l.nrec); c.ninj = std::max(c.ninj, l.ninj);
        c.nquad = std::max(c.nquad, l.nquad); c.nterm = std::max(c.nterm, l.nterm);
        exm = std::max(exm, (p->nelx + tx - 1) / tx); ezm = std::max(ezm, (p->nelz + tz - 1) / tz);
        ezl = std::max(ezl, p->nelz / tz);
        base[q][j] = v.ncta;
        v.ncta += tx * tz;
      }
      v.cta0 = cta0;
      cta0 += v.ncta;
      v.solves = &wv;
      v.L = res_layout(N, pk.vr, q, stc, exm, ezm, ezl, c);
      v.fn = res_kernel_for(N, pk.vr, q, stc);
      if (!res_shape(N, pk.vr, q, exm, ezm, ezl, q ? c.ninj : c.nrec, &v.h)) return SEM_ERR_UNSUPPORTED;
      v.cluster = res_clus(pk.vr) ? pk.tiles[wv[0]].tx * pk.tiles[wv[0]].tz : 0;
      int nb = 0;
      if (!res_fits(v.L) || raise_smem_limit((const void*)v.fn, (size_t)v.L.total * 4) != cudaSuccess ||
          (v.cluster > 8 && cudaFuncSetAttribute(v.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, v.fn, v.h.nc + v.h.nio, (size_t)v.L.total * 4) != cudaSuccess ||
          (long long)nb * sms < (v.cluster ? v.cluster : v.ncta)) {
        cudaGetLastError();
        return SEM_ERR_UNSUPPORTED;
      }
      if (!v.cluster) ll_words = std::max(ll_words, (long long)v.ncta * kResSlots * v.L.llw);
      if (q)
        for (int j : wv) wave_of[j] = (int)waves[q].size();
      else { b->last_tile_ex = exm; b->last_tile_ez = ezm; }
      waves[q].push_back(v);
    }
  }

  // ---- workspaces, descriptors
  std::vector<Workspace> ws(n);
  std::vector<int> nseg(n);
  long long total = 0;
  int max_seg = 1;
  for (int j = 0; j < n; ++j) {
    const sem_solve_t& s = sv[w.idx[j]];
    ws[j] = layout(s.plan, s.flags, w.k[j], &nseg[j]);
    total += ws[j].bytes;
    max_seg = std::max(max_seg, nseg[j]);
  }
  if (!at && total > b->arena_bytes) {
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
  const int nq = adj ? 2 : 1;  // descriptors: the forward waves', then the adjoint waves'
  b->h_solves.assign((size_t)n * nq, SolveDev{});
  b->h_cta.resize(cta0);
  b->h_io.clear();
  long long off = 0, max_pts = 1;
  for (int j = 0; j < n; ++j) {
    const sem_solve_t& s = sv[w.idx[j]];
    const sem_plan_s* p = s.plan;
    char* a = at ? at[w.idx[j]] : b->arena + off;
    SolveDev& d = b->h_solves[j];
    d.nelx = p->nelx; d.nelz = p->nelz; d.nxg = p->nxg; d.nzg = p->nzg; d.pitch = p->pitch;
    d.tiles_x = w.fwd.tiles[j].tx; d.tiles_z = w.fwd.tiles[j].tz;
    d.zchunk = p->nelz;
    d.tile_base = base[0][j];
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
      const ResLay& L = waves[1][wave_of[j]].L;
      if (int rc = encode_band_map(&b->h_tmaps[j], a, p, field_slots(ws[j], p, true), L.Wp, L.H)) return rc;
      d.tmap = b->d_tmaps + j;
    }
    d.D = p->D; d.beta = p->beta; d.tx = p->tx; d.tz = p->tz; d.src_term = p->src_term;
    d.rec_base = p->rec_base; d.rec_w = p->rec_w;
    d.rec_tile_off = lists[0][j].l.rec_off; d.rec_tile_ids = lists[0][j].l.rec_ids;
    d.rec_out = s.rec_out; d.yobs = s.y_obs;
    d.misfit = (double*)(a + ws[j].misfit);
    d.rmax = d.misfit + p->nrec;
    d.adj_scale = d.misfit + 2 * p->nrec;
    d.status = (int*)(a + ws[j].status);
    d.ws = (const float*)a;
    d.bnd_n = p->bnd_n; d.bnd_pitch = bnd_pitch_of(p);
    d.bnd_coef = p->bnd_n ? (const float*)(a + ws[j].bnd_coef) : nullptr;
    d.bnd_hist = ws[j].bnd_hist >= 0 ? (float*)(a + ws[j].bnd_hist) : nullptr;
    if (adj) {
      SolveDev& e = b->h_solves[n + j];
      const sem_plan_s::ResLists& l = lists[1][j];
      e = d;
      e.tiles_x = w.adj.tiles[j].tx; e.tiles_z = w.adj.tiles[j].tz;
      e.tile_base = base[1][j];
      e.rec_tile_off = l.l.rec_off; e.rec_tile_ids = l.l.rec_ids;
      e.inj_tile_off = l.l.inj_off; e.inj_tile_ids = l.l.inj_ids;
      e.iq_off = l.iq_off; e.iq_pos = l.iq_pos; e.iterm_off = l.iterm_off;
      e.iterm = l.iterm; e.iterm_w = l.iterm_w;
    }
    b->h_io.push_back(solve_io(s, ws[j], a));
    max_pts = std::max(max_pts, (long long)p->npoints);
    off += ws[j].bytes;
  }
  for (int q = 0; q < nq; ++q)
    for (const ResWave& v : waves[q])
      for (int j : *v.solves) {
        const SolveDev& d = b->h_solves[q * n + j];
        std::fill_n(b->h_cta.begin() + v.cta0 + d.tile_base, d.tiles_x * d.tiles_z, q * n + j);
      }
  if (n * nq > b->solves_cap) {
    cudaFree(b->d_solves);
    b->d_solves = nullptr;
    b->solves_cap = 0;
    CUDA_TRY(cudaMalloc((void**)&b->d_solves, sizeof(SolveDev) * n * nq));
    b->solves_cap = n * nq;
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
  const long long ll_bytes = ll_words * 8;
  if (ll_bytes > b->ll_cap) {
    cudaFree(b->d_ll);
    b->d_ll = nullptr;
    b->ll_cap = 0;
    CUDA_TRY(cudaMalloc((void**)&b->d_ll, ll_bytes));
    b->ll_cap = ll_bytes;
    CUDA_TRY(cudaMemsetAsync(b->d_ll, 0, ll_bytes, stream));
    b->ll_tag = 0;
  }
  // The launches of a captured run carry the same tags at every replay.  So the words are cleared before
  // them, and, since a replay leaves such tags behind at any time, before all later runs of this batch.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  CUDA_TRY(cudaStreamIsCapturing(stream, &cap));
  b->ll_recorded |= cap != cudaStreamCaptureStatusNone;
  if (b->ll_recorded && ll_bytes > 0) CUDA_TRY(cudaMemsetAsync(b->d_ll, 0, ll_bytes, stream));
  CUDA_TRY(cudaMemcpyAsync(b->d_solves, b->h_solves.data(), sizeof(SolveDev) * n * nq, cudaMemcpyHostToDevice, stream));
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
    const int q = kind == RES_ADJ;
    for (const ResWave& v : waves[q]) {
      int steps = 0;
      for (int j : *v.solves) {
        const SolveDev& d = b->h_solves[j];
        int seg, t0, t1;
        if (res_range(kind, idx, d.nt, d.k, d.nseg, d.it0, d.it1, seg, t0, t1)) steps = std::max(steps, t1 - t0);
      }
      if (steps == 0) continue;
      if (b->ll_tag > 0xf0000000u - (unsigned)steps) {
        if (b->d_ll) CUDA_TRY(cudaMemsetAsync(b->d_ll, 0, b->ll_cap, stream));
        b->ll_tag = 0;
      }
      cudaLaunchConfig_t lc = {};
      const bool drop = b->drop_tile && !v.cluster && v.ncta > 1;
      b->drop_tile = b->drop_tile && !drop;
      lc.gridDim = dim3((unsigned)(v.ncta - drop));
      lc.blockDim = dim3((unsigned)(v.h.nc + v.h.nio));
      lc.dynamicSmemBytes = (size_t)v.L.total * 4;
      lc.stream = stream;
      cudaLaunchAttribute at[1];
      if (v.cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)v.cluster;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
      }
      lc.attrs = at;
      lc.numAttrs = 1;
      CUDA_TRY(cudaLaunchKernelEx(&lc, v.fn, (const SolveDev*)b->d_solves, (const int*)b->d_cta + v.cta0, v.L, b->d_ll,
                                  b->ll_tag, kind, idx, v.h.nc, v.h.sw, v.h.ezc));
      b->ll_tag += (unsigned)steps + 2;
      b->last_launches++;
    }
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
  for (int q = 0; q < nq; ++q)
    for (const ResWave& v : waves[q]) {
      int prog = 0;
      for (int j : *v.solves) {
        const SolveDev& d = b->h_solves[j];
        prog = std::max(prog, q ? 1 + d.nt : d.nt + ((d.flags & F_SHIFT) ? 1 : 0) + (adj ? d.k * (d.nseg - 1) : 0));
      }
      b->last_ticks += prog;
    }
  for (int s0 = 0; s0 < n; s0 += 65535)
    batch_output_kernel<<<dim3(io_bx, (unsigned)std::min(65535, n - s0)), 256, 0, stream>>>(b->d_io, s0);
  b->last_launches++;
  CUDA_TRY(cudaGetLastError());
  b->last_kernel = 5;
  b->last_zchunk = 0;
  b->last_groups += (int)std::max(waves[0].size(), waves[1].size());
  return SEM_OK;
}

int sm_count(int device) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms;
}
// The class a solve runs resident in, or 0.  Adjoint solves too large for shared memory that were
// given a checkpoint interval keep the strip kernel, as they had it before (a replay with fields in
// memory was not timed).
int res_class(const sem_solve_t& s, int sms) {
  const int need = res_need(s.plan, s.flags & SEM_F_ADJOINT, sms);
  return need == RES_MEM && s.ckpt_k > 0 && s.ckpt_k < s.plan->nt ? 0 : need;
}

// Whether a class of solves runs faster by ticks, although it fits the SMs.  Times: 400 steps of solves
// with 20 m elements, by ticks -> resident.
bool ticks_win(const sem_solve_t* sv, const std::vector<int>& cls, int sms) {
  const sem_plan_s* p0 = sv[cls[0]].plan;
  const bool adj = sv[cls[0]].flags & SEM_F_ADJOINT, stc = p0->bnd_n > 0;
  long long elements = 0, chunks = 0, points = 0;
  int nt = 0, k = 0;  // longest solve, longest segment of one that is replayed in several
  for (int i : cls) {
    const sem_plan_s* p = sv[i].plan;
    if (p->nrec > std::min(kStripInj, kMaxInj)) return false;  // (strips and tiles may refuse more in one place)
    points += p->npoints;
    nt = std::max(nt, p->nt);
    k = std::max(k, adj && sv[i].ckpt_k > 0 && sv[i].ckpt_k < p->nt ? (int)sv[i].ckpt_k : INT_MAX);
    elements += (long long)p->nelx * p->nelz;
    chunks += (long long)strips_of(p, nullptr) * ((p->nelz + kMinChunk - 1) / kMinChunk);
  }
  const double each = (double)elements / cls.size();
  // A march has a prologue (20 us a wave of solves) that few steps do not pay for, the fewer the more waves
  // there are: forward, one 100x50, 1 step 0.05 -> 0.06 ms (5 steps 0.07, both); 32 of them, 5 steps
  // 0.25 -> 0.28 (12 steps 0.41 -> 0.35); 128 of them, 12 steps 1.19 -> 1.41 (24 steps 2.0, both); gradients
  // 0.14 -> 0.18 (0.19, both), 0.67 -> 0.80 (1.10 -> 1.02), 3.2 -> 3.6 (5.3 -> 5.0).
  if (nt <= 5.0 + 1.2e-6 * (double)points) return true;
  // So has each segment's replay and adjoint, which a short explicit interval repeats every k steps: 300
  // steps, k = 2, 40x20: order 2 4.8 -> 4.9 ms, order 3 4.9 -> 6.5 (k = 3: 4.9 -> 4.7), order 4 5.1 -> 5.7 (5.1
  // -> 4.4), order 5 5.8 -> 10.6 (k = 3: 5.8 -> 8.0; k = 4 and 4 models: 6.8, both); 30x15, order 6, k = 6
  // 5.7 -> 7.1 (k = 10: 5.7 -> 5.9, 4 models 7.5 -> 5.9), order 7, k = 10 6.2 -> 9.4 (k = 16, 4 models: 8.3 -> 8.7).
  static const int shortest[8] = {0, 2, 2, 3, 3, 4, 8, 16};
  if (k < shortest[p0->npol]) return true;
  if (p0->npol == 7) {
    // A lane's element of order 7 does not fit its registers (500 to 1200 bytes spilled): 6 us a forward
    // step and 10 an adjoint one, however small the tile.  Where a tick takes its least time too it is
    // faster: gradients 28x14 6.2 -> 8.0 ms, 23x11 6.4 -> 6.9 (but 11x6 6.6 -> 6.2, 57x29 8.4 -> 8.0, 4 of
    // 23x11 7.2 -> 6.9); with Stacey edges, gradients 23x11 6.4 -> 8.0, 4 of 16x8 6.7 -> 8.1 (6x3 8.2 -> 7.2,
    // 4 of 34x17 10.3 -> 8.2), forward 23x11 2.6 -> 2.9, 8 of 11x6 2.6 -> 2.8 (8 of 16x8 3.0 -> 2.7).
    if (stc ? (adj ? each >= 60 && elements < 2000 : elements < 1000) : adj && each >= 120 && elements < 800) return true;
    // And strips that fill the GPU hide what one warp waits for: sponge gradients, 2 of 157x79 12.5 -> 18.9,
    // 16 of 57x29 21.2 -> 23.9 (forward 8.0 -> 6.2; Stacey gradients 64 of 23x11 27.5 -> 19.8).
    if (adj && !stc && strip_fills(chunks, sms)) return true;
  }
  return false;
}

// Runs what can run resident and returns the solves that cannot in `rest`; unless `all`, those too that
// are faster by ticks.  at: see run_res_group.  ran: set for the solves that were launched, also when a
// later group fails.
int run_resident(sem_batch_t* b, const sem_solve_t* sv, char* const* at, int n, long long budget, bool all, cudaStream_t stream,
                 std::vector<int>* rest, std::vector<char>* ran = nullptr) {
  const int sms = sm_count(b->device);
  std::map<std::tuple<int, bool, bool, int>, std::vector<int>> classes;
  for (int i = 0; i < n; ++i) {
    const sem_plan_s* p = sv[i].plan;
    const bool adj = sv[i].flags & SEM_F_ADJOINT;
    const int need = res_class(sv[i], sms);
    if (!need) rest->push_back(i);
    else classes[std::make_tuple(p->npol, p->bnd_n > 0, adj, need)].push_back(i);
  }
  long long by_ticks = 0;  // bytes of the workspaces that the tick kernels then hold at once
  for (auto& kv : classes) {
    if (!all && ticks_win(sv, kv.second, sms)) {
      long long bytes = 0;
      int ns;
      for (int i : kv.second) {
        const bool adj = sv[i].flags & SEM_F_ADJOINT;
        const int k = adj ? std::max(2, std::min((int)sv[i].ckpt_k, sv[i].plan->nt)) : 2;
        if (!adj || sv[i].ckpt_k > 0) bytes += layout(sv[i].plan, sv[i].flags, k, &ns).bytes;
      }
      if (by_ticks + bytes <= budget) {  // (these split no batch without an automatic interval)
        by_ticks += bytes;
        rest->insert(rest->end(), kv.second.begin(), kv.second.end());
        continue;
      }
    }
    const std::vector<ResGroup> groups = res_plan(sv, kv.second, sms, budget);
    if (groups.empty()) { rest->insert(rest->end(), kv.second.begin(), kv.second.end()); continue; }
    for (const ResGroup& g : groups) {
      const int rc = run_res_group(b, sv, at, g, sms, stream);
      if (rc == SEM_ERR_UNSUPPORTED) rest->insert(rest->end(), g.idx.begin(), g.idx.end());
      else if (rc) return rc;
      else if (ran) for (int i : g.idx) (*ran)[i] = 1;
    }
  }
  std::sort(rest->begin(), rest->end());
  return SEM_OK;
}

}  // namespace
