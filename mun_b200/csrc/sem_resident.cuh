// sem_resident.cuh — resident kernels: one cooperative launch marches a wave of solves
// through all their time steps with the state held on chip.
//
// Included by sem_kernels.cu inside its anonymous namespace (uses SolveDev, the order
// constants c_D2 / c_B2, the ring and mbarrier helpers and the shared node arithmetic).
//
// Why.  A time step of one solve moves little and computes little (100x50 elements at
// N = 4: 80,601 nodes, 40 fp32 operations each: 0.1 us of the GPU), so a launch per step
// is bound by the launch chain (6 to 8 us a step measured for single solves), and for
// batches by re-reading every field from L2 or HBM through a pipeline of small bands
// (67 / 110 us per forward / adjoint step of 128 models).  Here each CTA owns a tile of
// elements of one solve for the whole sweep; displacement, increment, c^2 and the partial
// gradient stay in its shared memory, and a step exchanges only the tile's edge nodes with
// the four neighbours.  What still crosses HBM is the forward history (4 bytes per node and
// step, written once, read once).
//
// Exchange.  A neighbour's edge node travels as one 64-bit word {step tag, value} stored
// and polled with relaxed accesses: the tag arrives with the value in one atomic access, so
// no fence and no separate flag is on the path (one way 0.47 us measured between SMs;
// data + fence + flag: 1.2 us).  Four slots by tag: a CTA overwrites a slot only four steps
// later, after words that its readers sent when they were done with it (two steps
// suffice for direct neighbours, three for the corner node).
//
// Clusters.  A solve of at most 16 tiles can be one thread-block cluster: the words then go straight
// into the neighbours' shared memory and are polled there, without the way through L2, and no
// cooperative launch is needed (solves do not wait for one another).
//
// Threads.  A compute thread owns a column of elements, or of their halves: lane by lane the
// elements of a tile row, stepping down the element rows of its chunk.  All lines of an element
// are evaluated in registers; the carry into the element below stays in registers, the carry into
// the right neighbour goes by shuffle, and the first lane of a row is the left halo element,
// evaluated for its carry only.  A chunk starts with the z-lines of the element row above it, for
// their carry.  Nodes are advanced into the other of two buffers and each warp sends its own edge
// nodes, so a step needs one CTA barrier, when the halo words have arrived.  A few threads beyond
// the compute threads read out the receivers and form the adjoint source meanwhile.
//
// Large adjoint tiles (VG).  With displacement (two buffers), history (two), c^2, increment and
// partial gradient on chip an SM holds about 300 elements of order 4, so a 400x200 mesh's adjoint
// does not fit the GPU.  Increment and partial gradient are read and written once a step by the
// thread that owns them: kept in the solve's fields they cost 16 bytes a node and step of L2
// traffic, in flight during the x-lines, and 575 elements fit (forward + adjoint 15.7 us a step;
// strips 27.7).  Where the tiles fit anyway, keeping them on chip is as fast or faster.
//
// Arithmetic.  Per node the operations and roundings of the tile and strip kernels, in the
// same order: results are bitwise equal to theirs.

// most threads of a resident CTA, by order, lanes per element and kernel: up to 255 registers each
// with 256, 168 with 384, 128 with 512
__host__ __device__ constexpr int res_threads(int N, int lpe, bool adj) { return lpe == 2 ? 512 : adj || N > 4 ? 256 : 384; }
constexpr int kResSlots = 4;       // exchange slots by step tag

// Shared-memory layout (float offsets) and exchange layout (words) of one launch, by its
// largest tile; a kernel parameter, so every offset is a constant operand.
struct ResLay {
  int Wp, Cp;                    // pitches: haloed fields, owned fields
  int H;                         // rows of a haloed field (and of the history box)
  int reg;                       // floats of a haloed field
  int qx;                        // quads per owned row (injection map pitch)
  int w;                         // adjoint: forward-field tile, two buffers of wreg (128-byte aligned)
  int wreg;
  int b;                         // displacement (adjoint field): two buffers by step parity
  int c, v, g;                   // c^2, increment, partial gradient
  int tz;                        // row table: 1/m_z, 1/m_z, R_z, R_z, -d_z, -d_z, 0, 0
  int wi, wo;                    // exchange words received / sent: places
  int rs, ia, io, iq, ie, im;    // injection: residuals, node sums, term offsets, terms, weights, quad map
  int be, bd;                    // Stacey: edge coefficients, b_{t+2} - b_t
  int nrm, niq, Rm, Cm;          // most receivers and injection quads per tile, owned rows, columns
  int total;                     // floats
  int llw, ll_t, ll_r, ll_b, ll_c;  // exchange words per CTA and slot; offsets of the sides
  int sl;                        // clusters: the slots of arriving words; -1: they are in memory
};

enum : int { RES_FWD = 0, RES_REPLAY = 1, RES_ADJ = 2 };

__device__ __forceinline__ void ll_send(unsigned long long* p, float v, unsigned tag) {
  const unsigned long long q = ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(q) : "memory");
}
__device__ __forceinline__ unsigned long long ll_load(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// the same between the CTAs of a cluster: shared-memory address p of CTA `rank`, and of this CTA
__device__ __forceinline__ void ll_send_cluster(unsigned p, int rank, float v, unsigned tag) {
  const unsigned long long q = ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v);
  asm volatile("{ .reg .u32 a; mapa.shared::cluster.u32 a, %0, %1; st.relaxed.cluster.shared::cluster.u64 [a], %2; }"
               ::"r"(p), "r"(rank), "l"(q) : "memory");
}
__device__ __forceinline__ unsigned long long ll_load_shared(unsigned p) {
  unsigned long long v;
  asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"(p) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

// Exchange words' table entries.  In: place in this CTA's slot and region index.  Out: place among
// the words of the tile above on the left (and on from it) and region index.  Two ints; in the
// kernels that need the room one: 16 bits region index, two each dx + 1 and dz + 1 of the
// receiver's tile, 12 bits place in its slot (16 for arriving words).
__device__ __forceinline__ void word_in(int2& e, int place, int reg) { e = make_int2(place, reg); }
__device__ __forceinline__ void word_in(unsigned& e, int place, int reg) { e = (unsigned)place | (unsigned)reg << 16; }
__device__ __forceinline__ void word_out(int2& e, int place, int reg, int dx, int dz, int llc, int llr) {
  e = make_int2((dx + 1) * llc + (dz + 1) * llr + place, reg);
}
__device__ __forceinline__ void word_out(unsigned& e, int place, int reg, int dx, int dz, int, int) {
  e = (unsigned)(place | (dz + 1) << 12 | (dx + 1) << 14) | (unsigned)reg << 16;
}
__device__ __forceinline__ int word_reg(int2 e) { return e.y; }
__device__ __forceinline__ int word_reg(unsigned e) { return (int)(e >> 16); }
__device__ __forceinline__ int word_from(int2 e) { return e.x; }
__device__ __forceinline__ int word_from(unsigned e) { return (int)(e & 0xffff); }
__device__ __forceinline__ int word_to(int2 e, int, int) { return e.x; }
__device__ __forceinline__ int word_to(unsigned e, int llc, int llr) {
  return (int)(e >> 14 & 3) * llc + (int)(e >> 12 & 3) * llr + (int)(e & 0xfff);
}

__device__ __forceinline__ void res_barrier(int threads) {
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// N consecutive floats as pairs for packed arithmetic (N = 4: one 128-bit access; odd N: the
// last half is unused)
template <int N>
__device__ __forceinline__ void get2(const float* p, float2 (&u)[(N + 1) / 2]) {
  if constexpr (N == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    u[0] = make_float2(q.x, q.y);
    u[1] = make_float2(q.z, q.w);
  } else {
#pragma unroll
    for (int i = 0; i < (N + 1) / 2; ++i) u[i] = make_float2(p[2 * i], 2 * i + 1 < N ? p[2 * i + 1] : 0.f);
  }
}
template <int N>
__device__ __forceinline__ void put2(float* p, const float2 (&u)[(N + 1) / 2]) {
  if constexpr (N == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(u[0].x, u[0].y, u[1].x, u[1].y);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = (i & 1) ? u[i / 2].y : u[i / 2].x;
  }
}
template <int H>
__device__ __forceinline__ float lane_of(const float2 (&u)[H], int i) { return (i & 1) ? u[i / 2].y : u[i / 2].x; }

// the tile of this CTA
struct ResTile {
  int gx0, gz0;        // first owned node
  int EX, EZ, C, R;    // owned elements, columns and rows
  int off;             // region column of node gx0 - N
  int X0;              // node column of region column 0 (a multiple of 4)
  bool hl, hr, ht, hb; // neighbours
};
// first element of tile t of n over nel elements: the larger tiles come first, so the last tile,
// which owns the mesh's last line of nodes too, is never the largest of an uneven tiling
__host__ __device__ inline int res_start(int t, int nel, int n) { return (int)(((long long)t * nel + n - 1) / n); }

// Steps [t0, t1) of a launch for one solve: forward 0 .. nt - 1; replay and adjoint of the
// idx-th segment from the last.  Adjoint steps outside the misfit window are left out: above
// it1 the adjoint field is still zero, below it0 nothing is accumulated any more.
__host__ __device__ inline bool res_range(int kind, int idx, int nt, int k, int nseg, int it0, int it1,
                                          int& seg, int& t0, int& t1) {
  seg = nseg - 1 - idx;
  if (kind == RES_FWD) { t0 = 0; t1 = nt; return idx == 0; }
  if (seg < 0) return false;
  const int lo = seg * k > it0 ? seg * k : it0;
  int hi = (seg + 1) * k < nt ? (seg + 1) * k : nt;
  hi = hi < it1 ? hi : it1;
  if (lo >= hi) return false;
  t0 = kind == RES_REPLAY ? seg * k : lo;
  t1 = hi;
  return true;
}

// The z-lines of NQ pairs of an element's columns, a pair at a time as the halves of packed FFMA2 / FMUL2 (per
// half the scalar sequence), from its rows of nodes u (field), c (c^2) and, adjoint, w (forward
// field): segment results of row i in Z[i], sensitivities in S[i]; with CARRY only the last
// row's, for the element below.
template <int N, int NQ, bool ADJ, bool CARRY>
__device__ __forceinline__ void res_zlines(const float2 (&u)[N + 1][NQ], const float2 (&c)[N + 1][NQ],
                                           const float2 (&w)[N + 1][NQ], float2 (&Z)[N + 1][NQ],
                                           float2 (&S)[N + 1][NQ]) {
  constexpr int NP = N + 1;
#pragma unroll
  for (int p = 0; p < NQ; ++p) {
    // (the independent sums side by side, so that consecutive instructions do not wait)
    float2 d[NP], q[NP];
#pragma unroll
    for (int a = 0; a < NP; ++a) d[a] = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < NP; ++k)
#pragma unroll
      for (int a = 0; a < NP; ++a) d[a] = __ffma2_rn(c_D2[N][a * NP + k], u[k][p], d[a]);
#pragma unroll
    for (int a = 0; a < NP; ++a) q[a] = __fmul2_rn(c_B2[N][a], c[a][p]);
#pragma unroll
    for (int a = 0; a < NP; ++a) q[a] = __fmul2_rn(q[a], d[a]);
#pragma unroll
    for (int i = CARRY ? N : 0; i < NP; ++i) Z[i][p] = make_float2(0.f, 0.f);
#pragma unroll
    for (int a = 0; a < NP; ++a)
#pragma unroll
      for (int i = CARRY ? N : 0; i < NP; ++i) Z[i][p] = __ffma2_rn(c_D2[N][a * NP + i], q[a], Z[i][p]);
    if constexpr (ADJ) {
#pragma unroll
      for (int a = CARRY ? N : 0; a < NP; ++a) S[a][p] = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < NP; ++k)
#pragma unroll
        for (int a = CARRY ? N : 0; a < NP; ++a) S[a][p] = __ffma2_rn(c_D2[N][a * NP + k], w[k][p], S[a][p]);
#pragma unroll
      for (int a = CARRY ? N : 0; a < NP; ++a) S[a][p] = __fmul2_rn(__fmul2_rn(c_B2[N][a], S[a][p]), d[a]);
    }
  }
}

// One row's x-line segment from its N+1 nodes: results X (and sensitivity SX) of the element's
// own nodes, carries re (rs) into the next element's first column.
template <int N, bool ADJ>
__device__ __forceinline__ void res_xline(const float (&u)[N + 1], const float (&c)[N + 1], const float (&w)[N + 1],
                                          float2 (&X)[(N + 1) / 2], float2 (&SX)[(N + 1) / 2], float& re, float& rs) {
  constexpr int NP = N + 1, H2 = (N + 1) / 2;
  float q[NP], d[NP];
#pragma unroll
  for (int a = 0; a < NP; ++a) d[a] = 0.f;
#pragma unroll
  for (int k = 0; k < NP; ++k)
#pragma unroll
    for (int a = 0; a < NP; ++a) d[a] = fmaf(c_D[N][a * NP + k], u[k], d[a]);
#pragma unroll
  for (int a = 0; a < NP; ++a) q[a] = __fmul_rn(c_B[N][a], c[a]);
#pragma unroll
  for (int a = 0; a < NP; ++a) q[a] = __fmul_rn(q[a], d[a]);
  float r[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) r[i] = 0.f;
#pragma unroll
  for (int a = 0; a < NP; ++a)
#pragma unroll
    for (int i = 0; i < NP; ++i) r[i] = fmaf(c_D[N][a * NP + i], q[a], r[i]);
  re = r[N];
#pragma unroll
  for (int i = 0; i < H2; ++i) X[i] = make_float2(r[2 * i], 2 * i + 1 < N ? r[2 * i + 1] : 0.f);
  if constexpr (ADJ) {
#pragma unroll
    for (int a = 0; a < NP; ++a) r[a] = 0.f;
#pragma unroll
    for (int k = 0; k < NP; ++k)
#pragma unroll
      for (int a = 0; a < NP; ++a) r[a] = fmaf(c_D[N][a * NP + k], w[k], r[a]);
#pragma unroll
    for (int a = 0; a < NP; ++a) r[a] = sens_product(c_B[N][a], r[a], d[a]);
    rs = r[N];
#pragma unroll
    for (int i = 0; i < H2; ++i) SX[i] = make_float2(r[2 * i], 2 * i + 1 < N ? r[2 * i + 1] : 0.f);
  }
}

// CL: the solve's tiles are one cluster.  nc: compute threads (the first of the CTA); the rest serve the receivers.  sw: lanes per tile
// row (a power of two, at least the tile's columns of elements + 2: one for the left halo, one
// for the nodes on the right); ezc: element rows per chunk.
template <int N, int LPE, bool ADJ, bool STC, bool VG, bool CL>
__global__ void __launch_bounds__(res_threads(N, LPE, ADJ), 1)
    sem_resident_kernel(const SolveDev* __restrict__ solves, const int* __restrict__ cta_solve,
                        const __grid_constant__ ResLay L, unsigned long long* __restrict__ ll,
                        const unsigned tag0, const int kind, const int idx, const int nc, const int sw,
                        const int ezc) {
  constexpr int NP = N + 1, H2 = (N + 1) / 2;
  // two lanes per element (order 4): each has two columns' z-lines and two rows' x-lines and nodes
  static_assert(LPE == 1 || N == 4, "an element's halves");
  static_assert(!VG || (ADJ && LPE == 1), "large adjoint tiles");
  static_assert(!VG || !CL, "a cluster's tiles are small");  // (a switch at run time cost two lanes forward 4 %)
  constexpr int NJ = N / LPE, NQ = LPE == 2 ? 1 : H2;
  extern __shared__ __align__(128) float sm[];
  __shared__ SolveDev S;
  __shared__ int s_fail;
  __shared__ float s_src[2];  // the source term of this step and the next
  __shared__ double s_red[16];
  __shared__ int s_wo[18];
  __shared__ unsigned long long s_bar[2];
  const int tid = threadIdx.x, T = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = T >> 5;
  {
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(solves + cta_solve[blockIdx.x]);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(&S);
    for (int i = tid; i < (int)(sizeof(SolveDev) / 8); i += T) dst[i] = src[i];
  }
  if (tid == 0) s_fail = 0;
  if (ADJ && tid == 0) {
    mbar_init(s_bar, 1);
    mbar_init(s_bar + 1, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < L.total; i += T) sm[i] = 0.f;
  __syncthreads();
  int seg, t_lo, t_hi;
  if (kind != RES_FWD && !(S.flags & F_ADJ)) return;
  if (!res_range(kind, idx, S.nt, S.k, S.nseg, S.it0, S.it1, seg, t_lo, t_hi)) return;

  // ---------------- tile
  ResTile Q;
  const int lt = blockIdx.x - S.tile_base;
  {
    const int tx = lt % S.tiles_x, tz = lt / S.tiles_x;
    const int ex0 = res_start(tx, S.nelx, S.tiles_x), ex1 = res_start(tx + 1, S.nelx, S.tiles_x);
    const int ez0 = res_start(tz, S.nelz, S.tiles_z), ez1 = res_start(tz + 1, S.nelz, S.tiles_z);
    Q.EX = ex1 - ex0; Q.EZ = ez1 - ez0;
    Q.hl = ex0 > 0; Q.hr = ex1 < S.nelx; Q.ht = ez0 > 0; Q.hb = ez1 < S.nelz;
    Q.gx0 = ex0 * N; Q.gz0 = ez0 * N;
    Q.C = Q.EX * N + (Q.hr ? 0 : 1); Q.R = Q.EZ * N + (Q.hb ? 0 : 1);
    Q.X0 = (Q.gx0 - N) & ~3;
    Q.off = (Q.gx0 - N) - Q.X0;
  }
  const int off = Q.off;

  // ---------------- load the state (regions with their halo from the fields in memory)
  {
    const float* cur;
    const float* vin;
    if (ADJ) { cur = S.L + (long long)(t_hi & 1) * S.fstride; vin = S.Mu; }
    else if (kind == RES_FWD) { cur = fwd_b(S, 0); vin = fwd_v(S, 0); }
    else { cur = rep_b(S, seg, t_lo); vin = rep_v(S, seg, t_lo); }
    const int W = off + N + Q.C + (Q.hr ? 1 : 0), H = N + Q.R + (Q.hb ? 1 : 0);
    for (int i = tid; i < W * H; i += T) {
      const int r = i / W, cidx = i - r * W;
      const int gz = Q.gz0 - N + r, gx = Q.X0 + cidx;
      if (gz >= 0 && gx >= 0 && gz < S.nzg && gx < S.nxg) {
        const long long gi = (long long)gz * S.pitch + gx;
        sm[L.b + r * L.Wp + cidx] = cur[gi];
        sm[L.c + r * L.Wp + cidx] = S.c2[gi];
      }
    }
    for (int i = tid; i < Q.R * Q.C; i += T) {
      const int r = i / Q.C, cc = i - r * Q.C;
      const long long gi = (long long)(Q.gz0 + r) * S.pitch + Q.gx0 + cc;
      if (VG) break;
      sm[L.v + r * L.Cp + cc] = vin[gi];
      if (ADJ) sm[L.g + r * L.Cp + cc] = S.grad[gi];
    }
    for (int i = tid; i < Q.R; i += T)
      for (int q = 0; q < 3; ++q) {
        const float f = S.tz[q * S.nzg + Q.gz0 + i];
        sm[L.tz + 8 * i + 2 * q] = sm[L.tz + 8 * i + 2 * q + 1] = q < 2 ? f : -f;
      }
  }
  // ---------------- exchange words that arrive
  const unsigned slots = (unsigned)__cvta_generic_to_shared(sm + (CL ? L.sl : 0));
  typedef typename std::conditional<VG, unsigned, int2>::type Word;
  Word* const win = reinterpret_cast<Word*>(sm + L.wi);
  const int llc = kResSlots * L.llw, llr = llc * S.tiles_x;  // words of a tile, of a row of tiles
  const int nR = Q.R, nRN = Q.R * N, nC = Q.C, nCN = Q.C * N;
  const int n_in = (Q.hl ? nRN : 0) + (Q.ht ? nCN : 0) + (Q.hr ? nR : 0) + (Q.hb ? nC : 0) +
                   ((Q.hr && Q.hb && !ADJ) ? 1 : 0);
  const int o0 = N * L.Wp + off + N;  // region index of the first owned node
  {
    int n = 0;
    auto side = [&](bool has, int words, auto&& word) {
      if (!has) return;
      for (int w = tid; w < words; w += T) {
        const int2 e = word(w);
        word_in(win[n + w], e.x, e.y);
      }
      n += words;
    };
    side(Q.hl, nRN, [&](int w) { return make_int2(w, o0 + (w / N) * L.Wp - N + w % N); });
    side(Q.ht, nCN, [&](int w) { return make_int2(L.ll_t + (w / nC) * L.Cm + w % nC, o0 + (w / nC - N) * L.Wp + w % nC); });
    side(Q.hr, nR, [&](int w) { return make_int2(L.ll_r + w, o0 + w * L.Wp + Q.EX * N); });
    side(Q.hb, nC, [&](int w) { return make_int2(L.ll_b + w, o0 + nR * L.Wp + w); });
    side(Q.hr && Q.hb && !ADJ, 1, [&](int) { return make_int2(L.ll_c, o0 + nR * L.Wp + Q.EX * N); });
  }
  // and words that leave, by the warp that advances the node; s_wo: each warp's range
  Word* const wout = reinterpret_cast<Word*>(sm + L.wo);
  {
    const int n_r = Q.hr ? nRN : 0, n_b = Q.hb ? nCN : 0, n_l = Q.hl ? nR : 0, n_t = Q.ht ? nC : 0;
    const int n_out = n_r + n_b + n_l + n_t + ((Q.hl && Q.ht && !ADJ) ? 1 : 0);
    if (tid <= nw) s_wo[tid] = 0;
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
      for (int w = tid; w < n_out; w += T) {
        int q = w, r, cc, to, dx = 0, dz = 0;
        if (q < n_r) { r = q / N; cc = (Q.EX - 1) * N + q % N; to = q; dx = 1; }
        else if ((q -= n_r) < n_b) { r = nR - N + q / nC; cc = q % nC; to = L.ll_t + (q / nC) * L.Cm + cc; dz = 1; }
        else if ((q -= n_b) < n_l) { r = q; cc = 0; to = L.ll_r + q; dx = -1; }
        else if ((q -= n_l) < n_t) { r = 0; cc = q; to = L.ll_b + q; dz = -1; }
        else { r = 0; cc = 0; to = L.ll_c; dx = dz = -1; }
        const int wp = (((r / N) / ezc) * sw + (cc / N + 1) * LPE + (r % N) / NJ) >> 5;
        const int at = atomicAdd(&s_wo[pass ? wp : wp + 1], 1);
        if (pass) {
          if constexpr (CL)  // the receiver's rank and the place
            wout[at] = make_int2(to | (lt + dx + dz * S.tiles_x) << 16, o0 + r * L.Wp + cc);
          else
            word_out(wout[at], to, o0 + r * L.Wp + cc, dx, dz, llc, llr);
        }
      }
      __syncthreads();
      if (pass == 0 && tid == 0)
        for (int i = 0; i < nw; ++i) s_wo[i + 1] += s_wo[i];
      __syncthreads();
    }
    // the second pass left each warp's end where its start was
  }
  // Stacey edges of this tile: left column r, right column Rm + r, bottom row 2 Rm + c; rows
  // of the tables are 2 Rm + Cm floats (e1, e2, g)
  const int bn = 2 * L.Rm + L.Cm;
  auto edge_slot = [&](int k) -> int {  // the solve's boundary slot of local slot k, or -1
    if (k < L.Rm) return (!Q.hl && k < Q.R && Q.gz0 + k > 0) ? Q.gz0 + k : -1;
    if (k < 2 * L.Rm) return (!Q.hr && k - L.Rm < Q.R && Q.gz0 + k - L.Rm > 0) ? S.nzg + Q.gz0 + k - L.Rm : -1;
    const int c = k - 2 * L.Rm, gx = Q.gx0 + c;
    return (!Q.hb && c < Q.C && gx > 0 && gx < S.nxg - 1) ? 2 * S.nzg + gx : -1;
  };
  const bool stc_edge = STC && (!Q.hl || !Q.hr || !Q.hb);
  if (stc_edge)
    for (int k = tid; k < bn; k += T) {
      const int sl = edge_slot(k);
      for (int q = 0; q < 3; ++q)
        sm[L.be + q * bn + k] = sl >= 0 ? S.bnd_coef[(long long)q * S.bnd_pitch + sl] : (q < 2 ? 1.f : 0.f);
    }

  // ---------------- receivers: thread nc + q has the tile's receiver q
  const bool io = tid >= nc;
  const int it = tid - nc;
  const int loff = ADJ ? S.inj_tile_off[lt] : S.rec_tile_off[lt];
  const int cnt = (kind == RES_REPLAY) ? 0 : (ADJ ? S.inj_tile_off[lt + 1] : S.rec_tile_off[lt + 1]) - loff;
  const int my_r = (io && it < cnt) ? (ADJ ? S.inj_tile_ids : S.rec_tile_ids)[loff + it] : 0;
  const bool my_rec = io && it < cnt;
  const int shift = (S.flags & F_SHIFT) ? 1 : 0;
  const bool misfit_on = !ADJ && (S.flags & F_MISFIT);
  auto mis_tick = [&](int m) { return m >= S.it0 && m < S.it1 && (m - S.it0) % S.decim == 0; };
  auto y_at = [&](int m, int r) { return S.yobs[(long long)((m - S.it0) / S.decim) * S.nrec + r]; };
  int* const ioff = reinterpret_cast<int*>(sm + L.io);
  int* const s_iterm = reinterpret_cast<int*>(sm + L.iq);
  unsigned short* const imap = reinterpret_cast<unsigned short*>(sm + L.im);
  double ascale = 1.0;
  int niq = 0;               // injection: quads with receivers
  const int* iterm = nullptr;  // their terms and weights (VG: in memory, which leaves room for a larger tile)
  const float* iterm_w = nullptr;
  if (ADJ) {
    // the power of two that brings max|r| to ~1 (the tick kernels' scale tick)
    double m = 0.0;
    for (int r = tid; r < S.nrec; r += T) m = fmax(m, S.rmax[r]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) s_red[warp] = m;
    __syncthreads();
    for (int i = 0; i < nw; ++i) m = fmax(m, s_red[i]);
    ascale = (m > 0.0 && isfinite(m)) ? ldexp(1.0, -ilogb(m)) : 1.0;
    if (lt == 0 && tid == 0) *S.adj_scale = ascale;
    // injection lists of this tile: quads holding receiver nodes and their terms
    const int q0 = S.iq_off[lt];
    niq = S.iq_off[lt + 1] - q0;
    const int e0 = S.iterm_off[q0];
    for (int i = tid; i < niq; i += T) imap[(S.iq_pos[q0 + i] >> 16) * L.qx + (S.iq_pos[q0 + i] & 0xffff)] = i + 1;
    for (int i = tid; i <= niq; i += T) ioff[i] = S.iterm_off[q0 + i] - e0;
    const int ne = S.iterm_off[q0 + niq] - e0;
    iterm = S.iterm + e0;
    iterm_w = S.iterm_w + (long long)e0 * N;
    if (!VG) {
      for (int i = tid; i < ne; i += T) s_iterm[i] = iterm[i];
      for (int i = tid; i < ne * N; i += T) sm[L.ie + i] = iterm_w[i];
      iterm = s_iterm;
      iterm_w = sm + L.ie;
    }
  }
  auto residual = [&](int t) -> float {  // the adjoint source term of this thread's receiver at step t
    if (!mis_tick(t)) return 0.f;
    return (float)(((double)S.rec_out[(long long)t * S.nrec + my_r] - y_at(t, my_r)) * ascale);
  };
  // the tile's injection R^T r at step t, a quad per thread: per node the receivers' terms in their
  // order (a term: receiver and the mask of the nodes it reaches; residuals by t & 3)
  auto inject_sums = [&](int t, int first, int step) {
    const float* rs = sm + L.rs + (t & 3) * L.nrm;
    const bool on = mis_tick(t);
    for (int q = first; q < niq; q += step) {
      float acc[N];
#pragma unroll
      for (int i = 0; i < N; ++i) acc[i] = 0.f;
      if (on)
        for (int k = ioff[q]; k < ioff[q + 1]; ++k) {
          const int e = iterm[k];
          const float r = rs[e >> 8];
#pragma unroll
          for (int i = 0; i < N; ++i)
            if ((e >> i) & 1) acc[i] = __fmaf_rn(iterm_w[k * N + i], r, acc[i]);
        }
#pragma unroll
      for (int i = 0; i < N; ++i) sm[L.ia + (t & 1) * (L.niq * N) + q * N + i] = acc[i];
    }
  };
  // Stacey: b_{t+2} - b_t of the tile's edge nodes (the impedance term of step t), 4 at a time
  auto edge_diffs = [&](int t, int first, int step) {
    if (t > S.nt - 2) return;
    const float* const h2 = S.bnd_hist + (long long)(t + 2) * S.bnd_pitch;
    const float* const h0 = S.bnd_hist + (long long)t * S.bnd_pitch;
    for (int k0 = first; k0 < bn; k0 += 4 * step) {
      float a[4], c[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int sl = k0 + j * step < bn ? edge_slot(k0 + j * step) : -1;
        a[j] = sl >= 0 ? h2[sl] : 0.f;
        c[j] = sl >= 0 ? h0[sl] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (k0 + j * step < bn) sm[L.bd + (t & 1) * bn + k0 + j * step] = __fsub_rn(a[j], c[j]);
    }
  };
  if (ADJ) {
    if (my_rec) {
      sm[L.rs + ((t_hi - 1) & 3) * L.nrm + it] = residual(t_hi - 1);
      if (t_hi - 2 >= t_lo) sm[L.rs + ((t_hi - 2) & 3) * L.nrm + it] = residual(t_hi - 2);
    }
    __syncthreads();
    inject_sums(t_hi - 1, tid, T);
    if (stc_edge) edge_diffs(t_hi - 1, tid, T);
  }

  const int src_e = (S.src_gx - Q.gx0) / N;  // the source's quad, when this tile has it
  const int src_r = (!ADJ && S.src_gx >= Q.gx0 && S.src_gx < Q.gx0 + Q.C && S.src_gz >= Q.gz0 && S.src_gz < Q.gz0 + Q.R)
                        ? S.src_gz - Q.gz0 : -1;
  // the history box of step t's forward field (one tensor copy, two buffers by step parity)
  const int w_slot = (ADJ && tid == nc) ? (int)((S.ring - S.ws) / S.fstride) + 1 - seg * S.k : 0;
  auto fetch_w = [&](int t) {
    mbar_expect_tx(s_bar + (t & 1), (unsigned)(L.Wp * L.H) * 4u);
    tensor_load_3d(sm + L.w + (t & 1) * L.wreg, S.tmap, Q.X0, Q.gz0 - N, w_slot + t, s_bar + (t & 1));
  };
  if (src_r >= 0 && tid == 0) s_src[t_lo & 1] = S.src_term[t_lo];
  if (ADJ && tid == nc) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tile buffers were cleared above
    tensormap_acquire(S.tmap);
    fetch_w(t_hi - 1);
  }
  __syncthreads();
  if constexpr (CL) cluster_barrier();  // every CTA's slots are cleared before the first word is sent

  const bool fin = !ADJ && kind == RES_FWD && shift;  // one more read-out after the last step
  const int nst = t_hi - t_lo;                        // steps
  int n_fail = -1;
  const unsigned long long* const in0 = ll + (long long)blockIdx.x * llc;
  unsigned long long* const ll_out = ll + ((long long)blockIdx.x * llc - llc - llr);  // the tile above on the left
  // wait for the edge words of step n's field and put them into the halo (every thread takes part)
  auto receive = [&](const int n) {
    const unsigned tag = tag0 + (unsigned)n;
    const int so = (int)(tag & (kResSlots - 1)) * L.llw;
    float* const f = sm + L.b + (n & 1) * L.reg;
#pragma unroll 1
    for (int w0 = tid; w0 < n_in; w0 += 4 * T) {  // up to four words of a thread in flight
      Word e[4];
      unsigned long long v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) e[j] = win[w0 + j * T < n_in ? w0 + j * T : w0];
      long long since = 0;
      int spin = 0;
      for (;;) {
        bool ok = true;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j == 0 || w0 + j * T < n_in)
            v[j] = CL ? ll_load_shared(slots + 8u * (unsigned)(so + word_from(e[j]))) : ll_load(in0 + so + word_from(e[j]));
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j == 0 || w0 + j * T < n_in) ok &= (unsigned)(v[j] >> 32) == tag;
        if (ok) break;
        if ((++spin & 127) == 0) {
          const long long now = global_ns();
          if (spin == 128) since = now;
          if (now - since > kWaitNs || *(volatile int*)&s_fail) { s_fail = 1; break; }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j == 0 || w0 + j * T < n_in) f[word_reg(e[j])] = __uint_as_float((unsigned)v[j]);
    }
  };
  // ---------------- receiver threads' state
  const int rbase = my_rec && !ADJ ? L.b + (S.rec_base[2 * my_r + 1] - Q.gz0 + N) * L.Wp + S.rec_base[2 * my_r] - Q.X0 : 0;
  double mis = 0.0, rmx = 0.0, y_cur = 0.0;
  if (misfit_on && my_rec) {
    mis = S.misfit[my_r];
    rmx = S.rmax[my_r];
    if (mis_tick(-shift)) y_cur = y_at(-shift, my_r);
  }
  float rs_next = 0.f;
  if (ADJ && my_rec && nst > 2) rs_next = residual(t_hi - 3);

  // ---------------- compute threads: element column ec of the tile (the first of a row: the left
  // halo; after the last element: the nodes on its right, the mesh's last column or the right
  // neighbour's first)
  const int el = (tid & (sw - 1)) / LPE, h = tid % LPE, ch = tid / sw;
  const int ec = min(el - 1, Q.EX);             // lanes past that repeat it
  const bool full = el >= 1 && el <= Q.EX;
  const bool owner = full || (el == Q.EX + 1 && !Q.hr);
  const bool no_left = el == 1 && !Q.hl;
  const int EZ1 = Q.EZ + (Q.hb ? 0 : 1);        // rows of elements; the mesh's last line is one more
  const int er_lo = ch * ezc, er_hi = min(EZ1, er_lo + ezc);
  const bool damp = !STC && (!ADJ || (S.flags & F_EXACT));
  float2 nix[H2], Rx[H2], ndx[H2];  // -1/m_x, R_x, -d_x; 0 off the owned nodes, which keeps those at 0
  bool dxany = false;
#pragma unroll
  for (int i = 0; i < 2 * H2; ++i) {
    const int gx = Q.gx0 + ec * N + i;
    const bool in = i < N && (full || (owner && i == 0));
    const float a = in ? -S.tx[gx] : 0.f, r = in ? S.tx[S.nxg + gx] : 0.f, d = in && damp ? -S.tx[2 * S.nxg + gx] : 0.f;
    if (i & 1) { nix[i / 2].y = a; Rx[i / 2].y = r; ndx[i / 2].y = d; }
    else { nix[i / 2].x = a; Rx[i / 2].x = r; ndx[i / 2].x = d; }
    dxany |= d != 0.f;
  }
  const bool keep = (S.flags & F_ADJ) != 0;
  // where the forward's b goes: nowhere, a checkpoint (every k-th step) or the ring
  float* ring = nullptr;                                 // slot of step t + 1 in the ring
  int t_ring = 0x7fffffff, t_ck = 0x7fffffff, j_ck = 1;  // first t + 1 in the ring, next checkpoint
  if (!ADJ && keep) {
    const int k = S.k, r0 = kind == RES_REPLAY ? seg * k : (S.nseg - 1) * k;
    t_ring = max(r0, t_lo + 1);
    ring = S.ring + (long long)(t_ring - r0) * S.fstride;
    if (kind == RES_FWD && k < r0) t_ck = k;
  }
  const int src_i = (S.src_gx - Q.gx0) % N;
  const int pitch = S.pitch;
  // Stacey: local slot of this lane's first node of row 0 on an absorbing side, or -1
  const int side = !stc_edge ? -1 : (el == 1 && !Q.hl) ? 0 : (el == Q.EX + 1 && !Q.hr) ? L.Rm : -1;
  const int w_lo = warp > 0 ? s_wo[warp - 1] : 0, w_hi = s_wo[warp];  // exchange words this warp sends
  const int oc = N * L.Wp + off + N + ec * N;   // region offset of the column's first owned node

  // step n: forward t = t_lo + n, adjoint t = t_hi - 1 - n
  for (int n = 0; n < nst + (fin ? 1 : 0); ++n) {
    const int t = ADJ ? t_hi - 1 - n : t_lo + n;
    const bool more = n + 1 < nst;   // another step follows
    if (n > 0) receive(n);
    if (ADJ && !io)
      if (!mbar_wait(s_bar + (t & 1), (n >> 1) & 1)) s_fail = 1;
    res_barrier(T);  // the field of step n is complete; every thread is done with step n - 1
    if (s_fail) { n_fail = n; break; }
    if (io) {
      // ---- receivers; the next step's operands are in flight meanwhile
      if constexpr (!ADJ) {
        double y_next = 0.0;
        if (misfit_on && my_rec && mis_tick(t + 1 - shift)) y_next = y_at(t + 1 - shift, my_r);
        if (src_r >= 0 && it == 0 && t + 1 < t_hi) s_src[(t + 1) & 1] = S.src_term[t + 1];
        const int m = t - shift;
        if (my_rec && m >= 0) {
          const float v = rec_dot_tree<N>(S.rec_w + (long long)my_r * NP * NP, sm + rbase + (n & 1) * L.reg, L.Wp);
          S.rec_out[(long long)m * S.nrec + my_r] = v;
          if (misfit_on && mis_tick(m)) {
            const double res = (double)v - y_cur;
            mis = __dadd_rn(mis, __dmul_rn(res, res));
            rmx = fmax(rmx, fabs(res));
          }
        }
        y_cur = y_next;
      } else {
        if (more) {
          if (it == 0) fetch_w(t - 1);
          inject_sums(t - 1, it, T - nc);
          if (stc_edge) edge_diffs(t - 1, it, T - nc);
        }
        if (my_rec && n + 2 < nst) {
          sm[L.rs + ((t - 2) & 3) * L.nrm + it] = rs_next;
          if (n + 3 < nst) rs_next = residual(t - 3);
        }
      }
      continue;
    }
    if (n == nst) break;  // the last read-out
    float *bo = nullptr, *vo = nullptr;
    if constexpr (!ADJ) {
      if (t + 1 >= t_ring) {
        bo = ring;
        ring += S.fstride;
      } else if (t + 1 == t_ck) {
        bo = S.ckpt + (long long)(2 * j_ck) * S.fstride;
        vo = bo + S.fstride;
        ++j_ck;
        t_ck += S.k;
      }
    }
    const bool g_start = ADJ && grad_partial_starts(S, t);
    const bool g_fold = ADJ && grad_folds(S, t);
    const float* const fb = sm + L.b + (n & 1) * L.reg;        // the step's field
    float* const fn = sm + L.b + ((n + 1) & 1) * L.reg;        // and the next
    const float* const fw = sm + L.w + (t & 1) * L.wreg;

    // ---- down the chunk's element rows; the carry of the row above comes first.  The rows of
    // nodes stay in registers: an element's last row is the next one's first
    float2 u[NP][NQ], c[NP][NQ], w[NP][NQ];
    auto load = [&](const int a, const int o) {
      if constexpr (LPE == 2) {
        u[a][0] = *reinterpret_cast<const float2*>(fb + o);
        c[a][0] = *reinterpret_cast<const float2*>(sm + L.c + o);
        if (ADJ) w[a][0] = *reinterpret_cast<const float2*>(fw + o);
      } else {
        get2<N>(fb + o, u[a]);
        get2<N>(sm + L.c + o, c[a]);
        if (ADJ) get2<N>(fw + o, w[a]);
      }
    };
    const int oz = oc + (LPE == 2 ? 2 * h : 0);
    float2 zc[NQ], szc[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) { zc[i] = make_float2(0.f, 0.f); szc[i] = make_float2(0.f, 0.f); }
    {
      const int o = oz + min(er_lo, EZ1 - 1) * N * L.Wp;
      load(N, o);
      if (er_lo < er_hi && (er_lo > 0 || Q.ht)) {
        float2 Z[NP][NQ], SZ[NP][NQ];
#pragma unroll
        for (int a = 0; a < N; ++a) load(a, o + (a - N) * L.Wp);
        res_zlines<N, NQ, ADJ, true>(u, c, w, Z, SZ);
#pragma unroll
        for (int i = 0; i < NQ; ++i) { zc[i] = Z[N][i]; if (ADJ) szc[i] = SZ[N][i]; }
      }
    }
    // the next element's first node of a row is the next element's lane's
    auto beyond = [&](const float2 (&f)[H2]) { return __shfl_down_sync(0xffffffffu, f[0].x, LPE, sw); };
#pragma unroll 1
    for (int k = 0; k < ezc; ++k) {
      const int er = er_lo + k;
      // rows of lanes whose chunk has ended keep the warp's shuffles company
      const bool on = er < er_hi;
      if (!__any_sync(0xffffffffu, on)) break;
      const int e_ = min(er, EZ1 - 1), r0 = e_ * N + h * NJ;
      const bool vz = e_ == Q.EZ;  // the mesh's last line of nodes: one row, no lines below
#pragma unroll
      for (int i = 0; i < NQ; ++i) { u[0][i] = u[N][i]; c[0][i] = c[N][i]; if (ADJ) w[0][i] = w[N][i]; }
#pragma unroll
      for (int a = 1; a < NP; ++a) load(a, oz + (e_ * N + a) * L.Wp);
      // this lane's rows: N nodes each and the one beyond
      float2 xu[NJ][H2], xc[NJ][H2], xw[NJ][H2];
      float ux[NJ], cx[NJ], wx[NJ];
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        if constexpr (LPE == 2) {
          const int o = oc + (r0 + j) * L.Wp;
          get2<N>(fb + o, xu[j]);
          get2<N>(sm + L.c + o, xc[j]);
          if (ADJ) get2<N>(fw + o, xw[j]);
        } else {
#pragma unroll
          for (int i = 0; i < H2; ++i) { xu[j][i] = u[j][i]; xc[j][i] = c[j][i]; if (ADJ) xw[j][i] = w[j][i]; }
        }
        ux[j] = beyond(xu[j]);
        cx[j] = beyond(xc[j]);
        wx[j] = ADJ ? beyond(xw[j]) : 0.f;
      }
      float2 Z[NP][NQ], SZ[NP][NQ];
      res_zlines<N, NQ, ADJ, false>(u, c, w, Z, SZ);
#pragma unroll
      for (int i = 0; i < NQ; ++i) {
        Z[0][i] = vz ? zc[i] : __fadd2_rn(zc[i], Z[0][i]);
        zc[i] = Z[N][i];
        if (ADJ) {
          // scalar adds: a packed one is fused with the product before it
          SZ[0][i] = vz ? szc[i] : make_float2(__fadd_rn(szc[i].x, SZ[0][i].x), __fadd_rn(szc[i].y, SZ[0][i].y));
          szc[i] = SZ[N][i];
        }
      }
      // the z results of this lane's rows: two lanes per element swap the halves they have for each other
      float2 Zr[NJ][H2], SZr[NJ][H2];
      auto rows_of = [&](const float2 (&F)[NP][NQ], float2 (&R)[NJ][H2]) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          if constexpr (LPE == 2) {
            const float2 give = h ? F[j][0] : F[NJ + j][0], own = h ? F[NJ + j][0] : F[j][0];
            const float2 got = make_float2(__shfl_xor_sync(0xffffffffu, give.x, 1), __shfl_xor_sync(0xffffffffu, give.y, 1));
            R[j][0] = h ? got : own;
            R[j][H2 - 1] = h ? own : got;
          } else {
#pragma unroll
            for (int i = 0; i < H2; ++i) R[j][i] = F[j][i < NQ ? i : 0];
          }
        }
      };
      rows_of(Z, Zr);
      if (ADJ) rows_of(SZ, SZr);

      // ---- the element's rows of owned nodes: x-lines, then the update
      const int ri = oc + r0 * L.Wp, oi = r0 * L.Cp + ec * N;
      float2 X[NJ][H2], SX[NJ][H2];
      float re[NJ], rs[NJ];
      const bool mine = owner && on;
      float2 v[NJ][H2], g[NJ][H2];
      // a row of the increment or the partial gradient: in shared memory, or (VG) in the solve's fields
      auto vg_at = [&](int j, int o, float* f) { return VG ? f + (Q.gz0 + r0 + j) * pitch + Q.gx0 + ec * N : sm + o + oi + j * L.Cp; };
      auto vg_get = [&](float2 (&x)[NJ][H2], int o, float* f) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const float* const p = vg_at(j, o, f);
          if constexpr (!VG || N == 4) {
            if (!VG || (mine && (j == 0 || !vz))) get2<N>(p, x[j]);
          } else {
#pragma unroll
            for (int i = 0; i < N; ++i) {
              const float a = mine && (j == 0 || !vz) && (full || i == 0) ? p[i] : 0.f;
              if (i & 1) x[j][i / 2].y = a; else x[j][i / 2].x = a;
            }
          }
        }
      };
      auto vg_put = [&](float2 (&x)[NJ][H2], int o, float* f) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          float* const p = vg_at(j, o, f);
          if constexpr (!VG || N == 4) {
            if (!VG || j == 0 || !vz) put2<N>(p, x[j]);
          } else if (j == 0 || !vz) {
#pragma unroll
            for (int i = 0; i < N; ++i)
              if (full || i == 0) p[i] = lane_of(x[j], i);
          }
        }
      };
      if constexpr (VG) {  // (in flight during the x-lines)
        vg_get(v, L.v, S.Mu);
        vg_get(g, L.g, S.grad);
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        float lu[NP], lc[NP], lw[NP];
#pragma unroll
        for (int i = 0; i < N; ++i) { lu[i] = lane_of(xu[j], i); lc[i] = lane_of(xc[j], i); if (ADJ) lw[i] = lane_of(xw[j], i); }
        lu[N] = ux[j]; lc[N] = cx[j]; if (ADJ) lw[N] = wx[j];
        res_xline<N, ADJ>(lu, lc, lw, X[j], SX[j], re[j], rs[j]);
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        re[j] = __shfl_up_sync(0xffffffffu, re[j], LPE, sw);
        if (no_left) re[j] = 0.f;
        X[j][0].x = full ? __fadd_rn(re[j], X[j][0].x) : re[j];
        if (ADJ) {
          rs[j] = __shfl_up_sync(0xffffffffu, rs[j], LPE, sw);
          if (no_left) rs[j] = 0.f;
          SX[j][0].x = full ? __fadd_rn(rs[j], SX[j][0].x) : rs[j];
        }
      }
      // (nodes past the mesh's last line or column lie in this tile's arrays too and stay 0)
      float4 tz[NJ];   // 1/m_z and R_z, twice each
      float2 ndz[NJ];
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        tz[j] = *reinterpret_cast<const float4*>(sm + L.tz + 8 * (r0 + j));
        ndz[j] = *reinterpret_cast<const float2*>(sm + L.tz + 8 * (r0 + j) + 4);
      }
      if constexpr (ADJ) {
        if constexpr (!VG) vg_get(g, L.g, nullptr);
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int i = 0; i < H2; ++i)
            SX[j][i] = __ffma2_rn(make_float2(tz[j].z, tz[j].w), SX[j][i], __fmul2_rn(Rx[i], SZr[j][i]));  // sens_increment
        if (stc_edge && t <= S.nt - 2 && mine) {
          // g lambda (b_{t+2} - b_t) at the absorbing edges, rounded as bnd_sens
          auto sens = [&](int j, int i, int k) {
            float& f = (i & 1) ? SX[j][i / 2].y : SX[j][i / 2].x;
            f = __fadd_rn(f, __fmul_rn(__fmul_rn(sm[L.be + 2 * bn + k], lane_of(xu[j], i)), sm[L.bd + (t & 1) * bn + k]));
          };
#pragma unroll
          for (int j = 0; j < NJ; ++j)
            if (side >= 0 && r0 + j < Q.R && Q.gz0 + r0 + j > 0) sens(j, 0, side + r0 + j);
          if (vz && h == 0) {
#pragma unroll
            for (int i = 0; i < N; ++i)
              if (ec * N + i < Q.C && !(i == 0 && side >= 0)) sens(0, i, 2 * L.Rm + ec * N + i);
          }
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int i = 0; i < H2; ++i) g[j][i] = __fadd2_rn(g_start ? make_float2(0.f, 0.f) : g[j][i], SX[j][i]);
        if (mine) vg_put(g, L.g, S.grad);
      }
      if constexpr (!VG) vg_get(v, L.v, nullptr);
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < H2; ++i)
          X[j][i] = __ffma2_rn(make_float2(tz[j].z, tz[j].w), X[j][i], __fmul2_rn(Rx[i], Zr[j][i]));
      if (ADJ && niq > 0 && mine) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const int m = imap[(r0 + j) * L.qx + ec];
          if (m) {  // P (injection - K) + mu
            const float* ex = sm + L.ia + (t & 1) * (L.niq * N) + (m - 1) * N;
#pragma unroll
            for (int i = 0; i < N; ++i) {
              float& k = (i & 1) ? X[j][i / 2].y : X[j][i / 2].x;
              k = -__fsub_rn(ex[i], k);
            }
          }
        }
      }
      const bool here = !ADJ && src_r >= r0 && src_r < r0 + NJ && ec == src_e;  // the source's quad
      if constexpr (STC) {
        // as advance_node_stacey, two nodes at a time: w = v + F, and at the absorbing edges w = e1 v + e2 F
        const bool bottom = vz && h == 0 && mine && stc_edge, top = Q.gz0 + r0 == 0;
        const float* const be = sm + L.be;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const int ks = side >= 0 && mine && r0 + j < Q.R ? side + r0 + j : -1;
#pragma unroll
          for (int i = 0; i < H2; ++i) {
            const float2 np = __fmul2_rn(nix[i], make_float2(tz[j].x, tz[j].y));
            float2 f = ADJ ? __fmul2_rn(np, X[j][i]) : __ffma2_rn(np, X[j][i], make_float2(0.f, 0.f));
            if (here && r0 + j == src_r) {
              if (src_i == 2 * i) f.x = __fmaf_rn(np.x, X[j][i].x, s_src[t & 1]);
              if (src_i == 2 * i + 1) f.y = __fmaf_rn(np.y, X[j][i].y, s_src[t & 1]);
            }
            float2 w = make_float2(__fadd_rn(v[j][i].x, f.x), __fadd_rn(v[j][i].y, f.y));
            if (i == 0 && ks >= 0) w.x = __fmaf_rn(be[ks], v[j][i].x, __fmul_rn(be[bn + ks], f.x));
            if (j == 0 && bottom) {
              const int c0 = ec * N + 2 * i, k = 2 * L.Rm + c0;
              if (c0 < Q.C && !(i == 0 && side >= 0)) w.x = __fmaf_rn(be[k], v[j][i].x, __fmul_rn(be[bn + k], f.x));
              if (2 * i + 1 < N && c0 + 1 < Q.C) w.y = __fmaf_rn(be[k + 1], v[j][i].y, __fmul_rn(be[bn + k + 1], f.y));
            }
            if (j == 0 && top) w = make_float2(0.f, 0.f);
            X[j][i] = j == 0 && top ? w : __fadd2_rn(xu[j][i], w);
            v[j][i] = w;
          }
        }
        if (!ADJ && keep && stc_edge && mine) {
          float* const hist = S.bnd_hist + (long long)(t + 1) * S.bnd_pitch;
#pragma unroll
          for (int j = 0; j < NJ; ++j)
            if (side >= 0 && r0 + j < Q.R && Q.gz0 + r0 + j > 0) hist[(side ? S.nzg : 0) + Q.gz0 + r0 + j] = X[j][0].x;
          if (bottom) {
#pragma unroll
            for (int i = 0; i < N; ++i)
              if (ec * N + i < Q.C && !(i == 0 && side >= 0)) hist[2 * S.nzg + Q.gx0 + ec * N + i] = lane_of(X[0], i);
          }
        }
      } else {
        // as advance_node, two nodes at a time: w = v - P K (the products' signs are exact)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int i = 0; i < H2; ++i)
            v[j][i] = __ffma2_rn(__fmul2_rn(nix[i], make_float2(tz[j].x, tz[j].y)), X[j][i], v[j][i]);
        if (here) {
          const float s = s_src[t & 1];
#pragma unroll
          for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int i = 0; i < N; ++i)
              if (i == src_i && r0 + j == src_r) {
                if (i & 1) v[j][i / 2].y = __fadd_rn(v[j][i / 2].y, s); else v[j][i / 2].x = __fadd_rn(v[j][i / 2].x, s);
              }
        }
        bool dq = dxany;
#pragma unroll
        for (int j = 0; j < NJ; ++j) dq |= ndz[j].x != 0.f;
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int i = 0; i < H2; ++i) X[j][i] = __fadd2_rn(xu[j][i], v[j][i]);
        if (damp && dq) {
          // the sponge; elements outside it skip its operations (delta = 0 leaves w and s unchanged);
          // all signs turned: -delta = (-dx)(-dz) + ((-dx) + (-dz))
#pragma unroll
          for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int i = 0; i < H2; ++i) {
              const float2 nl = __ffma2_rn(ndx[i], ndz[j], __fadd2_rn(ndx[i], ndz[j]));
              v[j][i] = __ffma2_rn(nl, v[j][i], v[j][i]);
              X[j][i] = __ffma2_rn(nl, X[j][i], X[j][i]);
            }
        }
      }
      if (mine) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) put2<N>(fn + ri + j * L.Wp, X[j]);
        vg_put(v, L.v, S.Mu);
        if (!ADJ && bo) {
          float* const p = bo + (Q.gz0 + r0) * pitch + Q.gx0 + ec * N;
#pragma unroll
          for (int j = 0; j < NJ; ++j)
            if ((j == 0 && h == 0) || !vz) {
              if constexpr (N == 4) {  // (the row's padding takes the rest of the last node's quad)
                *reinterpret_cast<float4*>(p + j * pitch) = make_float4(X[j][0].x, X[j][0].y, X[j][H2 - 1].x, X[j][H2 - 1].y);
              } else {
#pragma unroll
                for (int i = 0; i < N; ++i)
                  if (full || i == 0) p[j * pitch + i] = lane_of(X[j], i);
              }
            }
        }
      }
    }
    // ---- the warp's edge nodes to the neighbours
    if (more || fin) {
      __syncwarp();
      const unsigned tag = tag0 + (unsigned)n + 1;
      unsigned long long* const p = ll_out + (int)(tag & (kResSlots - 1)) * L.llw;
      const float* const f = sm + L.b + ((n + 1) & 1) * L.reg;
#pragma unroll 1
      for (int w0 = w_lo + lane; w0 < w_hi; w0 += 128) {
        Word e[4];
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = wout[min(w0 + 32 * j, w_hi - 1)];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = f[word_reg(e[j])];
        if constexpr (CL) {
          const unsigned q = slots + 8u * ((tag & (kResSlots - 1)) * (unsigned)L.llw);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            ll_send_cluster(q + 8u * (unsigned)(word_from(e[j]) & 0xffff), word_from(e[j]) >> 16, v[j], tag);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)  // (past the end: the last word again)
            ll_send(p + word_to(e[j], llc, llr), v[j], tag);
        }
      }
    }
    // ---- now and then: v at a checkpoint, the gradient's partial sums into the float64 field (while
    // the words travel)
    if ((ADJ ? g_fold : vo != nullptr) && owner) {
#pragma unroll 1
      for (int q = er_lo * NJ; q < er_hi * NJ; ++q) {
        const int r = q / NJ * N + h * NJ + q % NJ;
        if (r >= Q.R) break;
        const int gi = (Q.gz0 + r) * pitch + Q.gx0 + ec * N, oi = r * L.Cp + ec * N;
        if (!ADJ) {
#pragma unroll 1
          for (int i = 0; i < (full ? N : 1); ++i) vo[gi + i] = sm[L.v + oi + i];
        } else {
          double a[N];
#pragma unroll
          for (int i = 0; i < N; ++i) a[i] = (full || i == 0) ? S.grad64[gi + i] : 0.0;
#pragma unroll
          for (int i = 0; i < N; ++i)
            if (full || i == 0) S.grad64[gi + i] = __dadd_rn(a[i], (double)(VG ? S.grad[gi + i] : sm[L.g + oi + i]));
        }
      }
    }
  }
  if constexpr (CL) cluster_barrier();  // no CTA leaves while a neighbour may still write to its slots
  if (misfit_on && my_rec && n_fail < 0) {
    S.misfit[my_r] = mis;
    S.rmax[my_r] = rmx;
  }
  if (n_fail >= 0) {
    if (tid == nc) {
      if (ADJ) mbar_wait(s_bar + ((t_hi - 1 - n_fail) & 1), (n_fail >> 1) & 1);  // the copy in flight lands first (bounded)
      atomicOr(S.status, SEM_ERR_TIMEOUT);
    }
    return;
  }
  __syncthreads();
  // ---------------- what the next launch reads, and the status
  bool bad = false;
  const bool more = ADJ && seg > 0 && t_lo == seg * S.k && t_lo > S.it0;  // another segment follows
  for (int i = tid; i < Q.R * Q.C; i += T) {
    const int r = i / Q.C, cc = i - r * Q.C;
    const float f = sm[L.b + (nst & 1) * L.reg + (N + r) * L.Wp + off + N + cc];
    bad |= !isfinite(f);  // a field that became non-finite stays so (b' = b + w)
    if (more) {
      const long long gi = (long long)(Q.gz0 + r) * S.pitch + Q.gx0 + cc;
      S.L[(long long)(t_lo & 1) * S.fstride + gi] = f;
      if (VG) continue;
      S.Mu[gi] = sm[L.v + r * L.Cp + cc];
      S.grad[gi] = sm[L.g + r * L.Cp + cc];
    }
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(S.status, SEM_ERR_NONFINITE);
}
