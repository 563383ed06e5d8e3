// LU-SGS sweep as a wavefront of warps (the default sweep).
//
// The (j,k) lines of a block are cut into tiles of 8 x 4 lines; one warp owns
// a tile, one lane a line, and a CTA owns FWJ x FWK tiles.  At step s lane
// (lj, lk) handles the cell I = s - lj - lk + 1 of its line, so the j and k
// neighbours' products are the ones other lanes of the CTA made in the step
// before: they pass through shared memory, one CTA barrier a step.  As in the
// reference (PREDGS imps4.f:345 / CORRGS imps4.f:76) every solved cell makes
// the split-Jacobian products for its three downstream neighbours; the
// triangular system is the reference's, so the result equals its slab order
// up to rounding.
//
// What bounds it.  A sweep is a serial chain of IMAX + JMAX + KMAX planes.
// One cluster with a barrier per plane took 2.3 us a plane, nearly all of it
// the cluster barrier.  Here nothing waits for a whole plane: a CTA starts as
// soon as its two upstream CTAs have passed its first cells and then runs at
// their pace.  A step of the chain is a warp's instructions for one cell a
// lane and a CTA barrier, 0.25 us in FP64 (a dependent multiply-add alone is
// ~25 cycles) and 0.21 us in FP32, and each CTA on the way adds the lag of its
// edge words, ~3 us.  The CTA's shape weighs the two: with 8 x 4 lines the
// lags cost more, with 16 x 8 lines the step, whose four warps then share the
// shared memory's bandwidth (one sweep of a 128x64x64 block with seven
// equations, FP64: 8 x 4 0.129 ms, 8 x 8 0.114 ms, 16 x 4 0.150 ms, 16 x 8
// 0.134 ms).  Loading the next record into registers a step ahead made the
// step longer (0.156 ms at 16 x 8), as did a step barrier split into arrival
// and wait on an mbarrier.  One sweep, B200: 128x64x64 cells, seven equations,
// 0.118 ms in FP64 and 0.103 ms in FP32 (cluster lines 0.588 ms); 64x32x32,
// five equations, 0.047 ms (0.223 ms); 248x136x72, seven, 0.251 ms (the mean of
// a hundred in a row; the shapes above were timed in one run of their own).
//
// Between CTAs the products of the edge lines go through global memory (L2)
// and carry their own arrival: every word of the edge buffer holds a mark (all
// bits set, no result of an arithmetic instruction; a value with that pattern
// is published as another NaN) until its value is stored, and the consumer
// writes the mark back once it has read the value.  No flags, no fences: a
// fence would put an L2 round trip into every step.  The words of a step are
// requested FPF steps before they are needed, so that the round trip is
// hidden once a CTA trails its upstream CTAs by that much.
//
// CTA tiles are taken from a counter in the order of their anti-diagonals, so
// a CTA only ever waits for tiles that other CTAs already hold: no
// co-residency is needed and any number of blocks' sweeps may run side by
// side.  Every wait is bounded; on time-out the error word is set, the tile
// finishes without waiting or starting copies, and waits once more, again
// with a bound, for the copies it has in flight.
//
// The cells' data is stored in the order of use: per tile and step one
// contiguous record of FlowRec<NV>::N rows of 32 values (a value of the 32
// lanes), fetched by one bulk copy per tile and step into a ring of FD slots.
// A record holds the right-hand side (replaced by the result), the
// state-dependent coefficients (k_flow_coef) and the face normals
// (k_flow_static).  Slots without a cell are zero and stay zero, so that
// every product a line starts from is zero without a test.
#pragma once

constexpr int FTJ = 8, FTK = 4;     // lines of a warp tile along j and k (32 lanes)
constexpr int FWJ = 1, FWK = 2;     // warp tiles of a CTA along j and k
constexpr int FW = FWJ * FWK, FBJ = FTJ * FWJ, FBK = FTK * FWK;   // its warps, its lines along j and k
constexpr int FIO = 64;             // threads that fetch, and that publish, the edge words
constexpr int FTHREADS = FW * 32 + 2 * FIO;
constexpr int FD = 6;               // ring slots: up to FD - 1 steps of record copies in flight
constexpr int FPF = 2;              // steps between an edge request and its use
constexpr int kFlowSpins = 1 << 22; // reads of a missing edge word before its wait gives up (seconds); records: 4 times
constexpr long kFlowDrain = 1L << 24;   // tries of the last wait for a CTA's copies after a time-out
constexpr int FHS = FW * 32 + (FBJ > FBK ? FBJ : FBK);   // products of one value: the CTA's lines + the incoming edge

// Rows of a record.  Solve: x = AL * rhs + B1 * yi + B2 * yj + B3 * yk, the
// pressure increment times SP.
//
// The product of a cell in direction d is SYM1I(diag(l1, l2, l1, l1, l5) *
// SYI(x)) with l1 = (rl -+ rmax)/2 -+ t, l2 = l1 + c/2, l5 = l1 - c/2 (rmax =
// |rl| + c is the same for all three waves, imps4.f:388-470), so the
// characteristic form collapses: with z = n . (x1, x2, x3)
//   out0 = l1 x0 + c^2/2 z,  out1..3 = l1 x1..3 + n x4 / (2 ro),
//   out4 = l1 x4 + ro c^2/2 z,  out5, 6 = l1 x5, 6
// and with k and omega the pressure row of SYM1KE, ydrp (out4 - drh ro out0 -
// .667 ro out5), is l1 w + K4 z with w = Y x4 - H3 x5 - H2 x0 taken once per
// cell.  15 multiply-adds a direction in place of 25, and 6 dependent ones in
// place of 13 from a neighbour's product to the cell's own: the step's chain.
template <int NV>
struct FlowRec {
  static constexpr int RHS = 0, AL = NV, B = NV + 1, SP = NV + 4, L = NV + 5, K0 = NV + 8, HR = NV + 9, K4 = NV + 10,
                       Y = NV + 11, H3 = NV + 12, H2 = NV + 13, F = NV == 7 ? NV + 14 : NV + 11, N = F + 9;
  static constexpr int EV = NV * (FBJ + FBK);   // edge words of a CTA and step: j edge (FBK lines), k edge (FBJ)
};

struct FlowGeom {
  int ntj, ntk, ntiles, ns;   // warp tiles along j and k, steps of a tile
  int nbj, nbk, nb, nbs;      // CTA tiles along j and k, steps of a CTA
};

__host__ __device__ inline FlowGeom flow_geom(int imax, int jmax, int kmax) {
  FlowGeom g;
  g.ntj = (jmax + FTJ - 1) / FTJ;
  g.ntk = (kmax + FTK - 1) / FTK;
  g.ntiles = g.ntj * g.ntk;
  g.ns = imax + FTJ + FTK - 2;
  g.nbj = (g.ntj + FWJ - 1) / FWJ;
  g.nbk = (g.ntk + FWK - 1) / FWK;
  g.nb = g.nbj * g.nbk;
  g.nbs = imax + FBJ + FBK - 2;
  return g;
}
inline size_t flow_rec_len(const FlowGeom& g, int nv) {
  return (size_t)g.ntiles * g.ns * (nv == 7 ? FlowRec<7>::N : FlowRec<5>::N) * 32;
}
inline size_t flow_edge_len(const FlowGeom& g, int nv) { return (size_t)g.nb * g.nbs * nv * (FBJ + FBK); }
__host__ __device__ constexpr size_t flow_smem_bytes(int nv, size_t elem) {
  return elem * ((size_t)FD * FW * (nv == 7 ? FlowRec<7>::N : FlowRec<5>::N) * 32 + 4 * (size_t)nv * FHS) + FD * 8;
}

// Slot -> cell: slot n = (tile * ns + s) * 32 + lane; false where the slot has none.
FF_DI bool flow_cell(const DevBlock& b, const FlowGeom& g, size_t n, int& I, int& J, int& K) {
  const int lane = (int)(n & 31);
  const unsigned r = (unsigned)(n >> 5), tile = r / (unsigned)g.ns, s = r - tile * g.ns;
  const int lj = lane % FTJ, lk = lane / FTJ;
  const unsigned tk = tile / (unsigned)g.ntj, tj = tile - tk * g.ntj;
  I = (int)s - lj - lk + 1;
  J = tj * FTJ + lj + 1;
  K = tk * FTK + lk + 1;
  return I >= 1 && I <= b.imax && J <= b.jmax && K <= b.kmax;
}

// The face normals of both sweeps' records: the products of the upper sweep
// (i+1 -> i) cross the cell's low faces, the lower sweep's its high faces.
// Metrics only, written once per block.
template <typename CT, int NV>
__global__ void k_flow_static(DevBlock b, FlowGeom g, CT* __restrict__ up, CT* __restrict__ lo) {
  using R = FlowRec<NV>;
  const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  int I, J, K;
  if (n >= (size_t)g.ntiles * g.ns * 32 || !flow_cell(b, g, n, I, J, K)) return;
  const size_t N = ix(b, I, J, K), o = (n >> 5) * (R::N * 32) + (n & 31);
  const int st[3] = {1, b.is, b.il};
#pragma unroll
  for (int d = 0; d < 3; d++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double* a = b.a[FF_A1XA + 4 * d + c];
      up[o + (R::F + 3 * d + c) * 32] = (CT)__ldg(a + N);
      lo[o + (R::F + 3 * d + c) * 32] = (CT)__ldg(a + N + st[d]);
    }
}

// TIME3, LOCDT and COPR (LOCDTK, IMSOKO, COPRKE), the state-dependent rows of
// both sweeps' records and the right-hand side of the upper sweep's (PREDGS
// imps4.f:388-470, DIAGGS 604-660, CORRGS 120-200): one pass over the state
// for both sweeps, whose diagonal factor needs the low and the high faces
// anyway.  Also rewinds the tile counters.
//
// A warp is 8 consecutive cells of 4 lines that are neighbours in j: a load is
// four runs of 64 bytes, and of a record's row, which holds the lines' cells
// of one diagonal, the four lanes of a diagonal of the warp write one sector.
// With one thread a slot, in record order, stores were whole lines but each
// load touched 32 sectors; turning the values in shared memory instead cost
// the occupancy that the chains of divisions need (128x64x64 cells, seven
// equations: 142 us in three passes with the time step and the conversion on
// their own, 165 us through shared memory, 104 us now).  Reciprocals are
// rcp's where the divisor cannot be zero or infinite.
template <typename CT, int NV>
__global__ void __launch_bounds__(256, 4) k_flow_coef(DevBlock b, ff_params p, ff::TimeConst tc, FlowGeom g, CT* __restrict__ up,
                                                   CT* __restrict__ lo, unsigned* ticket) {
  using R = FlowRec<NV>;
  if (blockIdx.x == 0 && threadIdx.x < 2) ticket[threadIdx.x] = 0u;
  const int nch = (b.imax + 7) / 8;
  const int tile = blockIdx.x / nch, i0 = (blockIdx.x - tile * nch) * 8;
  const int tk = tile / g.ntj, tj = tile - tk * g.ntj;
  const int line = threadIdx.x / 8, lj = line % FTJ, lk = line / FTJ, I = i0 + threadIdx.x % 8 + 1;
  const int J = tj * FTJ + lj + 1, K = tk * FTK + lk + 1;
  if (I > b.imax || J > b.jmax || K > b.kmax) return;
  const size_t N = ix(b, I, J, K), rec = ((size_t)tile * g.ns + I - 1 + lj + lk) * (R::N * 32) + line;
  CT *o = up + rec, *ol = lo + rec;
#define LD(s, m) __ldg(b.a[s] + (m))
  const double dtl = ff::time3_cell(b, p, tc, I, J, K, N), dt1 = p.theta * dtl;
  double x[NV];
  if constexpr (NV == 7) ff::coprke_cell(b, p, dtl, N, x);
  else ff::copr_cell(b, dtl, N, x);
#pragma unroll
  for (int q = 0; q < NV; q++) o[q * 32] = (CT)x[q];
  const double u = LD(FF_U, N), v = LD(FF_V, N), w = LD(FF_W, N), c = LD(FF_C, N), ro = LD(FF_RO, N);
  const double vol = LD(FF_VOL, N), mu = LD(FF_VIST, N) + LD(FF_VIS, N);
  const int st[3] = {1, b.is, b.il}, idi[3] = {p.idi1, p.idi2, p.idi3}, idx[3] = {I, J, K};
  double alo[3], ahi[3], su = 0., sl = 0., pu = 0., pl = 0., sd = 0.;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int ao = 4 * d;
    const size_t hi = N + st[d], lw = N - st[d];
    alo[d] = LD(FF_A1 + ao, N);
    ahi[d] = LD(FF_A1 + ao, hi);
    const double rlo = LD(FF_A1XA + ao, N) * u + LD(FF_A1YA + ao, N) * v + LD(FF_A1ZA + ao, N) * w;
    const double rhi = LD(FF_A1XA + ao, hi) * u + LD(FF_A1YA + ao, hi) * v + LD(FF_A1ZA + ao, hi) * w;
    double tu = 0., tl = 0.;
    if (idx[d] <= idi[d]) {
      tu = (idx[d] == 1 ? 8. : 4.) * alo[d] * rcp((vol + LD(FF_VOL, lw)) * (ro + LD(FF_RO, lw))) *
           (mu + LD(FF_VIST, lw) + LD(FF_VIS, lw));
      tl = 4. * alo[d] * rcp((vol + LD(FF_VOL, hi)) * (ro + LD(FF_RO, hi))) * (mu + LD(FF_VIST, hi) + LD(FF_VIS, hi));
    }
    const double rmu = fabs(rlo) + c, rml = fabs(rhi) + c;
    o[(R::L + d) * 32] = (CT)(dmin(rlo, 0.) - tu - .5 * c);
    ol[(R::L + d) * 32] = (CT)(dmax(rhi, 0.) + tl + .5 * c);
    su += (rmu + tu) * alo[d];
    sl += (rml + tl) * ahi[d];
    pu += rmu * alo[d];
    pl += rml * alo[d];
    sd += alo[d] * rmu + ahi[d] * rml;
  }
  const double du = vol + dt1 * su, dl = vol + dt1 * sl, scu = rcp(du), scl = rcp(dl);
  const double fd = 1. + dt1 * rcp(vol) * (.5 * sd);
  o[R::AL * 32] = (CT)(vol * scu);
  ol[R::AL * 32] = (CT)(vol * fd * scl);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    o[(R::B + d) * 32] = (CT)(-(dt1 * ahi[d]) * scu);
    ol[(R::B + d) * 32] = (CT)((dt1 * alo[d]) * scl);
  }
  o[R::SP * 32] = (CT)(du * rcp(vol + dt1 * pu));
  ol[R::SP * 32] = (CT)(dl * rcp(vol + dt1 * pl));
  auto both = [&](int row, double val) { o[row * 32] = ol[row * 32] = (CT)val; };
  const double k0 = .5 * (c * c), ypro = rcp(ro);
  both(R::K0, k0);
  both(R::HR, .5 * ypro);
  if constexpr (NV == 7) {
    const double rk = LD(FF_RK, N);
    const double ydrp = rcp(1. + .667 * rk * ypro * LD(FF_DRDP, N));
    const double h2 = ydrp * (.667 * rk * (ypro * ypro) * LD(FF_DRDH, N)) * ro;
    both(R::K4, ydrp * (ro * k0) - h2 * k0);
    both(R::Y, ydrp);
    both(R::H3, .667 * ro * ydrp);
    both(R::H2, h2);
  } else {
    both(R::K4, ro * k0);
  }
#undef LD
  b.a[FF_DTL][N] = dtl;
}

// The lower sweep's results from its records into DRO..DE(,DRK,DEPS): 32 cells
// of a tile's 32 lines a thread block, record rows in, runs along the lines out
// (128x64x64 cells, seven equations: 35 us with one thread a slot, 19 us).
constexpr int FOP = 36;   // shared-memory pitch of a line: a record row's lanes fall on different banks
template <typename CT, int NV>
__global__ void __launch_bounds__(256) k_flow_out(DevBlock b, FlowGeom g, const CT* __restrict__ lo) {
  using R = FlowRec<NV>;
  extern __shared__ __align__(128) unsigned char flow_smem[];
  CT* sv = reinterpret_cast<CT*>(flow_smem);   // [NV][32 lines][FOP]
  const int nch = (b.imax + 31) / 32;
  const int tile = blockIdx.x / nch, i0 = (blockIdx.x - tile * nch) * 32;
  const int tk = tile / g.ntj, tj = tile - tk * g.ntj;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NR = 32 + FTJ + FTK - 2;
  for (int r = warp; r < NR; r += 8) {
    const int i = r - lane % FTJ - lane / FTJ;
    if (i < 0 || i >= 32 || i0 + i >= b.imax) continue;
    const CT* row = lo + ((size_t)tile * g.ns + i0 + r) * (R::N * 32) + lane;
#pragma unroll
    for (int v = 0; v < NV; v++) sv[(v * 32 + lane) * FOP + i] = row[v * 32];
  }
  __syncthreads();
  if (i0 + lane >= b.imax) return;
  for (int l = warp; l < 32; l += 8) {
    const int J = tj * FTJ + l % FTJ + 1, K = tk * FTK + l / FTJ + 1;
    if (J > b.jmax || K > b.kmax) continue;
    const size_t N = ix(b, i0 + lane + 1, J, K);
#pragma unroll
    for (int v = 0; v < NV; v++) b.a[FF_DRO + v][N] = (double)sv[(v * 32 + l) * FOP + lane];
  }
}

// ---- edge words -------------------------------------------------------------
FF_DI double flow_ld(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
FF_DI float flow_ld(const float* p) {
  float v;
  asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
FF_DI void flow_st(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
FF_DI void flow_st(float* p, float v) {
  asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
FF_DI bool flow_mark(double v) { return __double_as_longlong(v) == -1LL; }
FF_DI bool flow_mark(float v) { return __float_as_int(v) == -1; }
FF_DI double flow_mark_of(double) { return __longlong_as_double(-1LL); }
FF_DI float flow_mark_of(float) { return __int_as_float(-1); }
// a value to publish: never the mark
FF_DI double flow_pub(double v) { return flow_mark(v) ? __longlong_as_double(0x7ff8000000000000LL) : v; }
FF_DI float flow_pub(float v) { return flow_mark(v) ? __int_as_float(0x7fc00000) : v; }

FF_DI void flow_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
FF_DI void flow_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// One sweep.  rec: this sweep's records; res: where row q of a slot's result
// goes, at the same slot and row (the lower sweep's records for the upper
// sweep, its own for the lower one).  grid = CTA tiles.  The first FW warps
// compute and do nothing else: with one warp doing everything its own
// instruction stream was the chain, 0.55 us a step.  The next FIO threads
// fetch the incoming edge words and wait for the records, one step ahead; the
// last FIO publish the outgoing edge words of the step before and start the
// record copies.
//
// HASTE: the same kernel with no patience (ff_sweep_haste): the CTAs that take
// an even ticket give up on their first record, every CTA on the first edge
// word that is not there yet.  A template parameter, because the limit as an
// argument cost the poll a register and the sweep 1 % (248x136x72 cells, seven
// equations: 254 -> 257 us).
template <typename CT, int NV, bool UP, bool HASTE>
__global__ void __launch_bounds__(FTHREADS) k_flow_sweep(const CT* rec, CT* res, CT* edge, FlowGeom g, int imax,
                                                         int jmax, int kmax, int drop, unsigned* ticket, int* err) {
  using R = FlowRec<NV>;
  constexpr int ROW = R::N * 32, EV = R::EV, NQ = (EV + FIO - 1) / FIO, PB = NV * FHS, NEVER = 1 << 28;
  constexpr uint32_t RB = ROW * sizeof(CT);
  extern __shared__ __align__(128) unsigned char flow_smem[];
  CT* ring = reinterpret_cast<CT*>(flow_smem);   // [FD][FW][N][32]
  CT* pj = ring + FD * FW * ROW;                 // [2][NV][FHS] products for the j neighbours
  CT* pk = pj + 2 * PB;                          // and for the k neighbours
  uint64_t* bars = reinterpret_cast<uint64_t*>(pk + 2 * PB);
  __shared__ int s_tile;
  __shared__ volatile int s_stop;   // 1 + the step whose record did not come: no record is waited for or copied any more
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t bar0 = pipe_smem_u32(bars), ring0 = pipe_smem_u32(ring);
  // the next CTA tile, in the order of the anti-diagonals (the counter wraps to 0 after the last one)
  if (threadIdx.x == 0) {
    s_tile = (int)atomicInc(ticket, (unsigned)g.nb - 1u);
    s_stop = 0;
    for (int q = 0; q < FD; q++) pipe_mbar_init(bar0 + 8 * q, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  for (int q = threadIdx.x; q < 4 * PB; q += FTHREADS) pj[q] = CT(0);
  __syncthreads();
  int t0 = s_tile, tj = 0, tk = 0;
  for (int d = 0;; d++) {
    const int k0 = max(0, d - g.nbj + 1), cnt = min(d, g.nbk - 1) - k0 + 1;
    if (t0 < cnt) { tk = k0 + t0; tj = d - tk; break; }
    t0 -= cnt;
  }
  // progress order: the lower sweep walks i, j, k upwards, the upper one downwards (tiles, lines and steps mirrored)
  const bool up_j = tj > 0, up_k = tk > 0, dn_j = tj < g.nbj - 1, dn_k = tk < g.nbk - 1;
  if (UP) { tj = g.nbj - 1 - tj; tk = g.nbk - 1 - tk; }
  const int tile = tk * g.nbj + tj, ns = g.ns, nbs = g.nbs;
  constexpr int sg = UP ? -1 : 1;
  const int s0 = UP ? nbs - 1 : 0;   // the CTA's first step in the edge buffer
  // warp tile w of the CTA: its number in the block (-1: outside) and the CTA step it starts at
  auto wtile = [&](int w, int& off) {
    const int wj = w % FWJ, wk = w / FWJ, bj = tj * FWJ + wj, bk = tk * FWK + wk;
    off = (UP ? FWJ - 1 - wj : wj) * FTJ + (UP ? FWK - 1 - wk : wk) * FTK;
    return bj < g.ntj && bk < g.ntk ? bk * g.ntj + bj : -1;
  };

  if (warp < FW) {
    // ---- solve and products ----
    int off;
    const int wt = wtile(warp, off);
    const int cj = (warp % FWJ) * FTJ + lane % FTJ, ck = (warp / FWJ) * FTK + lane / FTJ;   // line in the CTA tile
    const int mj = UP ? FBJ - 1 - cj : cj, mk = UP ? FBK - 1 - ck : ck;                     // mirrored
    const int J = tj * FBJ + cj + 1, K = tk * FBK + ck + 1;
    const bool line = J <= jmax && K <= kmax, any_drop = NV == 5 && UP && drop && (tj + 1) * FBJ >= jmax;
    auto place = [](int j, int k) { return ((k / FTK) * FWJ + j / FTJ) * 32 + (k % FTK) * FTJ + j % FTJ; };
    const CT* qj = pj + (mj == 0 ? FW * 32 + ck : place(cj - sg, ck));
    const CT* qk = pk + (mk == 0 ? FW * 32 + cj : place(cj, ck - sg));
    CT* nj = pj + warp * 32 + lane;
    CT* nk = pk + warp * 32 + lane;
    CT* o = res + ((size_t)max(wt, 0) * ns + (UP ? ns - 1 : 0)) * ROW + lane;
    CT yi[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) yi[v] = CT(0);
    __syncthreads();   // the record and the incoming words of step 0
    for (int T = 0; T < nbs; T++) {
      if (wt >= 0 && (unsigned)(T - off) < (unsigned)ns) {
        const CT* my = ring + ((T % FD) * FW + warp) * ROW + lane;
        const int bi = (T & 1) * PB, bo = PB - bi;
        const CT al = my[R::AL * 32], b1 = my[R::B * 32], b2 = my[(R::B + 1) * 32], b3 = my[(R::B + 2) * 32];
        CT x[NV];
#pragma unroll
        for (int v = 0; v < NV; v++) x[v] = al * my[v * 32] + b1 * yi[v];
#pragma unroll
        for (int v = 0; v < NV; v++) x[v] = (x[v] + b3 * qk[bi + v * FHS]) + b2 * qj[bi + v * FHS];
        x[4] = x[4] * my[R::SP * 32];
        const CT k0 = my[R::K0 * 32], k4 = my[R::K4 * 32], p = my[R::HR * 32] * x[4];
        CT w = x[4];
        if constexpr (NV == 7) w = (my[R::Y * 32] * x[4] - my[R::H3 * 32] * x[5]) - my[R::H2 * 32] * x[0];
        // the k and j products first: other lines wait for them
#pragma unroll
        for (int d = 2; d >= 0; d--) {
          const CT l = my[(R::L + d) * 32];
          const CT nx = my[(R::F + 3 * d) * 32], ny = my[(R::F + 3 * d + 1) * 32], nz = my[(R::F + 3 * d + 2) * 32];
          const CT z = nx * x[1] + ny * x[2] + nz * x[3];
          CT out[NV];
          out[0] = l * x[0] + k0 * z;
          out[1] = l * x[1] + nx * p;
          out[2] = l * x[2] + ny * p;
          out[3] = l * x[3] + nz * p;
          out[4] = l * w + k4 * z;
          if constexpr (NV == 7) {
            out[5] = l * x[5];
            out[6] = l * x[6];
          }
#pragma unroll
          for (int v = 0; v < NV; v++) {
            if (d == 0) yi[v] = out[v];
            else if (d == 1) nj[bo + v * FHS] = out[v];
            else nk[bo + v * FHS] = out[v];
          }
        }
        if (any_drop && J == jmax)   // PREDGS's dropped i+1 coupling (imps4.f:1460-1466)
#pragma unroll
          for (int v = 0; v < NV; v++) yi[v] = CT(0);
        if (line && (unsigned)(T - mj - mk) < (unsigned)imax)
#pragma unroll
          for (int v = 0; v < NV; v++) o[v * 32] = x[v];
        o += sg * ROW;
      }
      __syncthreads();
    }
    return;
  }

  const int io = threadIdx.x - FW * 32;
  if (io < FIO) {
    // ---- incoming edge words, records ----
    CT* ep[NQ];          // the word of step 0
    int eoff[NQ];        // wanted while 0 <= T - eoff < imax (NEVER: no upstream tile, no line)
    CT* ed[NQ];          // its place in buffer 0
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const int e = io + FIO * q;
      ep[q] = edge; eoff[q] = NEVER; ed[q] = pj;
      if (e < NV * FBK) {                      // from the j neighbour: value v of line row o
        const int v = e / FBK, o = e % FBK;
        ed[q] = pj + v * FHS + FW * 32 + o;
        if (up_j && tk * FBK + o < kmax) {
          eoff[q] = UP ? FBK - 1 - o : o;
          ep[q] = edge + ((long)(tile - sg) * nbs + s0 + sg * (FBJ - 1)) * EV + e;
        }
      } else if (e < EV) {                     // from the k neighbour: value v of line column o
        const int v = (e - NV * FBK) / FBJ, o = (e - NV * FBK) % FBJ;
        ed[q] = pk + v * FHS + FW * 32 + o;
        if (up_k && tj * FBJ + o < jmax) {
          eoff[q] = UP ? FBJ - 1 - o : o;
          ep[q] = edge + ((long)(tile - sg * g.nbj) * nbs + s0 + sg * (FBK - 1)) * EV + e;
        }
      }
    }
    auto want = [&](int q, int T) { return (unsigned)(T - eoff[q]) < (unsigned)imax; };
    bool dead = false;
    // words of step T (requested before, x) into the incoming places of buffer T & 1, waiting for those not there yet
    auto take = [&](int T, CT (&x)[NQ]) {
      const long at = (long)(sg * T) * EV;
      bool miss = false;
#pragma unroll
      for (int q = 0; q < NQ; q++) miss = miss || (want(q, T) && flow_mark(x[q]));
      if (__any_sync(0xffffffffu, miss)) {
        for (int it = 0; !dead; it++) {
          miss = false;
#pragma unroll
          for (int q = 0; q < NQ; q++)
            if (want(q, T) && flow_mark(x[q])) {
              x[q] = flow_ld(ep[q] + at);
              miss = miss || flow_mark(x[q]);
            }
          if (!__any_sync(0xffffffffu, miss)) break;
          if (HASTE || (it & 255) == 255) {
            int stop = HASTE || it >= kFlowSpins;
            if (stop && lane == 0) atomicExch(err, 3);
            stop = stop || *((volatile int*)err) != 0;
            dead = __any_sync(0xffffffffu, stop);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < NQ; q++)
        if (want(q, T)) {
          ed[q][(T & 1) * PB] = x[q];
          flow_st(ep[q] + at, flow_mark_of(x[q]));
        }
    };
    auto request = [&](int T, CT (&x)[NQ]) {
      const long at = (long)(sg * T) * EV;
#pragma unroll
      for (int q = 0; q < NQ; q++)
        if (want(q, T)) x[q] = flow_ld(ep[q] + at);
    };
    bool gone = io >= 32;   // one warp waits for the records, each lane up to its first time-out
    auto record = [&](int T) {
      if (gone || T >= nbs) return;
      for (long it = 0;; it++) {
        if (it >= (HASTE && (s_tile & 1) == 0 ? 0 : 4L * kFlowSpins)) { atomicExch(err, 4); s_stop = T + 1; gone = true; break; }
        if (pipe_try_wait(bar0 + 8 * (T % FD), (uint32_t)((T / FD) & 1))) break;
      }
    };
    CT ew[FPF][NQ];
#pragma unroll
    for (int u = 0; u < FPF; u++)
#pragma unroll
      for (int q = 0; q < NQ; q++) ew[u][q] = CT(0);
    request(0, ew[0]);
    take(0, ew[0]);
#pragma unroll
    for (int u = 1; u <= FPF; u++) request(u, ew[u % FPF]);
    record(0);
    __syncthreads();
    for (int tb = 0; tb < nbs; tb += FPF) {
#pragma unroll
      for (int u = 0; u < FPF; u++) {
        const int T = tb + u;
        if (T >= nbs) break;
        take(T + 1, ew[(u + 1) % FPF]);
        request(T + 1 + FPF, ew[(u + 1) % FPF]);
        record(T + 1);
        __syncthreads();
      }
    }
    return;
  }

  // ---- outgoing edge words, record copies ----
  const int po = io - FIO;
  int last = -1;             // the last step whose copies were started
  auto copy = [&](int T, int stop) {   // the records of CTA step T, one lane a warp tile
    if (po >= 32 || T >= nbs) return;
    int off = 0;
    const int wt = po < FW ? wtile(po, off) : -1;
    const bool act = !stop && wt >= 0 && (unsigned)(T - off) < (unsigned)ns;
    const unsigned n = __popc(__ballot_sync(0xffffffffu, act));
    const uint32_t bar = bar0 + 8 * (T % FD);
    if (po == 0 && (n || !stop)) { flow_expect(bar, n * RB); last = T; }
    __syncwarp();
    if (act)
      flow_bulk(ring0 + ((T % FD) * FW + po) * RB, rec + ((size_t)wt * ns + (UP ? ns - 1 - (T - off) : T - off)) * ROW, RB,
                bar);
  };
  for (int T = 0; T < FD; T++) copy(T, 0);
  CT* ep[NQ];          // the word of step 0
  int eoff[NQ];        // there while 0 <= T - eoff < imax (NEVER: no downstream tile, no line)
  const CT* es[NQ];    // its place in buffer 0
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const int e = po + FIO * q;
    ep[q] = edge + ((long)tile * nbs + s0) * EV + e; eoff[q] = NEVER; es[q] = pj;
    auto place = [](int j, int k) { return ((k / FTK) * FWJ + j / FTJ) * 32 + (k % FTK) * FTJ + j % FTJ; };
    if (e < NV * FBK) {                      // to the j neighbour: the last line of row o
      const int v = e / FBK, o = e % FBK;
      es[q] = pj + v * FHS + place(UP ? 0 : FBJ - 1, o);
      if (dn_j && tk * FBK + o < kmax) eoff[q] = (UP ? FBK - 1 - o : o) + FBJ - 1;
    } else if (e < EV) {                     // to the k neighbour: the last line of column o
      const int v = (e - NV * FBK) / FBJ, o = (e - NV * FBK) % FBJ;
      es[q] = pk + v * FHS + place(o, UP ? 0 : FBK - 1);
      if (dn_k && tj * FBJ + o < jmax) eoff[q] = (UP ? FBJ - 1 - o : o) + FBK - 1;
    }
  }
  auto publish = [&](int T) {   // the products of step T stand in buffer (T + 1) & 1
    const long at = (long)(sg * T) * EV;
#pragma unroll
    for (int q = 0; q < NQ; q++)
      if ((unsigned)(T - eoff[q]) < (unsigned)imax) flow_st(ep[q] + at, flow_pub(es[q][((T + 1) & 1) * PB]));
  };
  __syncthreads();
  for (int T = 0; T < nbs; T++) {
    if (T > 0) {
      const int stop = s_stop;
      publish(T - 1);
      copy(T - 1 + FD, stop);
    }
    __syncthreads();
  }
  publish(nbs - 1);
  if (po == 0 && s_stop)   // copies that nobody waited for must land before the CTA leaves
    for (int T = s_stop - 1; T <= last; T++)
      for (long it = 0; it < kFlowDrain && !pipe_try_wait(bar0 + 8 * (T % FD), (uint32_t)((T / FD) & 1)); it++) {}
}
