// Persistent batched kernel: one CTA (256 threads) per chain runs `moves` iterations of the
// move loop (gcmc.f:589-1380) entirely on the device.
//
// Per move: four warps set the move up side by side -- warp 0 takes the draws, chooses the move and
// builds the trial sites and the real-space work list, warp 1 finishes the last move's bookkeeping,
// warp 2 builds the phase tables, warp 3 the tail correction -- then all threads sweep their k-vectors
// (S(k), S_new, akk and the k-vector table are resident in shared memory for the whole launch) and
// their share of the real-space pair candidates, and every thread applies energy_eval to the warps'
// sums and commits its own k-vectors: two block barriers a move.
//
// A chain's move is a serial chain of latencies; what one costs, in SM cycles (16 chains, one an SM,
// K = 131, 510 atoms / 256 chains of 16 frameworks, two chains on most SMs): before the set-up and the
// bookkeeping were split over warps 23.8k / 30.0k (set-up 7.0k / 8.3k, sums 12.5k / 17.0k, acceptance,
// bookkeeping and commit 4.6k / 4.9k), now 14.8k / 19.2k.  Code that runs once a move comes through the
// instruction caches (32 KB, then 128 KB) each time, at up to ten cycles an instruction, so the set-up
// keeps one path for every move type and its rare parts out of line.
#include <cstring>
#include <map>
#include <mutex>

#include "fmc_batch.h"

namespace fmc {

namespace {

// The trial being evaluated: what the energy sums read, written while the move is set up.
struct MoveSmem {
  int mtype, g, nold, nnew, ns, ex_lo, ex_hi;
  int still;  // the trial leaves the molecule where it is (real_space_residue)
  double r[7], dis_delr, dis_rot;  // the trial's random numbers and step sizes (select_move)
  // trial sites (old ones first): position, charge factor q r4pie0 (negative for the old sites of a
  // displacement, whose energies are subtracted) and atom type, times types + 1 (a row of prow)
  double x[2 * kBatchMaxSites], y[2 * kBatchMaxSites], z[2 * kBatchMaxSites], cq[2 * kBatchMaxSites];
  int type[2 * kBatchMaxSites];
  // real-space work list, in chunks of 32 candidates: entry e < nsite is trial site e's voxel list {chunks
  // before it, first entry, length} (nfw chunks in all), entry nsite + e every guest site for it (gchunks)
  int4 list[2 * kBatchMaxSites];
  int nfw, gchunks, gpre[kMaxGuestTypes + 1];
  double lrc_term[kBatchMaxTab];
  // multi-jump (gcmc.f:1557-1785) across the two loop trips of one move: the first molecule's
  // choice and old sites, and (the bookkeeping warp's) its energy change and the energy before
  int mj_first, mj_lo;
  double mj_estep, mj_energy0;
  double mj_old[3 * kBatchMaxSites];
};

// What the acceptance test and the commit read.  Two copies in turn: the next move's set-up writes the
// other one while slower warps still commit this one.
struct MoveCtl {
  int mtype, g, ns, nmols, randchoice, need_lrc;
  int lo, seg_end;  // the moved molecule's first site, the end of its species' segment
  int mj_stage;     // multi-jump: 1 while the first jump is evaluated and kept, 2 for the second
  double rande;     // the draw the acceptance test takes if it draws
  double pref;      // the acceptance test's factor of exp(-beta dE) (insert, delete)
  int free_delete;  // no pressure: deletions are accepted
  double lrc, elrc; // tail correction with the trial's counts, and of the state before it
  double mj_estep;
};

// A decided move, kept for its bookkeeping (which runs beside the next move's set-up).
struct MoveDone {
  int mtype, g, randchoice, accepted, mj_stage, mv;
  double ewld1, ewld2, ewld3, vdw, delrc, estep, rande;
};

// A CTA's shared memory: the chain's control block, the move in progress and the system's constants,
// then the arrays sized by the batch (BatchArrays).  Every device function reaches it through
// batch_smem() instead of taking references, so that its accesses compile to shared-memory
// instructions also where the function is not inlined (a reference is a generic address there).
struct BatchSmem {
  ChainDev C;
  MoveSmem M;
  SysConst Y;
  MoveCtl ctl[2];
  MoveDone done;
  int st_nmol[kMaxGuestTypes];  // the bookkeeping warp's own copy of the molecule counts
  double red[3 * 16];  // per warp {sum akk d|S|^2, ewld2, vdw}
  int prow[(kBatchMaxTypes + 1) * (kBatchMaxTypes + 1)];
};

__device__ __forceinline__ BatchSmem& batch_smem() {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return *reinterpret_cast<BatchSmem*>(smem_raw);
}

constexpr int kBatchSmemBytes = ((int)sizeof(BatchSmem) + 15) & ~15;

// S(k), S_new, akk, the packed k-vectors and the trial's phase tables.
struct BatchArrays {
  double2 *Sk, *Sn;
  double* ak;
  int* kp;
  double2* tab;
};

__device__ __forceinline__ BatchArrays batch_arrays(int kmax_smem) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BatchArrays A;
  A.Sk = reinterpret_cast<double2*>(smem_raw + kBatchSmemBytes);
  A.Sn = A.Sk + kmax_smem;
  A.ak = reinterpret_cast<double*>(A.Sn + kmax_smem);
  A.kp = reinterpret_cast<int*>(A.ak + kmax_smem);
  A.tab = reinterpret_cast<double2*>(A.kp + ((kmax_smem + 3) & ~3));
  return A;
}

// The next 32 draws of duni (gcmc.f:2712-2805), one per lane.  The lagged Fibonacci part reads entries
// 33 and 97 draws back, so 32 draws do not depend on one another, and c steps through multiples of
// 2^-24 below cm, so lane i reaches its c in exact integer arithmetic; every draw equals duni's.
// Serially a draw is a chain of two dependent table reads, four additions and their tests (a move takes
// 2-11 of them, ~1.7k SM cycles); here all are ready after one such chain.
struct DrawWarp {
  float fresh, value, c;  // this lane's new table entry, its draw and c after it
  int slot, used;

  __device__ __forceinline__ void generate(const Duni& d, int lane) {
    constexpr int kCm = 16777213, kCd = 7654321;
    int i = d.ir - lane, j = d.jr - lane;
    if (i < 1) i += 97;
    if (j < 1) j += 97;
    slot = i - 1;
    float uni = d.u[i - 1] - d.u[j - 1];
    if (uni < 0.0f) uni = uni + 1.0f;
    fresh = uni;
    const int ci = ((int)(d.c * 16777216.0f) + (lane + 1) * (kCm - kCd)) % kCm;
    c = (float)ci * (1.0f / 16777216.0f);
    uni = uni - c;
    if (uni < 0.0f) uni = uni + 1.0f;
    value = uni;
    used = 0;
  }
  // Draw i of the 32 (every lane).
  __device__ __forceinline__ double at(int i) const { return (double)__shfl_sync(0xffffffffu, value, i); }
  // The state after the draws taken so far.
  __device__ __forceinline__ void commit(Duni& d, int lane) {
    if (used == 0) return;
    const float cl = __shfl_sync(0xffffffffu, c, used - 1);
    if (lane < used) d.u[slot] = fresh;
    if (lane == 0) {
      int i = d.ir - used, j = d.jr - used;
      d.ir = i < 1 ? i + 97 : i;
      d.jr = j < 1 ? j + 97 : j;
      d.c = cl;
    }
    __syncwarp();
  }
};

// Every 400 moves (gcmc.f:594-736): the end of production, the switch to production and the pressure
// equilibration; a rare path, kept out of line.
__device__ __noinline__ void check400() {
  BatchSmem& B = batch_smem();
  ChainDev& C = B.C;
  const SysConst& Y = B.Y;
  int totalguests = 0;
  for (int g = 0; g < Y.nspecies; g++) totalguests += B.st_nmol[g];
  if (C.production) {
    if (C.mcsteps < 0) {
      for (int t = 4; t > 0; t--) C.tick[t] = C.tick[t - 1];
      C.tick[0] = !(C.prodcount < (long long)(-C.mcsteps) * (totalguests + 1));
      bool all = true;
      for (int t = 0; t < 5; t++) all = all && C.tick[t];
      if (all) C.lgchk = 0;
    } else if (C.prodcount >= C.mcsteps) {
      C.lgchk = 0;
    }
  } else {
    if (C.despre > 0) {  // pressure equilibration (gcmc.f:637-696)
      for (int t = 4; t > 0; t--) C.tick[t] = C.tick[t - 1];
      C.tick[0] = !(C.prodcount < (long long)(-C.eqsteps) * (totalguests + 1) / 4);
      if (C.tick[0])
        pressure_adjust(Y.nspecies, C.press, &C.stats[0][0], 6, C.adspres, C.adsguen, C.packf, Y.volm, C.temp,
                        C.presrate, C.despre, C.gcmccount, C.prodcount, C.eqsteps);
    }
    if (C.eqsteps > 0) {
      if (C.gcmccount >= C.eqsteps && C.despre == 0) C.production = 1;
    } else if (C.eqsteps < 0) {
      for (int t = 4; t > 0; t--) C.tick[t] = C.tick[t - 1];
      C.tick[0] = !((long long)C.gcmccount < (long long)(-C.eqsteps) * (totalguests + 1));
      if (C.despre > 0) C.tick[0] = 0;
      bool all = true;
      for (int t = 0; t < 5; t++) all = all && C.tick[t];
      if (all) {
        C.production = 1;
        for (int t = 0; t < 5; t++) C.tick[t] = 0;
      }
    }
  }
}

__device__ __noinline__ void insertion_sample(int i, double estep) {
  ChainDev& C = batch_smem().C;
  window_insertion(C.win, i, estep, C.temp, C.accept_ins, C.stats[i]);
}

__device__ __noinline__ void close_window() {
  BatchSmem& B = batch_smem();
  ChainDev& C = B.C;
  window_close(C.win, B.Y.nspecies, C.nwind, C.temp, [&C](int i) { return (const double*)C.stats[i]; });
}

// One production move's averages (gcmc.f:1814-1928) by the bookkeeping warp: the five rolling averages and
// the five window means of a species take a lane each (their divisions, one after another, were a
// third of the bookkeeping); lane 0 stores the samples and takes the rare parts.  ins_g: species of an
// accepted insertion (-1: none).
__device__ __noinline__ void production_sample(int ins_g, bool counted, double estep, int lane) {
  BatchSmem& B = batch_smem();
  ChainDev& C = B.C;
  const int ns = B.Y.nspecies;
  const bool count = (C.laccsample && counted) || !C.laccsample;
  const long long prodcount = C.prodcount + (count ? 1 : 0);
  if (count) {
    const double pc = (double)prodcount;
    const int roll = C.win.rollcount + 1;
    __syncwarp();
    if (lane == 0) {
      C.prodcount = prodcount;
      C.win.rollcount = roll;
    }
#pragma unroll 1
    for (int i = 0; i < ns; i++) {
      const double dm = (double)(float)B.st_nmol[i], en = C.energy[i];
      if (lane == 0 && C.gasmol && prodcount <= kSampleCap + 1) {
        C.gasmol[(size_t)i * kSampleCap + prodcount - 1] = dm;
        C.gaseng[(size_t)i * kSampleCap + prodcount - 1] = en;
      }
      if (lane < 10) {
        const bool rolling = lane < 5;
        const int k = rolling ? lane : lane - 5;
        const double v = k == 0 ? dm : (k == 1 ? en : (k == 2 ? en * dm : (k == 3 ? dm * dm : en * en)));
        double* p = rolling ? &C.stats[i][k] : &C.win.avg[i][k];
        const double old = *p;
        const double q = (rolling ? v - old : (roll - 1) * old + v) / (rolling ? pc : (double)roll);
        *p = rolling ? old + q : q;
      }
      __syncwarp();
      if (lane == 0 && ins_g == i) insertion_sample(i, estep);
    }
  }
  __syncwarp();
  const bool closes = prodcount <= 0x7fffffffLL ? (int)prodcount % C.nwind == 0 : prodcount % C.nwind == 0;
  if (lane == 0 && (closes || !C.lgchk)) close_window();
}

// Bookkeeping of a decided move (gcmc.f:954-1380, 1796-1928) by one warp, beside the next move's
// set-up: running energies, the counters the set-up does not read, statistics, the trace record.
__device__ __noinline__ void finish_move(MoveRecord* trace, int lane) {
  BatchSmem& B = batch_smem();
  ChainDev& C = B.C;
  MoveSmem& M = B.M;
  __syncwarp();  // lane 0 wrote the decided move
  const MoveDone D = B.done;
  const int g = D.g, mtype = D.mtype;
  const bool accepted = D.accepted != 0;
  double estep = D.estep;
  const bool first_jump = mtype == kMultiJump && D.mj_stage == 1;
  if (mtype == kMultiJump && !first_jump) estep = M.mj_estep + estep;
  // flex / swap leave the reference's `accepted` as the previous move set it
  const bool counted = mtype == kNoop ? (C.last_accepted != 0) : accepted;
  __syncwarp();
  if (lane == 0) {
    if (first_jump) {
      // the first jump stands while the second is tried (gcmc.f:1697-1715); the move is counted
      // once, when the second jump is decided
      M.mj_energy0 = C.energy[g];
      M.mj_estep = estep;
      C.energy[g] = M.mj_energy0 + estep;
      C.jump_count++;
    } else if (mtype == kMultiJump) {
      if (accepted) C.accept_jump++;
      C.energy[g] = accepted ? M.mj_energy0 + estep : M.mj_energy0;
    } else if (mtype == kNoop) {
    } else {
      if (mtype == kInsert) C.ins_count++;
      else if (mtype == kDelete) C.del_count++;
      else if (mtype == kJump) C.jump_count++;
      if (accepted) {
        if (mtype == kInsert || mtype == kDelete) {
          if (mtype == kInsert) C.accept_ins++;
          else C.accept_del++;
          C.elrc = C.elrc + D.delrc;
          B.st_nmol[g] += mtype == kInsert ? 1 : -1;
        } else if (mtype == kJump) {
          C.accept_jump++;
        }
        C.energy[g] += estep;
      }
    }
    if (!first_jump) {
      if (mtype != kNoop) C.last_accepted = accepted;
      C.last_dE = accepted ? estep : 0.0;
      C.moves_done++;
    }
  }
  __syncwarp();
  if (first_jump) return;
  if (C.production) {
    production_sample(mtype == kInsert && accepted ? g : -1, counted, estep, lane);
  } else if (lane == 0 && C.despre > 0 && ((C.laccsample && counted) || !C.laccsample)) {
    // running loading while the pressures equilibrate (gcmc.f:1796-1808)
    C.prodcount++;
#pragma unroll 1
    for (int i = 0; i < B.Y.nspecies; i++)
      C.stats[i][0] = C.stats[i][0] + ((double)(float)B.st_nmol[i] - C.stats[i][0]) / (double)C.prodcount;
  }
  if (trace && lane == 0) {
    MoveRecord* rec = trace + D.mv;
    rec->step = C.gcmccount;
    rec->iguest = g;
    rec->mtype = mtype;
    rec->randchoice = D.randchoice;
    rec->accepted = counted;  // as the reference's `accepted` reads after the move
    rec->nmols_after = B.st_nmol[g];
    rec->pad0 = 0;
    rec->pad1 = 0;
    rec->ewld1 = D.ewld1;
    rec->ewld2 = D.ewld2;
    rec->ewld3 = D.ewld3;
    rec->vdw = D.vdw;
    rec->delrc = D.delrc;
    rec->estep = estep;
    rec->rande = D.rande;
    rec->energy_after = C.energy[g];
  }
  __syncwarp();
}

// Tail correction (gstlrcorrect, vdw_terms.f:684-745) by one warp, with the trial's molecule added to
// (d = 1) or taken from (-1) the counts: lane-parallel pair terms, summed by lane 0 in the reference's
// pair order.
__device__ __forceinline__ void lrc_warp(const BatchSmem& B, MoveSmem& M, int g, int d, double& lrc, int lane) {
  const ChainDev& C = B.C;
  const SysConst& Y = B.Y;
  const SpeciesConst& P = Y.sp[g];
  const int nt = Y.ntypes, ntab = nt * (nt + 1) / 2;
  const double twopi = 2.0 * kPi, v = Y.volm;
#pragma unroll 1
  for (int p = lane; p < ntab; p += 32) {
    int i = 1;
#pragma unroll 1
    while (i * (i + 1) / 2 <= p) i++;
    int j = p - (i - 1) * i / 2 + 1;
    int ni = C.numtyp[i], nj = C.numtyp[j];
#pragma unroll 1
    for (int s = 0; s < P.nsite; s++) {
      const int t = P.type[s];
      if (t == i) ni += d;
      if (t == j) nj += d;
    }
    double den = twopi * ((double)ni * (double)nj - (double)Y.numfrz[i] * (double)Y.numfrz[j]) / (v * v);
    M.lrc_term[p] = v * den * Y.steadd[p + 1];
  }
  __syncwarp();
  if (lane == 0) {
    double e = 0.0;
    if (Y.lrc_on)
#pragma unroll 4
      for (int p = 0; p < ntab; p++) e = e + M.lrc_term[p];
    lrc = e;
  }
}

// Device clock in nanoseconds (%globaltimer: one time base for every SM, unlike clock64).
__device__ __forceinline__ long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return (long long)t;
}

// One warp: phase tables of the trial sites (ewald.f:95-137).
__device__ __forceinline__ void build_phases(const BatchSmem& B, double2* tab, int stride, int lane) {
  const MoveSmem& M = B.M;
  const DevSystem& S = B.Y.S;
  const int nsite = M.nold + M.nnew, k1 = S.kmax[0], k2 = S.kmax[1];
#pragma unroll 1
  for (int w = lane; w < nsite * 3; w += 32) {
    int st = w / 3, ax = w % 3;
    double f[3];
    frac_coords(S.cell, M.x[st], M.y[st], M.z[st], f);
    int off = st * stride + (ax == 0 ? 0 : (ax == 1 ? k1 + 1 : k1 + k2 + 2));
    axis_phases(f[ax], S.kmax[ax], tab + off);
  }
}

// Past the 32nd draw (a multi-jump that keeps drawing its first molecule): the state moves on.
__device__ __noinline__ DrawWarp refill_draws(DrawWarp R, int lane) {
  Duni& d = batch_smem().C.rng;
  R.commit(d, lane);
  R.generate(d, lane);
  return R;
}

// Step-size adaptation (gcmc.f:794-834), every 50 or 100 attempts; out of line so that the set-up's code,
// run once a move, stays small (its instruction fetches are most of its time).
__device__ __noinline__ void adapt_steps(int g) {
  ChainDev& C = batch_smem().C;
  const int dc = C.disp_count[g], tc = C.tran_count[g], rc = C.rota_count;
  if (dc >= 1 && dc % 50 == 0) {
    const bool over = (C.accept_disp[g] / (double)dc) > C.disp_ratio[g];
    if (dc % 100 == 0) {
      if (over) C.delrdisp[g] = C.delrdisp[g] * 1.05;
      else if (C.delrdisp[g] > kDelrMin) C.delrdisp[g] = C.delrdisp[g] * 0.95;
    } else {
      if (over) C.rotangle = C.rotangle * 1.05;
      else if (C.rotangle > kMinAngle) C.rotangle = C.rotangle * 0.95;
    }
  }
  if (tc >= 1 && tc % 100 == 0) {
    if ((C.accept_tran[g] / (double)tc) > C.tran_ratio[g]) C.tran_delr[g] = C.tran_delr[g] * 1.05;
    else if (C.tran_delr[g] > kDelrMin) C.tran_delr[g] = C.tran_delr[g] * 0.95;
  }
  if (rc >= 1 && rc % 100 == 0) {
    if ((C.accept_rota / (double)rc) > C.rota_ratio) C.rota_rotangle = C.rota_rotangle * 1.05;
    else if (C.rota_rotangle > kMinAngle) C.rota_rotangle = C.rota_rotangle * 0.95;
  }
}

// Warp 0: the serial part of a move's set-up (gcmc.f:753-847): species and move choice, step-size
// adaptation, the counters it reads, and every random number of the trial in the reference's order
// (utility_pack.f:2545-3000), left in r for the warp to build the trial sites from.  Every lane
// takes the same branches and lane 0 writes.  `skip`: the last move's acceptance test took a draw.
__device__ __noinline__ void select_move(int par, int skip, bool second, int lane) {
  BatchSmem& B = batch_smem();
  ChainDev& C = B.C;
  const SysConst& Y = B.Y;
  MoveSmem& M = B.M;
  MoveCtl& T = B.ctl[par];
  DrawWarp R;
  R.generate(C.rng, lane);
  R.used = skip;
  int g = 0, mtype = kMultiJump, mj_stage = 2, mj_first = 0;
  if (second) {  // the second jump of a multi-jump: no count or selection
    g = M.g;
    mj_first = M.mj_first;
  } else {
    const int ng = Y.nspecies;
    if (ng > 1) g = (int)(R.at(R.used++) * ng);
    // the first cumulative frequency above the draw: insert, delete, displace, jump, flex and swap
    // (gcmc.f:1789-1795), translate, rotate, multi-jump; none: displace
    const double randmov = R.at(R.used++);
    const unsigned above = __ballot_sync(0xffffffffu, lane < 9 && randmov < C.mvcum[g][lane < 9 ? lane : 0]);
    constexpr unsigned long long kTypes = 0x854776321ULL;
    static_assert(kInsert == 1 && kDelete == 2 && kDisplace == 3 && kTranslate == 4 && kRotate == 5 && kJump == 6 &&
                      kNoop == 7 && kMultiJump == 8, "one digit of kTypes each");
    mtype = above ? (int)(kTypes >> (4 * (__ffs(above) - 1))) & 15 : (int)kDisplace;
    const int nmols = C.nmol[g];
    const unsigned dc = C.disp_count[g], tc = C.tran_count[g], rc = C.rota_count;
    if (nmols >= 1 && ((dc && dc % 50u == 0) || (tc && tc % 100u == 0) || (rc && rc % 100u == 0))) {
      if (lane == 0) adapt_steps(g);
      __syncwarp();
    }
    if (nmols == 0 || (nmols == 1 && mtype == kMultiJump)) mtype = kInsert;  // gcmc.f:837-847
    mj_stage = mtype == kMultiJump ? 1 : 0;
  }
  const int ns = Y.sp[g].nsite, nmols = C.nmol[g], seg = C.seg_off[g];
  const bool jump = mtype == kJump || mtype == kMultiJump, need_lrc = mtype == kInsert || mtype == kDelete;
  const bool full = mtype == kInsert && ((C.totatm - C.framatm) + ns >= C.maxguest || (nmols + 1) * ns > C.seg_cap[g]);
  int randchoice = 0;
  if (jump) {
    // long jump (gcmc.f:1389-1547): the choice first, then the seven draws of random_jump; the
    // second jump of a multi-jump draws until it hits a molecule other than the first
    do {
      if (R.used == 32) R = refill_draws(R, lane);
      randchoice = (int)(R.at(R.used++) * nmols) + 1;
    } while (randchoice == mj_first);
    if (mj_stage == 1) mj_first = randchoice;
    if (R.used > 24) R = refill_draws(R, lane);
  }
  // r[0..6], lane i's r[i]: a translation draws the first three, a rotation the last four
  const int lo = mtype == kRotate ? 3 : 0;
  const int nr = mtype == kDelete || mtype == kNoop || full ? 0 : (mtype == kTranslate ? 3 : 7 - lo);
  const double drawn = R.at((R.used + lane - lo) & 31);
  const double r = lane >= lo && lane < lo + nr ? drawn : (mtype == kRotate ? 0.5 : 0.0);
  R.used += nr;
  if (mtype == kDelete || mtype == kDisplace || mtype == kTranslate || mtype == kRotate)
    randchoice = (int)(R.at(R.used++) * nmols) + 1;
  const double rande = R.at(R.used);  // the draw the acceptance test would take (at most the 32nd)
  R.commit(C.rng, lane);
  if (lane < 7) M.r[lane] = r;
  if (lane == 0) {
    if (full) C.status = 75;
    double dis_delr = 0.0, dis_rot = 0.0;
    if (mtype == kTranslate) {
      C.tran_count[g]++;
      dis_delr = C.tran_delr[g];
    } else if (mtype == kRotate) {
      C.rota_count++;
      dis_rot = C.rota_rotangle;
    } else if (mtype == kDisplace) {
      C.disp_count[g]++;
      dis_delr = C.delrdisp[g];
      dis_rot = C.rotangle;
    }
    M.dis_delr = dis_delr;
    M.dis_rot = dis_rot;
    const int first = randchoice > 0 ? seg + (randchoice - 1) * ns : -1;
    M.mtype = mtype;
    M.g = g;
    M.nold = mtype == kInsert || mtype == kNoop ? 0 : ns;
    M.nnew = mtype == kDelete || mtype == kNoop || full ? 0 : ns;
    M.ns = ns;
    M.ex_lo = first;
    M.ex_hi = first < 0 ? -1 : first + ns;
    M.mj_first = mj_first;
    T.mtype = mtype;
    T.g = g;
    T.ns = ns;
    T.nmols = nmols;
    T.randchoice = randchoice;
    T.need_lrc = need_lrc;
    T.seg_end = seg + nmols * ns;
    T.lo = mtype == kInsert ? seg + nmols * ns : first;
    T.mj_stage = mj_stage;
    T.rande = rande;
  }
  __syncwarp();
}

// ------------------------------------------------------------------ the trial sites, one lane each
// The trial generators of fmc_common.h restated for a warp: lane i holds site i, so the moved
// molecule's sites load at once and each site takes the same arithmetic as there; the mass centre
// sums run over the sites in order in every lane (gathered by shuffles), so every lane holds the
// same centre.
__device__ __forceinline__ void com_lanes(const double* mass, int n, double x, double y, double z, double* c) {
  double w = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
#pragma unroll 1
  for (int j = 0; j < n; j++) {
    const double xj = __shfl_sync(0xffffffffu, x, j), yj = __shfl_sync(0xffffffffu, y, j),
                 zj = __shfl_sync(0xffffffffu, z, j);
    w = w + mass[j];
    sx = sx + xj * mass[j];
    sy = sy + yj * mass[j];
    sz = sz + zj * mass[j];
  }
  c[0] = sx / w;
  c[1] = sy / w;
  c[2] = sz / w;
}

// One site rotated by quaternion q (rotate_sites' matrix).
__device__ __forceinline__ void rotate_site(const double q[4], double& x, double& y, double& z) {
  const double q1 = q[0], q2 = q[1], q3 = q[2], q4 = q[3];
  const double Q0 = 2.0 * q2 * q2 + 2.0 * q1 * q1 - 1.0, Q1 = 2.0 * q2 * q3 - 2.0 * q1 * q4;
  const double Q2 = 2.0 * q2 * q4 + 2.0 * q1 * q3, Q3 = 2.0 * q2 * q3 + 2.0 * q1 * q4;
  const double Q4 = 2.0 * q1 * q1 + 2.0 * q3 * q3 - 1.0, Q5 = 2.0 * q3 * q4 - 2.0 * q1 * q2;
  const double Q6 = 2.0 * q2 * q4 - 2.0 * q1 * q3, Q7 = 2.0 * q3 * q4 + 2.0 * q1 * q2;
  const double Q8 = 2.0 * q4 * q4 + 2.0 * q1 * q1 - 1.0;
  const double tx = Q0 * x + Q1 * y + Q2 * z;
  const double ty = Q3 * x + Q4 * y + Q5 * z;
  const double tz = Q6 * x + Q7 * y + Q8 * z;
  x = tx;
  y = ty;
  z = tz;
}

// random_jump's frame (utility_pack.f:2766-2813): the site about the mass centre once it has moved to
// cm, and that centre.
__device__ __noinline__ void jump_frame(const double* mass, int ns, double& x, double& y, double& z, double* cm) {
  double c[3];
  com_lanes(mass, ns, x, y, z, c);
  const double xd = cm[0] - c[0], yd = cm[1] - c[1], zd = cm[2] - c[2];
  x = xd + x;
  y = yd + y;
  z = zd + z;
  com_lanes(mass, ns, x, y, z, cm);
  x = x - cm[0];
  y = y - cm[1];
  z = z - cm[2];
}

// Warp 0, after select_move: the trial sites (old sites read from the chain, new ones built by
// random_ins / random_disp + random_rot / random_jump), their charges and types -- from which warp 2
// builds the phase tables (named barrier 2) -- then their voxel lists and the real-space work list.
__device__ __noinline__ void build_trial(int lane) {
  BatchSmem& B = batch_smem();
  ChainDev& C = B.C;
  MoveSmem& M = B.M;
  const SysConst& Y = B.Y;
  const DevSystem& S = Y.S;
  const int mtype = M.mtype, ns = M.ns, nold = M.nold, nnew = M.nnew;
  const SpeciesConst& P = Y.sp[M.g];
  const bool mine = lane < ns;
  if (nold && mine) {
    const double4 a = C.gsite[M.ex_lo + lane];
    M.x[lane] = a.x;
    M.y[lane] = a.y;
    M.z[lane] = a.z;
    M.cq[lane] = (nnew ? -P.q[lane] : P.q[lane]) * kR4pie0;
    M.type[lane] = P.type[lane] * (S.ntypes + 1);
  }
  bool still = false;
  if (nnew) {
    // one code path for every move type, so that it stays small: the site about the centre of
    // rotation (vx, vy, vz), the centre, the angle
    const double* r = M.r;
    const double* h = S.cell.h;
    double vx = 0.0, vy = 0.0, vz = 0.0, cm[3], turn = 2.0 * kPi;
    if (mine) {
      vx = nold ? M.x[lane] : P.tx[lane];
      vy = nold ? M.y[lane] : P.ty[lane];
      vz = nold ? M.z[lane] : P.tz[lane];
    }
    if (!nold || mtype == kJump || mtype == kMultiJump) {
      // random_ins (utility_pack.f:2545-2650): template rotated, centred at fractional (r0, r1, r2)
      cm[0] = r[0] * h[0] + r[1] * h[3] + r[2] * h[6];
      cm[1] = r[0] * h[1] + r[1] * h[4] + r[2] * h[7];
      cm[2] = r[0] * h[2] + r[1] * h[5] + r[2] * h[8];
      // random_jump: the mass centre moved there, a new orientation about it
      if (nold) jump_frame(P.mass, ns, vx, vy, vz, cm);
    } else {
      // random_disp + random_rot (utility_pack.f:2679-2763, 2929-3000)
      const double half = M.dis_delr * 0.5;
      const double dx = (2.0 * r[0] - 1.0) * half, dy = (2.0 * r[1] - 1.0) * half, dz = (2.0 * r[2] - 1.0) * half;
      vx = dx + vx;
      vy = dy + vy;
      vz = dz + vz;
      com_lanes(P.mass, ns, vx, vy, vz, cm);
      const double* rh = S.cell.rh;
      double fx = rh[0] * cm[0] + rh[3] * cm[1] + rh[6] * cm[2];
      double fy = rh[1] * cm[0] + rh[4] * cm[1] + rh[7] * cm[2];
      double fz = rh[2] * cm[0] + rh[5] * cm[1] + rh[8] * cm[2];
      fx = fx - floor(fx);
      fy = fy - floor(fy);
      fz = fz - floor(fz);
      const double wx = h[0] * fx + h[3] * fy + h[6] * fz;
      const double wy = h[1] * fx + h[4] * fy + h[7] * fz;
      const double wz = h[2] * fx + h[5] * fy + h[8] * fz;
      const double shx = wx - cm[0], shy = wy - cm[1], shz = wz - cm[2];
      vx = vx + shx - wx;
      vy = vy + shy - wy;
      vz = vz + shz - wz;
      cm[0] = wx;
      cm[1] = wy;
      cm[2] = wz;
      turn = M.dis_rot;
      // draws are multiples of 2^-24, so an angle is now and then exactly zero
      still = (M.dis_delr == 0.0 || (r[0] == 0.5 && r[1] == 0.5 && r[2] == 0.5)) && (ns == 1 || r[3] == 0.0 || turn == 0.0);
    }
    double q[4];
    axis_angle_quat(r[3] * turn, r[4], r[5], r[6], q);
    rotate_site(q, vx, vy, vz);
    if (mine) {
      const int st = nold + lane;
      M.x[st] = vx + cm[0];
      M.y[st] = vy + cm[1];
      M.z[st] = vz + cm[2];
      M.cq[st] = P.q[lane] * kR4pie0;
      M.type[st] = P.type[lane] * (S.ntypes + 1);
    }
  }
  __syncwarp();
  asm volatile("bar.arrive 2, 64;" ::: "memory");
  // the work list (warp scan over the voxel lists' chunks; the guest lists have one length)
  const int nsite = nold + nnew;
  int b = 0, len = 0;
  if (lane < nsite) {
    const int v = voxel_of(S, M.x[lane], M.y[lane], M.z[lane]);
    b = S.vox_off[v];
    len = S.vox_off[v + 1] - b;
  }
  int gt = 0;
  if (lane == 0) M.gpre[0] = 0;
#pragma unroll 1
  for (int g = 0; g < Y.nspecies; g++) {
    gt += C.nmol[g] * Y.sp[g].nsite;
    if (lane == 0) M.gpre[g + 1] = gt;
  }
  const int mine_chunks = (len + 31) >> 5, gchunks = (gt + 31) >> 5;
  int w = mine_chunks;
#pragma unroll 1
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, w, o);
    if (lane >= o) w += u;
  }
  const int fw = __shfl_sync(0xffffffffu, w, 31);
  if (lane < nsite) M.list[lane] = make_int4(w - mine_chunks, b, len, 0);
  if (lane == 0) {
    M.nfw = fw;
    M.gchunks = gchunks;
    M.still = still;
  }
}

// ------------------------------------------------------------------ energy sums of a trial
// A thread's share of the reciprocal change (ewald.f:139-331): S_new(k) = S(k) + dS(k) to Sn, and akk
// and |S_new|^2 - |S|^2 (ewald.f:311-319) returned.  A thread takes k-vectors tid, tid + NT, ... and adds
// their terms in that order, KPT of them in flight.  Bound by the latency of its shared-memory reads and FP64
// chain with 1-4 k-vectors a thread.
//
// The arithmetic is fixed, fma by fma: S(k) goes through every accepted move, and its last bits decide the
// moves whose energy change is rounding alone (real_space_residue).  So the old and the new sites' terms are
// summed apart, each q e^{ik.r} formed before it is added, and (S - old) + new taken in that order, in every
// compiled tile.
__device__ __forceinline__ double flip_sign(double v, int mask) {
  return __hiloint2double(__double2hiint(v) ^ mask, __double2loint(v));
}

__device__ __forceinline__ double2 recip_term(int k, const double* charge, int nold, int nsite, int k1, int k2,
                                             int stride, const double2* tb, const int* kp, const double* ak,
                                             const double2* Sk, double2* Sn) {
  int l, m, n;
  kunpack(kp[k], l, m, n);
  const int o2 = k1 + 1 + (m < 0 ? -m : m), o3 = k1 + k2 + 2 + (n < 0 ? -n : n);
  const int sm = m & 0x80000000, sn = n & 0x80000000;
  double ax = 0.0, ay = 0.0, bx = 0.0, by = 0.0;  // the old sites' sum goes to b once it is complete
  const double2* t = tb;
  const double* qp = charge;
#pragma unroll 1
  for (int st = 0; st < nsite; st++, t += stride) {
    const double2 e1 = t[l], e2 = t[o2], e3 = t[o3];
    const double q = *qp++, y2 = flip_sign(e2.y, sm), y3 = flip_sign(e3.y, sn);
    const double px = fma(e1.x, e2.x, -(e1.y * y2)), py = fma(e1.y, e2.x, e1.x * y2);
    ax = fma(q, fma(px, e3.x, -(py * y3)), ax);
    ay = fma(q, fma(py, e3.x, px * y3), ay);
    if (st == nold - 1) {
      bx = ax;
      by = ay;
      ax = ay = 0.0;
      qp = charge;
    }
  }
  const double2 so = Sk[k], sw = make_double2((so.x - bx) + ax, (so.y - by) + ay);
  Sn[k] = sw;
  return make_double2(ak[k], fma(-so.y, so.y, fma(-so.x, so.x, fma(sw.x, sw.x, sw.y * sw.y))));
}

// One candidate of a chunk: its atom and type (-1: none in this lane), and the trial site the chunk
// belongs to (the same for every lane).
struct Cand {
  double x, y, z, q;
  int type, site;
};

// Chunk `chunk` of the work list: 32 candidates of one site.  Lane l holds where entries l and l + 32 of
// the list begin (`at0`, `at1`), so the entry is the number of those the chunk has reached, less one.
// What a lane without a candidate leaves in c does not matter: its type is -1.
__device__ __forceinline__ void load_chunk(const BatchSmem& B, int chunk, int nchunk, int nsite, int at0, int at1,
                                           Cand& c) {
  const MoveSmem& M = B.M;
  const DevSystem& S = B.Y.S;
  c.type = -1;
  if (chunk >= nchunk) return;  // the whole warp
  const int e = __popc(__ballot_sync(0xffffffffu, chunk >= at0)) + __popc(__ballot_sync(0xffffffffu, chunk >= at1)) - 1;
  const int lane = threadIdx.x & 31;
  const double4* p;
  const unsigned char* tp;
  int i;
  bool live;
  if (e < nsite) {
    const int4 d = M.list[e];
    const int j = ((chunk - d.x) << 5) + lane;
    i = d.y + j;
    live = j < d.z;
    p = S.vox_xyzq;
    tp = S.vox_type + i;
    c.site = e;
  } else {  // guest sites: a guest's type is the low byte of its int
    c.site = e - nsite;
    const int j = ((chunk - M.nfw - c.site * M.gchunks) << 5) + lane;
    live = j < M.gpre[B.Y.nspecies];
    i = B.C.seg_off[0] + j;
    if (B.Y.nspecies > 1)
#pragma unroll 1
      for (int g = 1; g < B.Y.nspecies; g++)
        if (j >= M.gpre[g]) i = B.C.seg_off[g] + (j - M.gpre[g]);
    live = live && (unsigned)(i - M.ex_lo) >= (unsigned)(M.ex_hi - M.ex_lo);
    p = B.C.gsite;
    tp = reinterpret_cast<const unsigned char*>(B.C.gtype + i);
  }
  p += i;
  if (live) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(c.x), "=d"(c.y), "=d"(c.z), "=d"(c.q) : "l"(p));
    c.type = *tp;
  }
}

// This warp's share of the real-space pairs (ewald2 + srfrce over guestlistgen's set): chunks warp,
// warp + NW, ... of the work list, each lane adding its pairs in that order.  The loop is bound by
// latency (two chains, 16 warps, share an SM): a pair is a candidate load, an image, a root, three
// table reads and two interpolations, each waiting for the last.  So U chunks are in flight: their
// distances first, then the next U chunks' loads, then their table reads, without a branch in
// between -- a lane whose candidate is missing or beyond the cut-off reads row 0 of the table (no vdW)
// at the cut-off and adds zero.  Energy sums of a move, SM cycles (one chain an SM / 256 chains, two on
// most SMs): one branching candidate a trip and separate tables 12.6k / 17.8k; U = 2 7.7k / 10.9k (0.3k / 0.4k
// more since the reciprocal terms keep their roundings), U = 3 7.3k / 10.8k with the whole launch 4% faster / 4%
// slower (larger code), U = 4 slower for both.
template <int KIND, int NT, int U>
__device__ __forceinline__ void real_space(const BatchSmem& B, double& v1, double& v2) {
  const MoveSmem& M = B.M;
  const DevSystem& S = B.Y.S;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NW = NT / 32;
  const int nold = M.nold, nsite = nold + M.nnew, nchunk = M.nfw + nsite * M.gchunks;
  auto begins = [&M, nsite](int e) {  // the chunk at which entry e begins
    return e < nsite ? M.list[e].x : (e < 2 * nsite ? M.nfw + (e - nsite) * M.gchunks : 0x7fffffff);
  };
  const int at0 = begins(lane), at1 = begins(lane + 32);
  const int nminus = M.nnew ? nold : 0;  // a displacement's old sites are subtracted
  const double rcut2 = S.rcut2;
  Cand c[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    c[u].x = c[u].y = c[u].z = c[u].q = 0.0;
    c[u].site = 0;
  }
#pragma unroll
  for (int u = 0; u < U; u++) load_chunk(B, warp + u * NW, nchunk, nsite, at0, at1, c[u]);
#pragma unroll 1
  for (int base = warp; base < nchunk; base += U * NW) {
    double rs[U], cq[U];
    int off[U], site[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int s = c[u].site;
      const double rsq = image_dist2<KIND>(S.cell, M.x[s] - c[u].x, M.y[s] - c[u].y, M.z[s] - c[u].z);
      const bool in = c[u].type >= 0 && rsq < rcut2;
      const double qq = M.cq[s] * c[u].q;
      rs[u] = in ? rsq : rcut2;
      cq[u] = in && fabs(qq) > 1e-10 ? qq : 0.0;  // ewald2 skips smaller products
      off[u] = in ? B.prow[M.type[s] + c[u].type] : 0;
      site[u] = s;
    }
#pragma unroll
    for (int u = 0; u < U; u++) load_chunk(B, base + (U + u) * NW, nchunk, nsite, at0, at1, c[u]);
#pragma unroll
    for (int u = 0; u < U; u++) {
      pair_table<KIND>(S, rs[u], cq[u], off[u], site[u] < nminus ? -1.0 : 1.0, v1, v2);
    }
  }
}

// A trial that leaves its molecule in place -- a single site's rotation, a rotation by a draw of exactly zero, a
// translation with no step size -- changes no energy: what is left of E_new - E_old is the rounding of two sums of
// the same pairs, yet its sign decides whether the acceptance test draws a random number (gcmc.f:1330-1338), and
// so where a seeded chain goes from there.  These pairs keep one fixed arithmetic and order of addition:
// candidates tid, tid + NT, ... of the old sites' lists, each followed by the guests, then the new sites', correctly
// rounded roots, one table at a time.
template <int NT>
__device__ __noinline__ void real_space_residue(double* vout) {
  const BatchSmem& B = batch_smem();
  const MoveSmem& M = B.M;
  const DevSystem& S = B.Y.S;
  const int gt = M.gpre[B.Y.nspecies], ns = M.ns, nsite = 2 * ns;
  double v1 = 0.0, v2 = 0.0;
  int s = 0, begin = 0;
#pragma unroll 1
  for (int t = threadIdx.x;; t += NT) {
    while (s < nsite && t >= begin + M.list[s].z + gt) begin += M.list[s++].z + gt;
    if (s >= nsite) break;
    const int j = t - begin;
    const double chgea = B.Y.sp[M.g].q[s < ns ? s : s - ns] * kR4pie0;
    double4 a;
    int type;
    const int4 d = M.list[s];
    if (j < d.z) {
      a = S.vox_xyzq[d.y + j];
      type = S.vox_type[d.y + j];
    } else {
      const int jg = j - d.z;
      int g = 0;
      while (g + 1 < B.Y.nspecies && jg >= M.gpre[g + 1]) g++;
      const int i = B.C.seg_off[g] + (jg - M.gpre[g]);
      if (i >= M.ex_lo && i < M.ex_hi) continue;
      a = B.C.gsite[i];
      type = B.C.gtype[i];
    }
    const int off = B.prow[M.type[s] + type];
    double ec = 0.0, ev = 0.0;
    double dx = M.x[s] - a.x, dy = M.y[s] - a.y, dz = M.z[s] - a.z;
    min_image(S.cell, dx, dy, dz);
    const bool xy = S.cell.imcon <= 3;
    const double rsq = fma(dz, dz, xy ? fma(dx, dx, dy * dy) : fma(dy, dy, dx * dx));
    if (rsq < S.rcut2) {
      const double r = sqrt(rsq), chgprd = chgea * a.w;
      auto interp = [r](const double* tab, double rdr) {
        const double x = __dmul_rn(r, rdr);
        const int l = (int)x;
        const double p = __dsub_rn(x, (double)l);
        const double t0 = tab[l], t1 = tab[l + 1], t2 = tab[l + 2];
        const double u1 = fma(t1 - t0, p, t0), u2 = fma(t2 - t1, p - 1.0, t1);
        return fma(__dmul_rn(u2 - u1, p), 0.5, u1);
      };
      if (fabs(chgprd) > 1e-10) ec = __dmul_rn(interp(S.erc, S.rdr_e), chgprd);
      if (off) ev = interp(S.vvv + off, S.rdr_v);
    }
    if (s < ns) {
      v1 -= ec;
      v2 -= ev;
    } else {
      v1 += ec;
      v2 += ev;
    }
  }
  vout[0] = v1;
  vout[1] = v2;
}

// Every thread: its share of {sum akk d|S|^2, ewld2, vdw}, summed over its warp into red.
template <int KIND, int NT, int KPT, int CPT>
__device__ __noinline__ void sums_kind(int kmax_smem, int stride) {
  BatchSmem& B = batch_smem();
  const BatchArrays A = batch_arrays(kmax_smem);
  const DevSystem& S = B.Y.S;
  const int tid = threadIdx.x, K = S.K, k1 = S.kmax[0], k2 = S.kmax[1], nold = B.M.nold, nsite = nold + B.M.nnew;
  const double* charge = B.Y.sp[B.M.g].q;
  double v0 = 0.0, v1 = 0.0, v2 = 0.0;
  auto term = [&](int k) {
    return recip_term(k, charge, nold, nsite, k1, k2, stride, A.tab, A.kp, A.ak, A.Sk, A.Sn);
  };
  int k = tid;
  if (KPT == 2)
#pragma unroll 1
    for (; k + NT < K; k += 2 * NT) {  // two independent k-vectors in flight, added in order
      const double2 a = term(k), b = term(k + NT);
      v0 = fma(b.x, b.y, fma(a.x, a.y, v0));
    }
#pragma unroll 1
  for (; k < K; k += NT) {
    const double2 a = term(k);
    v0 = fma(a.x, a.y, v0);
  }
  if (B.M.still) {
    double v[2];
    real_space_residue<NT>(v);
    v1 = v[0];
    v2 = v[1];
  } else {
    real_space<KIND, NT, kChunksPerTrip + CPT>(B, v1, v2);
  }
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) {
    v0 += __shfl_down_sync(0xffffffffu, v0, o);
    v1 += __shfl_down_sync(0xffffffffu, v1, o);
    v2 += __shfl_down_sync(0xffffffffu, v2, o);
  }
  if ((tid & 31) == 0) {
    double* red = B.red + 3 * (tid >> 5);
    red[0] = v0;
    red[1] = v1;
    red[2] = v2;
  }
}

template <int NT, int KPT, int CPT>
__device__ __forceinline__ void sums(const DevSystem& S, int kmax_smem, int stride) {
  const int kind = pair_kind(S);
  if (kind == kPairOrtho) sums_kind<kPairOrtho, NT, KPT, CPT>(kmax_smem, stride);
  else if (kind == kPairTriclinic) sums_kind<kPairTriclinic, NT, KPT, CPT>(kmax_smem, stride);
  else sums_kind<kPairGeneral, NT, KPT, CPT>(kmax_smem, stride);
}

// Energy assembly of the move (gcmc.f:946, 1112, 1328) from the block's sums {sum akk d|S|^2, ewld2, vdw}.
__device__ __forceinline__ void assemble(const SysConst& Y, const MoveCtl& T, double v0, double v1, double v2,
                                         double& ewld1, double& ewld3, double& delrc, double& estep) {
  const SpeciesConst& P = Y.sp[T.g];
  ewld1 = Y.S.recip_pref * v0;
  ewld3 = 0.0;
  delrc = 0.0;
  if (T.need_lrc) {
    delrc = T.lrc - T.elrc;
    ewld3 = P.ewald3en;
    const double sg = T.mtype == kInsert ? 1.0 : -1.0;
    ewld1 = ewld1 + sg * P.engsic;
    estep = (ewld1 + sg * v1 + sg * ewld3 + sg * v2 + delrc) / Y.engunit;
  } else {
    estep = (ewld1 + v1 + v2) / Y.engunit;
  }
}

// Acceptance (energy_eval, utility_pack.f:3049-3095, with the displacement shortcut of
// gcmc.f:1330-1338); `drawn`: the test took the move's acceptance draw, exactly where the reference
// draws it.
__device__ __forceinline__ bool decide(double beta, const MoveCtl& T, double e, bool& drawn) {
  drawn = false;
  if (T.mtype == kNoop) return false;    // nothing to accept or reject; no draw
  if (T.mj_stage == 1) return true;      // the first jump is kept for now
  if (T.mj_stage == 2) e = T.mj_estep + e;  // one test on the summed change (gcmc.f:1730-1739)
  if (!T.need_lrc && e < 0.0) return true;
  drawn = true;
  double test;
  if (-1 * beta * e > 700.0) {
    test = exp(700.0);
  } else {
    test = exp(-1.0 * beta * e);
    if (T.need_lrc) test = T.mtype == kDelete && T.free_delete ? 1.0 : T.pref * test;
  }
  return T.rande < test;
}

// Warp 0, once a move is decided: the counters the next set-up reads and the guest sites of an accepted
// insertion or displacement (an accepted deletion's shift is the whole block's).
__device__ __forceinline__ void commit_control(const MoveCtl& T, bool accepted, int lane) {
  BatchSmem& B = batch_smem();
  ChainDev& C = B.C;
  MoveSmem& M = B.M;
  const int mtype = T.mtype, g = T.g, ns = T.ns;
  const SpeciesConst& P = B.Y.sp[g];
  if (!accepted) {
    if (T.mj_stage == 2 && lane < ns)
      C.gsite[M.mj_lo + lane] =
          make_double4(M.mj_old[3 * lane], M.mj_old[3 * lane + 1], M.mj_old[3 * lane + 2], P.q[lane]);
    __syncwarp();
    return;
  }
  if (lane == 0) {
    if (T.need_lrc) {
      const int d = mtype == kInsert ? 1 : -1;
      C.nmol[g] += d;
      C.totatm += d * ns;
#pragma unroll 1
      for (int i = 0; i < ns; i++) C.numtyp[P.type[i]] += d;
    } else if (mtype == kTranslate) {
      C.accept_tran[g]++;
    } else if (mtype == kRotate) {
      C.accept_rota++;
    } else if (mtype == kDisplace) {
      C.accept_disp[g]++;
    }
    if (T.mj_stage == 1) M.mj_lo = T.lo;
  }
  if (lane < ns) {
    if (T.mj_stage == 1) {
      M.mj_old[3 * lane] = M.x[lane];
      M.mj_old[3 * lane + 1] = M.y[lane];
      M.mj_old[3 * lane + 2] = M.z[lane];
    }
    if (mtype != kDelete) {
      const int st = mtype == kInsert ? lane : ns + lane;
      C.gsite[T.lo + lane] = make_double4(M.x[st], M.y[st], M.z[st], P.q[lane]);
      C.gtype[T.lo + lane] = P.type[lane];
    }
  }
  __syncwarp();
}

// All threads, in production: storeprob (utility_pack.f:496-561) for the chain's state after the
// move, one guest molecule per thread, weights added to the plots' fixed-point grids.
__device__ __noinline__ void prob_store(const SysConst& Y, const ChainDev& C) {
  const int na = Y.ngrid[0], nb = Y.ngrid[1], nc = Y.ngrid[2];
  const long long cells = (long long)na * nb * nc;
  for (int g = 0; g < Y.nspecies; g++) {
    const SpeciesConst& P = Y.sp[g];
    const int ns = P.nsite, nmol = C.nmol[g];
    for (int m = threadIdx.x; m < nmol; m += blockDim.x) {
      double x[kBatchMaxSites], y[kBatchMaxSites], z[kBatchMaxSites];
      const double4* site = C.gsite + C.seg_off[g] + m * ns;
      for (int i = 0; i < ns; i++) {
        double4 a = site[i];
        x[i] = a.x;
        y[i] = a.y;
        z[i] = a.z;
      }
      double c[3], fc[3];
      centre_of_mass(P.mass, ns, x, y, z, 1, c);
      frac_wrap(Y.S.cell.rh, c[0], c[1], c[2], fc);
      for (int ip = 0; ip < Y.nplots; ip++) {
        if (Y.plot_guest[ip] != g) continue;
        unsigned long long* grid = C.prob + ip * cells;
        auto add = [grid](long long i, double w) {
          atomicAdd(grid + i, (unsigned long long)llrint(w * 4294967296.0));
        };
        for (int j = 0; j < Y.plot_nsite[ip]; j++) {
          const int s = Y.plot_site[ip][j];
          if (s == 0) {
            equitable_bin(na, nb, nc, fc[0], fc[1], fc[2], add);
          } else {
            double f[3];
            frac_wrap(Y.S.cell.rh, x[s - 1], y[s - 1], z[s - 1], f);
            equitable_bin(na, nb, nc, f[0], f[1], f[2], add);
          }
        }
      }
    }
  }
}

template <bool kProf, int NT, int KPT, int CPT>
__global__ void __launch_bounds__(NT, NT <= 128 ? 4 : (NT <= 256 ? 2 : 1)) fmc_batch_kernel(BatchLaunch L,
                                                                                           int tab_stride) {
  BatchSmem& B = batch_smem();
  ChainDev& C = B.C;
  MoveSmem& M = B.M;
  SysConst& Ysm = B.Y;
  DevSystem& S = Ysm.S;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((int)blockIdx.x >= L.nchains) return;
  const int cidx = L.order ? L.order[blockIdx.x] : (int)blockIdx.x;  // the chain this CTA runs
  if (!L.chains[cidx].active) return;
  const long long t_start = L.timing && tid == 0 ? global_ns() : 0;
  {
    const int* src = reinterpret_cast<const int*>(&L.chains[cidx]);
    int* dst = reinterpret_cast<int*>(&C);
    for (int i = tid; i < (int)(sizeof(ChainDev) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  {
    const int* src = reinterpret_cast<const int*>(&L.systems[C.sys]);
    int* dst = reinterpret_cast<int*>(&Ysm);
    for (int i = tid; i < (int)(sizeof(SysConst) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const SysConst& Y = Ysm;
  const int K = S.K, kmax_smem = L.kmax_smem;
  const int nt1 = S.ntypes + 1;
  // the offset of each pair's vdW row in the tables, 0 for pairs without one (row 0 is none's)
  for (int i = tid; i < nt1 * nt1; i += blockDim.x) B.prow[i] = max(S.pair_row[i], 0) * S.tab_stride;
  const BatchArrays A = batch_arrays(kmax_smem);
  double2 *const Sk = A.Sk, *const Sn = A.Sn, *const tab = A.tab;
  for (int k = tid; k < K; k += blockDim.x) {
    Sk[k] = C.sk[k];
    A.ak[k] = S.akk[k];
    A.kp[k] = S.kpack[k];
  }
  const int stride = S.kmax[0] + S.kmax[1] + S.kmax[2] + 3;
  (void)tab_stride;
  __syncthreads();
  long long t0 = 0, t1 = 0;
  constexpr bool prof = kProf;
  // a chain ends after the move on which its deck's equilibration + production budget ran
  // out (the reference's do-while(lgchk) loop, gcmc.f:589-736), or at its move budget
  long long nmoves = C.lgchk ? L.moves : 0;
  if (C.budget > 0) nmoves = min(nmoves, C.budget - C.moves_done);
  MoveRecord* trace = L.trace ? L.trace + (size_t)cidx * L.moves : nullptr;
  if (tid < kMaxGuestTypes) B.st_nmol[tid] = C.nmol[tid];
  __syncthreads();
  bool undone = false;  // the last trip's bookkeeping is still to be done
  bool second = false;  // the last trip was the first half of a multi-jump; the move goes on
  int skip = 0;         // the last acceptance test took a draw
  int par = 0;
  for (int mv = 0; mv < nmoves;) {
    MoveCtl& T = B.ctl[par];
    if (prof && tid == 0) t0 = clock64();
    // ---- set-up, four warps side by side: 0 draws, selects and builds the trial; 1 finishes the last
    // move and begins this one (the order of gcmc.f:589-736); 2 builds the phase tables from warp
    // 0's sites; 3 the tail correction from warp 0's counts.  Named barriers 1 and 2 are warp 0's
    // signals that the selection and the sites are there.
    if (warp == 0) {
      select_move(par, skip, second, lane);
      if (prof && lane == 0) C.prof[7] += clock64() - t0;
      asm volatile("bar.arrive 1, 96;" ::: "memory");
      if (prof && lane == 0) t1 = clock64();
      build_trial(lane);
      if (prof && lane == 0) C.prof[8] += clock64() - t1;
    } else if (warp == 1) {
      if (undone) finish_move(trace, lane);
      if (lane == 0 && !second) {
        C.gcmccount++;
        if (C.gcmccount % 400 == 0) check400();
      }
      __syncwarp();
      asm volatile("bar.sync 1, 96;" ::: "memory");
      if (lane == 0) {
        T.elrc = C.elrc;
        T.mj_estep = M.mj_estep;
        // energy_eval's factor (utility_pack.f:3049-3095) of exp(-beta dE)
        const double press = C.press[T.g];
        const bool ins = T.mtype == kInsert;
        const double vp = Y.statvolm * press, nt = (T.nmols + (ins ? 1 : 0)) * kBoltz * C.temp;
        T.pref = (ins ? vp : nt) / (ins ? nt : vp);
        T.free_delete = fabs(press) < 1e-7;
      }
    } else if (warp == 2) {
      asm volatile("bar.sync 2, 64;" ::: "memory");
      build_phases(B, tab, stride, lane);
    } else if (warp == 3) {
      asm volatile("bar.sync 1, 96;" ::: "memory");
      if (T.need_lrc) lrc_warp(B, M, T.g, T.mtype == kInsert ? 1 : -1, T.lrc, lane);
    }
    undone = false;
    __syncthreads();
    if (prof && tid == 0) {
      t1 = clock64();
      C.prof[0] += t1 - t0;
      t0 = t1;
    }
    if (C.status) {
      if (tid == 0) {  // the move that could not be tried was still counted
        if (T.mtype == kInsert) C.ins_count++;
        else if (T.mtype == kDelete) C.del_count++;
        else if (T.mtype == kJump || T.mj_stage == 1) C.jump_count++;
      }
      skip = 0;
      break;
    }
    // read before the sums: the bookkeeping of this move may change them while slow warps commit
    const bool last = !C.lgchk, store = Y.nplots && C.production;
    sums<NT, KPT, CPT>(S, kmax_smem, stride);
    if (prof && tid == 0) C.prof[6] += clock64() - t0;
    __syncthreads();
    if (prof && tid == 0) {
      t1 = clock64();
      C.prof[2] += t1 - t0;
      t0 = t1;
    }
    // ---- acceptance, by every thread from the warps' sums: no barrier before the commit
    const int mtype = T.mtype, g = T.g, mj_stage = T.mj_stage;
    bool accepted, drawn;
    {
      double v0 = 0.0, v1 = 0.0, v2 = 0.0;
#pragma unroll
      for (int w = 0; w < NT / 32; w++) {
        v0 += B.red[3 * w];
        v1 += B.red[3 * w + 1];
        v2 += B.red[3 * w + 2];
      }
      double ewld1, ewld3, delrc, e;
      assemble(Y, T, v0, v1, v2, ewld1, ewld3, delrc, e);
      accepted = decide(C.beta, T, e, drawn);
      if (tid == 32) {
        MoveDone& D = B.done;
        D.mtype = mtype;
        D.g = g;
        D.randchoice = T.randchoice;
        D.accepted = accepted;
        D.mj_stage = mj_stage;
        D.mv = mv;
        D.ewld1 = ewld1;
        D.ewld2 = v1;
        D.ewld3 = ewld3;
        D.vdw = v2;
        D.delrc = delrc;
        D.estep = e;
        D.rande = drawn ? T.rande : -1.0;
      }
    }
    skip = drawn;
    second = mj_stage == 1;
    undone = true;
    par ^= 1;
    if (prof && tid == 0) {
      t1 = clock64();
      C.prof[3] += t1 - t0;
      t0 = t1;
    }
    // ---- commit: every thread its own k-vectors, warp 0 the guest sites and the counts it reads
    if (second)  // park S(k) before the first jump of a multi-jump is committed
#pragma unroll 1
      for (int k = tid; k < K; k += NT) C.sk[k] = Sk[k];
    if (mj_stage == 2 && !accepted)  // rejected multi-jump: S(k) as it was
#pragma unroll 1
      for (int k = tid; k < K; k += NT) Sk[k] = C.sk[k];
    if (accepted)
#pragma unroll 1
      for (int k = tid; k < K; k += NT) Sk[k] = Sn[k];
    if (accepted && mtype == kDelete) {
      const int ns = T.ns, lo = T.lo, end = T.seg_end;
      for (int base = lo; base < end - ns; base += NT) {
        int i = base + tid;
        bool act = i < end - ns;
        double4 a = make_double4(0, 0, 0, 0);
        int t = 0;
        if (act) {
          a = C.gsite[i + ns];
          t = C.gtype[i + ns];
        }
        __syncthreads();
        if (act) {
          C.gsite[i] = a;
          C.gtype[i] = t;
        }
        __syncthreads();
      }
    }
    if (warp == 0) commit_control(T, accepted, lane);
    if (store && !second) {  // every production move (gcmc.f:1929-1931)
      __syncthreads();
      prob_store(Y, C);
    }
    if (prof && tid == 0) C.prof[4] += clock64() - t0;
    if (second) continue;
    if (last) break;
    mv++;
  }
  if (warp == 1 && undone) finish_move(trace, lane);
  if (tid == 0 && skip) duni_next(C.rng);
  __syncthreads();
  for (int k = tid; k < K; k += blockDim.x) C.sk[k] = Sk[k];
  if (tid == 0 && L.retire_finished && ((C.budget > 0 && C.moves_done >= C.budget) || !C.lgchk || C.status))
    C.active = 0;
  __syncthreads();
  {
    const int* src = reinterpret_cast<const int*>(&C);
    int* dst = reinterpret_cast<int*>(&L.chains[cidx]);
    for (int i = tid; i < (int)(sizeof(ChainDev) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
  }
  if (L.timing && tid == 0) {
    unsigned sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    L.timing[3 * cidx] = t_start;
    L.timing[3 * cidx + 1] = global_ns();
    L.timing[3 * cidx + 2] = sm;
  }
}

}  // namespace

int batch_smem_bytes(int kmax_K, int tab_sites, int tab_stride) {
  return kBatchSmemBytes + kmax_K * (int)(2 * sizeof(double2) + sizeof(double)) +
         ((kmax_K + 3) & ~3) * (int)sizeof(int) + tab_sites * tab_stride * (int)sizeof(double2);
}

namespace {
using BatchKernel = void (*)(BatchLaunch, int);
// the kernel of each tile of kBatchTiles, in the same order
constexpr BatchKernel kTileKernels[kNumBatchTiles] = {
    fmc_batch_kernel<false, 256, 1, 1>, fmc_batch_kernel<false, 256, 2, 1>, fmc_batch_kernel<false, 256, 1, 2>,
    fmc_batch_kernel<false, 256, 2, 2>, fmc_batch_kernel<false, 128, 1, 1>, fmc_batch_kernel<false, 128, 2, 1>,
    fmc_batch_kernel<false, 128, 1, 2>, fmc_batch_kernel<false, 128, 2, 2>, fmc_batch_kernel<false, 384, 1, 1>,
    fmc_batch_kernel<false, 384, 2, 1>, fmc_batch_kernel<false, 384, 1, 2>, fmc_batch_kernel<false, 384, 2, 2>};
constexpr BatchKernel kProfKernel = fmc_batch_kernel<true, 256, 1, 1>;
}  // namespace

// The dynamic shared-memory limit belongs to the kernel, shared by every batch and server of the
// process on the current device: it only ever rises, so that opening a batch with smaller tables
// cannot make the launches of one opened before it (with larger tables) exceed the limit.
cudaError_t configure_batch_kernel(int smem_bytes) {
  static std::mutex mu;
  static std::map<int, int> limit;  // device -> the limit set on it
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  int& have = limit[dev];
  if (smem_bytes <= have) return cudaSuccess;
  e = cudaFuncSetAttribute(kProfKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  for (int t = 0; t < kNumBatchTiles && e == cudaSuccess; t++)
    e = cudaFuncSetAttribute(kTileKernels[t], cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  if (e == cudaSuccess) have = smem_bytes;
  return e;
}

cudaError_t launch_batch(const BatchLaunch& L, int smem_bytes, int tab_stride, cudaStream_t st) {
  if (L.tile < 0 || L.tile >= kNumBatchTiles || (L.profile && L.tile != 0)) return cudaErrorInvalidValue;
  const BatchKernel k = L.profile ? kProfKernel : kTileKernels[L.tile];
  k<<<L.nchains, kBatchTiles[L.tile].threads, smem_bytes, st>>>(L, tab_stride);
  return cudaGetLastError();
}

}  // namespace fmc
