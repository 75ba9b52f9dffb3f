// FP64 kernels of the plain (one trial per launch) GPU path.
//
// fmc_pass_kernel   : one launch per trial move.  Blocks [0, nbk) compute the reciprocal
//                     change over all K k-vectors (ewald1_guest, ewald.f:32-365): per-site
//                     axis phase tables in shared memory, one k-vector per thread, S_new to
//                     scratch, akk*(|S_new|^2-|S_old|^2) reduced per block.  Blocks [nbk, ...)
//                     compute the real-space erfc Coulomb + tabulated vdW energy of one
//                     trial site each (ewald2 + srfrce over the neighbour set that
//                     guestlistgen would build).  Each block puts its sums, stamped, into pinned
//                     host memory; the host adds them in block order (deterministic).
// fmc_commit_kernel : S(k) <- S_new and the guest-site array update of an accepted move.
// fmc_recip_*       : full S(k) of a set of atoms (ewald1, ewald.f:368-630).
// fmc_sp_kernel     : per-guest-site real-space energies for the single-point energy.
// fmc_voxel_kernel  : the framework's per-voxel neighbour lists.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <type_traits>
#include <vector>

#include "fmc_device.cuh"
#include "fmc_kernels.h"

namespace fmc {

constexpr int kPassThreads = 256;

// A guest-site update by one block (all its threads): a delete removes [lo, lo+ns) and shifts
// the rest of the segment down in order; an insert writes at the segment end, a displacement
// over the molecule.
__device__ __forceinline__ void apply_commit(const PendingCommit& P, double4* site, int* type) {
  const int tid = threadIdx.x;
  if (P.op == kDelete) {
    const int ns = P.ns;
    for (int base = P.lo; base < P.seg_end - ns; base += blockDim.x) {
      const int i = base + tid;
      const bool act = i < P.seg_end - ns;
      double4 a = make_double4(0.0, 0.0, 0.0, 0.0);
      int t = 0;
      if (act) {
        a = site[i + ns];
        t = type[i + ns];
      }
      __syncthreads();
      if (act) {
        site[i] = a;
        type[i] = t;
      }
      __syncthreads();
    }
  } else if (tid < P.ns) {
    site[P.lo + tid] = P.site[tid];
    type[P.lo + tid] = P.type[tid];
  }
}

// ------------------------------------------------------------------------------ pass
struct PassSmem {
  double red[32 * 2];
  int prow[256];  // the vdW row's offset of the block's site with each type (at most 255 types)
  bool am_last;
};

// A word pair to pinned memory in one store.
__device__ __forceinline__ void publish(double* p, double a, double b) {
  asm volatile("st.volatile.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(a), "d"(b) : "memory");
}

// One block's share of a trial pass (block `blk` of `nblocks`): blocks [0, nbk) the reciprocal
// change of 256 k-vectors each, the next nsite blocks the real-space energy of one trial site each
// (further blocks idle).  Each writes its energy, stamped with the pass's number, to its own words of
// pinned memory, from which the host adds them up in order.  Where a guest-site update is pending
// (or `ticket` asks for it) the last block to finish then writes the update, every block having read
// the sites.  Returns (to every thread) whether this block was the last of a counted pass.
//
// A pass is one trial of one chain, some twenty blocks: it lasts as long as its chain of dependent reads.
// So what a block needs is read as early as its address is known -- the host finds each site's voxel
// list, a reciprocal block reads its k-vectors before it builds the phases, a real-space block its first
// candidates before the row offsets are there -- and nothing is combined on the device: a ticket with
// its fences took 0.8 us, reading the partials back and ordering the result behind them 1.2 us, of a
// kernel of 5 us (3,392 atoms, K = 4192); the stamp says on its own that a block's words have arrived.
template <class Args>
__device__ __forceinline__ bool pass_block(const DevSystem& S, const GuestView& G, const Args& A, const double2* sk,
                                           double2* sk_new, const PassScratch& W, int blk, int nblocks,
                                           double2* sm_tab, PassSmem& sm, bool ticket) {
  const int nsite = A.nold + A.nnew;
  const int nbk = A.nbk;
  const int tid = threadIdx.x;
  if (blk < nbk) {
    // ---- reciprocal space
    const int k1 = S.kmax[0], k2 = S.kmax[1], k3 = S.kmax[2];
    const int stride = (k1 + 1) + (k2 + 1) + (k3 + 1);
    const int k = blk * blockDim.x + tid;
    int kp = 0;
    double2 so = make_double2(0.0, 0.0);
    double ak = 0.0;
    if (k < S.K) {
      kp = S.kpack[k];
      so = sk[k];
      ak = S.akk[k];
    }
    for (int w = tid; w < nsite * 3; w += blockDim.x) {
      int s = w / 3, ax = w % 3;
      double f[3];
      frac_coords(S.cell, A.x[s], A.y[s], A.z[s], f);
      double2* t = sm_tab + s * stride + (ax == 0 ? 0 : (ax == 1 ? k1 + 1 : k1 + k2 + 2));
      axis_phases(f[ax], S.kmax[ax], t);
    }
    __syncthreads();
    double v[1] = {0.0};
    if (k < S.K) {
      int l, m, n;
      kunpack(kp, l, m, n);
      int am = m < 0 ? -m : m, an = n < 0 ? -n : n;
      // the arithmetic is fixed, fma by fma, and the old and new sites' terms are summed apart: S(k) goes through
      // every accepted move, and its last bits decide the moves whose energy change is rounding alone (plain_dist2)
      const int mneg = m & 0x80000000, nneg = n & 0x80000000;
      double ax = 0.0, ay = 0.0, bx = 0.0, by = 0.0;  // the old sites' sum goes to b once it is complete
#pragma unroll 3
      for (int s = 0; s < nsite; s++) {
        const double2* t = sm_tab + s * stride;
        const double2 e1 = t[l], e2 = t[k1 + 1 + am], e3 = t[k1 + k2 + 2 + an];
        const double q = A.q[s], y2 = __hiloint2double(__double2hiint(e2.y) ^ mneg, __double2loint(e2.y)),
                     y3 = __hiloint2double(__double2hiint(e3.y) ^ nneg, __double2loint(e3.y));
        const double px = fma(e1.x, e2.x, -(e1.y * y2)), py = fma(e1.y, e2.x, e1.x * y2);
        const double cp = fma(px, y3, py * e3.x), cm = fma(py, e3.x, px * y3);
        ax = fma(q, fma(px, e3.x, -(py * y3)), ax);
        ay = fma(q, nneg ? cm : cp, ay);
        if (s == A.nold - 1) {
          bx = ax;
          by = ay;
          ax = ay = 0.0;
        }
      }
      const double2 sn = make_double2((so.x - bx) + ax, (so.y - by) + ay);
      sk_new[k] = sn;
      v[0] = ak * fma(-so.y, so.y, fma(-so.x, so.x, fma(sn.x, sn.x, sn.y * sn.y)));
    }
    block_sum<1>(v, sm.red);
    if (tid == 0) publish(W.recip_slot(blk), v[0], pass_stamp(A.seq, v[0], 0.0));
  } else if (A.do_real && blk - nbk < nsite) {
    // ---- real space of one trial site
    const int s = blk - nbk;
    double v[2] = {0.0, 0.0};
    double ec_fw = 0.0, ev_fw = 0.0, ec_g = 0.0, ev_g = 0.0;
    const int row = tid <= S.ntypes ? max(S.pair_row[A.type[s] * (S.ntypes + 1) + tid], 0) * S.tab_stride : 0;
    auto rows = [&]() {
      if (tid <= S.ntypes) sm.prow[tid] = row;
      __syncthreads();
    };
    const int kind = pair_kind(S);
    auto pairs = [&](auto k) {
      site_pairs<decltype(k)::value>(S, G, A.pc, sm.prow, A.x[s], A.y[s], A.z[s], A.q[s], A.vb[s], A.vl[s], A.ex_lo,
                                     A.ex_hi, tid, blockDim.x, rows, ec_fw, ev_fw, ec_g, ev_g);
    };
    if (kind == kPairOrtho) pairs(std::integral_constant<int, kPairOrtho>());
    else if (kind == kPairTriclinic) pairs(std::integral_constant<int, kPairTriclinic>());
    else pairs(std::integral_constant<int, kPairGeneral>());
    v[0] = ec_g + ec_fw;
    v[1] = ev_g + ev_fw;
    block_sum<2>(v, sm.red);
    if (tid == 0) {
      publish(W.site_slot(s), v[0], v[1]);
      publish(W.site_slot(s) + 2, pass_stamp(A.seq, v[0], v[1]), 0.0);
    }
  }
  if (!ticket && !A.pc.op) return false;
  if (tid == 0) {
    // every thread's reads and writes of this pass come before the count (block_sum's barriers, or no
    // work at all), the update after it
    unsigned done;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(done) : "l"(W.counter) : "memory");
    sm.am_last = done == (unsigned)nblocks - 1;
    if (sm.am_last) *W.counter = 0u;
  }
  __syncthreads();
  if (!sm.am_last) return false;
  if (A.pc.op) apply_commit(A.pc, W.gsite, W.gtype);
  return true;
}

template <int N>
__global__ void __launch_bounds__(kPassThreads, 1) fmc_pass_kernel(DevSystem S, GuestView G, PassArgsT<N> A,
                                                                const double2* __restrict__ sk, double2* sk_new,
                                                                PassScratch W) {
  extern __shared__ double2 sm_tab[];
  __shared__ PassSmem sm;
  pass_block(S, G, A, sk, sk_new, W, (int)blockIdx.x, (int)gridDim.x, sm_tab, sm, false);
}

// ------------------------------------------------------------------------------ resident pass
// Every wait of the resident kernel is bounded on the device clock (%globaltimer, ns): block 0
// ends the kernel after `idle_ns` without a pass (the host passes the limit); the other blocks
// wait for block 0 up to 64 times as long, and for the previous pass's update up to kDoneNs:
// past either limit a block records why in host_words[1] and ends.
constexpr unsigned long long kDoneNs = 1000000000ULL;

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__global__ void __launch_bounds__(kPassThreads) fmc_pass_server_kernel(DevSystem S, const PassMailbox* mb,
                                                                       PassServerFlags* fl, int* host_words,
                                                                       PassScratch W, long long seq0,
                                                                       long long idle_ns) {
  extern __shared__ double2 sm_tab[];
  __shared__ PassSmem sm;
  __shared__ long long s_cmd;
  __shared__ PassArgsT<kSmallPassSites> A;
  __shared__ GuestView G;
  __shared__ const double2* s_sk;
  __shared__ double2* s_sk_new;
  const int tid = threadIdx.x;
  const bool leader = blockIdx.x == 0;
  long long seq = seq0;
  for (;;) {
    if (tid == 0) {
      // block 0 polls the mailbox in host memory, the other blocks block 0's flag in device memory
      const volatile long long* cmd = &mb->cmd;
      const volatile unsigned long long* go = &fl->go;
      const unsigned long long limit = (unsigned long long)(leader ? idle_ns : 64 * idle_ns);
      const unsigned long long t0 = now_ns();
      long long c = -1;
      for (;;) {
        c = leader ? *cmd : (long long)*go;
        if (c > seq) break;
        if (leader ? *(const volatile int*)&mb->quit != 0 : *(volatile int*)&fl->stop != 0) {
          c = -1;
          break;
        }
        if (now_ns() - t0 >= limit) {
          if (!leader) atomicExch(host_words + 1, 1);
          c = -1;
          break;
        }
        __nanosleep(leader ? 64 : 32);
      }
      if (c > seq) {
        // the previous pass's guest-site update is written before this pass reads the sites
        const unsigned long long t1 = now_ns();
        bool late = false;
        while (*(volatile unsigned long long*)&fl->done < (unsigned long long)(c - 1)) {
          if (now_ns() - t1 >= kDoneNs) {
            late = true;
            break;
          }
          __nanosleep(32);
        }
        if (late) {
          atomicExch(host_words + 1, 2);
          c = -1;
        }
      }
      if (c < 0 && leader) {
        *(volatile int*)&fl->stop = 1;
        __threadfence();
      }
      s_cmd = c;
    }
    __syncthreads();
    const long long c = s_cmd;
    if (c < 0) break;
    // the pass into shared memory: block 0 from the mailbox (host memory), which it then copies
    // to device memory for the others; the others from there
    {
      const volatile unsigned long long* src =
          reinterpret_cast<const volatile unsigned long long*>(leader ? (const void*)&mb->A : (const void*)&fl->A);
      unsigned long long* dst = reinterpret_cast<unsigned long long*>(&A);
      for (int i = tid; i < (int)(sizeof(A) / 8); i += blockDim.x) dst[i] = src[i];
      const volatile unsigned long long* gs =
          reinterpret_cast<const volatile unsigned long long*>(leader ? (const void*)&mb->G : (const void*)&fl->G);
      unsigned long long* gd = reinterpret_cast<unsigned long long*>(&G);
      for (int i = tid; i < (int)(sizeof(G) / 8); i += blockDim.x) gd[i] = gs[i];
      if (tid == 0) {
        s_sk = leader ? *(const double2* const volatile*)&mb->sk : *(const double2* const volatile*)&fl->sk;
        s_sk_new = leader ? *(double2* const volatile*)&mb->sk_new : *(double2* const volatile*)&fl->sk_new;
      }
    }
    __syncthreads();
    if (leader) {
      unsigned long long* dA = reinterpret_cast<unsigned long long*>(&fl->A);
      const unsigned long long* sA = reinterpret_cast<const unsigned long long*>(&A);
      for (int i = tid; i < (int)(sizeof(A) / 8); i += blockDim.x) dA[i] = sA[i];
      unsigned long long* dG = reinterpret_cast<unsigned long long*>(&fl->G);
      const unsigned long long* sG = reinterpret_cast<const unsigned long long*>(&G);
      for (int i = tid; i < (int)(sizeof(G) / 8); i += blockDim.x) dG[i] = sG[i];
      if (tid == 0) {
        fl->sk = s_sk;
        fl->sk_new = s_sk_new;
      }
      __threadfence();
      __syncthreads();
      if (tid == 0) *(volatile unsigned long long*)&fl->go = (unsigned long long)c;
    }
    const bool last = pass_block(S, G, A, s_sk, s_sk_new, W, (int)blockIdx.x, (int)gridDim.x, sm_tab, sm,
                                 true);
    if (last) {
      __syncthreads();  // the update is written by every thread of this block
      if (tid == 0) {
        __threadfence();
        *(volatile unsigned long long*)&fl->done = (unsigned long long)c;
      }
    }
    seq = c;
    __syncthreads();
  }
  // the last block to end tells the host
  if (tid == 0) {
    __threadfence();
    const unsigned n = atomicAdd(&fl->exit_count, 1u);
    if (n == gridDim.x - 1) {
      __threadfence_system();
      *(volatile int*)host_words = 1;
    }
  }
}

int pass_server_blocks(const DevSystem& S) { return pass_recip_blocks(S) + kServerBlocksExtra; }

cudaError_t launch_pass_server(const DevSystem& S, PassMailbox* mb, PassServerFlags* fl, int* host_words,
                               const PassScratch& W, long long seq0, long long idle_ns, cudaStream_t st) {
  static_assert(sizeof(PassArgsT<kSmallPassSites>) % 8 == 0 && sizeof(GuestView) % 8 == 0, "word copies");
  const int grid = pass_server_blocks(S);
  const int smem = pass_smem_bytes(S, kSmallPassSites);
  void* args[] = {(void*)&S, (void*)&mb, (void*)&fl, (void*)&host_words, (void*)&W, (void*)&seq0, (void*)&idle_ns};
  return cudaLaunchCooperativeKernel((const void*)fmc_pass_server_kernel, grid, kPassThreads, args, smem, st);
}

int pass_smem_bytes(const DevSystem& S, int nsite) {
  return nsite * ((S.kmax[0] + 1) + (S.kmax[1] + 1) + (S.kmax[2] + 1)) * (int)sizeof(double2);
}

int pass_recip_blocks(const DevSystem& S) { return (S.K + kPassThreads - 1) / kPassThreads; }

cudaError_t launch_pass(const DevSystem& S, const GuestView& G, const PassArgs& A, const double2* sk, double2* sk_new,
                        const PassScratch& W, cudaStream_t st) {
  int nsite = A.nold + A.nnew;
  int smem = A.nbk > 0 ? pass_smem_bytes(S, nsite) : 0;
  int grid = A.nbk + (A.do_real ? nsite : 0);
  if (grid == 0) return A.pc.op ? cudaErrorInvalidValue : cudaSuccess;  // a pending update needs a block
  if (nsite <= kSmallPassSites) {
    // the common case (molecules of up to 8 sites): a parameter block of ~1.3 KB instead of ~4 KB
    PassArgsT<kSmallPassSites> B;
    std::memcpy(&B, &A, offsetof(PassArgs, x));
    for (int i = 0; i < nsite; i++) {
      B.x[i] = A.x[i];
      B.y[i] = A.y[i];
      B.z[i] = A.z[i];
      B.q[i] = A.q[i];
      B.type[i] = A.type[i];
      B.vb[i] = A.vb[i];
      B.vl[i] = A.vl[i];
    }
    B.pc = A.pc;
    fmc_pass_kernel<kSmallPassSites><<<grid, kPassThreads, smem, st>>>(S, G, B, sk, sk_new, W);
  } else {
    fmc_pass_kernel<kMaxPassSites><<<grid, kPassThreads, smem, st>>>(S, G, A, sk, sk_new, W);
  }
  return cudaGetLastError();
}

cudaError_t configure_kernels() {
  cudaError_t e = cudaFuncSetAttribute(fmc_pass_kernel<kSmallPassSites>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       200 * 1024);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(fmc_pass_server_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(fmc_pass_kernel<kMaxPassSites>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  return e;
}


// ------------------------------------------------------------------------------ commit
__global__ void fmc_commit_kernel(int K, double2* sk, const double2* __restrict__ sk_new, CommitArgs C,
                                  double4* site, int* type) {
  if ((int)blockIdx.x < (int)gridDim.x - 1) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += (gridDim.x - 1) * blockDim.x) sk[k] = sk_new[k];
    return;
  }
  // last block: guest-site segment update
  const int tid = threadIdx.x;
  if (C.op == kDelete) {
    // remove [lo, lo+ns) and shift the rest of the segment down, preserving order
    const int ns = C.ns;
    for (int base = C.lo; base < C.seg_end - ns; base += blockDim.x) {
      int i = base + tid;
      double4 a;
      int t = 0;
      bool act = i < C.seg_end - ns;
      if (act) {
        a = site[i + ns];
        t = type[i + ns];
      }
      __syncthreads();
      if (act) {
        site[i] = a;
        type[i] = t;
      }
      __syncthreads();
    }
  } else if (tid < C.ns) {
    // insert writes at the segment end, displace overwrites the molecule
    site[C.lo + tid] = make_double4(C.x[tid], C.y[tid], C.z[tid], C.q[tid]);
    type[C.lo + tid] = C.type[tid];
  }
}

cudaError_t launch_commit(int K, double2* sk, const double2* sk_new, const CommitArgs& C, double4* site, int* type,
                          cudaStream_t st) {
  int nb = (K + 255) / 256;
  if (nb > 64) nb = 64;
  fmc_commit_kernel<<<nb + 1, 256, 0, st>>>(K, sk, sk_new, C, site, type);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------ full S(k)
// partial[c*K + k] = sum over the atoms of chunk c (in order) of q e^{i k.r}, the chunks then added in
// order: one fixed order of additions, on which the last bits of S(k) depend.
//
// Two forms with the same bits (products are written as the compiler contracted the plain expressions):
//
// fmc_recip_octet_kernel: a thread takes the k-vectors (l, +-m, +-n) and (l, +-m, +-n') of two |n|
// (S.koct): one read each of the three axes' phases serves all eight, and e^{i(lx +- my)} is formed
// once for four of them.  128-bit shared reads cost four cycles an SM whatever they hit, so one
// k-vector a thread is bound by them (12 cycles of reads a k-vector and warp against 5 of FP64); here
// two cycles of reads against 3.5 of FP64.
//
// fmc_recip_single_kernel: one k-vector a thread, for the sizes whose octets would leave SMs idle.
constexpr int kOctetThreads = 128, kSingleThreads = 256;

// Phase tables and charges of a chunk's atoms.
__device__ __forceinline__ void recip_phases(const DevSystem& S, const AtomSegs& atoms, int a0, int na, int stride,
                                             double2* tab, double* sq) {
  const int k1 = S.kmax[0], k2 = S.kmax[1];
  for (int w = threadIdx.x; w < na * 3; w += blockDim.x) {
    int s = w / 3, ax = w % 3, i = a0 + s;
    const double4* p = atoms.p[0];
#pragma unroll
    for (int g = 1; g <= kMaxGuestTypes; g++)
      if (i >= atoms.begin[g]) p = atoms.p[g] - atoms.begin[g];
    double4 a = p[i];
    double f[3];
    frac_coords(S.cell, a.x, a.y, a.z, f);
    double2* t = tab + s * stride + (ax == 0 ? 0 : (ax == 1 ? k1 + 1 : k1 + k2 + 2));
    axis_phases(f[ax], S.kmax[ax], t);
    if (ax == 0) sq[s] = a.w;
  }
  __syncthreads();
}

// acc += q e^{i(lx + my)} e3, e3 conjugated for n < 0.
template <bool kMinus>
__device__ __forceinline__ void recip_add(double px, double py, double2 e3, double q, double2& acc) {
  const double cx = kMinus ? fma(px, e3.x, py * e3.y) : fma(px, e3.x, -(py * e3.y));
  const double cy = kMinus ? fma(py, e3.x, -(e3.y * px)) : fma(e3.y, px, py * e3.x);
  acc.x = fma(q, cx, acc.x);
  acc.y = fma(q, cy, acc.y);
}

__global__ void __launch_bounds__(kOctetThreads) fmc_recip_octet_kernel(DevSystem S, AtomSegs atoms, int natoms,
                                                                        int chunk, double2* partial) {
  extern __shared__ double2 sm_tab[];
  __shared__ double sq[256];
  const int k1 = S.kmax[0], k2 = S.kmax[1], stride = k1 + k2 + S.kmax[2] + 3;
  const int c = blockIdx.y, a0 = c * chunk, na = min(chunk, natoms - a0);
  recip_phases(S, atoms, a0, na, stride, sm_tab, sq);
  const int run = blockIdx.x * blockDim.x + threadIdx.x;
  if (run >= S.noct) return;
  const KOctet& oct = S.koct[run];
  const double2 *t1 = sm_tab + oct.l, *t2 = sm_tab + k1 + 1 + oct.m, *t3 = sm_tab + k1 + k2 + 2 + oct.n[0],
                *t4 = sm_tab + k1 + k2 + 2 + oct.n[1];
  double2 acc[8];
#pragma unroll
  for (int i = 0; i < 8; i++) acc[i] = make_double2(0.0, 0.0);
  for (int s = 0; s < na; s++) {
    const int o = s * stride;
    const double2 e1 = t1[o], e2 = t2[o], e3 = t3[o], e4 = t4[o];
    const double q = sq[s];
    const double px = fma(e1.x, e2.x, -(e1.y * e2.y)), py = fma(e1.y, e2.x, e2.y * e1.x);
    const double mx = fma(e1.x, e2.x, e1.y * e2.y), my = fma(e1.y, e2.x, -(e2.y * e1.x));
    recip_add<false>(px, py, e3, q, acc[0]);
    recip_add<true>(px, py, e3, q, acc[1]);
    recip_add<false>(mx, my, e3, q, acc[2]);
    recip_add<true>(mx, my, e3, q, acc[3]);
    recip_add<false>(px, py, e4, q, acc[4]);
    recip_add<true>(px, py, e4, q, acc[5]);
    recip_add<false>(mx, my, e4, q, acc[6]);
    recip_add<true>(mx, my, e4, q, acc[7]);
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int k = oct.k[i];
    if (k >= 0) partial[(size_t)c * S.K + k] = acc[i];
  }
}

__global__ void __launch_bounds__(kSingleThreads) fmc_recip_single_kernel(DevSystem S, AtomSegs atoms, int natoms,
                                                                          int chunk, double2* partial) {
  extern __shared__ double2 sm_tab[];
  __shared__ double sq[256];
  const int k1 = S.kmax[0], k2 = S.kmax[1], stride = k1 + k2 + S.kmax[2] + 3;
  const int c = blockIdx.y, a0 = c * chunk, na = min(chunk, natoms - a0);
  recip_phases(S, atoms, a0, na, stride, sm_tab, sq);
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= S.K) return;
  int l, m, n;
  kunpack(S.kpack[k], l, m, n);
  const double2 *t1 = sm_tab + l, *t2 = sm_tab + k1 + 1 + (m < 0 ? -m : m),
                *t3 = sm_tab + k1 + k2 + 2 + (n < 0 ? -n : n);
  const int mneg = m & 0x80000000;
  const bool nneg = n < 0;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int s = 0; s < na; s++) {
    const int o = s * stride;
    const double2 e1 = t1[o], e2 = t2[o], e3 = t3[o];
    const double y2 = __hiloint2double(__double2hiint(e2.y) ^ mneg, __double2loint(e2.y));
    const double px = fma(e1.x, e2.x, -(e1.y * y2)), py = fma(e1.y, e2.x, y2 * e1.x);
    double2 a = acc, b = acc;
    recip_add<false>(px, py, e3, sq[s], a);
    recip_add<true>(px, py, e3, sq[s], b);
    acc.x = nneg ? b.x : a.x;
    acc.y = nneg ? b.y : a.y;
  }
  partial[(size_t)c * S.K + k] = acc;
}

// S[k] = sum_c partial[c][k] in order; energy sum akk |S|^2 per block into part[].  Bound by the latency
// of its reads: blocks of 32 k-vectors spread a few thousand of them over the SMs, and sixteen chunks
// are read before they are added.
constexpr int kRecipReduce = 32;

__global__ void __launch_bounds__(kRecipReduce) fmc_recip_reduce_kernel(DevSystem S, const double2* __restrict__ partial,
                                                                        int nchunk, double2* sk, double* part) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0.0;
  if (k < S.K) {
    double2 s = make_double2(0.0, 0.0);
    const double2* p = partial + k;
    int c = 0;
    for (; c + 16 <= nchunk; c += 16) {
      double2 a[16];
#pragma unroll
      for (int u = 0; u < 16; u++) a[u] = __ldcg(p + (size_t)(c + u) * S.K);
#pragma unroll
      for (int u = 0; u < 16; u++) {
        s.x += a[u].x;
        s.y += a[u].y;
      }
    }
    double2 a[15];
#pragma unroll
    for (int u = 0; u < 15; u++)
      if (c + u < nchunk) a[u] = __ldcg(p + (size_t)(c + u) * S.K);
#pragma unroll
    for (int u = 0; u < 15; u++)
      if (c + u < nchunk) {
        s.x += a[u].x;
        s.y += a[u].y;
      }
    sk[k] = s;
    v = S.akk[k] * (s.x * s.x + s.y * s.y);
  }
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
}

int recip_chunk(const DevSystem& S) {
  int stride = (S.kmax[0] + 1) + (S.kmax[1] + 1) + (S.kmax[2] + 1);
  int c = (40 * 1024) / (stride * (int)sizeof(double2));  // + 2 KB static charges < 48 KB
  if (c > 256) c = 256;
  return c < 1 ? 1 : c;
}

size_t recip_scratch_doubles(const DevSystem& S, int natoms) {
  int chunk = recip_chunk(S);
  int nchunk = (natoms + chunk - 1) / chunk;
  return (size_t)nchunk * S.K * 2 + 8;
}

int recip_nparts(const DevSystem& S) { return (S.K + kRecipReduce - 1) / kRecipReduce; }

cudaError_t launch_recip_full(const DevSystem& S, const AtomSegs& atoms, double2* sk, double* scratch, double* parts,
                              cudaStream_t st) {
  const int natoms = atoms.total();
  int chunk = recip_chunk(S);
  int nchunk = (natoms + chunk - 1) / chunk;
  if (nchunk == 0) {
    cudaMemsetAsync(sk, 0, sizeof(double2) * S.K, st);
    return cudaMemsetAsync(parts, 0, sizeof(double) * recip_nparts(S), st);
  }
  int stride = (S.kmax[0] + 1) + (S.kmax[1] + 1) + (S.kmax[2] + 1);
  double2* partial = reinterpret_cast<double2*>(scratch);
  const size_t smem = chunk * stride * sizeof(double2);
  // octets once their blocks give every SM one: below that the launch lasts as long as one thread's
  // atoms, eight times shorter with one k-vector a thread
  const int bx = (S.noct + kOctetThreads - 1) / kOctetThreads;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if ((long long)bx * nchunk >= sms)
    fmc_recip_octet_kernel<<<dim3(bx, nchunk), kOctetThreads, smem, st>>>(S, atoms, natoms, chunk, partial);
  else
    fmc_recip_single_kernel<<<dim3((S.K + kSingleThreads - 1) / kSingleThreads, nchunk), kSingleThreads, smem, st>>>(
        S, atoms, natoms, chunk, partial);
  fmc_recip_reduce_kernel<<<recip_nparts(S), kRecipReduce, 0, st>>>(S, partial, nchunk, sk, parts);
  return cudaGetLastError();
}

cudaError_t configure_recip_kernels() {
  cudaError_t e = cudaFuncSetAttribute(fmc_recip_single_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(fmc_recip_octet_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
  return e;
}

void recip_octets(const int* kpacked, int K, std::vector<KOctet>& out) {
  // quads (l, |m|, |n|) in table order, paired within an (l, |m|)
  struct Quad {
    int l, m, n, k[4];
  };
  std::vector<Quad> quads;
  std::vector<int> at(129 * 129, -1);  // (|m|, |n|) of the present l
  int l0 = -1;
  for (int k = 0; k < K; k++) {
    int l, m, n;
    kunpack(kpacked[k], l, m, n);
    if (l != l0) {
      std::fill(at.begin(), at.end(), -1);
      l0 = l;
    }
    const int am = m < 0 ? -m : m, an = n < 0 ? -n : n;
    int& q = at[am * 129 + an];
    if (q < 0) {
      q = (int)quads.size();
      quads.push_back({l, am, an, {-1, -1, -1, -1}});
    }
    quads[q].k[(m < 0 ? 2 : 0) + (n < 0 ? 1 : 0)] = k;
  }
  std::sort(quads.begin(), quads.end(), [](const Quad& a, const Quad& b) {
    return a.l != b.l ? a.l < b.l : (a.m != b.m ? a.m < b.m : a.n < b.n);
  });
  out.clear();
  for (size_t i = 0; i < quads.size();) {
    size_t e = i;
    while (e < quads.size() && quads[e].l == quads[i].l && quads[e].m == quads[i].m) e++;
    const size_t half = (e - i + 1) / 2;  // n and n + half together, so that neighbours read neighbours
    for (size_t j = 0; j < half; j++) {
      const Quad& a = quads[i + j];
      const bool two = i + j + half < e;
      const Quad& b = two ? quads[i + j + half] : a;
      KOctet o;
      o.l = (short)a.l;
      o.m = (short)a.m;
      o.n[0] = (short)a.n;
      o.n[1] = (short)b.n;
      for (int t = 0; t < 4; t++) {
        o.k[t] = a.k[t];
        o.k[4 + t] = two ? b.k[t] : -1;
      }
      out.push_back(o);
    }
    i = e;
  }
}

double recip_energy_from_parts(const DevSystem& S, const double* host_parts) {
  // 256 k-vectors at a time, whose sums are then added: the order that energies have always had
  double r = 0.0;
  const int n = recip_nparts(S);
  for (int b = 0; b < n;) {
    double s = 0.0;
    for (const int end = std::min(b + 256 / kRecipReduce, n); b < end; b++) s += host_parts[b];
    r += s;
  }
  return S.recip_pref * r;
}

// ------------------------------------------------------------------------------ single point
// Block b: guest site b of the segments in order; out[4*b + {0,1,2,3}] = {coulomb vs framework, vdw vs
// framework, coulomb vs other guests, vdw vs other guests}.
struct MolSites {
  int n[kMaxGuestTypes];  // sites per molecule of each species
};

template <int KIND>
__global__ void __launch_bounds__(256, 2) fmc_sp_kernel(DevSystem S, GuestView G, MolSites mol, double* out) {
  __shared__ double red[32 * 4];
  __shared__ int prow[256];
  int r = blockIdx.x, sg = 0;
  while (r >= G.seg_len[sg]) r -= G.seg_len[sg++];
  const int i = G.seg_off[sg] + r, lo = G.seg_off[sg] + r / mol.n[sg] * mol.n[sg], hi = lo + mol.n[sg];
  const double4 a = G.site[i];
  if ((int)threadIdx.x <= S.ntypes)
    prow[threadIdx.x] = max(S.pair_row[G.type[i] * (S.ntypes + 1) + threadIdx.x], 0) * S.tab_stride;
  const int v = voxel_of(S, a.x, a.y, a.z), vb = S.vox_off[v], vl = S.vox_off[v + 1] - vb;
  PendingCommit none;
  none.op = 0;
  none.seg = -1;
  none.lo = none.ns = none.seg_end = 0;
  double e[4] = {0.0, 0.0, 0.0, 0.0};
  site_pairs<KIND>(S, G, none, prow, a.x, a.y, a.z, a.w, vb, vl, lo, hi, threadIdx.x, blockDim.x,
                   [] { __syncthreads(); }, e[0], e[1], e[2], e[3]);
  block_sum<4>(e, red);
  if (threadIdx.x == 0)
    for (int k = 0; k < 4; k++) out[4 * blockIdx.x + k] = e[k];
}

cudaError_t launch_single_point_rs(const DevSystem& S, const GuestView& G, const int* nsite, double* out,
                                   cudaStream_t st) {
  MolSites mol;
  int n = 0;
  for (int g = 0; g < kMaxGuestTypes; g++) {
    mol.n[g] = g < G.nseg ? nsite[g] : 1;
    if (g < G.nseg) n += G.seg_len[g];
  }
  if (n == 0) return cudaSuccess;
  const int kind = pair_kind(S);
  if (kind == kPairOrtho) fmc_sp_kernel<kPairOrtho><<<n, 256, 0, st>>>(S, G, mol, out);
  else if (kind == kPairTriclinic) fmc_sp_kernel<kPairTriclinic><<<n, 256, 0, st>>>(S, G, mol, out);
  else fmc_sp_kernel<kPairGeneral><<<n, 256, 0, st>>>(S, G, mol, out);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------ voxel lists
// Every framework atom whose true minimum-image distance to a voxel's centre is below
// sqrt(lim2) (rcut + the voxel's circumradius), in ascending atom order.
__device__ __forceinline__ double true_dist2_dev(const CellGeom& c, double dx, double dy, double dz) {
  if (c.imcon == 4 || c.imcon == 5 || c.imcon == 7) return shifted_lattice_dist2(c, dx, dy, dz);
  if (c.imcon == 6) return slab_dist2(c, dx, dy, dz);
  min_image(c, dx, dy, dz);
  double best = dx * dx + dy * dy + dz * dz;
  if (c.imcon == 3) {
    for (int i = -1; i <= 1; i++)
      for (int j = -1; j <= 1; j++)
        for (int k = -1; k <= 1; k++) {
          double x = dx + i * c.h[0] + j * c.h[3] + k * c.h[6];
          double y = dy + i * c.h[1] + j * c.h[4] + k * c.h[7];
          double z = dz + i * c.h[2] + j * c.h[5] + k * c.h[8];
          best = fmin(best, x * x + y * y + z * z);
        }
  }
  return best;
}

__device__ __forceinline__ void voxel_centre(const CellGeom& c, int v, int n0, int n1, int n2, double* p) {
  int a = v / (n1 * n2), b = (v / n2) % n1, cc = v % n2;
  double fa = (a + 0.5) / n0, fb = (b + 0.5) / n1, fc = (cc + 0.5) / n2;
  if (c.imcon == 6) {  // slab: in-plane cell, z layers from zlo
    p[0] = fa * c.h[0] + fb * c.h[3];
    p[1] = fa * c.h[1] + fb * c.h[4];
    p[2] = c.zlo + (cc + 0.5) * c.dz;
    return;
  }
  p[0] = fa * c.h[0] + fb * c.h[3] + fc * c.h[6];
  p[1] = fa * c.h[1] + fb * c.h[4] + fc * c.h[7];
  p[2] = fa * c.h[2] + fb * c.h[5] + fc * c.h[8];
}

// A warp builds the lists of two consecutive voxels (one where a distance takes up to 27 images), 32 atoms
// at a time: no barriers, and an atom is read once for all of them.  In orthorhombic cells (imcon 1, 2) a
// distance is taken in float first, which decides all but the atoms within `margin` of the limit; those few
// are measured in double, so that the lists hold exactly the atoms of the double test.  The margin, with h
// the longest period and s the largest |atom| + |centre| + h of an axis: rounding the coordinates, their
// difference and n periods moves a separation by at most 3 * 2^-24 s and its square by h times that; where
// it picks the other of two images, the square moves by at most 2^-21 h s.  Three axes: 2.2e-6 h s in all,
// half of the margin.  Atoms 2^16 periods out and further are left to double.
// Bound by instructions issued (a test is some 20, and 3 for the atom's conversions) and, in the fill, by
// stores of the two or so of 32 atoms that are in a list.  5,928 atoms and 28,656 lists: count 238 us, fill 560
// us, against 517 and 1,112 with a block a voxel, a prefilter by voxel and four barriers every 128 atoms;
// 424 atoms: 28 us for both against 30.  Four voxels a warp: 250 and 523 us, but 34 us for 424 atoms; eight:
// 226 and 608, 41.
constexpr int kVoxThreads = 128;

template <bool kOrtho>
constexpr int kVoxPerWarp = kOrtho ? 2 : 1;

struct VoxelCell {  // an orthorhombic cell's side of the float test, converted on the host: conversions are slow
  float h[3], r[3], lim, scale, far;  // scale: 4.4e-6 h; far: 2^16 h, beyond which double decides alone
};

struct VoxelCentre {
  float x, y, z, lo, hi;  // lo, hi: the limit less and plus the margin's part that is not the atom's
  double p[3];
};

// Flags, for each of the warp's voxels, of this lane's atom (live: there is one).
template <bool kOrtho>
__device__ __forceinline__ void voxel_flags(const CellGeom& c, const VoxelCell& f, const double4& a, bool live,
                                            double lim2, const VoxelCentre* t, bool* flag) {
  constexpr int V = kVoxPerWarp<kOrtho>;
  bool open[V], some = false;
  if (kOrtho) {
    constexpr float kRound = 12582912.0f;  // 1.5 * 2^23: adding it rounds to the nearest integer
    const float ax = (float)a.x, ay = (float)a.y, az = (float)a.z;
    const float out = fmaxf(fabsf(ax), fmaxf(fabsf(ay), fabsf(az)));
    const float margin = out < f.far ? f.scale * out : __int_as_float(0x7f800000);
#pragma unroll
    for (int u = 0; u < V; u++) {
      float dx = t[u].x - ax, dy = t[u].y - ay, dz = t[u].z - az;
      dx = fmaf(-f.h[0], fmaf(f.r[0], dx, kRound) - kRound, dx);
      dy = fmaf(-f.h[1], fmaf(f.r[1], dy, kRound) - kRound, dy);
      dz = fmaf(-f.h[2], fmaf(f.r[2], dz, kRound) - kRound, dz);
      const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      flag[u] = live && d2 < t[u].lo - margin;
      open[u] = live && !flag[u] && !(d2 > t[u].hi + margin);
      some = some || open[u];
    }
    if (!__any_sync(0xffffffffu, some)) return;
  } else {
#pragma unroll
    for (int u = 0; u < V; u++) {
      flag[u] = false;
      open[u] = live;
    }
  }
#pragma unroll
  for (int u = 0; u < V; u++)
    if (open[u]) {
      double dx = t[u].p[0] - a.x, dy = t[u].p[1] - a.y, dz = t[u].p[2] - a.z;
      if (kOrtho) {  // true_dist2_dev without its other cells: a quarter of the code
        if (c.imcon == 1) min_image_t<1>(c, dx, dy, dz);
        else min_image_t<2>(c, dx, dy, dz);
        flag[u] = dx * dx + dy * dy + dz * dz < lim2;
      } else {
        flag[u] = true_dist2_dev(c, dx, dy, dz) < lim2;
      }
    }
}

// The lists' lengths (counts), or the lists themselves at off.
template <bool kOrtho, bool kFill>
__global__ void __launch_bounds__(kVoxThreads) fmc_voxel_kernel(CellGeom cell, VoxelCell f, int n0, int n1, int n2,
                                                                const double4* __restrict__ fw,
                                                                const int* __restrict__ ftype, int nf, double lim2,
                                                                int* __restrict__ counts, const int* __restrict__ off,
                                                                int* __restrict__ atoms,
                                                                unsigned short* __restrict__ atoms16,
                                                                double4* __restrict__ xyzq,
                                                                unsigned char* __restrict__ vtype, long long cap) {
  constexpr int V = kVoxPerWarp<kOrtho>;
  const int lane = threadIdx.x & 31, nv = n0 * n1 * n2;
  const int v0 = (blockIdx.x * (kVoxThreads / 32) + (threadIdx.x >> 5)) * V;
  if (v0 >= nv || nf < 1) return;
  VoxelCentre t[V];
  int at[V], end[V];
#pragma unroll
  for (int u = 0; u < V; u++) {
    const int v = min(v0 + u, nv - 1);
    voxel_centre(cell, v, n0, n1, n2, t[u].p);
    t[u].x = (float)t[u].p[0];
    t[u].y = (float)t[u].p[1];
    t[u].z = (float)t[u].p[2];
    const float h = fmaxf(f.h[0], fmaxf(f.h[1], f.h[2]));
    const float margin = f.scale * (h + fmaxf(fabsf(t[u].x), fmaxf(fabsf(t[u].y), fabsf(t[u].z))));
    t[u].lo = f.lim - margin;
    t[u].hi = f.lim + margin;
    at[u] = kFill ? off[v] : 0;
    // beyond the capacity: the caller compares off[nv] with cap and rebuilds
    end[u] = kFill && v0 + u < nv ? (int)min((long long)off[v + 1], cap) : 0;
  }
  double4 a = fw[min(lane, nf - 1)], next = a;
#pragma unroll 1
  for (int base = 0; base < nf; base += 32, a = next) {
    const int j = base + lane;
    const bool live = j < nf;
    next = fw[min(j + 32, nf - 1)];
    bool flag[V];
    voxel_flags<kOrtho>(cell, f, a, live, lim2, t, flag);
    if (!kFill) {
#pragma unroll
      for (int u = 0; u < V; u++) at[u] += flag[u];
      continue;
    }
    const int type = ftype[min(j, nf - 1)];
#pragma unroll
    for (int u = 0; u < V; u++) {
      const unsigned mask = __ballot_sync(0xffffffffu, flag[u]);
      const int pos = at[u] + __popc(mask & ((1u << lane) - 1u));
      at[u] += __popc(mask);
      if (flag[u] && pos < end[u]) {
        if (atoms) atoms[pos] = j;
        if (atoms16) atoms16[pos] = (unsigned short)j;
        xyzq[pos] = a;
        vtype[pos] = (unsigned char)type;
      }
    }
  }
  if (!kFill)
#pragma unroll
    for (int u = 0; u < V; u++) {
      const int n = __reduce_add_sync(0xffffffffu, at[u]);
      if (lane == 0 && v0 + u < nv) counts[v0 + u] = n;
    }
}

namespace {
template <bool kFill>
cudaError_t launch_voxels(const CellGeom& cell, const int* nvox, const double4* fw, const int* ftype, int nf,
                          double lim2, int* counts, const int* off, int* atoms, unsigned short* atoms16, double4* xyzq,
                          unsigned char* vtype, long long cap, cudaStream_t st) {
  const int nv = nvox[0] * nvox[1] * nvox[2], warps = kVoxThreads / 32;
  const bool ortho = cell.imcon == 1 || cell.imcon == 2;
  VoxelCell f = {};
  if (ortho) {
    double h = 0.0;
    for (int a = 0; a < 3; a++) {
      const int i = cell.imcon == 1 ? 0 : a;
      f.h[a] = (float)cell.h[4 * i];
      f.r[a] = (float)cell.inv[i];
      h = std::max(h, std::fabs(cell.h[4 * i]));
    }
    f.lim = (float)lim2;
    f.scale = (float)(4.4e-6 * h);
    f.far = (float)(65536.0 * h);
  }
  const int per = warps * (ortho ? kVoxPerWarp<true> : kVoxPerWarp<false>);
  const auto k = ortho ? fmc_voxel_kernel<true, kFill> : fmc_voxel_kernel<false, kFill>;
  k<<<(nv + per - 1) / per, kVoxThreads, 0, st>>>(cell, f, nvox[0], nvox[1], nvox[2], fw, ftype, nf, lim2, counts, off,
                                                  atoms, atoms16, xyzq, vtype, cap);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_voxel_count(const CellGeom& cell, const int* nvox, const double4* fw, int nf, double lim2,
                               int* counts, cudaStream_t st) {
  if (nf < 1) return cudaMemsetAsync(counts, 0, sizeof(int) * nvox[0] * nvox[1] * nvox[2], st);
  return launch_voxels<false>(cell, nvox, fw, nullptr, nf, lim2, counts, nullptr, nullptr, nullptr, nullptr, nullptr, 0, st);
}

cudaError_t launch_voxel_fill(const CellGeom& cell, const int* nvox, const double4* fw, const int* ftype, int nf,
                              double lim2, const int* off, int* atoms, unsigned short* atoms16, double4* xyzq,
                              unsigned char* vtype, long long cap, cudaStream_t st) {
  return launch_voxels<true>(cell, nvox, fw, ftype, nf, lim2, nullptr, off, atoms, atoms16, xyzq, vtype, cap, st);
}

namespace {
constexpr int kScanThreads = 1024;

// Exclusive prefix sum of n counts into off[0..n] (off[n] = total) by one CTA: each thread sums
// a contiguous chunk, the chunk sums are scanned across the block, then each thread writes its
// chunk's offsets.
__global__ void __launch_bounds__(kScanThreads) fmc_exclusive_scan_kernel(const int* __restrict__ counts, int n,
                                                                          int* __restrict__ off) {
  __shared__ int wsum[kScanThreads / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int chunk = (n + kScanThreads - 1) / kScanThreads;
  const int lo = min(n, t * chunk), hi = min(n, lo + chunk);
  int sum = 0;
  for (int i = lo; i < hi; i++) sum += counts[i];
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = wsum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  int run = incl - sum + (warp ? wsum[warp - 1] : 0);
  for (int i = lo; i < hi; i++) {
    off[i] = run;
    run += counts[i];
  }
  if (t == kScanThreads - 1) off[n] = wsum[kScanThreads / 32 - 1];
}
}  // namespace

namespace {
__global__ void __launch_bounds__(256) fmc_pack_tables_kernel(const double* __restrict__ erc,
                                                              const double* __restrict__ vvv, int stride, int n,
                                                              double2* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = make_double2(erc[i % stride], i < stride ? 0.0 : vvv[i]);
}
}  // namespace

cudaError_t launch_pack_tables(const double* erc, const double* vvv, int stride, int rows, double2* out,
                               cudaStream_t st) {
  const int n = rows * stride;
  if (n > 0) fmc_pack_tables_kernel<<<(n + 255) / 256, 256, 0, st>>>(erc, vvv, stride, n, out);
  return cudaGetLastError();
}

cudaError_t launch_exclusive_scan(const int* counts, int n, int* off, cudaStream_t st) {
  fmc_exclusive_scan_kernel<<<1, kScanThreads, 0, st>>>(counts, n, off);
  return cudaGetLastError();
}

}  // namespace fmc
