// akb_patch.cu -- the fused explicit step (AKB_MODE_FP64, AKB_MODE_FP32_BULK).
//
// k_fan_step (FP64 triangles, tetrahedra, hexahedra: plans on fan records): a
// resident grid over the patches, a fan of elements per thread; described
// below, before its layout.
// k_patch_step (FP32, segments, plans too large for a fan record's shared
// memory): one CTA per patch (akb_patch.cuh for the node order, the
// predicted displacement w and the shared-node protocol).
//   1. stage: thread 0 starts TMA bulk copies of the interior nodes' X and w
//      (two contiguous slices) and of the first chunk records, and prefetches
//      the interior nodes' v, a, 1/M and blocked flags into L2; every thread
//      starts cp.async copies of its shared nodes' X and w and zeroes the
//      force accumulators;
//   2. element forces in chunks of blockDim elements from shared memory
//      (akb_fastmath.cuh), each corner vector written to its contribution
//      slot; one thread per node run adds the run (ascending local element
//      order) to the node's accumulator (the -1 scatter of
//      dof_manager.cc:83-137, without atomics). The record of the next chunk
//      is copied while this one is used (two buffers, when they fit);
//   3. finish: each shared node's partial force goes to its slot; the
//      interior nodes get the residual, lumped solve and corrector
//      (non_linear_solver_lumped.cc:85-98, newmark-beta.cc:176-210) and the
//      next predictor (newmark-beta.cc:60-89), written back as u, v, a and w.
// Every wait on a bulk copy is bounded: past it the CTA flags the error
// (P.err, read by the host on its next synchronisation), waits again (bounded)
// for the copies it issued and stops.
// k_finish_list: one thread per (listed node, component) adds the partials
// of the shared nodes in patch order and finishes them the same way, and the
// nodes of no element (after the exchange between parts, for a partitioned
// mesh).
#include <cfloat>
#include <mutex>

#include "akb_fastmath.cuh"
#include "akb_patch.cuh"

namespace akb {
namespace {

constexpr int kThreads = 256;

struct SmemLayout {
  size_t xs, ws, fs, contrib, sslot, buf, buf_stride, mbar, total;
};

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~size_t(15); }
__host__ __device__ inline size_t align128(size_t x) { return (x + 127) & ~size_t(127); }

// Shared-memory layout: node arrays X and w row-major ([position][i], 16
// bytes of slack in front for the offset of the interior slice), force
// accumulators component-major ([i][position], row stride LM), the chunk's
// element vectors (CH slots, cidx), the partial slot of each shared node
// (SHmax uint32), nbuf chunk record buffers of CB bytes, three mbarriers (two
// record buffers, the node staging).
__host__ __device__ inline SmemLayout layout(int LM, int CH, int CB, int Lmax, int SHmax, int d,
                                             int sbytes, int nbuf) {
  SmemLayout s;
  const size_t nb = align16(16 + (size_t)Lmax * d * sizeof(double));
  s.xs = 0;
  s.ws = s.xs + nb;
  s.fs = s.ws + nb;
  s.contrib = s.fs + align16((size_t)LM * d * sizeof(double));
  s.sslot = align16(s.contrib + (size_t)CH * d * sbytes);
  s.buf = align128(s.sslot + (size_t)SHmax * sizeof(uint32_t));
  s.buf_stride = align128((size_t)CB);
  s.mbar = s.buf + nbuf * s.buf_stride;
  s.total = s.mbar + 24;
  return s;
}
__host__ __device__ inline SmemLayout layout(const DevPatches& p, int d, int sbytes, int nbuf) {
  return layout(p.node_stride, p.contrib_slots, p.chunk_bytes, p.max_nodes, p.max_shared, d, sbytes,
                nbuf);
}

// The n local indices of element el (uint16, n per element): one vector load
// when n * 2 bytes is a power of two (2, 4 and 8 corners), else n loads.
template <int n>
__device__ inline void load_corners(const uint16_t* base, int el, int* out) {
  if (n == 2 || n == 4 || n == 8) {
    uint32_t w[4];
    if (n == 2) {
      w[0] = reinterpret_cast<const uint32_t*>(base)[el];
    } else if (n == 4) {
      const uint2 q = reinterpret_cast<const uint2*>(base)[el];
      w[0] = q.x;
      w[1] = q.y;
    } else {
      const uint4 q = reinterpret_cast<const uint4*>(base)[el];
      w[0] = q.x;
      w[1] = q.y;
      w[2] = q.z;
      w[3] = q.w;
    }
#pragma unroll
    for (int a = 0; a < n; ++a) out[a] = (int)((w[a >> 1] >> (16 * (a & 1))) & 0xffffu);
  } else {
#pragma unroll
    for (int a = 0; a < n; ++a) out[a] = base[el * n + a];
  }
}

// Differences of an element's corner coordinates and predicted
// displacements to its first corner, in FP64 before any rounding to S. Node
// arrays are row-major; in 2D a node's two components are one 16-byte load.
template <int d, int n, typename S>
__device__ inline void gather_differences(const double* xs, const double* ws, const int* lc,
                                          double* dX, S* du) {
  if constexpr (d == 2) {
    const double2 x0 = reinterpret_cast<const double2*>(xs)[lc[0]];
    const double2 u0 = reinterpret_cast<const double2*>(ws)[lc[0]];
    dX[0] = dX[1] = 0.0;
    du[0] = du[1] = S(0);
#pragma unroll
    for (int a = 1; a < n; ++a) {
      const double2 x = reinterpret_cast<const double2*>(xs)[lc[a]];
      const double2 u = reinterpret_cast<const double2*>(ws)[lc[a]];
      dX[a * 2] = x.x - x0.x;
      dX[a * 2 + 1] = x.y - x0.y;
      du[a * 2] = S(u.x - u0.x);
      du[a * 2 + 1] = S(u.y - u0.y);
    }
  } else {
#pragma unroll
    for (int i = 0; i < d; ++i) {
      dX[i] = 0;
      du[i] = 0;
      const double x0 = xs[d * lc[0] + i], u0 = ws[d * lc[0] + i];
#pragma unroll
      for (int a = 1; a < n; ++a) {
        dX[a * d + i] = xs[d * lc[a] + i] - x0;
        du[a * d + i] = S(ws[d * lc[a] + i] - u0);
      }
    }
  }
}

// Where component i of contribution slot k sits: 3D contributions are rows
// of three (one address per slot; 3 is invertible mod 16 and mod 32, so
// slots at distinct residues keep distinct banks), 1D and 2D ones
// component-major ([i][slot], 16-byte loads in 2D would otherwise pair slots
// on one bank group).
template <int d>
__device__ inline int cidx(int k, int i, int CH) {
  return d == 3 ? 3 * k + i : i * CH + k;
}

// CTAs per SM each instantiation is built for (register budget).
template <int T, typename S> struct PatchOccupancy { static constexpr int value = 3; };
template <> struct PatchOccupancy<AKB_HEXAHEDRON_8, float> { static constexpr int value = 2; };
template <> struct PatchOccupancy<AKB_HEXAHEDRON_8, double> { static constexpr int value = 1; };
// FP32-bulk tetrahedra (FP32 contributions, 768-element patches, one record
// buffer: <= 56 KB), 2D and 1D patches of <= 1024 elements take <= 56 KB of
// shared memory: four CTAs per SM when the registers allow it (<= 64 per
// thread; the FP64 tetrahedron at 64 registers measured slower)
template <> struct PatchOccupancy<AKB_TETRAHEDRON_4, float> { static constexpr int value = 4; };
template <typename S> struct PatchOccupancy<AKB_TRIANGLE_3, S> { static constexpr int value = 4; };
template <typename S> struct PatchOccupancy<AKB_SEGMENT_2, S> { static constexpr int value = 4; };

// DOFs handled per thread per round of the finishing loop: their global
// loads are issued together.
constexpr int kBatch = 4;
constexpr uint32_t kWaitLimit = 1u << 22;

__device__ inline uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The step's kernels are launched with programmatic stream serialization
// (launch_pdl): k_patch_step waits before its first read of the node state,
// k_finish_list before its first read of the partials.
__device__ inline void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}
// L2 prefetch of [lo, hi) rounded out to 16-byte boundaries (inside the
// allocation: nodal arrays carry 16 bytes of slack at their end).
__device__ inline void prefetch_l2(const void* base, size_t lo, size_t hi) {
  const size_t a = lo & ~size_t(15), b = (hi + 15) & ~size_t(15);
  if (b <= a) return;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((const char*)base + a),
               "r"((uint32_t)(b - a))
               : "memory");
}
__device__ inline void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(saddr(dst)), "l"(src) : "memory");
}
__device__ inline void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr(dst)), "l"(src) : "memory");
}
__device__ inline void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}
__device__ inline bool mbar_wait(uint32_t a, uint32_t parity) {
  for (uint32_t it = 0; it < kWaitLimit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ inline void expect_tx(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(mbar),
               "r"(bytes)
               : "memory");
}
__device__ inline void arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

// Corrector of one free DOF from its total force r (with f_ext), and the
// next predictor: u = w (the predicted displacement this step's forces were
// evaluated at), v* = v + dt a recomputed bit for bit, then
// x = r / M - a, v = v* + dt/2 x, a += x (u += 0 x only when x is not
// finite); w' = u + dt v + dt^2/2 a.
// M v^2 of one DOF from its inverse lumped mass, for masses above
// DBL_EPSILON (the test of getKineticEnergy, solid_mechanics_model.cc:547-561).
__device__ inline double ke_term(double v, double im) {
  const double M = 1.0 / im;
  return M > DBL_EPSILON ? v * v * M : 0.0;
}

// The same of a node from its sum of v^2 (one mass for all components).
__device__ inline double ke_sum(double v2, double im) {
  const double M = 1.0 / im;
  return M > DBL_EPSILON ? v2 * M : 0.0;
}

// Sum of the CTA's per-thread values in a fixed order (lanes by an xor
// tree, then warps in order), by thread 0; every thread must call it.
__device__ inline double cta_sum(double x, double* warp_sums) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();  // warp_sums free (a previous use is read)
  if ((threadIdx.x & 31) == 0) warp_sums[w] = x;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < nw; ++k) s += warp_sums[k];
  return s;
}

__device__ inline void finish_dof(double dt, double r, double im, double w, double& v, double& a,
                                  double& u, double& wn) {
  u = w;
  v = __dadd_rn(v, __dmul_rn(dt, a));
  fast::correct(dt, r, im, u, v, a);
  wn = u;
  double vn = v;
  fast::predict(dt, wn, vn, a);
}

// One patch p, by the whole CTA. uses: chunk records this CTA has consumed
// before (it picks the buffer and the mbarrier phase); stages: patches it
// staged before (the phase of the staging mbarrier). Returns false when a
// bounded wait gave up.
template <int T, typename S, bool FEXT>
__device__ __forceinline__ bool patch_body(const DevModel& m, const DevPatches& P, double dt0,
                                           int p, unsigned char* smem, uint32_t& uses,
                                           uint32_t& stages) {
  constexpr int d = ET<T>::dim, n = ET<T>::nnpe;
  static_assert(kChunk == kThreads, "one element per thread per chunk");
  const double dt = P.inst_dt ? P.inst_dt[P.patch_inst[p]] : dt0;
  const int ib = P.ibeg[p], nint = P.nint[p];
  const int s0 = P.sh_ptr[p], nsh = P.sh_ptr[p + 1] - s0;
  const int L = nint + nsh;
  const int eb = P.elem_ptr[p];
  const int ne = P.elem_ptr[p + 1] - eb;
  const int nchunks = (ne + kChunk - 1) / kChunk;
  const int ch0 = P.chunk_base[p];
  const int LM = P.node_stride, CH = P.contrib_slots;
  const bool two = P.nbuf == 2;  // buffers: 1 or 2
  const SmemLayout lay = layout(P, d, sizeof(S), two ? 2 : 1);
  // the interior slice [ib, ib + nint) of X and w is bulk-copied from the
  // 16-byte boundary at or below its start (the bytes before it land in the
  // slack in front of the array; o: the slice's offset in doubles) to the
  // boundary at or below its end; the remaining tail (one double at most)
  // comes by cp.async, so that nothing is written past the slice, where the
  // shared nodes go
  const size_t row = (size_t)d * sizeof(double);
  const size_t s_lo = (size_t)ib * row, s_hi = (size_t)(ib + nint) * row;
  const size_t c_lo = s_lo & ~size_t(15), c_hi = s_hi & ~size_t(15);
  const int o = (int)((s_lo - c_lo) / sizeof(double));
  double* xs = reinterpret_cast<double*>(smem + lay.xs) + o;  // node at position j: xs[d j + i]
  double* ws = reinterpret_cast<double*>(smem + lay.ws) + o;
  double* fs = reinterpret_cast<double*>(smem + lay.fs);      // fs[i LM + j]
  S* contrib = reinterpret_cast<S*>(smem + lay.contrib);
  const int tid = threadIdx.x;
  const uint32_t mb0 = saddr(smem + lay.mbar), mbs = mb0 + 16;

  // record k (counted over the CTA's chunks) uses buffer k % nbuf, and the
  // (k / nbuf)-th phase of that buffer's mbarrier
  auto buffer = [&](uint32_t k) { return two ? (k & 1u) : 0u; };
  auto phase = [&](uint32_t k) { return (two ? (k >> 1) : k) & 1u; };
  auto issue = [&](int c) {  // chunk c's record, by thread 0
    const uint2 cd = __ldg(reinterpret_cast<const uint2*>(&P.chunks[ch0 + c]));  // off16, bytes
    const uint32_t b = buffer(uses + c), bar = mb0 + 8 * b;
    expect_tx(bar, cd.y);
    bulk_copy(saddr(smem + lay.buf + b * lay.buf_stride), P.cdata + (size_t)cd.x * 8, cd.y, bar);
  };

  // 1. staging
  // the interior nodes' finishing inputs go to the spare record buffer (the
  // one the next chunk would use) at the start of the last chunk, when two
  // buffers are used and they fit; the finish then reads shared memory
  bool pre;
  {
    uint32_t f_off[5], f_bytes[5];
    size_t f_lo[5];
    pre = two && nint > 0 &&
          finish_regions<d, FEXT>(ib, nint, f_off, f_lo, f_bytes) <= lay.buf_stride;
  }
  const uint32_t spare = buffer(uses + nchunks);
  auto issue_finish = [&]() {  // by thread 0
    const void* src[5] = {m.v, m.a, m.inv_mass, m.blocked, m.fext};
    uint32_t f_off[5], f_bytes[5];
    size_t f_lo[5];
    const uint32_t total = finish_regions<d, FEXT>(ib, nint, f_off, f_lo, f_bytes);
    const uint32_t dst = saddr(smem + lay.buf + spare * lay.buf_stride);
    expect_tx(mbs, total);
    uint32_t at = 0;
#pragma unroll
    for (int k = 0; k < (FEXT ? 5 : 4); ++k) {
      bulk_copy(dst + at, reinterpret_cast<const char*>(src[k]) + f_lo[k], f_bytes[k], mbs);
      at += f_bytes[k];
    }
  };
  if (tid == 0) {
    // the previous patch's generic-proxy accesses of these buffers (ordered
    // before this point by the CTA barrier) come before the bulk copies
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (nint > 0 && c_hi > c_lo) {
      const uint32_t bytes = (uint32_t)(c_hi - c_lo);
      expect_tx(mbs, 2 * bytes);
      bulk_copy(saddr(smem + lay.xs), reinterpret_cast<const char*>(m.X) + c_lo, bytes, mbs);
      bulk_copy(saddr(smem + lay.ws), reinterpret_cast<const char*>(P.w) + c_lo, bytes, mbs);
    } else {
      arrive(mbs);
    }
    if (nchunks > 0) issue(0);
    if (two && nchunks > 1) issue(1);
    if (nint > 0 && !pre) {  // inputs of the interior nodes' finish
      prefetch_l2(m.v, s_lo, s_hi);
      prefetch_l2(m.a, s_lo, s_hi);
      prefetch_l2(m.inv_mass, (size_t)ib * 8, (size_t)(ib + nint) * 8);
      prefetch_l2(m.blocked, (size_t)ib * d, (size_t)(ib + nint) * d);
      if (FEXT) prefetch_l2(m.fext, s_lo, s_hi);
    }
  }
  if (tid == kThreads - 1 && nint > 0 && c_hi < s_hi && c_hi >= s_lo) {  // the tail double
    const size_t k = (c_hi - s_lo) / sizeof(double);
    cp_async8(xs + k, m.X + (size_t)ib * d + k);
    cp_async8(ws + k, P.w + (size_t)ib * d + k);
  } else if (tid == kThreads - 1 && nint > 0 && c_hi < s_lo) {  // slice within one 16 bytes
    for (size_t k = 0; k < (size_t)nint * d; ++k) {
      cp_async8(xs + k, m.X + (size_t)ib * d + k);
      cp_async8(ws + k, P.w + (size_t)ib * d + k);
    }
  }
  uint32_t* sslot = reinterpret_cast<uint32_t*>(smem + lay.sslot);
  for (int t = tid; t < nsh; t += kThreads) {
    const int64_t g = P.sgid[s0 + t];
    sslot[t] = P.sslot[s0 + t];  // for the finish
    const int j = nint + t;
    if constexpr (d == 2) {
      cp_async16(xs + 2 * j, m.X + g * 2);
      cp_async16(ws + 2 * j, P.w + g * 2);
    } else {
#pragma unroll
      for (int i = 0; i < d; ++i) {
        cp_async8(xs + d * j + i, m.X + g * d + i);
        cp_async8(ws + d * j + i, P.w + g * d + i);
      }
    }
  }
  for (int k = tid; k < L * d; k += kThreads) {
    const int i = k / L, j = k - i * L;
    fs[i * LM + j] = 0.0;
  }
  cp_async_wait_all();
  {
    const bool ok = mbar_wait(mbs, stages & 1u);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        atomicExch(P.err, 1);
        mbar_wait(mbs, stages & 1u);
        for (int k = 0; k < min(nchunks, two ? 2 : 1); ++k)
          mbar_wait(mb0 + 8 * buffer(uses + k), phase(uses + k));
      }
      return false;
    }
  }
  ++stages;
  if (pre && nchunks <= 1 && tid == 0) issue_finish();  // the second buffer is free already

  // 2. element forces chunk by chunk: each element writes its corner vectors
  //    to their contribution slots, then one thread per node run adds the
  //    run (ascending element order) to that node
  for (int c = 0; c < nchunks; ++c) {
    // one buffer: chunk c's record goes where chunk c-1's was, once every
    // thread is done with it
    if (!two && c > 0) {
      __syncthreads();
      if (tid == 0) issue(c);
    }
    // with two buffers this barrier also ends chunk c-1: past it no thread
    // reads chunk c-1's record or contributions any more
    const uint32_t b = buffer(uses + c);
    const bool ok = mbar_wait(mb0 + 8 * b, phase(uses + c));
    if (__syncthreads_or(!ok)) {  // bounded: flag, drain what was issued, stop
      if (tid == 0) {
        atomicExch(P.err, 1);
        const int last = min(nchunks - 1, (two && c == 0) ? 1 : c);
        for (int k = c; k <= last; ++k) mbar_wait(mb0 + 8 * buffer(uses + k), phase(uses + k));
        if (pre && nchunks <= 1) mbar_wait(mbs, stages & 1u);  // the finishing inputs
      }
      return false;
    }
    if (two && tid == 0 && c > 0 && c + 1 < nchunks) issue(c + 1);  // into chunk c-1's buffer
    if (pre && tid == 0 && c > 0 && c + 1 == nchunks) issue_finish();  // ditto
    const int c0 = c * kChunk, nec = min(kChunk, ne - c0);
    const uint32_t A = (uint32_t)align16((size_t)nec * n * 2);
    if (tid < nec) {
      const uint16_t* lcs = reinterpret_cast<const uint16_t*>(smem + lay.buf + b * lay.buf_stride + 16);
      int lc[n], sl[n];
      load_corners<n>(lcs, tid, lc);
      load_corners<n>(lcs + A / 2, tid, sl);
      const MatParams& mp = (P.emat ? m.mat_table[P.emat[(size_t)eb + c0 + tid]] : m.mats[0]);
      double dX[3 * 8];
      S du[3 * 8];
      gather_differences<d, n, S>(xs, ws, lc, dX, du);
      S fe[3 * 8];
      fast::element_force<T, S>(mp, dX, du, fe);
#pragma unroll
      for (int a = 0; a < n; ++a)
#pragma unroll
        for (int i = 0; i < d; ++i) contrib[cidx<d>(sl[a], i, CH)] = fe[a * d + i];
    }
    __syncthreads();
    // one thread per run (a node's contributions of this chunk, ascending
    // element order) adds the run to the node's accumulator; runs are sorted
    // by length, so a warp's threads loop about as long
    const unsigned char* buf = smem + lay.buf + b * lay.buf_stride;
    const uint4 hd = *reinterpret_cast<const uint4*>(buf);  // header: 8 x uint16
    {
      constexpr int G = sizeof(S) == 8 ? 16 : 32;  // runs per group
      // header words: x = R | ng << 16, y = runs | goff << 16, z = idx | G << 16
      const int R = (int)(hd.x & 0xffff);
      const uint32_t* runs = reinterpret_cast<const uint32_t*>(buf + (hd.y & 0xffff));
      const uint16_t* goff = reinterpret_cast<const uint16_t*>(buf + (hd.y >> 16));
      const uint16_t* idx = reinterpret_cast<const uint16_t*>(buf + (hd.z & 0xffff));
      for (int q = tid; q < R; q += kThreads) {
        const uint32_t w = runs[q];
        const int len = (int)(w >> 16), jp = (int)(w & 0xffff);
        if (len == 0) continue;
        const uint16_t* ix = idx + goff[q / G] + (q % G);
        double f[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
        for (int t = 0; t < len; ++t) {
          const int k = ix[t * G];
#pragma unroll
          for (int i = 0; i < d; ++i) f[i] += double(contrib[cidx<d>(k, i, CH)]);
        }
#pragma unroll
        for (int i = 0; i < d; ++i) fs[i * LM + jp] -= f[i];
      }
    }
  }
  {
    // the sums of the last chunk are in (and the finishing inputs)
    const bool ok = !pre || mbar_wait(mbs, stages & 1u);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        atomicExch(P.err, 1);
        mbar_wait(mbs, stages & 1u);
      }
      return false;
    }
  }
  if (pre) ++stages;
  uses += nchunks;
  const unsigned char* fin = smem + lay.buf + spare * lay.buf_stride;
  uint32_t f_off[5];
  {
    size_t f_lo[5];
    uint32_t f_bytes[5];
    finish_regions<d, FEXT>(ib, nint, f_off, f_lo, f_bytes);
  }

  // 3. finish: the shared nodes' partials to their slots (the second pass
  //    adds them), the interior nodes finished here, one thread per DOF,
  //    contiguous in the global arrays
  grid_launch_dependents();  // the second pass may start launching (it waits for this grid)
  for (int k = tid; k < nsh * d; k += kThreads) {
    const int t = k / d, i = k - t * d;
    P.partial[(size_t)sslot[t] * d + i] = fs[i * LM + nint + t];
  }
  const int items = nint * d;
  double ke = 0.0;  // M v^2 of this thread's DOFs after the step
  for (int base = 0; base < items; base += kThreads * kBatch) {
    double v[kBatch], a[kBatch], im[kBatch], fx[kBatch];
    uint8_t bl[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int k = base + b * kThreads + tid;
      if (k < items) {
        if (pre) {
          v[b] = *reinterpret_cast<const double*>(fin + f_off[0] + 8 * k);
          a[b] = *reinterpret_cast<const double*>(fin + f_off[1] + 8 * k);
          im[b] = *reinterpret_cast<const double*>(fin + f_off[2] + 8 * (k / d));
          bl[b] = fin[f_off[3] + k];
          fx[b] = FEXT ? *reinterpret_cast<const double*>(fin + f_off[4] + 8 * k) : 0.0;
        } else {
          const int64_t q = (int64_t)ib * d + k;
          bl[b] = m.blocked[q];
          v[b] = m.v[q];
          a[b] = m.a[q];
          im[b] = m.inv_mass[ib + k / d];
          fx[b] = FEXT ? m.fext[q] : 0.0;
        }
      }
    }
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int k = base + b * kThreads + tid;
      if (k >= items) continue;
      if (!bl[b]) {  // blocked DOFs keep u, v, a (and w = u)
        const int j = k / d, i = k - j * d;
        const int64_t q = (int64_t)ib * d + k;
        const double f = fs[i * LM + j];
        double u, wn;
        finish_dof(dt, FEXT ? f + fx[b] : f, im[b], ws[k], v[b], a[b], u, wn);
        m.u[q] = u;
        m.v[q] = v[b];
        m.a[q] = a[b];
        P.w[q] = wn;
      }
      ke += ke_term(v[b], im[b]);
    }
  }
  if (P.ke_part) {
    __shared__ double warp_sums[kThreads / 32];
    const double s = cta_sum(ke, warp_sums);
    if (tid == 0) P.ke_part[p] = s;
  }
  return true;
}

// One CTA per patch, or (PERSIST) a grid smaller than the patch count whose
// CTAs stride over the patches. The loop is a separate instantiation: kept
// out of the one-patch kernel it would raise that kernel's register pressure.
template <int T, typename S, bool FEXT, bool PERSIST>
__global__ void __launch_bounds__(kThreads, (PatchOccupancy<T, S>::value))
    k_patch_step(DevModel m, DevPatches P, double dt0) {
  extern __shared__ __align__(128) unsigned char smem[];
  {
    const SmemLayout lay = layout(P, ET<T>::dim, sizeof(S), P.nbuf);
    if (threadIdx.x == 0) {
      for (int b = 0; b < 3; ++b)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(smem + lay.mbar + 8 * b))
                     : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
  }
  grid_wait();  // the previous step's (or update's) writes of w, v, a, u
  uint32_t uses = 0, stages = 0;
  if constexpr (PERSIST) {
    for (int p = blockIdx.x; p < P.npatch; p += gridDim.x) {
      if (p != (int)blockIdx.x) __syncthreads();  // shared memory of the previous patch is free
      if (!patch_body<T, S, FEXT>(m, P, dt0, p, smem, uses, stages)) return;
    }
  } else {
    patch_body<T, S, FEXT>(m, P, dt0, blockIdx.x, smem, uses, stages);
  }
}

// ------------------------------------------------------------- fan records
// The fused step on fan records (akb_patch.cuh: FP64 triangles, tetrahedra and
// hexahedra). As k_patch_step, with two differences:
//  - triangles and tetrahedra: a thread computes a fan, a row of elements around
//    a hinge, keeping the last ring node in registers: each further element loads
//    one node, re-reads the hinge and writes one contribution. A tetrahedron costs
//    about 105 FP64 operations (the hinge's cross products are shared between
//    neighbours). Hexahedra are fans of one element (hex_force_f64);
//  - all contributions of the patch stay in shared memory, so that the node
//    sums run once per patch and feed the finish directly: two barriers a
//    patch instead of two per 256 elements, and no force accumulators.

// Shared memory: X and w of the patch's nodes (row-major, 16 bytes of slack in
// front), the contributions, the record, the interior nodes' finishing inputs
// (finish_regions), two buffers of the shared entries (node, partial slot)
// and three of the patch descriptor, two mbarriers (staging, finishing inputs).
struct FanLayout {
  size_t xs, ws, c, rec, fin, sh, sh_stride, desc, mbar, total;
};
__host__ __device__ inline FanLayout fan_layout(int Lmax, int Imax, int SHmax, int slots,
                                                int rec_bytes, int d, bool fext) {
  FanLayout s;
  const size_t nb = align16(16 + (size_t)Lmax * d * sizeof(double));
  s.xs = 0;
  s.ws = nb;
  s.c = 2 * nb;
  s.rec = align128(s.c + (size_t)slots * d * sizeof(double));
  s.fin = align128(s.rec + (size_t)rec_bytes);
  // v, a, 1 / M, the flags and f_ext, each rounded out to 16 bytes on both sides
  s.sh = s.fin + align16((size_t)Imax * ((fext ? 3 : 2) * 8 * d + 8 + d)) + 5 * 32;
  s.sh_stride = align16((size_t)SHmax * sizeof(uint2));
  s.desc = s.sh + 2 * s.sh_stride;
  s.mbar = s.desc + 3 * sizeof(FanDesc);
  s.total = s.mbar + 16;
  return s;
}
__host__ __device__ inline FanLayout fan_layout(const DevPatches& p, int d, bool fext) {
  return fan_layout(p.max_nodes, p.max_interior, p.max_shared, p.contrib_slots, p.chunk_bytes, d,
                    fext);
}

// Threads of a CTA and CTAs per SM each instantiation is built for. A thread
// computes a fan, so a patch has about as many fans as its CTA has threads:
// larger patches share fewer nodes, smaller ones overlap their phases better.
// Tetrahedra at 128 registers (16 warps an SM either way; more spill): 256
// threads 140.6 us a step on the 6 M-element cube, 128 threads 145.3, 192
// threads 148.7. Triangles (512 plates): 128 threads 47.9 us, 256 threads 48.4.
// LIN: every material small-strain elastic (simplices), every element a
// parallelepiped (hexahedra).
template <int TY, bool LIN> struct FanBuild;
template <bool LIN> struct FanBuild<AKB_TETRAHEDRON_4, LIN> {
  static constexpr int threads = 256, ctas = 2;
};
template <bool LIN> struct FanBuild<AKB_TRIANGLE_3, LIN> {
  static constexpr int threads = 128, ctas = LIN ? 6 : 5;
};
// Hexahedra: FP64 issue bound, 255 registers for the signed sums and the 36
// accumulators, so 8 warps an SM; 128-thread CTAs (a 128-element patch each)
// overlap one patch's staging and finish with the other's elements. 64^3
// neo-Hookean block: 77.1 us a step, and 79.5 when the others were measured
// (256-element chunks in one 256-thread CTA 95.1; 4 x 64 threads 81.4; 1 x 256
// threads 126; 3 x 128 at 168 registers, spilling, 86.8); 37 x 31 x 33 distorted
// 16.7 against 31.3.
template <bool PAR> struct FanBuild<AKB_HEXAHEDRON_8, PAR> {
  static constexpr int threads = 128, ctas = 2;
};

// w P of one element from G = det * grad u (row-major), P the Cauchy (small
// strain) or first Piola stress, w the reference volume of the simplex. A
// small-strain elastic material's P is rounded the same whether or not the model
// has others (LIN): an instance of a batch steps as it does alone.
template <int d, bool LIN>
__device__ inline void fan_stress(const MatParams& mp, const double* G, double det, double* P) {
  constexpr double w = d == 3 ? 1.0 / 6.0 : 0.5;
  if (LIN || !mp.finite) {
    const double s = w * (1.0 / det), mu = mp.mu * s;
    double tr = G[0] + G[d + 1];
    if (d == 3) tr += G[2 * d + 2];
    tr *= mp.lambda * s;
#pragma unroll
    for (int i = 0; i < d; ++i) {
      P[i * d + i] = fma(2.0 * mu, G[i * d + i], tr);
#pragma unroll
      for (int j = 0; j < i; ++j) P[i * d + j] = P[j * d + i] = mu * (G[i * d + j] + G[j * d + i]);
    }
  } else {
    const double idet = 1.0 / det;
    double g[d * d];
#pragma unroll
    for (int k = 0; k < d * d; ++k) g[k] = G[k] * idet;
    fast::stress_P<d, double>(mp, g, P);
#pragma unroll
    for (int k = 0; k < d * d; ++k) P[k] *= w;
  }
}

__device__ inline void cross3(const double* a, const double* b, double* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

// Contributions of fan t of a staged patch. The simplex (hinge, r_t, r_{t+1})
// has the edges e1 (tetrahedra: to the hinge's second node), e2, e3 from the
// hinge's first node; the columns of the adjugate of J are e2 x e3, e3 x e1 =
// -c3 and e1 x e2 = c2, c3 being the next element's c2.
template <int d, bool LIN>
__device__ __forceinline__ void fan_forces(const uint16_t* rec, int t, const double* xs,
                                           const double* ws, double* C, const MatParams& mp0,
                                           const MatParams* table, const uint32_t* emat) {
  constexpr int H = d - 1;
  const uint16_t* ro = rec + rec[2];
  // per entry: position | slot << 16
  const uint32_t* node = reinterpret_cast<const uint32_t*>(rec + rec[3]);
  const uint32_t info = reinterpret_cast<const uint32_t*>(rec + rec[4])[t];
  const int k = (int)(info & 0x7fff);
  const bool closed = info & 0x8000;
  const uint32_t first = node[ro[H] + t];  // r_0
  const int ja = (int)(node[t] & 0xffff);
  double e1[3], d1[3], e2[d], d2[d], c2[3], fa[d], fb[3], ft[d];
  auto load = [&](int j, double* x, double* u) {
    if constexpr (d == 2) {
      const double2 p = reinterpret_cast<const double2*>(xs)[j];
      const double2 q = reinterpret_cast<const double2*>(ws)[j];
      x[0] = p.x;
      x[1] = p.y;
      u[0] = q.x;
      u[1] = q.y;
    } else {
#pragma unroll
      for (int i = 0; i < d; ++i) {
        x[i] = xs[d * j + i];
        u[i] = ws[d * j + i];
      }
    }
  };
  auto edge = [&](int j, double* e, double* u) {  // (the hinge re-read: 12 registers less)
    double xa[d], ua[d];
    load(ja, xa, ua);
    load(j, e, u);
#pragma unroll
    for (int i = 0; i < d; ++i) {
      e[i] -= xa[i];
      u[i] -= ua[i];
    }
  };
  auto store = [&](int s, const double* f) {
    if constexpr (d == 2) {
      reinterpret_cast<double2*>(C)[s] = make_double2(f[0], f[1]);
    } else {
#pragma unroll
      for (int i = 0; i < d; ++i) C[d * s + i] = f[i];
    }
  };
  edge((int)(first & 0xffff), e2, d2);
  if constexpr (d == 3) {
    edge((int)(node[ro[1] + t] & 0xffff), e1, d1);
    cross3(e1, e2, c2);
  }
#pragma unroll
  for (int i = 0; i < d; ++i) fa[i] = ft[i] = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) fb[i] = 0.0;
  uint32_t at = first;
#pragma unroll 1  // (the ring node's registers swap roles: no moves)
  for (int s = 0; s < k; ++s) {
    const uint32_t next = closed && s == k - 1 ? first : node[ro[H + 1 + s] + t];
    const int jn = (int)(next & 0xffff);
    const MatParams& mp = emat ? table[emat[(info >> 16) + s]] : mp0;
    double e3[d], d3[d], fn[d], G[d * d], P[d * d];
    edge(jn, e3, d3);
    if constexpr (d == 3) {
      double x[3], c3[3];
      cross3(e2, e3, x);
      cross3(e1, e3, c3);
      const double det = e1[0] * x[0] + e1[1] * x[1] + e1[2] * x[2];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) G[i * 3 + j] = d1[i] * x[j] - d2[i] * c3[j] + d3[i] * c2[j];
      fan_stress<d, LIN>(mp, G, det, P);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        fb[i] += P[i * 3] * x[0] + P[i * 3 + 1] * x[1] + P[i * 3 + 2] * x[2];
        ft[i] -= P[i * 3] * c3[0] + P[i * 3 + 1] * c3[1] + P[i * 3 + 2] * c3[2];
        fn[i] = P[i * 3] * c2[0] + P[i * 3 + 1] * c2[1] + P[i * 3 + 2] * c2[2];
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) c2[i] = c3[i];
    } else {
      const double det = e2[0] * e3[1] - e2[1] * e3[0];
#pragma unroll
      for (int i = 0; i < 2; ++i) {  // adjugate columns (e3y, -e3x), (-e2y, e2x)
        G[i * 2] = d2[i] * e3[1] - d3[i] * e2[1];
        G[i * 2 + 1] = d3[i] * e2[0] - d2[i] * e3[0];
      }
      fan_stress<d, LIN>(mp, G, det, P);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        ft[i] += P[i * 2] * e3[1] - P[i * 2 + 1] * e3[0];
        fn[i] = P[i * 2 + 1] * e2[0] - P[i * 2] * e2[1];
      }
    }
    store((int)(at >> 16), ft);
    at = next;
#pragma unroll
    for (int i = 0; i < d; ++i) {  // the forces of an element add up to zero
      fa[i] -= ft[i];
      ft[i] = fn[i];
      e2[i] = e3[i];
      d2[i] = d3[i];
    }
  }
#pragma unroll
  for (int i = 0; i < d; ++i) {
    fa[i] -= ft[i];
    if (d == 3) fa[i] -= fb[i];
  }
  if (closed) {  // r_0's contribution, written by this thread above
#pragma unroll
    for (int i = 0; i < d; ++i) C[d * (int)(first >> 16) + i] += ft[i];
  } else {
    store((int)(at >> 16), ft);
  }
  store((int)(node[t] >> 16), fa);
  if constexpr (d == 3) store((int)(node[ro[1] + t] >> 16), fb);
}

// Contributions of hexahedron t of a staged patch (fan records of single
// elements, row a its corner a).
template <bool PAR>
__device__ __forceinline__ void hex_forces(const uint16_t* rec, int t, const double* xs,
                                           const double* ws, double* C, const MatParams& mp0,
                                           const MatParams* table, const uint32_t* emat) {
  constexpr int d = 3, n = 8;
  const int nf = rec[0];
  const uint32_t* node = reinterpret_cast<const uint32_t*>(rec + rec[3]) + t;
  const bool affine = rec[rec[4] + 2 * t] & kFanAffine;
  const MatParams& mp = emat ? table[emat[t]] : mp0;
  double dX[d * n], du[d * n], fe[d * n];
  {
    int lc[n];
#pragma unroll
    for (int a = 0; a < n; ++a) lc[a] = (int)(node[a * nf] & 0xffff);
    gather_differences<d, n, double>(xs, ws, lc, dX, du);
  }
  fast::hex_force_f64<PAR>(mp, dX, du, fe, affine);
#pragma unroll
  for (int a = 0; a < n; ++a) {
    const int s = (int)(node[a * nf] >> 16);
#pragma unroll
    for (int i = 0; i < d; ++i) C[d * s + i] = fe[a * d + i];
  }
}

// A node's d values at position j of a row-major array.
template <int d>
__device__ inline void get_row(const double* p, int j, double* x) {
  if constexpr (d == 2) {
    const double2 q = reinterpret_cast<const double2*>(p)[j];
    x[0] = q.x;
    x[1] = q.y;
  } else {
#pragma unroll
    for (int i = 0; i < d; ++i) x[i] = p[d * j + i];
  }
}
template <int d>
__device__ inline void put_row(double* p, int j, const double* x) {
  if constexpr (d == 2) {
    reinterpret_cast<double2*>(p)[j] = make_double2(x[0], x[1]);
  } else {
#pragma unroll
    for (int i = 0; i < d; ++i) p[d * j + i] = x[i];
  }
}

// The CTAs stride over the patches (one each when the grid covers them). The
// staging of a patch needs its descriptor, then its shared entries, then the
// nodes these name: three dependent trips to memory, so the descriptor is
// fetched two patches ahead and the shared entries one, and the patch's slices
// and record are prefetched into L2. What does not change between steps (X,
// record, entries of the CTA's first patch) is staged before the previous
// grid in the stream has finished.
template <int TY, bool LIN, bool FEXT>
__global__ void __launch_bounds__(FanBuild<TY, LIN>::threads, (FanBuild<TY, LIN>::ctas))
    k_fan_step(DevModel m, DevPatches P, double dt0) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int d = ET<TY>::dim, T = FanBuild<TY, LIN>::threads;
  __shared__ double warp_sums[T / 32];
  const FanLayout lay = fan_layout(P, d, FEXT);
  const int tid = threadIdx.x, G = gridDim.x;
  const uint32_t mb = saddr(smem + lay.mbar);
  FanDesc* descs = reinterpret_cast<FanDesc*>(smem + lay.desc);
  double* C = reinterpret_cast<double*>(smem + lay.c);
  const uint16_t* rec = reinterpret_cast<const uint16_t*>(smem + lay.rec);
  auto entries = [&](int it) {
    return reinterpret_cast<uint2*>(smem + lay.sh + (it & 1) * lay.sh_stride);
  };
  auto fetch_desc = [&](int p, int b) {
    if (p < P.npatch && tid < (int)(sizeof(FanDesc) / 16))
      cp_async16(reinterpret_cast<char*>(descs + b) + 16 * tid,
                 reinterpret_cast<const char*>(P.desc + p) + 16 * tid);
  };
  auto fetch_entries = [&](int s0, int nsh, int it) {
    uint2* e = entries(it);
    for (int t = tid; t < nsh; t += T) cp_async8(e + t, P.entries + s0 + t);
  };
  if (tid == 0) {
    for (int b = 0; b < 2; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb + 8 * b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fetch_desc(blockIdx.x, 0);
  fetch_desc(blockIdx.x + G, 1);
  cp_async_wait_all();
  __syncthreads();
  fetch_entries(descs[0].s0, descs[0].nsh, 0);
  cp_async_wait_all();
  __syncthreads();
  int it = 0;
  constexpr size_t row = (size_t)d * sizeof(double);
  // the offset in doubles of an interior slice behind its 16-byte boundary
  auto offset = [](int ib) { return d == 3 ? (int)(ib & 1) : 0; };
  auto nodes = [&](size_t at, int ib) { return reinterpret_cast<double*>(smem + at) + offset(ib); };
  int cur = 0;  // the current descriptor's buffer
  for (int p = blockIdx.x; p < P.npatch; p += G, ++it, cur = cur == 2 ? 0 : cur + 1) {
    // each phase reads the descriptor again: few registers live across the
    // element loop
    {  // 1. staging
      const FanDesc D = descs[cur];
      const int ib = D.ibeg, nint = D.nint, nsh = D.nsh;
      const uint2* ent = entries(it);
      // the interior slices of X and w (see patch_body) and the record
      const size_t s_lo = (size_t)ib * row, s_hi = s_lo + nint * row;
      const size_t c_lo = s_lo & ~size_t(15), c_hi = s_hi & ~size_t(15);
      const uint32_t slice = nint > 0 && c_hi > c_lo ? (uint32_t)(c_hi - c_lo) : 0;
      // the doubles of a slice past its last whole 16 bytes, and the shared nodes
      auto gather = [&](double* to, const double* from) {
        if (d == 3 && tid == T - 1 && nint > 0)
          for (size_t k = slice ? (c_hi - s_lo) / sizeof(double) : 0; k < (size_t)nint * d; ++k)
            cp_async8(to + k, from + (size_t)ib * d + k);
        for (int t = tid; t < nsh; t += T) {
          const int64_t g = ent[t].x;
          const int j = nint + t;
          if constexpr (d == 2) {
            cp_async16(to + 2 * j, from + g * 2);
          } else {
#pragma unroll
            for (int i = 0; i < d; ++i) cp_async8(to + d * j + i, from + g * d + i);
          }
        }
      };
      if (tid == 0) {
        // the previous patch's generic-proxy accesses of these buffers (ordered
        // before this point by the CTA barrier) come before the bulk copies
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        expect_tx(mb, 2 * slice + D.rec_bytes);
        bulk_copy(saddr(rec), P.cdata + (size_t)D.rec_off16 * 8, D.rec_bytes, mb);
        if (slice)
          bulk_copy(saddr(smem + lay.xs), reinterpret_cast<const char*>(m.X) + c_lo, slice, mb);
      }
      gather(nodes(lay.xs, ib), m.X);
      if (it == 0) grid_wait();  // the previous step's (or update's) writes of w, v, a, u
      if (tid == 0) {
        if (slice)
          bulk_copy(saddr(smem + lay.ws), reinterpret_cast<const char*>(P.w) + c_lo, slice, mb);
        if (nint > 0) {  // inputs of the interior nodes' finish
          const void* src[5] = {m.v, m.a, m.inv_mass, m.blocked, m.fext};
          uint32_t off[5], nbytes[5];
          size_t lo[5];
          expect_tx(mb + 8, finish_regions<d, FEXT>(ib, nint, off, lo, nbytes));
          uint32_t at = saddr(smem + lay.fin);
#pragma unroll
          for (int k = 0; k < (FEXT ? 5 : 4); ++k) {
            bulk_copy(at, reinterpret_cast<const char*>(src[k]) + lo[k], nbytes[k], mb + 8);
            at += nbytes[k];
          }
        } else {
          arrive(mb + 8);
        }
      }
      gather(nodes(lay.ws, ib), P.w);
      cp_async_wait_all();
      const bool ok = mbar_wait(mb, it & 1);
      if (__syncthreads_or(!ok)) {
        if (tid == 0) {
          atomicExch(P.err, 1);
          mbar_wait(mb, it & 1);
          mbar_wait(mb + 8, it & 1);
        }
        return;
      }
    }
    if (p + G < P.npatch) {
      // ahead: the descriptor two patches on, the next patch's entries, its
      // slices and record to L2
      const FanDesc& N = descs[cur == 2 ? 0 : cur + 1];
      fetch_entries(N.s0, N.nsh, it + 1);
      if (tid == 0) {
        const size_t lo = (size_t)N.ibeg * row, hi = lo + N.nint * row;
        prefetch_l2(P.cdata, (size_t)N.rec_off16 * 16, (size_t)N.rec_off16 * 16 + N.rec_bytes);
        if (N.nint > 0) {
          prefetch_l2(m.X, lo, hi);
          prefetch_l2(P.w, lo, hi);
          prefetch_l2(m.v, lo, hi);
          prefetch_l2(m.a, lo, hi);
        }
      }
      fetch_desc(p + 2 * G, cur == 0 ? 2 : cur - 1);
    }
    {  // 2. element forces, one thread per fan (or element)
      const FanDesc& D = descs[cur];
      const bool mixed = D.mat == kMixed;
      const MatParams& mp = P.emat && !mixed ? m.mat_table[D.mat] : m.mats[0];
      const uint32_t* emat = mixed ? P.emat + D.elem0 : nullptr;
      const double *xs = nodes(lay.xs, D.ibeg), *ws = nodes(lay.ws, D.ibeg);
      const int nf = rec[0];
      for (int t = tid; t < nf; t += T) {
        if constexpr (TY == AKB_HEXAHEDRON_8)
          hex_forces<LIN>(rec, t, xs, ws, C, mp, m.mat_table, emat);
        else
          fan_forces<d, LIN>(rec, t, xs, ws, C, mp, m.mat_table, emat);
      }
    }
    {
      const bool ok = mbar_wait(mb + 8, it & 1);  // finishing inputs
      if (__syncthreads_or(!ok)) {
        cp_async_wait_all();
        if (tid == 0) {
          atomicExch(P.err, 1);
          mbar_wait(mb + 8, it & 1);
        }
        return;
      }
    }
    // the second pass may start launching (it waits for this grid)
    if (p + G >= P.npatch) grid_launch_dependents();
    asm volatile("" ::: "memory");
    // 3. finish, one thread per node, all of it in shared memory: an interior
    // node's v and a are updated where they were staged, its u is this step's w
    // (finish_dof) where w was staged, its next w takes X's place, and the four
    // slices go out by bulk copies (blocked DOFs as they were: w = u there). A
    // shared node's partial goes to its slot (the second pass adds them).
    const FanDesc D = descs[cur];
    const int ib = D.ibeg, nint = D.nint, nsh = D.nsh;
    const double dt = P.inst_dt ? P.inst_dt[D.inst] : dt0;
    const uint2* ent = entries(it);
    const uint16_t* cnt = rec + rec[5];
    const uint16_t* goff = rec + rec[6];
    uint32_t off[5];
    {
      size_t lo[5];
      uint32_t nbytes[5];
      finish_regions<d, FEXT>(ib, nint, off, lo, nbytes);
    }
    unsigned char* fin = smem + lay.fin;
    double* xs = nodes(lay.xs, ib);
    double* ws = nodes(lay.ws, ib);
    double* vs = reinterpret_cast<double*>(fin + off[0]);
    double* as = reinterpret_cast<double*>(fin + off[1]);
    const double* ims = reinterpret_cast<const double*>(fin + off[2]);
    const double* fxs = reinterpret_cast<const double*>(fin + off[4]);
    double ke = 0.0;  // M v^2 of this thread's DOFs after the step
    for (int j = tid; j < nint + nsh; j += T) {
      double f[d];
#pragma unroll
      for (int i = 0; i < d; ++i) f[i] = 0.0;
      const int n = cnt[j];
      const uint16_t* ix = rec + goff[j >> 5] + (j & 31);
#pragma unroll 2
      for (int q = 0; q < n; ++q) {
        double c[d];
        get_row<d>(C, ix[32 * q], c);
#pragma unroll
        for (int i = 0; i < d; ++i) f[i] -= c[i];
      }
      if (j < nint) {
        const double im = ims[j];
        double w[d], v[d], a[d], u[d], wn[d], v2 = 0.0;
        get_row<d>(ws, j, w);
        get_row<d>(vs, j, v);
        get_row<d>(as, j, a);
#pragma unroll
        for (int i = 0; i < d; ++i) {
          u[i] = wn[i] = w[i];
          if (!fin[off[3] + d * j + i])
            finish_dof(dt, FEXT ? f[i] + fxs[d * j + i] : f[i], im, w[i], v[i], a[i], u[i], wn[i]);
          v2 += v[i] * v[i];
        }
        put_row<d>(vs, j, v);
        put_row<d>(as, j, a);
        put_row<d>(xs, j, wn);
#pragma unroll
        for (int i = 0; i < d; ++i)
          if (!(u[i] == w[i])) ws[d * j + i] = u[i];  // only where u is not finite
        ke += ke_sum(v2, im);
      } else {
        put_row<d>(P.partial, (int)ent[j - nint].y, f);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before the bulk copies read
    const double s = cta_sum(ke, warp_sums);  // (also the barrier before the copies)
    if (tid == 0 && P.ke_part) P.ke_part[p] = s;
    // the slices' whole 16-byte units by bulk copies, the double before or after
    // them by itself
    const size_t s_lo = (size_t)ib * row, s_hi = s_lo + nint * row;
    const size_t b_lo = (s_lo + 15) & ~size_t(15), b_hi = s_hi & ~size_t(15);
    double* const dst[4] = {m.u, m.v, m.a, P.w};
    const double* const src[4] = {ws, vs, as, xs};
    if (tid == 0 && b_hi > b_lo) {
      const size_t at = (b_lo - s_lo) / sizeof(double);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                         reinterpret_cast<char*>(dst[k]) + b_lo),
                     "r"(saddr(src[k] + at)), "r"((uint32_t)(b_hi - b_lo))
                     : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    } else if (d == 3 && tid >= 32 && tid < 40 && nint > 0) {
      const int k = (tid - 32) & 3;
      const size_t q = tid < 36 ? s_lo : s_hi - 8;  // the slice's first and last double
      if ((tid < 36 && b_lo > s_lo) || (tid >= 36 && b_hi < s_hi))
        dst[k][q / sizeof(double)] = src[k][(q - s_lo) / sizeof(double)];
    }
    if (p + G < P.npatch) {
      cp_async_wait_all();  // the entries and the descriptor ahead
      __syncthreads();      // shared memory of this patch is free
    }
  }
}

// Listed nodes, one thread per (entry, component): the sum of the entry's
// partials in rank order (none for a node of no element), then the same
// finish as in the fused step, from the node's stored w; and the block's sum
// of M v^2 after the step (a kinetic-energy partial). The entry's own state
// (v, a, w, 1/M, blocked flag, f_ext) is not written by the fused step, and
// every kernel before the fused step has completed when this grid launches
// (the fused step waited for them before letting it launch): it is loaded
// before waiting for the fused step, through L2 (no L1 line of an earlier
// grid), so only the partials wait.
template <int D, bool FEXT>
__global__ void k_finish_list(DevModel m, DevPatches P, double dt0) {
  constexpr int d = D;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool on = t < P.nlist * d;
  const int64_t e = on ? t / d : 0;
  const int i = (int)(t - e * d);
  const bool sh = on && e < (int64_t)P.nshared;
  int64_t q = 0;
  uint32_t k = 0;
  uint8_t bl = 1;
  double dt = dt0, im = 1.0, w = 0.0, fx = 0.0, v = 0.0, a = 0.0;
  if (on) {
    // a single mesh's shared nodes are one block: no index to load
    const int64_t g = sh && P.shared_contig ? (int64_t)P.shared_base + e : (int64_t)P.list_gid[e];
    q = g * d + i;
    k = P.list_k[e];
    if (P.inst_dt) dt = P.inst_dt[P.list_inst[e]];
    bl = __ldcg(m.blocked + q);
    im = __ldcg(m.inv_mass + g);
    w = __ldcg(P.w + q);
    if (FEXT) fx = __ldcg(m.fext + q);
    v = __ldcg(m.v + q);
    a = __ldcg(m.a + q);
  }
  grid_wait();               // the fused step's partials
  grid_launch_dependents();  // the next step may start launching (it waits for this grid)
  double ke = 0.0;
  if (on) {
    double f = 0.0;
    if (sh) {  // ranks 0 and 1 in the dense rows at known addresses
      const double p0 = P.partial[(size_t)e * d + i];
      const double p1 = P.partial[((size_t)P.nshared + e) * d + i];  // zero when k = 1
      f += p0;
      if (k > 1) f += p1;
      if (k > 2) {
        const uint32_t over = P.list_part[e];
        for (uint32_t r = 2; r < k; ++r) f += P.partial[(size_t)(over + r - 2) * d + i];
      }
    }
    if (!bl) {
      double u, wn;
      finish_dof(dt, FEXT ? f + fx : f, im, w, v, a, u, wn);
      m.u[q] = u;
      m.v[q] = v;
      m.a[q] = a;
      P.w[q] = wn;
    }
    ke = ke_term(v, im);
  }
  if (P.ke_part) {
    __shared__ double warp_sums[kThreads / 32];
    const double s = cta_sum(ke, warp_sums);
    if (threadIdx.x == 0) P.ke_part[P.npatch + blockIdx.x] = s;
  }
}

// w = u + dt v + dt^2/2 a on free DOFs, w = u on blocked ones; one thread per
// DOF (batches: the node's instance by bisection of the node ranges).
__global__ void k_refresh_w(DevModel m, DevPatches P, double dt0) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= m.nn * m.dim) return;
  double u = m.u[q];
  if (!m.blocked[q]) {
    double dt = dt0;
    if (P.inst_dt) {
      const int64_t node = q / m.dim;
      int lo = 0, hi = P.ninst;  // node_off[lo] <= node < node_off[hi]
      while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (P.node_off[mid] <= node) lo = mid; else hi = mid;
      }
      dt = P.inst_dt[lo];
    }
    double v = m.v[q];
    fast::predict(dt, u, v, m.a[q]);
  }
  P.w[q] = u;
}

// Interface nodes of a partitioned mesh, one thread per (node, component):
// the sum of the node's partials in order (export), or the total over all
// parts written as its only partial (import).
// Component i of the partial of rank r of shared node s.
__device__ inline double& partial_of(const DevPatches& P, uint32_t s, uint32_t r, int d, int i) {
  return P.partial[(size_t)partial_slot(P.nshared, s, P.list_part[s], r) * d + i];
}

__global__ void k_iface_export(DevPatches P, const uint32_t* shared, const uint32_t* ks, int64_t n,
                               int d, double* out) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n * d) return;
  const int64_t e = t / d;
  const int i = (int)(t % d);
  const uint32_t s = shared[e], k = ks[e];
  double f = 0.0;
  for (uint32_t r = 0; r < k; ++r) f += partial_of(P, s, r, d, i);
  out[t] = f;
}

__global__ void k_iface_import(DevPatches P, const uint32_t* shared, const uint32_t* ks, int64_t n,
                               int d, const double* in) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n * d) return;
  const int64_t e = t / d;
  const int i = (int)(t % d);
  const uint32_t s = shared[e], k = ks[e];
  for (uint32_t r = 0; r < k; ++r) partial_of(P, s, r, d, i) = r == 0 ? in[t] : 0.0;
}

// One thread per (packed row, component); the own value of a row is the sum
// of its partial slots, as k_iface_export forms it.
__global__ void k_iface_pack(DevPatches P, const uint32_t* shared, const uint32_t* ks,
                             ExchangePlan x, int d, double* out) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= x.n_send * d) return;
  const int64_t j = t / d;
  const int i = (int)(t - j * d);
  const uint32_t e = x.send_rows[j];
  const uint32_t s = shared[e], k = ks[e];
  double f = 0.0;
  for (uint32_t r = 0; r < k; ++r) f += partial_of(P, s, r, d, i);
  out[t] = f;
}

// One thread per (interface row, component): the terms in the plan's order,
// then the total written as the row's only partial.
__global__ void k_iface_sum_import(DevPatches P, const uint32_t* shared, const uint32_t* ks,
                                   ExchangePlan x, int d, const double* recv) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= x.n_rows * d) return;
  const int64_t e = t / d;
  const int i = (int)(t - e * d);
  const uint32_t s = shared[e], k = ks[e];
  double own = 0.0;
  for (uint32_t r = 0; r < k; ++r) own += partial_of(P, s, r, d, i);
  double acc = 0.0;
  for (uint32_t j = x.sum_ptr[e]; j < x.sum_ptr[e + 1]; ++j) {
    const int32_t src = x.sum_src[j];
    acc += src < 0 ? own : recv[(int64_t)src * d + i];
  }
  for (uint32_t r = 0; r < k; ++r) partial_of(P, s, r, d, i) = r == 0 ? acc : 0.0;
}

__global__ void k_mass_pack(DevModel m, const uint32_t* nodes, ExchangePlan x, double* out) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= x.n_send) return;
  out[t] = m.mass[(int64_t)nodes[x.send_rows[t]] * m.dim];
}

__global__ void k_mass_sum_import(DevModel m, const uint32_t* nodes, ExchangePlan x,
                                  const double* recv) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= x.n_rows) return;
  const int64_t g = nodes[e];
  const double own = m.mass[g * m.dim];
  double M = 0.0;
  for (uint32_t j = x.sum_ptr[e]; j < x.sum_ptr[e + 1]; ++j) {
    const int32_t src = x.sum_src[j];
    M += src < 0 ? own : recv[src];
  }
  for (int c = 0; c < m.dim; ++c) m.mass[g * m.dim + c] = M;
  m.inv_mass[g] = 1. / M;
}

__global__ void k_mass_export(DevModel m, const uint32_t* nodes, int64_t n, double* out) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  out[t] = m.mass[(int64_t)nodes[t] * m.dim];
}

__global__ void k_mass_import(DevModel m, const uint32_t* nodes, int64_t n, const double* in) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int64_t g = nodes[t];
  const double M = in[t];
  for (int c = 0; c < m.dim; ++c) m.mass[g * m.dim + c] = M;
  m.inv_mass[g] = 1. / M;
}

template <typename V>
__global__ void k_permute_rows(const uint32_t* perm, int64_t n, int width, const V* in, V* out,
                               bool scatter) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n * width) return;
  const int64_t i = t / width;
  const int c = (int)(t - i * width);
  const int64_t j = perm[i];
  if (scatter)
    out[j * width + c] = in[t];
  else
    out[t] = in[j * width + c];
}

// grid of the patch kernel: one CTA per patch, or a persistent grid of
// P.grid CTAs that stride over the patches
inline int grid_of(const DevPatches& p) {
  return (p.grid > 0 && p.grid < p.npatch) ? p.grid : p.npatch;
}

inline int blocks_of(int64_t n) { return (int)((n + kThreads - 1) / kThreads); }

template <int T, typename S>
cudaError_t launch_patch(const DevModel& m, const DevPatches& p, double dt, bool fext,
                         cudaStream_t s) {
  const SmemLayout lay = layout(p, ET<T>::dim, sizeof(S), p.nbuf);
  const int grid = grid_of(p);
  if (grid < p.npatch)
    return fext ? launch_pdl(k_patch_step<T, S, true, true>, grid, kThreads, lay.total, s, m, p, dt)
                : launch_pdl(k_patch_step<T, S, false, true>, grid, kThreads, lay.total, s, m, p, dt);
  return fext ? launch_pdl(k_patch_step<T, S, true, false>, grid, kThreads, lay.total, s, m, p, dt)
              : launch_pdl(k_patch_step<T, S, false, false>, grid, kThreads, lay.total, s, m, p, dt);
}

// The dynamic shared memory limit is an attribute of the kernel function in
// the device's context, shared by every model of the process: it is only ever
// raised, so that a model built later with smaller patches cannot lower it
// below what an earlier model launches with.
std::mutex g_attr_mutex;

template <typename K>
cudaError_t raise_smem_limit(K kernel, size_t bytes) {
  cudaFuncAttributes attr;
  cudaError_t e = cudaFuncGetAttributes(&attr, kernel);
  if (e != cudaSuccess) return e;
  if ((size_t)attr.maxDynamicSharedSizeBytes >= bytes) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// f(kernel, threads) for the fan step's instantiation of a plan.
template <int TY, bool LIN, typename F>
cudaError_t with_fan_kernel(bool fext, F f) {
  constexpr int threads = FanBuild<TY, LIN>::threads;
  return fext ? f(k_fan_step<TY, LIN, true>, threads) : f(k_fan_step<TY, LIN, false>, threads);
}
template <typename F>
cudaError_t with_fan_kernel(int type, bool lin, bool fext, F f) {
  switch (type) {
  case AKB_TRIANGLE_3:
    return lin ? with_fan_kernel<AKB_TRIANGLE_3, true>(fext, f)
               : with_fan_kernel<AKB_TRIANGLE_3, false>(fext, f);
  case AKB_TETRAHEDRON_4:
    return lin ? with_fan_kernel<AKB_TETRAHEDRON_4, true>(fext, f)
               : with_fan_kernel<AKB_TETRAHEDRON_4, false>(fext, f);
  default:
    return lin ? with_fan_kernel<AKB_HEXAHEDRON_8, true>(fext, f)
               : with_fan_kernel<AKB_HEXAHEDRON_8, false>(fext, f);
  }
}

cudaError_t launch_fan(const DevModel& m, const DevPatches& p, double dt, bool fext,
                       cudaStream_t s) {
  const size_t bytes = fan_layout(p, m.dim, fext).total;
  return with_fan_kernel(m.type, p.linear, fext, [&](auto kernel, int threads) {
    const int grid = p.grid > 0 ? p.grid : p.resident[fext];
    return launch_pdl(kernel, std::min(grid, p.npatch), threads, bytes, s, m, p, dt);
  });
}

template <int T, typename S>
cudaError_t configure(const DevPatches& p) {
  const SmemLayout lay = layout(p, ET<T>::dim, sizeof(S), p.nbuf);
  std::lock_guard<std::mutex> lock(g_attr_mutex);
  cudaError_t e;
  if ((e = raise_smem_limit(k_patch_step<T, S, true, false>, lay.total)) != cudaSuccess) return e;
  if ((e = raise_smem_limit(k_patch_step<T, S, false, false>, lay.total)) != cudaSuccess) return e;
  if ((e = raise_smem_limit(k_patch_step<T, S, true, true>, lay.total)) != cudaSuccess) return e;
  return raise_smem_limit(k_patch_step<T, S, false, true>, lay.total);
}

}  // namespace

size_t patch_smem_bytes(const DevPatches& p, int dim, bool fp32, int nbuf) {
  return layout(p, dim, fp32 ? 4 : 8, nbuf).total;
}

size_t fan_smem_bytes(const PatchHost& p, int dim) {
  return fan_layout(p.max_nodes, p.max_interior, p.max_shared, p.contrib_slots, p.chunk_bytes, dim,
                    true).total;
}

cudaError_t fan_configure(const DevModel& m, const DevPatches& p, int device, int* resident) {
  int sms = 0, per_sm = 0;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_attr_mutex);
  for (int k = 0; k < 2; ++k) {
    const size_t bytes = fan_layout(p, m.dim, k).total;
    e = with_fan_kernel(m.type, p.linear, k, [&](auto kernel, int threads) {
      const cudaError_t r = raise_smem_limit(kernel, bytes);
      return r != cudaSuccess
                 ? r
                 : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, bytes);
    });
    if (e != cudaSuccess) return e;
    resident[k] = sms * per_sm;
  }
  return cudaSuccess;
}

int patch_buffers(const DevPatches& p, int type, bool fp32) {
  // CTAs per SM: 228 KB of shared memory, 1 KB reserved per CTA, and the
  // register budget the instantiation is built for
  int regs;
  switch (type) {
  case AKB_HEXAHEDRON_8: regs = fp32 ? PatchOccupancy<AKB_HEXAHEDRON_8, float>::value
                                     : PatchOccupancy<AKB_HEXAHEDRON_8, double>::value; break;
  case AKB_TETRAHEDRON_4: regs = fp32 ? PatchOccupancy<AKB_TETRAHEDRON_4, float>::value
                                      : PatchOccupancy<AKB_TETRAHEDRON_4, double>::value; break;
  case AKB_TRIANGLE_3: regs = fp32 ? PatchOccupancy<AKB_TRIANGLE_3, float>::value
                                   : PatchOccupancy<AKB_TRIANGLE_3, double>::value; break;
  default: regs = fp32 ? PatchOccupancy<AKB_SEGMENT_2, float>::value
                       : PatchOccupancy<AKB_SEGMENT_2, double>::value; break;
  }
  const int dim = type == AKB_SEGMENT_2 ? 1 : type == AKB_TRIANGLE_3 ? 2 : 3;
  auto ctas = [&](int nbuf) {
    const size_t s = layout(p, dim, fp32 ? 4 : 8, nbuf).total + 1024;
    return std::min<int>(regs, (int)((228 * 1024) / s));
  };
  return ctas(2) >= ctas(1) ? 2 : 1;
}

cudaError_t patch_configure(const DevModel& m, const DevPatches& p, bool fp32) {
  switch (m.type) {
  case AKB_SEGMENT_2: return fp32 ? configure<AKB_SEGMENT_2, float>(p) : configure<AKB_SEGMENT_2, double>(p);
  case AKB_TRIANGLE_3: return fp32 ? configure<AKB_TRIANGLE_3, float>(p) : configure<AKB_TRIANGLE_3, double>(p);
  case AKB_TETRAHEDRON_4: return fp32 ? configure<AKB_TETRAHEDRON_4, float>(p) : configure<AKB_TETRAHEDRON_4, double>(p);
  default: return fp32 ? configure<AKB_HEXAHEDRON_8, float>(p) : configure<AKB_HEXAHEDRON_8, double>(p);
  }
}

cudaError_t patch_step(const DevModel& m, const DevPatches& p, double dt, bool fp32,
                       bool fext, cudaStream_t s) {
  if (p.npatch == 0) return cudaSuccess;
  if (p.fans) return launch_fan(m, p, dt, fext, s);
  switch (m.type) {
  case AKB_SEGMENT_2:
    return fp32 ? launch_patch<AKB_SEGMENT_2, float>(m, p, dt, fext, s)
                : launch_patch<AKB_SEGMENT_2, double>(m, p, dt, fext, s);
  case AKB_TRIANGLE_3:
    return fp32 ? launch_patch<AKB_TRIANGLE_3, float>(m, p, dt, fext, s)
                : launch_patch<AKB_TRIANGLE_3, double>(m, p, dt, fext, s);
  case AKB_TETRAHEDRON_4:
    return fp32 ? launch_patch<AKB_TETRAHEDRON_4, float>(m, p, dt, fext, s)
                : launch_patch<AKB_TETRAHEDRON_4, double>(m, p, dt, fext, s);
  default:
    return fp32 ? launch_patch<AKB_HEXAHEDRON_8, float>(m, p, dt, fext, s)
                : launch_patch<AKB_HEXAHEDRON_8, double>(m, p, dt, fext, s);
  }
}

cudaError_t patch_finish_list(const DevModel& m, const DevPatches& p, double dt, bool fext,
                              cudaStream_t s) {
  if (p.nlist <= 0) return cudaSuccess;
  const int blocks = blocks_of(p.nlist * m.dim);
  switch (m.dim) {
  case 1: return fext ? launch_pdl(k_finish_list<1, true>, blocks, kThreads, 0, s, m, p, dt)
                      : launch_pdl(k_finish_list<1, false>, blocks, kThreads, 0, s, m, p, dt);
  case 2: return fext ? launch_pdl(k_finish_list<2, true>, blocks, kThreads, 0, s, m, p, dt)
                      : launch_pdl(k_finish_list<2, false>, blocks, kThreads, 0, s, m, p, dt);
  default: return fext ? launch_pdl(k_finish_list<3, true>, blocks, kThreads, 0, s, m, p, dt)
                       : launch_pdl(k_finish_list<3, false>, blocks, kThreads, 0, s, m, p, dt);
  }
}

int64_t patch_ke_parts(const DevPatches& p, int dim) {
  return p.npatch + (p.nlist > 0 ? blocks_of(p.nlist * dim) : 0);
}

cudaError_t patch_refresh_w(const DevModel& m, const DevPatches& p, double dt, cudaStream_t s) {
  if (m.nn == 0) return cudaSuccess;
  k_refresh_w<<<blocks_of(m.nn * m.dim), kThreads, 0, s>>>(m, p, dt);
  return cudaGetLastError();
}

cudaError_t patch_iface_export(const DevModel& m, const DevPatches& p, const uint32_t* shared,
                               const uint32_t* k, int64_t n, double* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_iface_export<<<blocks_of(n * m.dim), kThreads, 0, s>>>(p, shared, k, n, m.dim, out);
  return cudaGetLastError();
}

cudaError_t patch_iface_import(const DevModel& m, const DevPatches& p, const uint32_t* shared,
                               const uint32_t* k, int64_t n, const double* in, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_iface_import<<<blocks_of(n * m.dim), kThreads, 0, s>>>(p, shared, k, n, m.dim, in);
  return cudaGetLastError();
}

cudaError_t mass_export(const DevModel& m, const uint32_t* nodes, int64_t n, double* out,
                        cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_mass_export<<<blocks_of(n), kThreads, 0, s>>>(m, nodes, n, out);
  return cudaGetLastError();
}

cudaError_t mass_import(const DevModel& m, const uint32_t* nodes, int64_t n, const double* in,
                        cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_mass_import<<<blocks_of(n), kThreads, 0, s>>>(m, nodes, n, in);
  return cudaGetLastError();
}

cudaError_t patch_iface_pack(const DevModel& m, const DevPatches& p, const uint32_t* shared,
                             const uint32_t* k, const ExchangePlan& x, double* out,
                             cudaStream_t s) {
  if (x.n_send <= 0) return cudaSuccess;
  k_iface_pack<<<blocks_of(x.n_send * m.dim), kThreads, 0, s>>>(p, shared, k, x, m.dim, out);
  return cudaGetLastError();
}

cudaError_t patch_iface_sum_import(const DevModel& m, const DevPatches& p, const uint32_t* shared,
                                   const uint32_t* k, const ExchangePlan& x, const double* recv,
                                   cudaStream_t s) {
  if (x.n_rows <= 0) return cudaSuccess;
  k_iface_sum_import<<<blocks_of(x.n_rows * m.dim), kThreads, 0, s>>>(p, shared, k, x, m.dim, recv);
  return cudaGetLastError();
}

cudaError_t mass_pack(const DevModel& m, const uint32_t* nodes, const ExchangePlan& x,
                      double* out, cudaStream_t s) {
  if (x.n_send <= 0) return cudaSuccess;
  k_mass_pack<<<blocks_of(x.n_send), kThreads, 0, s>>>(m, nodes, x, out);
  return cudaGetLastError();
}

cudaError_t mass_sum_import(const DevModel& m, const uint32_t* nodes, const ExchangePlan& x,
                            const double* recv, cudaStream_t s) {
  if (x.n_rows <= 0) return cudaSuccess;
  k_mass_sum_import<<<blocks_of(x.n_rows), kThreads, 0, s>>>(m, nodes, x, recv);
  return cudaGetLastError();
}

cudaError_t permute_rows(const uint32_t* perm, int64_t n, int width, const double* in,
                         double* out, bool scatter, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_permute_rows<double><<<blocks_of(n * width), kThreads, 0, s>>>(perm, n, width, in, out, scatter);
  return cudaGetLastError();
}

cudaError_t permute_rows_u8(const uint32_t* perm, int64_t n, int width, const uint8_t* in,
                            uint8_t* out, bool scatter, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_permute_rows<uint8_t><<<blocks_of(n * width), kThreads, 0, s>>>(perm, n, width, in, out, scatter);
  return cudaGetLastError();
}

}  // namespace akb
