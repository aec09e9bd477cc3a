// K4-C: the blockwise Jacobi SVD with each coupled sector spread over a thread-block
// cluster.
//
// The same method as block_svd_kernel (tnb_svd.cu) -- one-sided Jacobi, the same round-robin
// order of column pairs, the same rotations -- with a warp per column pair, so that all
// ceil(c / 2) pairs of a step run at once on up to 16 SMs.  What bounds the method is the
// chain of steps, (c - 1) per sweep and 10-25 sweeps: a decaying spectrum takes 20 or more.
// In one CTA of 16 warps a step of 58 pairs is four rounds of dot products, shuffles and a
// dependent divide / square root chain, between two CTA barriers.
//
// Round robin as a systolic array: pair k > 0 of step s holds columns (s + k) and (s - k)
// modulo n1 = cp - 1, pair 0 holds the fixed column n1 and column s.  From one step to the
// next every column moves to a neighbouring pair (slot A of pair k to pair k - 1, slot B to
// pair k + 1, turning round at the ends), so a pair's warp writes its two rotated columns
// straight into its neighbours' shared memory and signals the receiver's mbarrier; no step
// has a barrier.  Within a CTA that is a plain store and an arrive, across CTAs st.async,
// whose bytes complete the receiver's mbarrier themselves: a store followed by an arrive
// with cluster-scope release cost 1,500-1,900 clocks a step.  Buffers alternate between two
// slots: a neighbour sends its step-s columns only after it has read its own step-s buffers, and
// this warp writes those buffers again only after receiving them, so two slots suffice.  One
// cluster barrier per sweep decides convergence.  A warp whose wait gives up leaves the sweep,
// sends nothing more and says so at that barrier: the whole cluster then stops and the
// sector's info word is -TNB_ETIMEOUT.  (Its vote, behind the loads of the received columns,
// takes 1 % of the launch; before them 5 %.)
//
// Measured on B200 (the whole launch, before: block_svd_kernel): ten SU(2) sectors up to 116
// x 116, 2.4 ms (16.5); two 128 x 128 sectors, 2.7 ms (18.9); sectors up to 49 x 49, 0.68
// ms (2.18); up to 22 x 22, 0.24 ms (0.34); up to 5 x 5, 30 us (32) -- the same sweeps and the
// same bits.  A step of 128 columns is about 1,800 clocks: dot products and their shuffles
// 350, the divide / square root chain 470, rotation and sends 300, and the rest the
// hand-over between CTAs.  Sending W ahead of V (V's rotation then overlaps W's way) measured
// slower, 3.2 against 2.35 ms: every mbarrier wait costs some 250 clocks even when it is ready.
//
// Limits: max(m, n) <= 512 and min(m, n) <= 256 (the columns of at most eight pairs, two
// slots each, in one CTA's shared memory); larger sectors, and those it is slower for
// (linalg.cluster_sectors), take block_svd_kernel.
#include <string>
#include <type_traits>

#include "tnb_common.cuh"

namespace tnb {

constexpr int kScMaxR = 512, kScMaxC = 256, kScMaxWarps = 8, kScMaxCluster = 16;
constexpr int kScRow = 8;  // m, n, a_off, u_off, s_off, vt_off, (w_off), pad
constexpr int kScMaxSweeps = 64;
constexpr double kScTol = 1e-15;  // rotate while |a_i . a_j| > tol * |a_i| |a_j|
constexpr long long kScWaitCycles = 4000000000LL;  // ~2 s at the boost clock
constexpr long long kScDrainCycles = 200000;  // ~0.1 ms: copies in flight land in microseconds

__device__ __forceinline__ double sc_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ uint32_t sc_smem(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint32_t sc_mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ void sc_cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Wait for a phase whose data came from this CTA (`remote` false) or partly from a peer.
__device__ __forceinline__ bool sc_test(uint32_t mbar, uint32_t parity, bool remote) {
  uint32_t done;
  if (remote)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
  return done != 0;
}
__device__ __forceinline__ bool sc_wait(uint32_t mbar, uint32_t parity, bool remote,
                                        long long limit) {
  if (sc_test(mbar, parity, remote)) return true;
  const long long t0 = clock64();
  while (!sc_test(mbar, parity, remote))
    if (clock64() - t0 > limit) return false;
  return true;
}

// Two elements of a column to a slot of this CTA, or of a peer CTA (whose mbarrier counts
// the bytes).
__device__ __forceinline__ void sc_put(uint32_t addr, double x, double y) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" :: "r"(addr), "d"(x), "d"(y) : "memory");
}
__device__ __forceinline__ void sc_put_remote(uint32_t addr, double x, double y, uint32_t mbar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];"
      :: "r"(addr), "d"(x), "d"(y), "r"(mbar) : "memory");
}

__device__ __forceinline__ void sc_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" :: "r"(mbar) : "memory");
}

// One column slot's destination in the next step.
struct ScDest {
  uint32_t data, mbar;  // slot 0's addresses (shared::cta, or mapped to the peer)
  bool remote;
};

// Whether a pair is rotated: |ga| > tol sqrt(al) sqrt(be), neither norm zero.  Squares decide
// it unless they come within 1e-12 of each other or al be leaves [1e-200, 1e200]; the two
// square roots in the chain of every step cost more than the rest of the test.
__device__ __forceinline__ bool sc_rotates(double al, double be, double ga) {
  const double q = al * be, g2 = ga * ga, th = (kScTol * kScTol) * q;
  if (q > 1e-200 && q < 1e200) {
    if (g2 > th * (1.0 + 1e-12)) return true;
    if (g2 < th * (1.0 - 1e-12)) return false;
  }
  return fabs(ga) > kScTol * sqrt(al) * sqrt(be) && al != 0.0 && be != 0.0;
}

// The rotation of block_svd_kernel on a lane's elements of two columns, with that kernel's
// fused operations: near a tie of two columns' norms a last-bit difference can turn a
// rotation the other way and with it the sign of a singular pair.
template <int E>
__device__ __forceinline__ void sc_rotate(double cs, double sn, double (&lo)[E], double (&hi)[E]) {
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const double x = lo[e], y = hi[e];
    lo[e] = fma(cs, x, -__dmul_rn(sn, y));
    hi[e] = fma(sn, x, __dmul_rn(cs, y));
  }
}

template <int E>
__global__ void __launch_bounds__(kScMaxWarps * 32)
block_svd_cluster_kernel(const int64_t* __restrict__ rows, int64_t n_rows,
                         const double* __restrict__ a, int64_t n_a, double* __restrict__ u,
                         int64_t n_u, double* __restrict__ s, int64_t n_s,
                         double* __restrict__ vt, int64_t n_vt, int32_t* __restrict__ info,
                         int64_t smem_doubles, int cl, long long wait_cycles) {
  extern __shared__ __align__(16) double sc_buf[];
  __shared__ __align__(8) uint64_t mbar[kScMaxWarps][2];
  // what a sweep's pairs found (1: a rotation, 2: a wait gave up), three sweeps in turn, and the
  // same for the hand-over after the last sweep
  __shared__ unsigned rotated[4];
  __shared__ double sig[kScMaxC];
  __shared__ double red[kScMaxWarps];
  const int rank = static_cast<int>(blockIdx.x) % cl;
  const int64_t b = blockIdx.x / cl;
  if (b >= n_rows) return;
  const int64_t* row = rows + b * kScRow;
  const int64_t m = row[0], n = row[1], a_off = row[2], u_off = row[3], s_off = row[4],
                vt_off = row[5];
  const bool trans = m < n;
  const int64_t r64 = trans ? n : m, c64 = trans ? m : n;  // W = A or A^T: r x c, r >= c
  const int nw = blockDim.x / 32;
  // (every CTA of the cluster takes the same branch: the conditions are the row's)
  const bool ok = m >= 0 && n >= 0 && c64 <= kScMaxC && r64 <= 32 * E && r64 <= kScMaxR &&
                  a_off >= 0 && a_off + m * n <= n_a && u_off >= 0 && u_off + m * c64 <= n_u &&
                  s_off >= 0 && s_off + c64 <= n_s && vt_off >= 0 && vt_off + c64 * n <= n_vt;
  const int r = static_cast<int>(r64), c = static_cast<int>(c64);
  const int K = (c + 1) / 2, n1 = 2 * K - 1;  // pairs; steps per sweep
  const int pw = ok ? (K + cl - 1) / cl : 0;  // pairs (warps) per CTA
  // a column in a slot: 32-element groups of W, then of V, two groups interleaved so that a
  // lane's elements of both are one 16-byte access; an odd last group has an empty partner
  const int ew = (r + 63) / 64, ev = (c + 63) / 64, ld = 64 * (ew + ev);
  if (!ok || pw > nw || static_cast<int64_t>(pw) * 4 * ld > smem_doubles) {
    if (threadIdx.x == 0 && rank == 0) {
      raise_bounds();
      info[b] = -1;
    }
    return;
  }
  if (c == 0) {
    if (threadIdx.x == 0 && rank == 0) info[b] = 0;
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k = rank * pw + warp;  // this warp's pair
  const bool active = warp < pw && k < K;

  // incoming columns from this CTA arrive once each; those from a peer are counted in bytes,
  // announced by this warp's own arrival
  const int from_a = k == 0 || k == K - 1 ? k : k + 1;
  const int from_b = k == 0 ? (K == 1 ? 0 : 1) : k - 1;
  const int remote_in = (from_a / pw != rank) + (from_b / pw != rank);
  if (active && lane == 0) {
    const int count = 2 - remote_in + (remote_in > 0);
    for (int q = 0; q < 2; ++q)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;"
                   :: "r"(sc_smem(&mbar[warp][q])), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 4) rotated[tid] = 0;

  // where slot A (col 0) and slot B (col 1) of this pair go: pair, then slot of the receiver
  const uint32_t slot_bytes = static_cast<uint32_t>(2 * ld * 8);  // one buffer: both columns
  auto dest = [&](int pair, int col) {
    ScDest d;
    const int cta = pair / pw, w = pair % pw;
    const uint32_t data = sc_smem(sc_buf) + static_cast<uint32_t>(w) * 2 * slot_bytes +
                          static_cast<uint32_t>(col * ld * 8);
    const uint32_t mb = sc_smem(&mbar[w][0]);
    d.remote = cta != rank;
    d.data = d.remote ? sc_mapa(data, static_cast<uint32_t>(cta)) : data;
    d.mbar = d.remote ? sc_mapa(mb, static_cast<uint32_t>(cta)) : mb;
    return d;
  };
  ScDest da{}, db{};
  if (active) {
    da = k <= 1 ? dest(0, k) : dest(k - 1, 0);
    db = K == 1 ? dest(0, 1) : (k == K - 1 ? dest(k, 0) : dest(k + 1, 1));
  }
  const double* const mine = sc_buf + static_cast<size_t>(warp) * 4 * ld;
  const uint32_t mb0 = sc_smem(&mbar[warp < kScMaxWarps ? warp : 0][0]);
  const uint32_t flag0 = sc_mapa(sc_smem(&rotated[0]), 0);

  // this pair's columns, a lane's elements q = lane + 32 e of each
  double wa[E], wb[E], va[E], vb[E];
  auto home = [&](int col, int st) {  // the column in slot A / B of pair k at step st
    if (k == 0) return col == 0 ? n1 : st;
    int x = col == 0 ? st + k : st - k;
    if (x >= n1) x -= n1;
    if (x < 0) x += n1;
    return x;
  };
  {
    const int ia = active ? home(0, 0) : c, ib = active ? home(1, 0) : c;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int q = lane + 32 * e;
      auto load = [&](int j) -> double {
        if (j >= c || q >= r) return 0.0;
        return trans ? __ldg(a + a_off + static_cast<int64_t>(j) * n + q)
                     : __ldg(a + a_off + static_cast<int64_t>(q) * n + j);
      };
      wa[e] = load(ia);
      wb[e] = load(ib);
      va[e] = q == ia ? 1.0 : 0.0;
      vb[e] = q == ib ? 1.0 : 0.0;
    }
  }
  sc_cluster_sync();  // every CTA's mbarriers are ready

  auto announce = [&](uint32_t slot) {  // the bytes that peers will send to `slot`
    if (remote_in && lane == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                   :: "r"(mb0 + 8u * slot), "r"(static_cast<uint32_t>(remote_in * ld * 8))
                   : "memory");
  };
  if (active) announce(1);
  bool dead = wait_cycles == 0;  // a wait gave up
  uint32_t t = 0;          // steps done; the buffer in use is t & 1
  auto receive = [&]() {   // step t's columns
    const uint32_t slot = t & 1u;
    if (!dead && !sc_wait(mb0 + 8u * slot, ((t - 1) >> 1) & 1u, remote_in > 0, wait_cycles))
      dead = true;
    const double* p = mine + slot * 2 * ld + 2 * lane;
    auto load = [&](const double* q, int groups, double (&x)[E]) {
#pragma unroll
      for (int e = 0; e < E; e += 2) {
        if (e < groups) {
          const double2 v = *reinterpret_cast<const double2*>(q + 32 * e);
          x[e] = v.x;
          if (e + 1 < E) x[e + 1] = v.y;
        }
      }
    };
    load(p, 2 * ew, wa);
    load(p + ld, 2 * ew, wb);
    load(p + 64 * ew, 2 * ev, va);
    load(p + ld + 64 * ew, 2 * ev, vb);
    dead = __any_sync(0xffffffffu, dead);  // the whole warp's
    if (!dead) announce(slot ^ 1u);
  };
  auto report = [&](int word, bool any) {  // to rank 0's words
    const unsigned found = (any ? 1u : 0u) | (dead ? 2u : 0u);
    if (found != 0u && lane == 0)
      asm volatile("red.shared::cluster.or.b32 [%0], %1;" :: "r"(flag0 + 4u * word), "r"(found)
                   : "memory");
  };
  auto reported = [&](int word) {
    uint32_t f;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(f) : "r"(flag0 + 4u * word) : "memory");
    return f;
  };
  // a column to the next step's slot (t already counts that step)
  auto send = [&](const ScDest& d, const double (&w)[E], const double (&v)[E]) {
    const uint32_t off = d.data + (t & 1u) * slot_bytes + 16u * lane;
    const uint32_t mb = d.mbar + 8u * (t & 1u);
    auto put = [&](uint32_t to, int groups, const double (&x)[E]) {
#pragma unroll
      for (int e = 0; e < E; e += 2) {
        if (e < groups) {
          const double hi = e + 1 < E ? x[e + 1 < E ? e + 1 : e] : 0.0;
          if (d.remote)
            sc_put_remote(to + 256u * e, x[e], hi, mb);
          else
            sc_put(to + 256u * e, x[e], hi);
        }
      }
    };
    put(off, 2 * ew, w);
    put(off + 512u * ew, 2 * ev, v);
  };

  int sweep = 0;
  bool converged = c == 1, gave_up = false;
  for (; sweep < kScMaxSweeps && !converged && !gave_up; ++sweep) {
    bool any = false;
    if (active) {
#pragma unroll 1
      for (int step = 0; step < n1; ++step) {
        if (t > 0) {
          receive();
          if (dead) break;
        }
        const int ia = home(0, step), ib = home(1, step);
        if (ia < c && ib < c) {  // (else one is the padding column)
          double aa = 0.0, bb = 0.0, ga = 0.0;
#pragma unroll
          for (int e = 0; e < E; ++e) {
            aa = fma(wa[e], wa[e], aa);
            bb = fma(wb[e], wb[e], bb);
            ga = fma(wa[e], wb[e], ga);
          }
          aa = sc_warp_sum(aa);
          bb = sc_warp_sum(bb);
          ga = sc_warp_sum(ga);
          // the pair in column order: al the lower column's, be the higher one's
          const bool swap = ia > ib;
          const double al = swap ? bb : aa, be = swap ? aa : bb;
          if (sc_rotates(al, be, ga)) {
            const double zeta = (be - al) / (2.0 * ga);
            const double tt = fabs(zeta) > 1e150
                                  ? 0.5 / zeta
                                  : copysign(1.0, zeta) / (fabs(zeta) + sqrt(fma(zeta, zeta, 1.0)));
            const double cs = 1.0 / sqrt(fma(tt, tt, 1.0)), sn = cs * tt;
            if (swap) {
              sc_rotate<E>(cs, sn, wb, wa);
              sc_rotate<E>(cs, sn, vb, va);
            } else {
              sc_rotate<E>(cs, sn, wa, wb);
              sc_rotate<E>(cs, sn, va, vb);
            }
            any = true;
          }
        }
        ++t;
        send(da, wa, va);
        send(db, wb, vb);
        __syncwarp();
        if (lane == 0) {
          if (!da.remote) sc_arrive(da.mbar + 8u * (t & 1u));
          if (!db.remote) sc_arrive(db.mbar + 8u * (t & 1u));
        }
      }
      report(sweep % 3, any);
    }
    if (rank == 0 && tid == 0) rotated[(sweep + 1) % 3] = 0;
    sc_cluster_sync();
    const uint32_t f = reported(sweep % 3);  // (the same in every CTA)
    converged = f == 0;
    gave_up = (f & 2u) != 0;
  }

  // singular values: the column norms, to every CTA of the cluster
  const int ia = active ? home(0, 0) : c, ib = active ? home(1, 0) : c;
  if (active && t > 0 && !gave_up) {
    receive();
    report(3, false);
  }
  double na = 0.0, nb = 0.0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    na = fma(wa[e], wa[e], na);
    nb = fma(wb[e], wb[e], nb);
  }
  na = sqrt(sc_warp_sum(na));
  nb = sqrt(sc_warp_sum(nb));
  if (lane < cl) {
    const uint32_t p = sc_mapa(sc_smem(sig), static_cast<uint32_t>(lane));
    if (ia < c)
      asm volatile("st.shared::cluster.f64 [%0], %1;" :: "r"(p + 8u * ia), "d"(na) : "memory");
    if (ib < c)
      asm volatile("st.shared::cluster.f64 [%0], %1;" :: "r"(p + 8u * ib), "d"(nb) : "memory");
  }
  sc_cluster_sync();
  if (gave_up || reported(3) != 0u) {  // (the same in every CTA)
    const long long t0 = clock64();
    while (clock64() - t0 < kScDrainCycles) {
    }
    if (rank == 0 && tid == 0) {
      atomicCAS(&g_device_error, 0, TNB_ETIMEOUT);
      info[b] = -TNB_ETIMEOUT;
    }
    sc_cluster_sync();  // no CTA leaves while a peer may still read its shared memory
    return;
  }

  // outputs in descending order (ties by column index): column j goes to position p(j)
  auto position = [&](int j) {
    const double v = sig[j];
    int p = 0;
    for (int q = lane; q < c; q += 32) p += (sig[q] > v || (sig[q] == v && q < j)) ? 1 : 0;
    return static_cast<int>(__reduce_add_sync(0xffffffffu, static_cast<unsigned>(p)));
  };
  double* const wout = trans ? vt + vt_off : u + u_off;   // W's columns
  double* const vout = trans ? u + u_off : vt + vt_off;   // V's columns
  const int64_t w_col = trans ? n : 1, w_el = trans ? 1 : c;
  const int64_t v_col = trans ? 1 : n, v_el = trans ? c : 1;
  auto emit = [&](int j, double v, const double* w, const double* z) {
    if (j >= c) return;
    const int64_t p = position(j);
    if (lane == 0) s[s_off + p] = v;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int q = lane + 32 * e;
      // (a norm that is NaN leaves its column as it is; a zero one is completed below)
      if (q < r && v != 0.0) wout[p * w_col + q * w_el] = v > 0.0 ? w[e] / v : w[e];
      if (q < c) vout[p * v_col + q * v_el] = z[e];
    }
  };
  if (active) {
    emit(ia, na, wa, va);
    emit(ib, nb, wb, vb);
  }
  // columns of exactly zero norm: an orthonormal completion in column order, by rank 0 from
  // the columns written above (a unit vector orthogonalised twice against every column
  // ranked before it)
  bool zero = false;
  for (int q = lane; q < c; q += 32) zero = zero || sig[q] == 0.0;
  zero = __any_sync(0xffffffffu, zero);
  sc_cluster_sync();  // also: no CTA leaves while a peer may still read its shared memory
  if (rank == 0 && zero) {
    double* const wz = sc_buf;  // r doubles: the column being completed
    auto cta_sum = [&](double v) {
      v = sc_warp_sum(v);
      __syncthreads();
      if (lane == 0) red[warp] = v;
      __syncthreads();
      double x = 0.0;
      for (int w = 0; w < nw; ++w) x += red[w];
      return x;
    };
    for (int jz = 0; jz < c; ++jz) {
      if (sig[jz] != 0.0) continue;
      const int64_t pz = position(jz);
      for (int cand = 0; cand < r; ++cand) {
        __syncthreads();
        for (int q = tid; q < r; q += blockDim.x) wz[q] = q == cand ? 1.0 : 0.0;
        __syncthreads();
        for (int pass = 0; pass < 2; ++pass) {
          for (int64_t p = 0; p < pz; ++p) {
            const double* wp = wout + p * w_col;
            double d = 0.0;
            for (int q = tid; q < r; q += blockDim.x) d = fma(__ldcg(wp + q * w_el), wz[q], d);
            d = cta_sum(d);
            for (int q = tid; q < r; q += blockDim.x) wz[q] -= d * __ldcg(wp + q * w_el);
            __syncthreads();
          }
        }
        double nn = 0.0;
        for (int q = tid; q < r; q += blockDim.x) nn = fma(wz[q], wz[q], nn);
        nn = cta_sum(nn);
        if (nn > 0.25) {
          const double inv = 1.0 / sqrt(nn);
          for (int q = tid; q < r; q += blockDim.x) __stcg(wout + pz * w_col + q * w_el, wz[q] * inv);
          __syncthreads();
          break;
        }
      }
    }
  }
  if (rank == 0 && tid == 0) info[b] = converged ? 0 : sweep;
}

// Cluster size, warps per CTA and dynamic shared memory of a launch whose sectors have
// max(m, n) <= r and min(m, n) <= c; false when the kernel does not take them.
struct ScShape {
  int cl, warps;
  size_t smem;
};
static bool sc_shape(int64_t r, int64_t c, ScShape* out) {
  if (r < 0 || c < 0 || c > r || r > kScMaxR || c > kScMaxC) return false;
  const int64_t pairs = c < 2 ? 1 : (c + 1) / 2;
  // four pairs per CTA, a warp on each of the SM's schedulers, up to 16 CTAs (two or eight
  // per CTA: within 1 % and 5-10 % slower at 64 pairs, all within 3 % up to 15 pairs)
  int cl = 1;
  while (cl < kScMaxCluster && pairs > 4 * cl) cl *= 2;
  out->cl = cl;
  out->warps = static_cast<int>((pairs + cl - 1) / cl);
  out->smem = static_cast<size_t>(out->warps) * 4 * 64 * ((r + 63) / 64 + (c + 63) / 64) * 8;
  return out->warps <= kScMaxWarps && out->smem <= 220 * 1024;
}

template <int E>
static cudaError_t sc_config(const ScShape& sh, unsigned grid, cudaStream_t stream,
                             cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr) {
  static PerDeviceOnce opted;
  const cudaError_t e = opted.once([] {
    cudaError_t x = cudaFuncSetAttribute(block_svd_cluster_kernel<E>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         220 * 1024);
    if (x == cudaSuccess)
      x = cudaFuncSetAttribute(block_svd_cluster_kernel<E>,
                               cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return x;
  });
  if (e != cudaSuccess) return e;
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(grid);
  cfg->blockDim = dim3(static_cast<unsigned>(sh.warps * 32));
  cfg->dynamicSmemBytes = sh.smem;
  cfg->stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(sh.cl);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  return cudaSuccess;
}

// f(std::integral_constant-like tag) for the elements per lane a column of r rows needs.
template <class F>
static auto sc_dispatch(int64_t r, F&& f) {
  if (r <= 32) return f(std::integral_constant<int, 1>{});
  if (r <= 64) return f(std::integral_constant<int, 2>{});
  if (r <= 128) return f(std::integral_constant<int, 4>{});
  if (r <= 256) return f(std::integral_constant<int, 8>{});
  return f(std::integral_constant<int, 16>{});
}

}  // namespace tnb

extern "C" int tnb_block_svd_cluster_ok(int64_t max_r, int64_t max_c) {
  return tnb_block_svd_cluster_count(max_r, max_c) > 0 ? 1 : 0;
}

extern "C" int64_t tnb_block_svd_cluster_count(int64_t max_r, int64_t max_c) {
  tnb::ScShape sh;
  if (!tnb::sc_shape(max_r, max_c, &sh)) return 0;
  return tnb::sc_dispatch(max_r, [&](auto tag) {
    constexpr int E = decltype(tag)::value;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    int n = 0;
    if (tnb::sc_config<E>(sh, static_cast<unsigned>(sh.cl), nullptr, &cfg, attr) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, tnb::block_svd_cluster_kernel<E>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return n;
  });
}

extern "C" int tnb_block_svd_cluster(const int64_t* rows, int64_t n_rows, const double* a,
                                     int64_t n_a, double* u, int64_t n_u, double* s, int64_t n_s,
                                     double* vt, int64_t n_vt, int32_t* info, int64_t max_r,
                                     int64_t max_c, void* stream) {
  return tnb_block_svd_cluster_bounded(rows, n_rows, a, n_a, u, n_u, s, n_s, vt, n_vt, info, max_r,
                                       max_c, tnb::kScWaitCycles, stream);
}

extern "C" int tnb_block_svd_cluster_bounded(const int64_t* rows, int64_t n_rows, const double* a,
                                             int64_t n_a, double* u, int64_t n_u, double* s,
                                             int64_t n_s, double* vt, int64_t n_vt, int32_t* info,
                                             int64_t max_r, int64_t max_c, int64_t wait_cycles,
                                             void* stream) {
  TNB_REQUIRE(n_rows >= 0 && n_a >= 0 && n_u >= 0 && n_s >= 0 && n_vt >= 0 && wait_cycles >= 0,
              "tnb_block_svd_cluster: negative size");
  tnb::ScShape sh;
  TNB_REQUIRE(tnb::sc_shape(max_r, max_c, &sh),
              "tnb_block_svd_cluster: sectors larger than 512 x 256");
  if (n_rows == 0) return TNB_OK;
  TNB_REQUIRE(rows && a && u && s && vt && info, "tnb_block_svd_cluster: null pointer");
  TNB_REQUIRE(n_rows < (1ll << 26), "tnb_block_svd_cluster: too many sectors");
  const cudaError_t e = tnb::sc_dispatch(max_r, [&](auto tag) {
    constexpr int E = decltype(tag)::value;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    const cudaError_t x = tnb::sc_config<E>(sh, static_cast<unsigned>(n_rows * sh.cl),
                                            tnb::as_stream(stream), &cfg, attr);
    if (x != cudaSuccess) return x;
    return cudaLaunchKernelEx(&cfg, tnb::block_svd_cluster_kernel<E>, rows, n_rows, a, n_a, u,
                              n_u, s, n_s, vt, n_vt, info,
                              static_cast<int64_t>(sh.smem / 8), sh.cl,
                              static_cast<long long>(wait_cycles));
  });
  if (e != cudaSuccess) {
    tnb::set_error(std::string("tnb_block_svd_cluster: ") + cudaGetErrorString(e));
    return TNB_ECUDA;
  }
  return tnb::check_launch("tnb_block_svd_cluster");
}
