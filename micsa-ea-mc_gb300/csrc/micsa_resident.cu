/*
 * Small lattices resident in shared memory: a cluster of C blocks holds one
 * sample's state of one 32-replica word -- spins, demon planes, couplings in
 * registers -- for a whole launch of up to 1024 iterations; device memory is
 * touched only at the ends.  Layout and walk convention: micsa_kernels.cuh.
 */
#include <type_traits>

#include "micsa_device.cuh"
#include "micsa_kernels.cuh"

namespace {

/* ------------------------------------------------ cluster shared memory */
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}
/* the address of this block's shared word `a` in block `rank` of the cluster */
__device__ __forceinline__ uint32_t peer_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
/* two words into a peer's shared memory, counted on its mbarrier */
__device__ __forceinline__ void push2(uint32_t dst, uint2 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];"
               ::"r"(dst), "r"(v.x), "r"(v.y), "r"(bar) : "memory");
}
__device__ __forceinline__ void push4(uint32_t dst, uint4 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar) : "memory");
}
/* word w of two adjacent sites of W words at a (an even site: 8-byte aligned
 * at W = 1, 16-byte aligned at W = 2) */
__device__ __forceinline__ uint2 word_pair(const uint32_t *a, int W, int w) {
  if (W == 2) {
    const uint4 v = *(const uint4 *)a;
    return w ? make_uint2(v.y, v.w) : make_uint2(v.x, v.z);
  }
  if (W == 1) return *(const uint2 *)a;
  return make_uint2(a[w], a[W + w]);
}
__device__ __forceinline__ bool try_phase(uint32_t bar, uint32_t phase) {
  uint32_t done;
  asm volatile("{ .reg .pred q; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 q, [%1], %2; "
               "selp.u32 %0, 1, 0, q; }"
               : "=r"(done) : "r"(bar), "r"(phase) : "memory");
  return done;
}
/* Waits of the cluster exchange.  Bounded by tries, which count only while the
 * cluster runs; once a wait of the context has run out the others give up at
 * their 1024th.
 *
 * A thread whose wait ran out (a peer that never pushed) counts it in the
 * context's word, which the host looks at whenever it has waited for the stream,
 * and ends: barriers wait for the threads that are left, nothing is pushed or
 * re-armed on the strength of words that did not come, and the threads that
 * depend on its own words run out in turn.  It ends late, by a millisecond or
 * so, since a block's shared memory must outlast the pushes to it: a neighbour
 * issues its last ones within an iteration (10 us) of the first word it misses. */
__device__ __noinline__ void halo_lost(unsigned *ran_out) {
  atomicAdd_system(ran_out, 1u);
  for (int i = 0; i < 1000; i++) __nanosleep(2000);
  asm volatile("exit;");
}
__device__ __forceinline__ void halo_tries(uint32_t bar, uint32_t phase, const micsa_waits *wt) {
  for (int i = 0;; i++) {
    if (try_phase(bar, phase)) return;
    if ((i & 1023) == 1023 && (i >= wt->tries || *(volatile unsigned *)wt->ran_out)) break;
  }
  halo_lost(wt->ran_out);
}
__device__ __noinline__ void halo_tries_call(uint32_t bar, uint32_t phase, const micsa_waits *wt) {
  halo_tries(bar, phase, wt);
}
/* CALL: one try in line, the others out of it, which shortens the half-sweep's
 * code: us per iteration, all tries in line and so, L=16 x 1 by 8 blocks 3.02 and
 * 2.88, by 4 4.01 and 3.97, L=32 x 2 9.77 and 9.56.  Where the threads next to a
 * neighbour do not fill their warps and hold two pairs, the call costs more than
 * it saves: L=24 x 2 by 4 blocks 8.68 and 9.55. */
template <bool CALL> __device__ __forceinline__ void halo_wait(uint64_t *bar, uint32_t phase, const micsa_waits *wt) {
  const uint32_t a = smem_addr(bar);
  if (!CALL) halo_tries(a, phase, wt);
  else if (!try_phase(a, phase)) halo_tries_call(a, phase, wt);
}

/* ---------------------------------------------------------------- shape */
/* A block owns the Zc = L/C z planes [rank*Zc, (rank+1)*Zc) of both colours,
 * and a thread one or two (PPT) x-adjacent same-colour site pairs per colour,
 * the same (y, x) in planes KZ apart.  With two, the first (k = 0) is inside
 * the slab and only the second may touch a neighbouring block, so that the
 * first one's work covers the wait for the neighbour's words: thread group
 * gamma has the planes outer(gamma) and inner(gamma) = outer +- KZ.  The spin
 * planes lie in shared memory in that order (all outer, then all inner ones),
 * which puts a thread's two pairs a constant distance apart. */
template <int L, int C, int PPT> struct rcfg {
  static constexpr int Lh = L / 2, R = Lh / 2, PL = L * Lh; /* pairs per row, sites per plane */
  static constexpr int Zc = L / C, NPP = L * R;             /* planes, pairs per plane */
  static constexpr int T = Zc * NPP / PPT, KZ = Zc / PPT;
  static constexpr int HZ = C > 1 ? Zc + 2 : Zc; /* spin planes with their halos */
  static constexpr bool CALL = PPT == 1 || NPP % 32 == 0; /* see halo_wait */
  static_assert(L % C == 0 && Zc >= 2 && Zc % PPT == 0 && PPT <= 2 && T <= 1024, "shape");
  /* at most one pair of a thread leaves along z, an inner plane is no edge */
  static_assert(C == 1 || PPT == 1 || KZ >= 2, "shape");
  static constexpr size_t smem(int nc) {
    return sizeof(uint32_t) * PL * (2 * (size_t)HZ + 4 * (size_t)nc * Zc);
  }
  /* slab plane of thread group g's pair k (k = PPT - 1: the outer one) */
  static __host__ __device__ constexpr int plane(int g, int k) {
    const int o = C == 1 || PPT == 1 || g == 0 ? g : (g == 1 ? Zc - 1 : g - 1);
    return k == PPT - 1 ? o : (C > 1 && g == 1 ? o - KZ : o + KZ);
  }
  /* slab plane at position pos of the stack, and back */
  static __host__ __device__ constexpr int at_pos(int pos) {
    return pos < KZ ? plane(pos, PPT - 1) : plane(pos - KZ, 0);
  }
  static __host__ __device__ constexpr int pos_of(int z) {
    int r = 0;
    for (int i = 0; i < Zc; i++)
      if (at_pos(i) == z) r = i;
    return r;
  }
};

/* A launch's share of a call of `total` iterations of `units` (sample,
 * replica word) pairs in `rounds` rounds: cluster i takes place first + i of
 * the sequence (round 0 of every unit, round 1 of every unit, ...). */
struct slice {
  int total, rounds, units, first;
};

/* n iterations of one sample and replica word by one cluster along
 * blockIdx.x: all of the call's, or one round's (see slice).
 *
 * Shared memory: sp[2][HZ][PL] spins (with C > 1 a halo plane below and
 * above the slab), then the demon planes [(p, ic)][Zc][PL][D0, D1].  A
 * thread keeps its own spins of both colours and its couplings (as masks) in
 * registers; of a pair's neighbours it holds the two words at the same index
 * of the other colour itself and reads the z+-1, y+-1 pairs and one more
 * x word.
 *
 * Order: half-sweep j updates colour p = j & 1 and reads the other colour.
 * Inside a block a barrier ends it; between blocks only the slab's outer
 * planes matter: the threads that update them also push the new words into
 * the neighbour's halo plane (st.async, counted on the neighbour's mbarrier
 * of that colour), and a thread that reads a halo waits for that mbarrier's
 * phase.  A neighbour sends half-sweep j + 1's words of a plane only after
 * reading the halo of j next to it, and this block sends j + 2's only after
 * receiving all of j + 1's, so a halo is never overwritten before it is read
 * and a mbarrier never sees two phases at once.
 *
 * The demon walk along x and y (and z when C = 1) is an address translation
 * inside the block, as in the other kernels.  Along z with C > 1 the demons
 * of two planes leave for the neighbouring block every iteration: the plane
 * of site z' sits in slot (z' - sgn 2t) mod Zc after t iterations, so the
 * two slots that leave are the two that enter, and each thread pushes its
 * pair's new demons of half-sweep j into the same slot of the neighbour at
 * the start of j + 3: the halo words of j + 1, received during j + 2, show
 * that the neighbour has ended j, hence has read that slot.  The neighbour
 * waits for them an iteration later.  The last iteration keeps its demons and
 * the final copy stores them at their place.
 *
 * Waits are bounded; see halo_lost.
 *
 * What bounds it: with one block per sample the integer ALU pipe (75% busy at
 * L=16, 58 of 86 instructions per pair and half-sweep; the 15 ... 35 us of a
 * launch's ends aside, 0.59 us per half-sweep against 0.93 for a kernel that
 * reads every word from shared memory).  With clusters the exchange adds to it
 * (L=16 by 8 blocks, 0.24 us per half-sweep: the pipe 30% busy).  L=32, C=8 ran
 * 0.84 us per half-sweep when 0.60 were left without the exchange (0.19 the
 * demons' pushes and their wait, 0.05 the halos), and runs 0.80 since the waits'
 * further tries are out of line.  Tried for the exchange, L=32, against 0.84:
 * whole-plane bulk copies after the barrier 0.93, plain peer stores with a fence
 * and an arrival 0.88, 8-byte pushes of D0 and D1 apart 0.87, the pushes spread
 * over three half-sweeps 0.86; one pair per thread (64 registers) 1.16; a state
 * carried past each wait instead of ending the thread 0.87 to 0.97.  Measured
 * against the half-sweep launches: L=16, one sample x 64 replicas 11.3 -> 2.9 us
 * per iteration; L=24, 2 x 32, nc=5 23.1 -> 5.1; L=32, 24 x 64 65 -> 32 (15
 * clusters of 221 KB per block fit the GPU at once; see resident_rounds). */
template <int L, int C, int PPT>
__global__ void __launch_bounds__((rcfg<L, C, PPT>::T), 1)
k_resident(const micsa_geo g, const slice sl, uint32_t *__restrict__ spin,
           uint32_t *__restrict__ d0, uint32_t *__restrict__ d1, const uint8_t *__restrict__ jb,
           const int *__restrict__ walk, const __grid_constant__ micsa_waits wt) {
  using K = rcfg<L, C, PPT>;
  constexpr int Lh = K::Lh, R = K::R, PL = K::PL, Zc = K::Zc, NPP = K::NPP, T = K::T, KZ = K::KZ,
                HZ = K::HZ, P = L * PL;
  constexpr bool CL = C > 1;
  constexpr int H0 = CL ? 1 : 0;                /* the slab's first plane among the HZ */
  constexpr uint32_t PB = PL * 4; /* bytes of a spin plane */
  extern __shared__ uint4 smem_raw[];
  __shared__ uint64_t bars[6]; /* halo of colour 0, 1; demons of (ic 2, p), (ic 5, p) */
  const int rank = CL ? (int)blockIdx.x : 0, W = g.W, nc = g.nc;
  const int place = sl.first + (int)(blockIdx.z * gridDim.y + blockIdx.y), round = place / sl.units, unit = place - round * sl.units;
  const int w = unit % W, s = unit / W;
  const int share = sl.total / sl.rounds, more = sl.total % sl.rounds;
  const int n = share + (round < more), done = round * share + (round < more ? round : more);
  if (micsa_frozen(g, s)) return; /* the whole cluster */
  char *const sm = (char *)smem_raw;
  uint32_t *const sp = (uint32_t *)smem_raw;
  uint2 *const sd = (uint2 *)(sp + 2 * HZ * PL); /* [2*nc][Zc][PL] (D0, D1) */
  const int tid = threadIdx.x, z0 = rank * Zc;
  const size_t sbase = (size_t)s * 2 * P, dbase = (size_t)s * 2 * nc * P;
  const int k0 = (walk[s] + done) % Lh;

  /* spins of the slab (and its halos); demons, the planes that the walk
   * moves along z already in the frame of their sites: a pair of sites per
   * step, in one or two vector loads where a site has one or two words */
#pragma unroll 4
  for (int i = tid; i < HZ * PL; i += T) {
    const int p = i / (HZ * PL / 2), r = 2 * (i % (HZ * PL / 2));
    const int h = r / PL - H0; /* -1 and Zc: the halos */
    int z = z0 + (h < 0 || h >= Zc ? h : K::at_pos(h));
    z += z < 0 ? L : (z >= L ? -L : 0);
    *(uint2 *)(sp + p * (HZ * PL) + r) = word_pair(spin + (sbase + (size_t)p * P + z * PL + r % PL) * W, W, w);
  }
#pragma unroll 4
  for (int i = tid; i < nc * Zc * PL; i += T) {
    const int pi = i / (Zc * PL / 2), r = 2 * (i % (Zc * PL / 2)), ic = pi % nc;
    int z = z0 + r / PL;
    if (CL && (ic == 2 || ic == 5)) {
      z += ((pi < nc) == (ic < 3)) ? -2 * k0 : 2 * k0;
      z += z < 0 ? L : (z >= L ? -L : 0);
    }
    const size_t o = (dbase + (size_t)pi * P + z * PL + r % PL) * W;
    const uint2 u = word_pair(d0 + o, W, w), v = word_pair(d1 + o, W, w);
    *(uint4 *)(sd + pi * (Zc * PL) + r) = make_uint4(u.x, v.x, u.y, v.y);
  }

  /* this thread's pairs: planes zp[k], (y, 2j); byte offsets in the stack of
   * spin planes: at + (PPT - 1 - k)*KZ*PB is pair k itself */
  const int zt = tid / NPP, y = (tid % NPP) / R, j2 = 2 * (tid % R);
  int zp[PPT];
  uint32_t atU[PPT], atD[PPT];
  const uint32_t in = 4u * (uint32_t)(y * Lh + j2), at = in + (uint32_t)(H0 + zt) * PB;
#pragma unroll
  for (int k = 0; k < PPT; k++) {
    zp[k] = K::plane(zt, k);
    const int u = zp[k] + 1, d = zp[k] - 1;
    atU[k] = in + (uint32_t)(u < Zc ? H0 + K::pos_of(u) : (CL ? Zc + 1 : K::pos_of(0))) * PB;
    atD[k] = in + (uint32_t)(d >= 0 ? H0 + K::pos_of(d) : (CL ? 0 : K::pos_of(Zc - 1))) * PB;
  }
  const int par0 = (y + z0 + zp[PPT - 1]) & 1; /* x = 2*(x/2) + ro(k, p), ro = par0 ^ p ^ (k's z) */
  const uint32_t atN = (y + 1 == L) ? at - 4 * (L - 1) * Lh : at + 4 * Lh;
  const uint32_t atS = (y == 0) ? at + 4 * (L - 1) * Lh : at - 4 * Lh;
  /* the other x neighbours of the pair's sites where x = 2*(x/2) + ro: the
   * next (ro = 1) or the previous word of the row; even and odd par */
  uint32_t atX[2][2];
  {
    const uint32_t next = (j2 + 2 == Lh) ? at - 4 * j2 : at + 8, prev = (j2 == 0) ? at + 4 * (Lh - 1) : at - 4;
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const bool ro = par0 ^ e;
      atX[e][0] = ro ? at + 4 : prev;
      atX[e][1] = ro ? next : at;
    }
  }
  /* couplings as masks: the bond to the word at the same index of the other
   * colour, the other x bond, +y, +z, -y, -z */
  uint32_t m[PPT][2][2][6];
#pragma unroll
  for (int k = 0; k < PPT; k++)
#pragma unroll
    for (int p = 0; p < 2; p++) {
      const uint32_t v = *(const uint16_t *)(jb + sbase + (size_t)p * P + (z0 + zp[k]) * PL + y * Lh + j2);
      const bool ro = par0 ^ p ^ (((PPT - 1 - k) * KZ) & 1);
#pragma unroll
      for (int t = 0; t < 2; t++) {
        const uint32_t b = v >> (8 * t);
        const uint32_t mE = jmask(b, 0), mO = jmask(b, 3);
        m[k][p][t][0] = ro ? mO : mE;
        m[k][p][t][1] = ro ? mE : mO;
        m[k][p][t][2] = jmask(b, 1);
        m[k][p][t][3] = jmask(b, 2);
        m[k][p][t][4] = jmask(b, 4);
        m[k][p][t][5] = jmask(b, 5);
        /* kept as registers: derived again from the byte, each mask would cost
         * an extract and a select per use */
#pragma unroll
        for (int d = 0; d < 6; d++) asm volatile("" : "+r"(m[k][p][t][d]));
      }
    }
  constexpr uint32_t HALO_BYTES = 2 * PB, DEM_BYTES = 4 * PB;
  if (CL && tid == 0) {
    for (int b = 0; b < 6; b++) mbar_init(bars + b, 1 + wt.withheld);
    mbar_fence_init();
    for (int b = 0; b < 2; b++) mbar_expect_tx(bars + b, HALO_BYTES);
    for (int b = 2; b < 6; b++) mbar_expect_tx(bars + b, DEM_BYTES);
  }
  if (CL) cluster_sync();
  else __syncthreads();

#define AT4(off) (*(uint4 *)(sm + (off)))
#define AT2(off) (*(uint2 *)(sm + (off)))
#define AT1(off) (*(uint32_t *)(sm + (off)))
  uint2 own[PPT][2];
#pragma unroll
  for (int k = 0; k < PPT; k++)
#pragma unroll
    for (int p = 0; p < 2; p++) own[k][p] = AT2(at + p * HZ * PB + (PPT - 1 - k) * KZ * PB);
  /* the neighbours' shared memory and mbarriers (an address moves with its base) */
  const uint32_t sm_at = smem_addr(sm), bar_at = smem_addr(bars);
  const int up = CL && rank + 1 < C ? rank + 1 : 0, dn = CL && rank == 0 ? C - 1 : rank - 1;
  uint32_t sm_up = 0, sm_dn = 0, bar_up = 0, bar_dn = 0;
  if (CL) {
    sm_up = peer_addr(sm_at, (uint32_t)up);
    sm_dn = peer_addr(sm_at, (uint32_t)dn);
    bar_up = peer_addr(bar_at, (uint32_t)up);
    bar_dn = peer_addr(bar_at, (uint32_t)dn);
  }
  const bool low = CL && zp[PPT - 1] == 0, high = CL && zp[PPT - 1] == Zc - 1;

  /* demons of this thread on their way to the neighbour, per colour: their
   * words and offset in the neighbour's memory (0: none); since when and of
   * which plane (the same in the whole cluster) */
  uint4 out[2];
  uint32_t out_at[2] = {0, 0}, out_j[2] = {1u << 30, 1u << 30};
  int out_ic[2] = {0, 0};

  int kw = k0;     /* walk: x and y translations */
  int tz = 0;      /* 2t mod Zc: z slots (C > 1) */
  uint32_t jn = 0; /* half-sweeps done */
  for (int it = 0; it < n; it++) {
    for (int ic = 0; ic < nc; ic++) {
      const int axis = ic < 3 ? ic : ic - 3;
      const bool zx = CL && axis == 2; /* demons that change blocks */
      auto half = [&](auto PC) {
        constexpr int p = decltype(PC)::value, q = p ^ 1;
        const bool plus = (p == 0) == (ic < 3);
        /* the walk as shifts in x/2, y and z (one of them not zero), taken
         * off the pair's position modulo the sides */
        const int sh = plus ? kw : -kw;
        const int shx = axis == 0 ? sh : 0, shy = axis == 1 ? 2 * sh : 0;
        const int shz = axis != 2 ? 0 : (CL ? (plus ? tz : -tz) : 2 * sh);
        if (CL && out_j[q] + 3 == jn && out_at[q]) { /* demons that left three half-sweeps ago */
          const bool lp = (q == 0) == (out_ic[q] < 3);
          push4((lp ? sm_up : sm_dn) + out_at[q], out[q],
                (lp ? bar_up : bar_dn) + 8 * (2 + (out_ic[q] == 5 ? 2 : 0) + q));
          out_at[q] = 0;
        }
        if (zx && it > 0) { /* the planes that entered since the last iteration */
          uint64_t *b = bars + 2 + (ic == 5 ? 2 : 0) + p;
          halo_wait<K::CALL>(b, (uint32_t)(it - 1) & 1, &wt);
          if (tid == 0) mbar_expect_tx(b, DEM_BYTES);
        }
        int xd = j2 - shx, yd = y - shy;
        xd += xd < 0 ? Lh : (xd >= Lh ? -Lh : 0);
        yd += yd < 0 ? L : (yd >= L ? -L : 0);
        const uint32_t drow = 2 * HZ * PB + 8u * (uint32_t)((p * nc + ic) * (Zc * PL) + yd * Lh + xd);
        const bool pair = !(shx & 1);
        uint32_t da[PPT], db[PPT];
        uint4 a[PPT]; /* D0, D1 of the two sites */
#pragma unroll
        for (int k = 0; k < PPT; k++) {
          int zs = zp[k] - shz;
          zs += zs < 0 ? Zc : (zs >= Zc ? -Zc : 0);
          da[k] = drow + (uint32_t)zs * (2 * PB);
          db[k] = da[k] + (xd + 1 == Lh ? -8 * (Lh - 1) : 8);
        }
        if (pair) {
#pragma unroll
          for (int k = 0; k < PPT; k++) a[k] = AT4(da[k]);
        } else {
#pragma unroll
          for (int k = 0; k < PPT; k++) {
            const uint2 u = AT2(da[k]), v = AT2(db[k]);
            a[k] = make_uint4(u.x, u.y, v.x, v.y);
          }
        }
#pragma unroll
        for (int k = 0; k < PPT; k++) {
          if (CL && k == PPT - 1 && jn > 0 && (low || high)) {
            halo_wait<K::CALL>(bars + q, ((jn - 1) >> 1) & 1, &wt);
            if (tid == 0) mbar_expect_tx(bars + q, HALO_BYTES);
          }
          constexpr uint32_t oq = q * HZ * PB;
          const uint32_t zk = (PPT - 1 - k) * KZ * PB + oq;
          const int e = (p ^ ((PPT - 1 - k) * KZ)) & 1;
          const uint2 vN = AT2(atN + zk), vS = AT2(atS + zk);
          const uint2 vU = AT2(atU[k] + oq), vD = AT2(atD[k] + oq);
          const uint32_t xA = AT1(atX[e][0] + zk), xB = AT1(atX[e][1] + zk);
          const uint2 c = own[k][q];
          uint2 v = own[k][p];
          {
            const uint32_t *M = m[k][p][0];
            const uint32_t f0 = xor3(v.x, c.x, M[0]), f1 = xor3(v.x, xA, M[1]);
            const uint32_t f2 = xor3(v.x, vN.x, M[2]), f3 = xor3(v.x, vU.x, M[3]);
            const uint32_t f4 = xor3(v.x, vS.x, M[4]), f5 = xor3(v.x, vD.x, M[5]);
            v.x ^= isi_update(xor3(f0, f1, f2), maj3(f0, f1, f2), xor3(f3, f4, f5),
                              maj3(f3, f4, f5), a[k].x, a[k].y);
          }
          {
            const uint32_t *M = m[k][p][1];
            const uint32_t f0 = xor3(v.y, c.y, M[0]), f1 = xor3(v.y, xB, M[1]);
            const uint32_t f2 = xor3(v.y, vN.y, M[2]), f3 = xor3(v.y, vU.y, M[3]);
            const uint32_t f4 = xor3(v.y, vS.y, M[4]), f5 = xor3(v.y, vD.y, M[5]);
            v.y ^= isi_update(xor3(f0, f1, f2), maj3(f0, f1, f2), xor3(f3, f4, f5),
                              maj3(f3, f4, f5), a[k].z, a[k].w);
          }
          own[k][p] = v;
          AT2(at + (PPT - 1 - k) * KZ * PB + p * HZ * PB) = v;
        }
        if (low) /* into the halo above the lower neighbour's slab */
          push2(sm_dn + in + (p * HZ + Zc + 1) * PB, own[PPT - 1][p], bar_dn + 8 * p);
        if (high) /* into the halo below the upper neighbour's */
          push2(sm_up + in + p * HZ * PB, own[PPT - 1][p], bar_up + 8 * p);
        if (zx && it + 1 < n) {
          /* the two planes that leave: one pair of some threads */
#pragma unroll
          for (int k = 0; k < PPT; k++) {
            if (plus ? zp[k] >= Zc - 2 : zp[k] < 2) {
              out[p] = a[k];
              out_at[p] = da[k];
            } else {
              AT4(da[k]) = a[k];
            }
          }
          out_j[p] = jn;
          out_ic[p] = ic;
        } else if (pair) {
#pragma unroll
          for (int k = 0; k < PPT; k++) AT4(da[k]) = a[k];
        } else {
#pragma unroll
          for (int k = 0; k < PPT; k++) {
            AT2(da[k]) = make_uint2(a[k].x, a[k].y);
            AT2(db[k]) = make_uint2(a[k].z, a[k].w);
          }
        }
        jn++;
        __syncthreads();
      };
      half(std::integral_constant<int, 0>());
      half(std::integral_constant<int, 1>());
    }
    kw = (kw + 1 == Lh) ? 0 : kw + 1;
    if (CL && it + 1 < n) {
      tz += 2;
      tz -= tz >= Zc ? Zc : 0;
    }
  }
#undef AT1
#undef AT2
#undef AT4

  /* the last half-sweep's words must have arrived before this block ends */
  if (CL) {
    halo_wait<K::CALL>(bars + 1, ((jn - 1) >> 1) & 1, &wt);
    cluster_sync();
  }
#pragma unroll 4
  for (int i = tid; i < 2 * Zc * PL; i += T) {
    const int p = i / (Zc * PL), r = i % (Zc * PL);
    spin[(sbase + (size_t)p * P + (size_t)(z0 + K::at_pos(r / PL)) * PL + r % PL) * W + w] =
        sp[(p * HZ + H0) * PL + r];
  }
  /* demons: the slot of site plane z in the last iteration's frame (walk kl) */
  const int kl = (int)(((int64_t)k0 + n - 1) % Lh);
#pragma unroll 4
  for (int i = tid; i < nc * Zc * PL; i += T) {
    const int pi = i / (Zc * PL / 2), r = 2 * (i % (Zc * PL / 2)), ic = pi % nc;
    int z = z0 + r / PL, slot = r;
    if (CL && (ic == 2 || ic == 5)) {
      const bool plus = (pi < nc) == (ic < 3);
      int zs = r / PL + (plus ? -tz : tz);
      zs += zs < 0 ? Zc : (zs >= Zc ? -Zc : 0);
      slot = zs * PL + r % PL;
      z += plus ? -2 * kl : 2 * kl;
      z += z < 0 ? L : (z >= L ? -L : 0);
    }
    const size_t o = (dbase + (size_t)pi * P + z * PL + r % PL) * W;
    const uint4 v = *(const uint4 *)(sd + pi * (Zc * PL) + slot);
    if (W == 1) {
      *(uint2 *)(d0 + o) = make_uint2(v.x, v.z);
      *(uint2 *)(d1 + o) = make_uint2(v.y, v.w);
    } else {
      d0[o + w] = v.x;
      d0[o + W + w] = v.z;
      d1[o + w] = v.y;
      d1[o + W + w] = v.w;
    }
  }
}

/* ------------------------------------------------------------- launches */
constexpr size_t STATIC_SMEM = 64; /* at least the kernel's mbarriers */
using kern_t = void (*)(micsa_geo, slice, uint32_t *, uint32_t *, uint32_t *, const uint8_t *,
                        const int *, micsa_waits);
struct variant {
  int L, C, T;
  size_t (*smem)(int);
  kern_t k;
};
template <int L, int C, int PPT> variant make_variant() {
  return {L, C, rcfg<L, C, PPT>::T, [](int nc) { return rcfg<L, C, PPT>::smem(nc); },
          k_resident<L, C, PPT>};
}
/* by lattice side, cluster sizes ascending */
const variant *variants(int *n) {
  static const variant v[] = {make_variant<8, 1, 1>(),  make_variant<16, 1, 2>(),
                              make_variant<16, 2, 2>(), make_variant<16, 4, 1>(),
                              make_variant<16, 8, 1>(), make_variant<24, 4, 2>(),
                              make_variant<24, 8, 1>(), make_variant<32, 8, 2>()};
  *n = (int)(sizeof v / sizeof v[0]);
  return v;
}
void config(const variant &v, int nc, int W, int ns, cudaStream_t st, cudaLaunchAttribute *at,
            cudaLaunchConfig_t *c) {
  *c = {};
  c->gridDim = dim3((unsigned)v.C, (unsigned)W, (unsigned)ns);
  c->blockDim = dim3((unsigned)v.T);
  c->dynamicSmemBytes = v.smem(nc);
  c->stream = st;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)v.C;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  c->attrs = at;
  c->numAttrs = 1;
}
/* The limit of a kernel's dynamic shared memory belongs to the function, not to
 * the launch or the context: it is raised to what the deepest context (nc = 6,
 * or fewer where the device has less) may ask for, always to the same value,
 * so that contexts of other threads never lower it between each other's
 * launches. */
cudaError_t raise_limit(const variant &v, int optin) {
  int nc = 6;
  while (nc > 1 && v.smem(nc) + STATIC_SMEM > (size_t)optin) nc--;
  return cudaFuncSetAttribute(v.k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem(nc));
}

} /* namespace */

/* Blocks per cluster for a context: the most that still run all of its
 * (sample, word) clusters at once -- more SMs per sample shorten every
 * half-sweep (L=16, one sample: 7.1, 5.1, 4.0 and 2.9 us per iteration with
 * 1, 2, 4 and 8 blocks; L=24 x 2, nc = 5: 7.4 and 5.3 with 4 and 8) -- else the fewest,
 * which spend least on the exchange (L=24, 60 samples x 64 replicas: 30 us
 * with 4 blocks; before rounds, 36 with 4 and 52 with 8).  pin > 0 asks for that size.
 *
 * *min_n: the least number of iterations in a call that pays for copying the
 * state in and out.  A launch of v waves of clusters costs about v times
 * (15 to 35 us + its iterations), the half-sweep launches 23 to 115 us per
 * iteration; measured, they meet at n = v or just above it for L = 24 and 32:
 * one wave at L = 24 wins from n = 1 (L=24 x 2: 22 against 24 us), at L = 32
 * from n = 2 (48 against 62; n = 1: 38 against 31), four waves (L=32 x 24
 * samples) from n = 5 (n = 4: 245 against 243 us, n = 8: 399 against 486).  At
 * L <= 16 n = 2 pays for any number of waves (L=16 x 100 samples, two waves: 83
 * against 91 us; x 300, four: 175 against 187; n = 1: 97 by half-sweeps).
 *
 * `beside`: contexts at work side by side fill the gaps of each other's
 * half-sweep launches, not of launches that hold whole SMs.  us per call, three
 * contexts, resident and half-sweeps: L=32 x 24 samples (four waves) n = 8 321
 * and 288, 12 441 and 433, 16 562 and 577; L=32 x 10 (two) 4 82 and 79, 6 107 and
 * 118; L=32 x 60 (eight) 12 1099 and 920, 24 2000 and 1830; L=24 x 60 (four) 8 316
 * and 313, 11 402 and 430; L=16 x 300 (four) 3 194 and 215, 4 222 and 295, 2 166
 * and 146. */
cudaError_t micsa_resident_shape(int L, int nc, int W, int ns, int optin, int pin, bool beside,
                                 int *cluster, int *at_once, int64_t *min_n) {
  *cluster = 0;
  *at_once = 0;
  *min_n = 1;
  int n;
  const variant *v = variants(&n);
  for (int i = 0; i < n; i++) {
    if (v[i].L != L || v[i].smem(nc) + STATIC_SMEM > (size_t)optin || (pin > 0 && v[i].C != pin)) continue;
    cudaLaunchAttribute at;
    cudaLaunchConfig_t c;
    int fit = 0;
    config(v[i], nc, W, ns, 0, &at, &c);
    cudaError_t e = raise_limit(v[i], optin);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&fit, v[i].k, &c);
    if (e != cudaSuccess) return e;
    if (fit < 1) continue;
    const int64_t waves = ((int64_t)W * ns + fit - 1) / fit;
    if (*cluster == 0 || waves == 1) {
      *cluster = v[i].C;
      *at_once = pin > 0 ? 0 : fit;
      if (pin > 0) *min_n = 1;
      else if (waves == 1) *min_n = 1 + (L > 24);
      else if (L <= 16) *min_n = beside && waves > 2 ? 3 : 2;
      else *min_n = beside ? (L > 24 ? 3 : 2) * waves : waves + 1;
    }
  }
  return cudaSuccess;
}

/* Rounds for a call of n iterations.  U clusters of which M run at once take
 * ceil(U / M) waves, the last one mostly idle when U is a little more than a
 * multiple of M; in R rounds of n / R iterations, laid end to end and cut
 * into launches of M, only the last of ceil(R*U / M) launches is.  A wave
 * costs its iterations and about four more (its share of copying the state
 * in and out, the launch).  us per iteration at 256 iterations: L=32, 24
 * samples x 64 replicas (U = 48, M = 15; 16 launches of 51 iterations for 4
 * waves of 256) 38.9 -> 32.8; L=32, 10 x 64 19.4 -> 13.5; L=24, 24 x 64 17.9 ->
 * 12.2; L=16, 100 x 64 14.4 -> 9.8.  Launches side by side on two streams
 * gained another 1% and were left out. */
static int resident_rounds(int64_t U, int64_t M, int n) {
  if (M < 1 || U <= M) return 1;
  int best = 1;
  double cost = 0.97 * (double)((U + M - 1) / M) * (n + 4); /* 3% less, or not worth it */
  for (int R = 2; R <= 8 && R <= n; R++) {
    const double c = (double)((R * U + M - 1) / M) * ((double)n / R + 4);
    if (c < cost) cost = c, best = R;
  }
  return best;
}

cudaError_t micsa_launch_resident(const micsa_geo &g, int cluster, int at_once, int n, uint32_t *spin,
                                  uint32_t *d0, uint32_t *d1, const uint8_t *jb, int *walk,
                                  const micsa_waits &wt, cudaStream_t st, int64_t *launches) {
  int nv;
  const variant *v = variants(&nv);
  const int U = g.W * g.ns, R = resident_rounds(U, at_once, n), M = R > 1 ? at_once : U;
  for (int i = 0; i < nv; i++) {
    if (v[i].L != g.L || v[i].C != cluster) continue;
    cudaLaunchAttribute at;
    cudaLaunchConfig_t c;
    if (R > 1) config(v[i], g.nc, M, 1, st, &at, &c);
    else config(v[i], g.nc, g.W, g.ns, st, &at, &c);
    cudaError_t e = cudaSuccess;
    for (int first = 0; first < R * U && e == cudaSuccess; first += M) {
      /* exactly the places that are left: a test for them in the kernel cost
       * its half-sweeps 8% (L=32) */
      if (R > 1) c.gridDim.y = (unsigned)(R * U - first < M ? R * U - first : M);
      e = cudaLaunchKernelEx(&c, v[i].k, g, slice{n, R, U, first}, spin, d0, d1, jb, (const int *)walk,
                             wt);
      ++*launches;
    }
    if (e != cudaSuccess) return e;
    ++*launches;
    return micsa_launch_walk_add(g, walk, n, st);
  }
  return cudaErrorInvalidValue;
}
