// Multi-step kernel: one cooperative launch advances a specimen by many timesteps.  Shared by the
// FP64 form (dem_run.cu, built with --fmad=false) and the FP32-force form (dem_run_fp32.cu).
//
// A timestep launched on its own is a chain of latencies: launch, step counter, flags, adjacency
// range, adjacency entry, partner, law, damping, the last block's epilogue, the next launch.  Here
// each block (one per SM) keeps its particles for the whole launch, the wall planes and the pairs
// that matter stay in shared memory, and only what a partner reads (position, velocity, spin) goes
// through L2 between steps.  One grid barrier a step replaces launch and epilogue: the
// double-buffered state needs no second one, and requests (to stop for the host's neighbour
// search, to prune again) travel in the barrier's own word.
//
// Pruned lists.  Most pairs of a Verlet list are nowhere near touching: the list reaches verletDist
// beyond contact so that it lasts for hundreds of steps.  Every particle is therefore given an
// allowance of movement, and the block keeps the adjacency entries of its particles whose gap is
// below the two particles' allowances.  Those alone are evaluated until some particle has used its
// allowance up: until then no other pair can touch, and a pair that does not touch contributes
// nothing and keeps a zero history.  Then all blocks prune again from the full list at the start
// of the next step.  The allowance is verletDist / 16, or what the particle's speed covers in
// RunArgs::horizon steps where that is more (at most verletDist / 2); both double when prunes come
// at less than kRunPruneSteps steps.
//
// Entry-parallel evaluation.  The law is a chain of dependent FP64 divisions and square roots
// (about 2,400 cycles) behind one L2 round trip (about 1,000), so a thread that walks its
// particle's contacts one after another, and a warp that waits for its longest list, spend most of
// the step in latency.  The block's entries are dealt to its threads instead, whoever owns them;
// each result goes to shared memory and the particle's own thread adds its entries in adjacency
// order.  Every sum is then the one k_step forms with one lane per particle: the FP64 states are
// bit-identical to its single-step launches.
//
// Measured (200 steps, a sheared cell of 250,000): 8.6 -> 4.6 ms in the FP32 form and 10.4 -> 4.9 ms in
// FP64 against single-step launches; 31,000 particles, 100 steps: 2.0 -> 0.9 ms; 180 particles take
// 2 us a step.  Bound by the chain of a step (L2 round trip, law, sums, grid barrier): at 250,000 in
// FP64 24 % of the issue slots, 10 % of the FP64 pipe, 26 % of L2.
#pragma once
#include "dem_step.cuh"

namespace dem {

constexpr int kRunPruneSteps = 8;      // prunes closer than this many steps double the allowances
enum : int { RUN_STOP = 1, RUN_PRUNE = 2, RUN_LOST = 4 };

// The grid barrier number k of the launch, on word k & 1 of two: bits 0..31 count arrivals, 32..47
// the blocks that asked to stop, 48..63 those that asked to prune (modulo 2^16).  A block may arrive
// at barrier k + 1 while another still polls for barrier k, but never at k + 2, so each word is
// steady when a barrier on it is passed, and its requests are what the counts grew by since the
// barrier before on the same word.  Barriers x blocks stays below 2^32.
struct RunBarrier {
  unsigned long long* word;  // [2]
  unsigned nblocks;
  int polls;
  int k = 0;
  unsigned seen[2] = {0u, 0u};  // upper halves
  // Arrival with this block's requests; one thread, after a __syncthreads.
  __device__ __forceinline__ void arrive(int ask) const {
    unsigned long long add = 1ull;
    if (ask & RUN_STOP) add += 1ull << 32;
    if (ask & RUN_PRUNE) add += 1ull << 48;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word + (k & 1)), "l"(add) : "memory");
  }
  // The wait of the same thread for every block; everything written before the arrivals is then
  // visible at L2.  Returns the union of the requests, or RUN_LOST when the wait ran out.
  __device__ __forceinline__ int wait() {
    const unsigned target = (unsigned)((k >> 1) + 1) * nblocks;
    const int w = k & 1;
    ++k;
    for (int it = 0; it < polls; ++it) {
      unsigned long long v;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word + w) : "memory");
      if ((unsigned)v >= target) {
        const unsigned now = (unsigned)(v >> 32), was = seen[w];
        seen[w] = now;
        return ((now & 0xffffu) != (was & 0xffffu) ? RUN_STOP : 0) | ((now >> 16) != (was >> 16) ? RUN_PRUNE : 0);
      }
    }
    return RUN_LOST;
  }
};

// Records that other SMs write within the launch are read at L2 (ldcg4): neither the read-only path
// nor L1 is coherent with them.

// kAdjHeld marks bond-held entries, which a specimen without bonds does not have: a pruned entry
// uses the bit for its dynamic group's index.
static_assert(kMaxDyn <= 2, "a pruned entry's group index is one bit");

// A block's shared memory (sizes: run_layout in dem_device.cuh).  Particle arrays are indexed by
// the block's local particle number, entry arrays by the pruned entry's place.
template <bool ROT, int FEAT, bool FP32, bool ONE>
struct RunSmem {
  using RT = typename std::conditional<FP32, float, double>::type;
  static constexpr bool FRIC = (FEAT & (F_FRIC | F_NFRIC)) != 0;   // two force contributions per entry
  static constexpr bool MOM = ROT && (FEAT & F_FRIC) != 0;         // and a moment
  double* state;           // ONE: [RUN_STATE..][particle]
  double* coef;            // [3][pool]: the pair's scaled stiffnesses and contact-point ratio
  RT* res;                 // [9 / 6 / 3][room]: contributions to the owner
  int2* entry;             // [pool]
  float* limit;            // [particle]: the displacement bound at which the particle's allowance is used up
  float* bound;            // [particle]
  unsigned* flags;         // [particle]
  unsigned short* at;      // [particle + 1]: first entry
  unsigned short* owner;   // [pool]
  int ppb, pool, room;
  __device__ __forceinline__ RunSmem(unsigned char* base, const RunArgs& ra) : ppb(ra.ppb), pool(ra.pool), room(ra.room) {
    const RunLayout L = run_layout(ROT, FRIC, MOM, FP32, ONE, ra.ppb, ra.pool, ra.room);
    state = reinterpret_cast<double*>(base);
    coef = reinterpret_cast<double*>(base + L.coef);
    res = reinterpret_cast<RT*>(base + L.res);
    entry = reinterpret_cast<int2*>(base + L.entry);
    limit = reinterpret_cast<float*>(base + L.limit);
    bound = limit + ppb;
    flags = reinterpret_cast<unsigned*>(bound + ppb);
    at = reinterpret_cast<unsigned short*>(base + L.at);
    owner = reinterpret_cast<unsigned short*>(base + L.owner);
  }
  // ONE: a particle's records, 4 doubles each (0 position and radius, 1 velocity and mass, 2 the
  // walls' force on the position and 1/m, 3 spin and inertia, 4 orientation), and 1/I at 20
  __device__ __forceinline__ double4 get(int rec, int l) const {
    const double* p = state + (size_t)(4 * rec) * ppb + l;
    return make_double4(p[0], p[ppb], p[2 * ppb], p[3 * ppb]);
  }
  __device__ __forceinline__ void put(int rec, int l, const double4& v) const {
    double* p = state + (size_t)(4 * rec) * ppb + l;
    p[0] = v.x; p[ppb] = v.y; p[2 * ppb] = v.z; p[3 * ppb] = v.w;
  }
  __device__ __forceinline__ double& inv_inertia(int l) const { return state[(size_t)20 * ppb + l]; }
  __device__ __forceinline__ void put_res(int k, int q, const V3<RT>& v) const {
    res[(size_t)(3 * k) * room + q] = v.x; res[(size_t)(3 * k + 1) * room + q] = v.y; res[(size_t)(3 * k + 2) * room + q] = v.z;
  }
  __device__ __forceinline__ V3<RT> get_res(int k, int q) const {
    return mk(res[(size_t)(3 * k) * room + q], res[(size_t)(3 * k + 1) * room + q], res[(size_t)(3 * k + 2) * room + q]);
  }
};

// Damping of one of a particle's two motions, linear or rotational (damp's order): u its velocity
// or spin, f the accumulated force or moment, s = 1/m or 1/I, m the mass or inertia.
__device__ __forceinline__ void damp_one(const StepArgs& a, bool lin, const V& u, double s, double m, V& f) {
  if (lin && a.damp_loc && a.loc_before_lin) f += local_damping_force(u, f, a.visc_loc);
  if (lin ? a.damp_lin : a.damp_rot)
    f += damping_force(u, f, s, m, lin ? a.visc_lin : a.visc_rot, lin ? a.dt_lin : a.dt_rot,
                       lin ? a.iter_lin : a.iter_rot);
  if (lin ? (a.damp_loc && !a.loc_before_lin) : a.damp_rotloc)
    f += local_damping_force(u, f, lin ? a.visc_loc : a.visc_rotloc);
}

// The wall forces on a particle without the walls' reactions.
__device__ __forceinline__ V run_walls(int nwall, const WallDev* walls, unsigned pf, const double4& p4) {
  V F = mk(0.0, 0.0, 0.0);
  if (pf & (0xffu << PF_WALL_SHIFT))
    for (int w = 0; w < nwall; ++w) {
      if (!(pf & (1u << (PF_WALL_SHIFT + w)))) continue;
      const WallDev W = walls[w];
      V f;
      if (law_wall(W.k, mk(W.ox, W.oy, W.oz), mk(W.nx, W.ny, W.nz), xyz(p4), p4.w, f)) F += f;
    }
  return F;
}

// The planes a step read, kept for its reactions; then the native wall loader moves wall w.
__device__ __forceinline__ void run_move_wall(const StepArgs& a, WallDev* walls, WallDev* walls_in, int w) {
  const double vx = a.wall_vel[3 * w], vy = a.wall_vel[3 * w + 1], vz = a.wall_vel[3 * w + 2];
  WallDev& W = walls[w];
  walls_in[w] = W;
  if (vx != 0.0 || vy != 0.0 || vz != 0.0) {
    W.ox += vx * a.dt;
    W.oy += vy * a.dt;
    W.oz += vz * a.dt;
  }
}

// Exclusive prefix of the block's `n` counts at[1..n] (in place, at[0] = 0), by all threads;
// returns the total.  Counts and total stay below 65536 or the total is returned as that.
__device__ __forceinline__ int run_scan(unsigned short* at, int n, int* s_warp) {
  const int per = (n + kRunThreads - 1) / kRunThreads, l0 = 1 + threadIdx.x * per, l1 = min(n + 1, l0 + per);
  int sum = 0;
  for (int l = l0; l < l1; ++l) sum += at[l];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if ((threadIdx.x & 31) >= o) incl += v;
  }
  if ((threadIdx.x & 31) == 31) s_warp[threadIdx.x >> 5] = incl;
  __syncthreads();
  int before = 0, total = 0;
  for (int w = 0; w < kRunThreads / 32; ++w) {
    if (w < (int)(threadIdx.x >> 5)) before += s_warp[w];
    total += s_warp[w];
  }
  int run = before + incl - sum;
  for (int l = l0; l < l1; ++l) {
    run += at[l];
    at[l] = (unsigned short)min(run, 65535);
  }
  if (threadIdx.x == 0) at[0] = 0;
  __syncthreads();
  return total;
}

// Blocks of kRunThreads threads, one per SM; block b owns the particles of every gridDim.x-th
// group of `chunk` consecutive slots (sorted packings spread evenly).  ONE: the particles' own
// records stay in shared memory for the launch; otherwise they are read back from L2 each step.
template <bool ROT, int FEAT, bool FP32, bool ONE>
__global__ void __launch_bounds__(kRunThreads, 1) k_run(const StepArgs a, const RunArgs ra) {
  using Smem = RunSmem<ROT, FEAT, FP32, ONE>;
  using RT = typename Smem::RT;
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ double s_red[kRunThreads / 32][kMaxWalls][3];
  __shared__ WallDev s_wall[kMaxWalls], s_wall_in[kMaxWalls];  // this step's planes; the last step's
  __shared__ int s_ask, s_got, s_scan[kRunThreads / 32];
  __shared__ bool s_last;
  const Smem S(s_dyn, ra);
  constexpr int kBarrierThread = kRunThreads - 32;  // of the warp with the least other work
  const int ppb = ra.ppb, tid = threadIdx.x, wlane = tid & 31, warp = tid >> 5;
  const unsigned nb = gridDim.x;
  const long long t0 = *a.step_counter;
  auto slot_of = [&](int l) { return ((l / ra.chunk) * (int)nb + (int)blockIdx.x) * ra.chunk + l % ra.chunk; };
  // with few particles per block the two motions of a particle run side by side, in two halves of the block
  const bool split = ROT && ppb <= kRunThreads / 2;
  const int l_first = split ? tid & (kRunThreads / 2 - 1) : tid;
  const bool do_lin = !split || tid < kRunThreads / 2, do_rot = ROT && (!split || tid >= kRunThreads / 2);

  for (int k = tid; k < (kRunThreads / 32) * kMaxWalls * 3; k += kRunThreads) (&s_red[0][0][0])[k] = 0.0;
  if (tid < a.nwall) s_wall[tid] = a.walls[tid];
  if (tid == 0) s_ask = s_got = 0;
  __syncthreads();
  for (int l = tid; l < ppb; l += kRunThreads) {
    const int i = slot_of(l);
    const unsigned pf = i < a.P.n ? a.P.pflags[i] : 0u;
    S.flags[l] = pf;
    if (!(pf & PF_ALIVE)) continue;
    S.bound[l] = a.P.dbound[i];
    if (ONE) {
      const ParticleBuf in = a.P.buf[a.cur];
      const double4 p4 = in.pr[i], v4 = in.vm[i];
      S.put(0, l, p4);
      S.put(1, l, v4);
      S.put(2, l, d4(run_walls(a.nwall, s_wall, pf, p4), v4.w != 0.0 ? 1.0 / v4.w : 0.0));
      if (ROT) {
        const double4 w4 = in.wi[i];
        S.put(3, l, w4);
        S.put(4, l, in.qq[i]);
        S.inv_inertia(l) = 1.0 / w4.w;
      }
    }
  }
  __syncthreads();  // a prune deals particles to other threads

  const float allow_max = (float)(0.5 * a.g.alpha);
  float half = ra.half, reach_t = ra.horizon * (float)a.dt;
  auto allowance = [&](const double4& v) {
    const float vx = (float)v.x, vy = (float)v.y, vz = (float)v.z;
    return fminf(allow_max, fmaxf(half, reach_t * sqrtf(vx * vx + vy * vy + vz * vz)));
  };
  const int lanes = ppb <= kRunThreads / 4 ? 8 : 4;  // per particle in a prune
  RunBarrier barrier{a.run_word, nb, ra.polls};  // used by kBarrierThread
  int ran = 0, pruned_at = 0, used = 0, full = 0;
  bool prune = true;
  while (true) {
    const long long step = t0 + ran + 1;
    const int c = (a.cur + ran) & 1;
    const bool swapped = (ran & 1) != 0;
    const ParticleBuf in = a.P.buf[c], out = a.P.buf[c ^ 1];

    if (prune) {
      if (ran && ran - pruned_at < kRunPruneSteps) { half = fminf(2.f * half, allow_max); reach_t *= 2.f; }
      pruned_at = ran;
      // pass 0 counts every particle's entries within reach, pass 1 writes them
      for (int pass = 0; pass < 2; ++pass) {
        for (int base = 0; base < ppb * lanes; base += kRunThreads) {
          const int l = (base + tid) / lanes, g = (base + tid) % lanes;
          const bool on = l < ppb && (S.flags[l] & PF_ALIVE);
          const int i = on ? slot_of(l) : 0;
          double4 p4 = make_double4(0, 0, 0, 0);
          float mine = 0.f;
          if (on) {
            p4 = ldcg4(in.pr + i);
            mine = allowance(ldcg4(in.vm + i));
          }
          int q = 0;  // entries of the particle so far
          for (int d = 0; d < a.ndyn; ++d) {
            const DynDev& G = a.dyn[d];
            const int e0 = on ? __ldg(G.adj_start + i) : 0, e1 = on ? __ldg(G.adj_start + i + 1) : 0;
            const int rounds = __reduce_max_sync(0xffffffffu, (e1 - e0 + lanes - 1) / lanes);
            for (int it = 0; it < rounds; ++it) {
              const int e = e0 + it * lanes + g;
              bool near = false, isp1 = false;
              int2 en = make_int2(0, 0);
              double4 pa, pb;
              if (e < e1) {
                en = __ldg(G.adj + e);
                const double4 pj = ldcg4(in.pr + en.x), vj = ldcg4(in.vm + en.x);
                isp1 = en.y < 0;
                pa = isp1 ? p4 : pj;
                pb = isp1 ? pj : p4;
                const V x1 = xyz(pa), x2 = image_of(a.g, x1, xyz(pb));
                const V D = x1 - x2;
                const double reach = pa.w + pb.w + ((double)mine + (double)allowance(vj));
                near = dot(D, D) < reach * reach;
              }
              const unsigned m = (__ballot_sync(0xffffffffu, near) >> (wlane - g)) & ((1u << lanes) - 1u);
              if (near) {
                if (pass) {
                  const int place = S.at[l] + q + __popc(m & ((1u << g) - 1u));
                  S.entry[place] = make_int2(en.x, en.y | (d ? kAdjHeld : 0));
                  S.owner[place] = (unsigned short)l;
                  double k0 = 0.0, k1 = 0.0;
                  if (G.kind == 0) k0 = elastic_k(G.k, G.scaling, pa.w, pb.w);
                  else if (G.kind == 1) friction_k(G.k, G.ks, G.scaling, G.meanR, pa.w, pb.w, k0, k1);
                  else if (G.kind == 2) nfriction_k(G.k, G.ks, G.scaling, pa.w, pb.w, k0, k1);
                  S.coef[place] = k0;
                  S.coef[S.pool + place] = k1;
                  S.coef[2 * S.pool + place] = pb.w / (pa.w + pb.w);
                }
              } else if (e < e1 && !pass && isp1 && G.kind != 0) {  // no contact, no history, in either buffer
                const int k = en.y & kAdjIndex;
                if (FP32) {
                  const_cast<float4*>(G.hist32_in)[k] = G.hist32_out[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                } else {
                  const_cast<double4*>(G.hist_in)[k] = G.hist_out[k] = make_double4(0.0, 0.0, 0.0, 0.0);
                }
              }
              q += __popc(m);
            }
          }
          if (!pass && l < ppb && g == 0) {
            S.limit[l] = __fadd_rd(S.bound[l], __fmul_rd(mine, 0.99999f));
            S.at[l + 1] = (unsigned short)(q <= S.room ? q : 65535);  // one particle beyond the room: full
          }
        }
        __syncthreads();
        if (!pass) {
          used = run_scan(S.at, ppb, s_scan);
          // more entries than some block can hold: every block leaves before this step
          if (tid == kBarrierThread) {
            const int ask = used > S.pool ? RUN_STOP : 0;
            if (nb > 1) {
              barrier.arrive(ask);
              s_got = barrier.wait();
            } else {
              s_got = ask;
            }
          }
          __syncthreads();
          if (s_got) { full = 1; break; }
        }
      }
      if (full) break;
    }

    for (int l0 = 0, l1 = 0; l0 < ppb; l0 = l1) {
      // the particles whose entries' results fit the room together (mostly: all of them)
      const int q0 = S.at[l0];
      l1 = ppb;
      if (used - q0 > S.room) {
        int lo = l0 + 1, hi = ppb;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (S.at[mid] - q0 <= S.room) lo = mid; else hi = mid - 1;
        }
        l1 = lo;
      }
      const int q1 = S.at[l1];

      // 3. dynamic pair groups: every entry evaluated for its owner
      for (int q = q0 + tid; q < q1; q += kRunThreads) {
        const int2 en = S.entry[q];
        const int l = S.owner[q], i = slot_of(l), j = en.x, k = en.y & kAdjIndex;
        const bool isp1 = en.y < 0;
        const DynDev& G = a.dyn[a.ndyn > 1 && (en.y & kAdjHeld) ? 1 : 0];
        const bool history = Smem::FRIC && G.kind != 0;
        // the partner's records and the history, all on their way at once
        const double4 pj = ldcg4(in.pr + j);
        double4 vj, wj, hj;
        float4 hf;
        if (Smem::FRIC) vj = ldcg4(in.vm + j);
        if (Smem::MOM) wj = ldcg4(in.wi + j);
        if (history) {
          if (FP32) hf = __ldcg((swapped ? G.hist32_out : G.hist32_in) + k);
          else hj = ldcg4((swapped ? G.hist_out : G.hist_in) + k);
        }
        double4 p4, v4, w4;
        if (ONE) {
          p4 = S.get(0, l);
          if (Smem::FRIC) v4 = S.get(1, l);
          if (Smem::MOM) w4 = S.get(3, l);
        } else {
          p4 = ldcg4(in.pr + i);
          if (Smem::FRIC) v4 = ldcg4(in.vm + i);
          if (Smem::MOM) w4 = ldcg4(in.wi + i);
        }
        double4* const hist_out = swapped ? const_cast<double4*>(G.hist_in) : G.hist_out;
        float4* const hist32_out = swapped ? const_cast<float4*>(G.hist32_in) : G.hist32_out;
        // canonical orientation: p1 = lower id
        const double4 pa = isp1 ? p4 : pj, pb = isp1 ? pj : p4;
        const V x1 = xyz(pa), x2 = image_of(a.g, x1, xyz(pb));
        const V D = x1 - x2;
        const double eq_dist = pa.w + pb.w;
        const bool touching = dot(D, D) < (eq_dist * eq_dist);  // the laws' contact test
        const int at = q - q0;
        if (!touching) {  // zero contributions
          const V3<RT> z = mk(RT(0), RT(0), RT(0));
          S.put_res(0, at, z);
          if (Smem::FRIC) S.put_res(1, at, z);
          if (Smem::MOM) S.put_res(2, at, z);
          if (history && isp1) {
            if (FP32) hist32_out[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            else hist_out[k] = make_double4(0.0, 0.0, 0.0, 0.0);
          }
          continue;
        }
        const double k0 = S.coef[q], k1 = S.coef[S.pool + q], part = S.coef[2 * S.pool + q];
        if (G.kind == 0) {
          if constexpr ((FEAT & F_ELASTIC) != 0) {
            if constexpr (!FP32) {
              V f;
              law_elastic(k0, x1, pa.w, x2, pb.w, f);
              S.put_res(0, at, isp1 ? -1.0 * f : f);
            } else {
              Vf f;
              law_elastic_f32(k0, D, pa.w, pb.w, f);
              S.put_res(0, at, isp1 ? -f : f);
            }
            if constexpr (Smem::FRIC) S.put_res(1, at, mk(RT(0), RT(0), RT(0)));
            if constexpr (Smem::MOM) S.put_res(2, at, mk(RT(0), RT(0), RT(0)));
          }
        } else if (G.kind >= 2) {
          if constexpr (!FP32 && (FEAT & F_NFRIC) != 0) {
            const double4 va = isp1 ? v4 : vj, vb = isp1 ? vj : v4;
            FricOut o;
            if (G.kind == 2) {
              law_nfriction(k0, k1, G.mu_s, G.dt, x1, pa.w, xyz(va), x2, pb.w, xyz(vb), mk(hj.x, hj.y, hj.z), o);
            } else if (G.kind == 3) {
              law_hertz_mindlin(G.k, G.ks, G.mu_s, G.dt, x1, pa.w, xyz(va), x2, pb.w, xyz(vb), mk(hj.x, hj.y, hj.z), o);
              o.fn = -1.0 * o.fn;
            } else {
              law_hertz_mindlin_visco(G.k, G.ks, G.mu_s, G.mu_d, G.dt, x1, pa.w, va.w, xyz(va), x2, pb.w, vb.w, xyz(vb), o);
              o.fn = -1.0 * o.fn;
            }
            S.put_res(0, at, isp1 ? -1.0 * o.fn : o.fn);
            S.put_res(1, at, isp1 ? o.Ffric : -1.0 * o.Ffric);
            if constexpr (Smem::MOM) S.put_res(2, at, mk(RT(0), RT(0), RT(0)));  // forces only
            if (isp1)
              st4(hist_out + k, d4(o.Ffric, (o.slipping ? 1.0 : 0.0) + (o.touching ? 2.0 : 0.0)));
          }
        } else {
          if constexpr (Smem::MOM) {
            if constexpr (!FP32) {
              const double4 va = isp1 ? v4 : vj, vb = isp1 ? vj : v4;
              const double4 wa = isp1 ? w4 : wj, wb = isp1 ? wj : w4;
              FricOut o;
              law_friction_at<double>(k0, k1, part, G.mu_s, G.mu_d, G.dt, x1, pa.w, xyz(va), xyz(wa), x2, pb.w, xyz(vb),
                                      xyz(wb), mk(hj.x, hj.y, hj.z), (((int)hj.w) & 1) != 0, o);
              S.put_res(0, at, isp1 ? -1.0 * o.fn : o.fn);
              S.put_res(1, at, isp1 ? o.Ffric : -1.0 * o.Ffric);
              S.put_res(2, at, isp1 ? o.M1 : o.M2);
              if (isp1)
                st4(hist_out + k, d4(o.Ffric, (o.slipping ? 1.0 : 0.0) + (o.touching ? 2.0 : 0.0)));
            } else {
              const Vf vi = mk((float)v4.x, (float)v4.y, (float)v4.z), vo = mk((float)vj.x, (float)vj.y, (float)vj.z);
              const Vf wi = mk((float)w4.x, (float)w4.y, (float)w4.z), wo = mk((float)wj.x, (float)wj.y, (float)wj.z);
              FricOutF o;
              law_friction_f32_at(k0, k1, part, G.mu_s, G.mu_d, (float)G.dt, D, pa.w, pb.w, isp1 ? vi : vo,
                                  isp1 ? wi : wo, isp1 ? vo : vi, isp1 ? wo : wi, mk(hf.x, hf.y, hf.z),
                                  (((int)hf.w) & 1) != 0, o);
              S.put_res(0, at, isp1 ? -o.fn : o.fn);
              S.put_res(1, at, isp1 ? o.Ffric : -o.Ffric);
              S.put_res(2, at, isp1 ? o.M1 : o.M2);
              if (isp1)
                hist32_out[k] = make_float4(o.Ffric.x, o.Ffric.y, o.Ffric.z,
                                            (o.slipping ? 1.f : 0.f) + (o.touching ? 2.f : 0.f));
            }
          }
        }
      }
      __syncthreads();

      // the particles: their entries' contributions in adjacency order, walls, body forces, damping, integration
      struct Own { double4 p4, v4, w4, q4; };
      auto load = [&](int l, Own& o) {
        if (l >= l1 || !(S.flags[l] & PF_ALIVE)) return;
        const int i = slot_of(l);
        o.p4 = ldcg4(in.pr + i);
        o.v4 = ldcg4(in.vm + i);
        if (ROT) { o.w4 = ldcg4(in.wi + i); o.q4 = ldcg4(in.qq + i); }
      };
      const int stride = split ? kRunThreads / 2 : kRunThreads;
      int l = l0 + l_first;
      Own cur_o, next_o;
      if (!ONE) load(l, next_o);
      for (; l < l1; l += stride) {
        if (!ONE) {
          cur_o = next_o;
          load(l + stride, next_o);
        }
        const unsigned pf = S.flags[l];
        if (!(pf & PF_ALIVE)) continue;
        const int i = slot_of(l);
        // a few entries' contributions are loaded before they are added, in order
        V Fp = mk(0.0, 0.0, 0.0), Mp = Fp;
        const int e1 = S.at[l + 1] - q0;
        KSum3 Fk, Mk;
        Fk.zero();
        Mk.zero();
        constexpr int kAhead = 3;
        const V3<RT> z = mk(RT(0), RT(0), RT(0));
        if (do_lin)
          for (int q = S.at[l] - q0; q < e1; q += kAhead) {
            V3<RT> f0[kAhead], f1[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
              f0[u] = q + u < e1 ? S.get_res(0, q + u) : z;
              f1[u] = Smem::FRIC && q + u < e1 ? S.get_res(1, q + u) : z;
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
              if constexpr (FP32) {
                Fk.add(f0[u]);
                if (Smem::FRIC) Fk.add(f1[u]);
              } else {
                Fp += f0[u];
                if (Smem::FRIC) Fp += f1[u];
              }
            }
          }
        if (Smem::MOM && do_rot)
          for (int q = S.at[l] - q0; q < e1; q += kAhead) {
            V3<RT> m[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) m[u] = q + u < e1 ? S.get_res(2, q + u) : z;
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
              if constexpr (FP32) Mk.add(m[u]);
              else Mp += m[u];
            }
          }
        if constexpr (FP32) {
          Fp = Fk.value() + Fp;
          Mp = Mk.value() + Mp;
        }
        const bool forces = a.store_forces && (a.force_step < 0 || step == a.force_step);
        if (do_lin) {
          const double4 p4 = ONE ? S.get(0, l) : cur_o.p4, v4 = ONE ? S.get(1, l) : cur_o.v4;
          V F;
          double inv_m;
          if (ONE) {
            const double4 f = S.get(2, l);
            F = xyz(f);
            inv_m = f.w;
          } else {
            F = run_walls(a.nwall, s_wall, pf, p4);
            inv_m = v4.w != 0.0 ? 1.0 / v4.w : 0.0;
          }
          for (int k = 0; k < a.ngrav; ++k) F += mk(a.grav[k][0], a.grav[k][1], a.grav[k][2]) * v4.w;
          F += Fp;
          damp_one(a, true, xyz(v4), inv_m, v4.w, F);
          const V xi = xyz(p4);
          V v = xyz(v4), x = xi;
          integrate_lin(pf, a.dt, inv_m, F, v, x);
          const double4 pn = d4(x, p4.w), vn = d4(v, v4.w);
          st4(out.pr + i, pn);
          st4(out.vm + i, vn);
          if (ONE) { S.put(0, l, pn); S.put(1, l, vn); }
          if (forces) a.P.force[i] = d4(F, 0.0);
          float b = S.bound[l];
          if (displaced(a, i, xi, x, b)) atomicOr(&s_ask, RUN_STOP);
          else if (b > S.limit[l]) atomicOr(&s_ask, RUN_PRUNE);
          S.bound[l] = b;
        }
        if (do_rot) {
          const double4 w4 = ONE ? S.get(3, l) : cur_o.w4;
          const double inv_i = ONE ? S.inv_inertia(l) : 1.0 / w4.w;
          V M = mk(0.0, 0.0, 0.0);
          M += Mp;
          damp_one(a, false, xyz(w4), inv_i, w4.w, M);
          V w = xyz(w4);
          integrate_spin(pf, a.dt, inv_i, M, w);
          const double4 wn = d4(w, w4.w);
          st4(out.wi + i, wn);
          if (forces) a.P.moment[i] = d4(M, 0.0);
          if (ONE) {
            S.put(3, l, wn);
          } else {
            double4 q4 = cur_o.q4;
            turn_quat(pf, a.dt, w, q4);
            st4(out.qq + i, q4);
          }
        }
      }
      if (l1 < ppb) __syncthreads();  // the next particles' results take the room
    }

    // ONE: the walls' forces of this step are taken already, so their planes can move
    if (ONE && tid < a.nwall) run_move_wall(a, s_wall, s_wall_in, tid);
    __syncthreads();
    ++ran;
    if (tid == kBarrierThread && nb > 1) barrier.arrive(s_ask);
    // while the arrivals travel: what no other block waits for
    if (ONE) {
      for (int l = l_first; l < ppb; l += split ? kRunThreads / 2 : kRunThreads) {
        const unsigned pf = S.flags[l];
        if (!(pf & PF_ALIVE)) continue;
        if (do_rot) {
          double4 q4 = S.get(4, l);
          turn_quat(pf, a.dt, xyz(S.get(3, l)), q4);
          S.put(4, l, q4);
        }
        if (do_lin && (pf & (0xffu << PF_WALL_SHIFT))) {
          const double inv_m = S.get(2, l).w;
          S.put(2, l, d4(run_walls(a.nwall, s_wall, pf, S.get(0, l)), inv_m));
        }
      }
    } else if (tid < a.nwall) {
      run_move_wall(a, s_wall, s_wall_in, tid);
    }
    if (tid == kBarrierThread) {
      s_got = nb > 1 ? barrier.wait() : s_ask;
      if (!(s_ask & RUN_STOP)) s_ask = 0;
    }
    __syncthreads();
    if ((s_got & (RUN_STOP | RUN_LOST)) || ran == ra.nsteps) break;
    prune = (s_got & RUN_PRUNE) != 0;
  }

  // own records back, and the last step's wall reactions from the positions and planes it read
  const ParticleBuf last_in = a.P.buf[(a.cur + ran + 1) & 1], last_out = a.P.buf[(a.cur + ran) & 1];
  for (int l = tid; l - tid < ppb; l += kRunThreads) {
    const int i = l < ppb ? slot_of(l) : 0;
    const unsigned pf = l < ppb ? S.flags[l] : 0u;
    const bool on = (pf & PF_ALIVE) != 0;
    if (on) {
      if (ONE && ROT && ran) last_out.qq[i] = S.get(4, l);
      a.P.dbound[i] = S.bound[l];
    }
    if (ran) {
      const double4 p = on ? ldcg4(last_in.pr + i) : make_double4(0, 0, 0, 0);
      V F = mk(0.0, 0.0, 0.0);
      wall_forces<false>(a.nwall, s_wall_in, on, pf, xyz(p), p.w, wlane, warp, s_red, F);
    }
  }
  if (tid == 0) {
    if (s_got & RUN_LOST) atomicOr(a.ctrl, CTRL_LOST);
    if (full) atomicOr(a.ctrl, CTRL_FULL);
    if (s_ask & RUN_STOP) atomicOr(a.ctrl, CTRL_REBUILD);
  }
  // the last block closes the launch
  if (!block_partials<kRunThreads / 32>(a, blockIdx.x, gridDim.x, a.block_counter, s_red, &s_last)) return;
  if (!ran) return;
  wall_totals(a, t0 + ran, gridDim.x, wlane, warp);
  if (tid < a.nwall) a.walls[tid] = s_wall[tid];
  if (tid == 0) *a.step_counter = t0 + ran;
}

template <bool R, int FEAT, bool FP32, bool ONE>
inline cudaError_t launch_run_as(const StepArgs& a, RunArgs ra, cudaStream_t s) {
  const void* fn = reinterpret_cast<const void*>(k_run<R, FEAT, FP32, ONE>);
  using Smem = RunSmem<R, FEAT, FP32, ONE>;
  const size_t smem = run_layout(R, Smem::FRIC, Smem::MOM, FP32, ONE, ra.ppb, ra.pool, ra.room).bytes;
  // the attribute is the function's, not the launch's: every handle and host thread sets the same value
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunSmem);
  if (e != cudaSuccess) return e;
  StepArgs arg = a;
  void* p[] = {&arg, &ra};
  return cudaLaunchCooperativeKernel(fn, dim3(ra.blocks), dim3(kRunThreads), p, smem, s);
}

template <bool R, int FEAT, bool FP32>
inline cudaError_t launch_run_any(const StepArgs& a, const RunArgs& ra, cudaStream_t s) {
  return ra.one ? launch_run_as<R, FEAT, FP32, true>(a, ra, s) : launch_run_as<R, FEAT, FP32, false>(a, ra, s);
}

}  // namespace dem
