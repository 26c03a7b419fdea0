/*
 * The walk kernel: the reference's voxelized transport (MCd3D,
 * CUDAMCFLtransport.cu:286-447) as a persistent loop of whole warps, for
 * plain media: every label of the grid scatters, none is isotropic, all share
 * one refractive index, and no drop of a weight is zero or above half of it
 * (decided on the host when a medium is created).  Included by
 * transport.cuh, whose device functions it uses.
 *
 * What bounds it: a full GPU is bound by instruction issue and by the latency
 * of the label gather, and the end of every launch, when only the
 * longest-lived photons are left, by the latency of one pass.
 *
 *   - One branch per pass.  A pass is "common" when nothing of it needs a
 *     decision: a positive step that ends inside the slab, with a weight that
 *     no roulette follows.  Each lane states whether its pass is special in
 *     one predicate, one warp vote decides, and the common pass runs as
 *     straight-line code with no divergence, no reconvergence and no vote for
 *     lanes that ended.  Only an iteration with a special lane leaves the
 *     loop for the event code, which runs the reference's sequence lane by
 *     lane.
 *   - Random numbers off the critical path: the step length's logarithm for
 *     the next pass, the azimuth and the deflection draw depend on the stream
 *     alone and are computed while the end point's label is on its way.
 *   - Photons set up ahead.  A launch costs several hundred instructions
 *     (stream hashing, source sampling, label lookup) that one or two lanes
 *     of a warp used to run alone; here half of a warp's lanes set up a queue
 *     of 16 photons at once in shared memory (32 gave no more), and a free
 *     lane takes the next in a dozen loads.
 *   - The launch's end in few warps.  Once all tickets are drawn, the warps of
 *     a block meet every kTailPasses passes and move their photons together,
 *     so that the long-lived photons do not keep every warp issuing passes for
 *     one or two lanes.
 *   - The absorbed weight is not summed pass by pass: what a photon loses
 *     between two events is the difference of its weights there, exactly.
 *   - What only the event code needs of a lane or a warp lives in shared
 *     memory, so that the loop's state fits the registers.
 *
 * Measured on a GB300 against the transport kernel, calls as a user makes
 * them: 1999 + 2000 strict-math photons 17.6 -> 13.2 ms, 20011 fast photons
 * without the hitting density 4.64 -> 2.08 ms, 1e6 + 2.5e5 photons on 50^3
 * voxels 23.8 -> 11.5 ms, 4e6 wide-field photons on 256 x 256 x 128 voxels
 * 34.5 -> 21.6 ms.  2e7 + 2e7 photons on 128 x 128 x 64 voxels, launches: 105
 * -> 85 ms and 169 -> 124 ms.  On 200 x 200 x 100 voxels (256 x 5) 175 and 140
 * instead of 213 and 190 warp instructions per 32 passes, 84 and 82 % of the
 * issue slots used.
 */

constexpr uint32_t kTailPasses = 256u; /* passes between two meetings of a block's warps */
constexpr uint32_t kTailWarps = 2u;    /* warps a block keeps while it has photons for them */
constexpr uint32_t kSpreadWarps = 12u; /* warps of an SM that a run of few photons is spread over */
constexpr uint32_t kMixedPool = 64u;   /* photons that move at one meeting, mixed media */

/* Photons set up ahead per warp: rows of kN entries in shared memory (reals:
 * position, direction, -log of the next step draw; words: stream state,
 * multiplier, label and kQueuePassed, job, weight, source entry). */
constexpr uint32_t kQueuePassed = 0x100u; /* the photon has made its first pass */
struct WalkQueue {
  static constexpr int kN = 16;
  static constexpr int kReals = 7, kWords = 7;
  static constexpr size_t kBytes = (size_t)kN * (kReals * sizeof(real) + kWords * 4);
  real *f;
  uint32_t *u;
  __device__ __forceinline__ WalkQueue(unsigned char *base, unsigned warp) {
    f = reinterpret_cast<real *>(base + warp * kBytes);
    u = reinterpret_cast<uint32_t *>(f + kReals * kN);
  }
};

/* 1/mu_t of a label that draws no step length, as the common pass sees it:
 * no step is positive. */
__device__ __forceinline__ real walk_no_step() { return (real)__int_as_float(0xff800000); }

/* One rounding each, whatever the compiler makes of the code around them: a
 * lane's pass may run as the common pass or in the event code, by what the
 * other lanes of its warp do, and both have to give the same bits.  In strict
 * math a multiply-add is two roundings, as on the host. */
#if MCFL_EXACT_MATH
__device__ __forceinline__ real fp_mul(real a, real b) { return __fmul_rn(a, b); }
__device__ __forceinline__ real fp_add(real a, real b) { return __fadd_rn(a, b); }
__device__ __forceinline__ real fp_fma(real a, real b, real c) { return __fadd_rn(__fmul_rn(a, b), c); }
#else
__device__ __forceinline__ real fp_mul(real a, real b) { return __fmul_rn(a, b); }
__device__ __forceinline__ real fp_add(real a, real b) { return __fadd_rn(a, b); }
__device__ __forceinline__ real fp_fma(real a, real b, real c) { return __fmaf_rn(a, b, c); }
#endif

/* 1 - v^2 */
__device__ __forceinline__ real fp_one_minus_sq(real v) { return fp_fma(-v, v, MCFL_C(1.0)); }

/* spin() with the azimuth's sine and cosine, q = 1 - dz^2 and the uniform
 * given.  kAxis: the direction can lie on the z axis.  kSplit:
 * sin(theta)^2 with two roundings, as the transport kernel's 128 x 9 shape has
 * it in fast math: runs in that shape keep their tallies, which differ from the
 * other shapes' (they agree statistically). */
template <bool kAxis, bool kSplit>
__device__ __forceinline__ void walk_spin(Photon &p, const Rec &c, real u_hg, real cosp, real sinp, real q) {
  const real two_g = c.b.x;
  const real temp = c.a.z / fp_fma(two_g, u_hg, c.a.w);
#if MCFL_EXACT_MATH
  const real cost = fp_fma(-temp, temp, c.b.y) / two_g;
  const real sint = MCFL_SQRT(fp_one_minus_sq(cost));
  const real so = MCFL_SQRT(q); /* sin(theta_old) */
  real dx, dy, dz;
  if (!kAxis || so != MCFL_C(0.0)) {
    dx = fp_fma(p.dx, cost, fp_mul(sint, fp_fma(fp_mul(p.dx, p.dz), cosp, -fp_mul(p.dy, sinp))) / so);
    dy = fp_fma(p.dy, cost, fp_mul(sint, fp_fma(fp_mul(p.dy, p.dz), cosp, fp_mul(p.dx, sinp))) / so);
    dz = fp_fma(p.dz, cost, fp_mul(fp_mul(-sint, cosp), so));
  } else {
    dx = fp_mul(sint, cosp);
    dy = fp_mul(sint, sinp);
    dz = MCFL_COPYSIGN(cost, p.dz * cost);
  }
  const real nrm = MCFL_RSQRTF(fp_fma(dz, dz, fp_fma(dy, dy, fp_mul(dx, dx))));
#else
  const real cost = fp_mul(fp_fma(-temp, temp, c.b.y), c.b.z);
  const real sint = MCFL_SQRT(kSplit ? fp_add(MCFL_C(1.0), -fp_mul(cost, cost)) : fp_one_minus_sq(cost));
  real dx, dy, dz;
  if (!kAxis || q > MCFL_C(0.0)) {
    const real st = fp_mul(sint, rsqrtf(q)); /* sin(theta) / sin(theta_old) */
    const real a = fp_mul(st, cosp), b = fp_mul(st, sinp);
    const real mx = fp_mul(p.dx, p.dz), my = fp_mul(p.dy, p.dz);
    dx = fp_fma(p.dx, cost, fp_fma(a, mx, -fp_mul(b, p.dy)));
    dy = fp_fma(p.dy, cost, fp_fma(a, my, fp_mul(b, p.dx)));
    dz = fp_fma(p.dz, cost, -fp_mul(a, q));
  } else {
    dx = fp_mul(sint, cosp);
    dy = fp_mul(sint, sinp);
    dz = MCFL_COPYSIGN(cost, p.dz * cost);
  }
  const real nrm = rsqrtf(fp_fma(dz, dz, fp_fma(dx, dx, fp_mul(dy, dy))));
#endif
  p.dx = fp_mul(dx, nrm);
  p.dy = fp_mul(dy, nrm);
  p.dz = fp_mul(dz, nrm);
}

/* The draws of a deflection: its uniform, and the azimuth's sine and cosine
 * (sin goes to cosp and cos to sinp, as in CUDAMCFLtransport.cu:603). */
__device__ __forceinline__ void walk_draw(Rng &r, real &u_hg, real &cosp, real &sinp) {
  u_hg = fp_mul(r.raw(), MCFL_C(0x1p-32));
#if MCFL_EXACT_MATH
  MCFL_SINCOSF(fp_mul(MCFL_C(2.0) * kPi, fp_mul(r.raw(), MCFL_C(0x1p-32))), &cosp, &sinp);
#else
  __sincosf(fp_mul(MCFL_C(2.0) * kPi * MCFL_C(0x1p-32), r.raw()), &cosp, &sinp);
#endif
}

/* -log of the next draw */
__device__ __forceinline__ real walk_depth(Rng &r) {
  return -MCFL_LOGF(fp_fma(r.raw(), -MCFL_C(0x1p-32), MCFL_C(1.0)));
}

/* reflect(), one rounding at a time. */
__device__ __forceinline__ bool walk_reflect(Photon &p, real n1, real n2, Rng &r) {
  const real ci = MCFL_FABS(p.dz);
  if (n1 == n2) return true;
  const real s2 = fp_add(MCFL_C(1.0), -fp_mul(ci, ci)), n1s = fp_mul(n1, n1), n2s = fp_mul(n2, n2);
  if (n2s < fp_mul(n1s, s2)) {
    p.dz = -p.dz;
    return false;
  }
  if (ci == MCFL_C(1.0)) {
    const real rr = fp_add(n1, -n2) / fp_add(n1, n2);
    if (fp_mul(r.raw(), MCFL_C(0x1p-32)) <= fp_mul(rr, rr)) {
      p.dz = -p.dz;
      return false;
    }
    return true;
  }
  real e = fp_mul(n1s / n2s, s2);
  const real g = fp_mul(MCFL_C(2.0), MCFL_SQRT(fp_mul(fp_mul(fp_mul(fp_mul(s2, fp_add(MCFL_C(1.0), -e)), e), ci), ci)));
  e = fp_fma(fp_mul(ci, ci), fp_fma(-MCFL_C(2.0), e, MCFL_C(1.0)), e);
  const real f = fp_add(MCFL_C(1.0), -e);
  const real rr = fp_mul(e, fp_add(f, -g) / fp_mul(fp_add(f, g), fp_add(e, g)));
  if (fp_mul(r.raw(), MCFL_C(0x1p-32)) <= rr) {
    p.dz = -p.dz;
    return false;
  }
  const real k = n1 / n2;
  p.dx = fp_mul(p.dx, k);
  p.dy = fp_mul(p.dy, k);
  p.dz = MCFL_COPYSIGN(MCFL_SQRT(fp_fma(-fp_mul(k, k), s2, MCFL_C(1.0))), p.dz);
  return true;
}

/* The x-fastest grid index of a point, clamped: always a voxel, the point's own
 * where the point lies in the grid. */
__device__ __forceinline__ uint32_t walk_voxel(const Med &m, real x, real y, real z) {
  const uint32_t i = MCFL_R2U_RZ(fp_mul(fp_add(x, m.hx), m.gx)) +
                     m.nx * (MCFL_R2U_RZ(fp_mul(fp_add(y, m.hy), m.gy)) + m.ny * MCFL_R2U_RZ(fp_mul(z, m.gz)));
  return min(i, m.total - 1u);
}

/* The media above and below the slab (labels 0 and last). */
__device__ __forceinline__ bool walk_outside(uint32_t label, uint32_t last) { return label - 1u >= last - 1u; }

/* move_to_first_boundary() out of line: none of its registers in the kernel's
 * loop (in a plain medium only photons of a source below the slab take it). */
struct GlassEnd {
  real x, y, z;
  uint32_t label;
  uint64_t tof;
};
template <bool kTime>
__device__ __noinline__ GlassEnd walk_glass(Photon p, Med m, real max_s) {
  const uint32_t label = move_to_first_boundary<kTime>(p, m, max_s);
  return GlassEnd{p.x, p.y, p.z, label, p.tof};
}

/* What a warp keeps between its events (all lanes write the same values). */
struct WalkWarp {
  unsigned long long seen; /* single medium: the last ticket number seen */
  uint32_t q_head, q_cnt;  /* single medium: what is left in the warp's queue */
  /* passes the warp makes before it looks up: a bound below what any of its
   * photons may still make before the pass cap, and what is left until the
   * next meeting (the launch's end) or the next look at a slice's end; the
   * smaller of the two at the last entry into the loop */
  uint32_t cap_left, period_left, common;
  uint32_t it; /* slices: passes of the warp */
};

/* A photon's state while it moves between warps: 7 real rows, then words. */
constexpr int kPoolReals = 7;
__host__ __device__ constexpr size_t walk_pool_entry(bool time) { return kPoolReals * sizeof(real) + (time ? 10 : 8) * 4; }

/* Shared memory of a block: static (per-thread words) and dynamic (label
 * records and queues, or the mixed-media pool). */
constexpr size_t walk_static(int threads) { return (size_t)threads * (4 * 4 + 8) + (size_t)threads * 2; }
static size_t walk_dynamic(bool uniform, bool time, int block, uint32_t n_labels) {
  if (!uniform) return kMixedPool * walk_pool_entry(time);
  return (size_t)n_labels * 2 * sizeof(real4) + (size_t)(block / 32) * WalkQueue::kBytes;
}

/* kUniform: the medium comes from the launch parameters and the label records
 * from shared memory; otherwise (mixed media) both come from the photon's
 * job.  kTime: carries the time of flight.  kTally: how the hitting density
 * is tallied. */
template <bool kUniform, bool kTime, int kTally, int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) MCFL_WALK_NAME(McflLaunch L) {
  constexpr bool kNoPhd = kTally == kWalkNone, kRuns = kTally == kWalkRuns;
  constexpr bool kDirs = kNoPhd && !kTime; /* only these launches have emitting voxels */
  constexpr bool kPhd = kUniform && !kTime && !kNoPhd; /* such a launch always tallies it */
  /* After a pass with decisions in which no photon ended, back to the common
   * passes at once (true) or by way of the warp's bookkeeping.  Measured:
   * 1999 strict-math photons 7.5 against 8.4 ms (excitation); but 20011 fast
   * photons 2.8 against 1.8 ms, 2e7 fast emission photons 131 against 124 ms
   * and 30 beams in one launch 30.3 against 28.4 ms, where the compiler keeps
   * less of the common pass's state in registers. */
  constexpr bool kStay = MCFL_EXACT_MATH || !kUniform;
  constexpr bool kSplit = kUniform && kThreads == 128;
  using Queue = WalkQueue;
  extern __shared__ __align__(16) unsigned char s_mem[];
  real4 *s_lab = reinterpret_cast<real4 *>(s_mem);
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  const size_t gtid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned char *s_rest = s_mem + (kUniform ? (size_t)L.med.n_labels * 2 * sizeof(real4) : 0);
  Queue queue(s_rest, warp);
  /* the photons that move at a meeting (single medium: through the queues,
   * which are empty by then) */
  real *pool_f = reinterpret_cast<real *>(s_rest);
  const uint32_t pool_size =
      kUniform ? (uint32_t)((n_warps * Queue::kBytes) / walk_pool_entry(kTime)) : kMixedPool;
  uint32_t *pool_u = reinterpret_cast<uint32_t *>(pool_f + kPoolReals * pool_size);
  /* per lane: the job, and of the job since the last flush the photons
   * ended, their passes and the weight absorbed */
  __shared__ uint32_t s_job[kThreads], s_done[kThreads], s_steps[kThreads];
  __shared__ unsigned long long s_absorbed[kThreads];
  __shared__ uint32_t s_src[kDirs ? kThreads : 1];
  __shared__ uint32_t s_live[kThreads / 32];
  __shared__ WalkWarp s_warp[kThreads / 32];
  volatile WalkWarp &w = s_warp[warp];
  uint32_t &job = s_job[threadIdx.x], &done = s_done[threadIdx.x];
  uint32_t &steps = s_steps[threadIdx.x], &src_idx = s_src[kDirs ? threadIdx.x : 0];
  unsigned long long &absorbed = s_absorbed[threadIdx.x];
  job = 0xffffffffu;
  done = 0;
  steps = 0;
  absorbed = 0ull;

  Photon p = {};
  Rng r = {};
  Med m = {};
  if (kUniform) {
    m.labels = L.med.labels;
    m.lab = (const float4 *)L.med.lab;
    m.fhd = L.med.fhd;
    m.hx = L.med.hx;
    m.hy = L.med.hy;
    m.esp = L.med.esp;
    m.gx = L.med.gx;
    m.gy = L.med.gy;
    m.gz = L.med.gz;
    m.nx = L.med.nx;
    m.ny = L.med.ny;
    m.total = L.med.total;
    m.last = L.med.last_label;
    for (uint32_t i = threadIdx.x; i < L.med.n_labels; i += blockDim.x) {
      Rec q = load_rec(m, i);
      if (!(q.a.x != FLT_MAX)) q.a.x = walk_no_step();
      s_lab[2 * i] = q.a;
      s_lab[2 * i + 1] = q.b;
    }
    __syncthreads();
  }
  /* the record of a label, as the common pass sees it */
  auto rec_of_label = [&](uint32_t label) -> Rec {
    if (kUniform) return Rec{s_lab[2 * label], s_lab[2 * label + 1]};
    return load_rec(m, label);
  };

  const uint32_t w_event = L.w_event, pst_event = L.step_cap - 1u;
  /* common passes that any new photon may make: it may have made its first */
  const uint32_t fresh_left = max(pst_event, 1u) - 1u;
  const uint8_t *tiles = nullptr;
  uint32_t tile_y = 0, tile_z = 0, tile_last = 0;
  if (kUniform) {
    tiles = L.med.tiles;
    tile_y = L.med.tile_y;
    tile_z = L.med.tile_z;
    tile_last = L.med.tile_bytes - 1u;
  }
  auto ticket_end_of = [&]() -> uint64_t { return L.ticket_end_dev ? __ldg(L.ticket_end_dev) : L.ticket_end; };
  bool alive = false;
  /* mixed media: the warp's ticket queue; which queues it found exhausted
   * (warp-uniform; a missing second queue counts as exhausted) */
  const bool two_queues = !kUniform && L.order2 != nullptr;
  const uint32_t period = L.express_period ? L.express_period : 4u;
  uint32_t tq = two_queues ? (((uint32_t)(gtid >> 5) % period) != 0u ? 1u : 0u) : 0u;
  bool ex0 = false, ex1 = !two_queues;
  bool first = true; /* the first photons are still to be drawn */
  bool tail = false; /* the launch's end: all tickets drawn */
  w.seen = 0;
  w.q_head = 0;
  w.q_cnt = 0;
  w.cap_left = fresh_left;
  w.period_left = 0;
  w.it = 0;
  __syncwarp();

  real nl = MCFL_C(1.0);     /* -log of the pass's step draw */
  real mutr = MCFL_C(0.0);   /* 1/mu_t of the photon's label */
  uint32_t pst = 0;          /* the photon's passes */
  uint32_t run_at = 0;       /* kWalkRuns: the voxel and the weight summed there */
  unsigned long long run_w = 0ull;
  uint32_t pst0 = 0;         /* slices: passes before this one */
  uint64_t k = 0;
  auto job_of = [&]() -> const McflJob * { return &L.jobs[job]; };
  auto flush_stats = [&]() {
    if (job == 0xffffffffu) return;
    unsigned long long *st = (unsigned long long *)__ldg((const unsigned long long *)&job_of()->stats);
    if (done) atomicAdd(&st[MCFL_ST_DONE], (unsigned long long)done);
    if (steps) atomicAdd(&st[MCFL_ST_STEPS], (unsigned long long)steps);
    if (absorbed) atomicAdd(&st[MCFL_ST_ABSORBED], absorbed);
    done = 0;
    steps = 0;
    absorbed = 0ull;
  };
  auto ev_add = [&](int e, unsigned long long v) {
    if (v) atomicAdd((unsigned long long *)__ldg((const unsigned long long *)&job_of()->stats) + e, v);
  };
  /* takes up the photon's label; a label without scattering draws no step */
  auto enter_label = [&]() {
    mutr = kUniform ? s_lab[2 * p.label].x : load_rec(m, p.label).a.x;
    if (!kUniform && !(mutr != FLT_MAX)) mutr = walk_no_step();
  };
  auto next_depth = [&]() -> real { return mutr != walk_no_step() ? walk_depth(r) : MCFL_C(1.0); };

  /* a slice of a served run: photons in flight are parked at its end and
   * resumed by the next slice */
  const bool sliced = !kUniform && (L.max_iters || L.slice_ns) && L.saved;
  uint32_t t_begin = 0; /* the low word of the clock: slices last under 2^32 ns */
  if (!kUniform && L.slice_ns) t_begin = __shfl_sync(kFull, (uint32_t)global_ns(), 0);
  if (sliced) {
    const McflSaved sv = L.saved[gtid];
    if (sv.alive) {
      job = sv.job;
      load_med(job_of(), m);
      p = Photon{sv.x, sv.y, sv.z, sv.dx, sv.dy, sv.dz, sv.weight, sv.label};
      p.tof = sv.tof;
      r.x = sv.rng_x;
      r.a = sv.rng_a;
      k = sv.k;
      pst = sv.steps;
      pst0 = pst;
      absorbed = p.weight;
      alive = true;
      enter_label();
      nl = next_depth();
    }
    w.cap_left = __reduce_min_sync(kFull, alive ? pst_event - pst : fresh_left);
    __syncwarp();
  }

  for (;;) {
    if (sliced && w.period_left == 0u) {
      const uint32_t it = w.it;
      if (L.max_iters && it >= L.max_iters) break;
      /* a served slice ends when its time is up or its stop flag is raised
       * (a request arrived, or one finished); lane 0 reads the clock and the
       * flag every 64 passes */
      if (L.slice_ns || L.stop_flag) {
        int stop = 0;
        if (lane == 0)
          stop = (L.slice_ns && (uint32_t)global_ns() - t_begin >= (uint32_t)L.slice_ns) ||
                 (L.stop_flag && *(volatile const unsigned int *)L.stop_flag != 0u);
        if (__shfl_sync(kFull, stop, 0)) break;
      }
      __syncwarp();
      w.period_left = L.max_iters ? min(64u, L.max_iters - it) : 64u;
      __syncwarp();
    }
    unsigned dead = __ballot_sync(kFull, !alive);
    if (!sliced && ex0 && ex1 && (tail || dead) && w.q_cnt == 0) {
      const bool meet = !tail || w.period_left == 0u || dead == kFull;
      tail = true;
      if (meet) {
        /* ---- a meeting: the block's photons are shared out evenly among
         * its first `keep` warps, in an order that starts at another warp in
         * each block of an SM (so that the schedulers share them).  Enough
         * warps to hold them, and kTailWarps while there are photons for
         * these: a lane waits for the events of its warp's other lanes, so
         * few lanes per warp are as good as the issue slots allow. ---- */
        const unsigned start = L.sm_count ? (blockIdx.x / L.sm_count) % n_warps : 0u;
        const unsigned order = (warp + n_warps - start) % n_warps;
        if (lane == 0) s_live[order] = 32u - (uint32_t)__popc(dead);
        __syncthreads();
        uint32_t total = 0;
        for (unsigned i = 0; i < n_warps; ++i) total += s_live[i];
        if (total == 0u) break;
        const uint32_t keep = min(n_warps, max((total + 31u) >> 5, kTailWarps));
        const uint32_t per = (total + keep - 1u) / keep;
        uint32_t give = 0, give_at = 0, room = 0, take_at = 0;
        for (unsigned i = 0; i < n_warps; ++i) {
          const uint32_t l = s_live[i], most = i < keep ? per : 0u;
          const uint32_t over = l > most ? l - most : 0u, under = l < most ? most - l : 0u;
          if (i < order) {
            give_at += over;
            take_at += under;
          }
          give += over;
          room += under;
        }
        give = min(min(give, room), pool_size);
        const uint32_t mine = s_live[order], most = order < keep ? per : 0u;
        const uint32_t above = __popc(~dead & ((1u << lane) - 1u)), free_above = __popc(dead & ((1u << lane) - 1u));
        if (alive && above >= most && give_at + (above - most) < give) {
          const uint32_t e = give_at + (above - most);
          pool_f[e] = p.x;
          pool_f[pool_size + e] = p.y;
          pool_f[2 * pool_size + e] = p.z;
          pool_f[3 * pool_size + e] = p.dx;
          pool_f[4 * pool_size + e] = p.dy;
          pool_f[5 * pool_size + e] = p.dz;
          pool_f[6 * pool_size + e] = nl;
          pool_u[e] = p.weight;
          pool_u[pool_size + e] = p.label;
          pool_u[2 * pool_size + e] = (uint32_t)r.x;
          pool_u[3 * pool_size + e] = (uint32_t)(r.x >> 32);
          pool_u[4 * pool_size + e] = r.a;
          pool_u[5 * pool_size + e] = job;
          pool_u[6 * pool_size + e] = pst;
          if constexpr (kDirs) pool_u[7 * pool_size + e] = src_idx;
          if constexpr (kTime) {
            pool_u[8 * pool_size + e] = (uint32_t)p.tof;
            pool_u[9 * pool_size + e] = (uint32_t)(p.tof >> 32);
          }
          alive = false;
        }
        __syncthreads();
        if ((dead >> lane & 1u) && mine + free_above < most && take_at + free_above < give) {
          const uint32_t e = take_at + free_above;
          const uint32_t j = pool_u[5 * pool_size + e];
          if (j != job) {
            flush_stats();
            job = j;
            if (!kUniform) load_med(job_of(), m);
          }
          p.x = pool_f[e];
          p.y = pool_f[pool_size + e];
          p.z = pool_f[2 * pool_size + e];
          p.dx = pool_f[3 * pool_size + e];
          p.dy = pool_f[4 * pool_size + e];
          p.dz = pool_f[5 * pool_size + e];
          nl = pool_f[6 * pool_size + e];
          p.weight = pool_u[e];
          p.label = pool_u[pool_size + e];
          r.x = ((uint64_t)pool_u[3 * pool_size + e] << 32) | pool_u[2 * pool_size + e];
          r.a = pool_u[4 * pool_size + e];
          pst = pool_u[6 * pool_size + e];
          if constexpr (kDirs) src_idx = pool_u[7 * pool_size + e];
          if constexpr (kTime) p.tof = ((uint64_t)pool_u[9 * pool_size + e] << 32) | pool_u[8 * pool_size + e];
          enter_label();
          alive = true;
        }
        __syncthreads();
        w.period_left = kTailPasses;
        w.cap_left = __reduce_min_sync(kFull, alive ? pst_event - pst : fresh_left);
        __syncwarp();
      }
    } else if (dead && ((uint32_t)__popc(dead) >= L.relaunch_min || dead == kFull)) {
      if constexpr (kUniform) {
        uint32_t want = __popc(dead), q_head = w.q_head, q_cnt = w.q_cnt;
        const uint64_t ticket_end = ticket_end_of();
        if (first && L.sm_count) {
          /* few photons: as many per warp as spread them over kSpreadWarps
           * warps of each SM (they share its issue slots either way; fewer
           * lanes per warp have fewer special passes to wait for) */
          const uint64_t spread = (uint64_t)kSpreadWarps * L.sm_count, share = (ticket_end + spread - 1u) / spread;
          if (share < want) want = (uint32_t)share;
        }
        first = false;
        while (want) {
          if (q_cnt == 0) {
            if (ex0) break;
            __syncwarp();
            /* set up the photons wanted now, and ahead of them half of the
             * warp's share of what is left */
            const uint64_t seen = w.seen, left = ticket_end > seen ? ticket_end - seen : 0ull;
            const uint32_t warps = gridDim.x * n_warps;
            uint32_t fill = left >= (uint64_t)warps * (2 * Queue::kN) ? (uint32_t)Queue::kN
                                                                     : (uint32_t)left / (2u * warps);
            fill = min(max(fill, want), (uint32_t)Queue::kN);
            unsigned long long base = 0ull;
            if (lane == 0) base = atomicAdd(L.ticket_counter, (unsigned long long)fill);
            base = __shfl_sync(kFull, base, 0);
            w.seen = base + fill;
            const uint32_t got =
                base >= ticket_end ? 0u : (uint32_t)min((unsigned long long)fill, (unsigned long long)ticket_end - base);
            if (got < fill) ex0 = true;
            if (lane < got) {
              const uint64_t t = base + lane;
              const uint32_t j = find_job(L.jobs, L.order, L.n_jobs, t);
              if (j != 0xffffffffu) {
                const McflJob *J = &L.jobs[j];
                const uint64_t kk = __ldg((const unsigned long long *)&J->photon_base) +
                                    (t - __ldg((const unsigned long long *)&J->ticket_begin));
                Photon f;
                Rng fr;
                uint32_t src = 0;
                launch_photon<0, kDirs>(J, m, kk, L.mult, f, fr, src);
                real fnl = MCFL_C(1.0);
                uint32_t passed = 0u;
                if (s_lab[2 * f.label].x != walk_no_step()) {
                  fnl = walk_depth(fr);
                  /* a beam starts along the z axis, where the deflection has
                   * a form of its own: its first pass, when it is common
                   * otherwise, is made here, for all the photons set up */
                  const real fs = fp_mul(fnl, s_lab[2 * f.label].x), fz = fp_fma(fs, f.dz, f.z);
                  const real fq = fp_one_minus_sq(f.dz);
                  if (!kTime && !(fq > MCFL_C(0.0)) && fminf(fz, fs) > MCFL_C(0.0) && fz < m.esp && f.weight > w_event &&
                      pst_event > 0u) {
                    const uint32_t w0 = f.weight;
                    f.x = fp_fma(f.dx, fs, f.x);
                    f.y = fp_fma(f.dy, fs, f.y);
                    f.z = fz;
                    const bool in = MCFL_FABS(f.x) < m.hx && MCFL_FABS(f.y) < m.hy;
                    const uint32_t v = walk_voxel(m, f.x, f.y, f.z);
                    f.label = in ? (uint32_t)m.labels[v] : 1u;
                    if (kPhd && in) atomicAdd(&m.fhd[v], (unsigned long long)w0);
                    real u_hg, cosp, sinp;
                    walk_draw(fr, u_hg, cosp, sinp);
                    const Rec c = rec_of_label(f.label);
                    f.weight -= MCFL_R2U_RU(fp_mul(c.a.y, MCFL_U2R_RN(w0)));
                    walk_spin<true, kSplit>(f, c, u_hg, cosp, sinp, fq);
                    fnl = walk_depth(fr);
                    passed = kQueuePassed;
                  }
                }
                queue.f[0 * Queue::kN + lane] = f.x;
                queue.f[1 * Queue::kN + lane] = f.y;
                queue.f[2 * Queue::kN + lane] = f.z;
                queue.f[3 * Queue::kN + lane] = f.dx;
                queue.f[4 * Queue::kN + lane] = f.dy;
                queue.f[5 * Queue::kN + lane] = f.dz;
                queue.f[6 * Queue::kN + lane] = fnl;
                queue.u[0 * Queue::kN + lane] = (uint32_t)fr.x;
                queue.u[1 * Queue::kN + lane] = (uint32_t)(fr.x >> 32);
                queue.u[2 * Queue::kN + lane] = fr.a;
                queue.u[3 * Queue::kN + lane] = f.label | passed;
                queue.u[5 * Queue::kN + lane] = f.weight;
                queue.u[6 * Queue::kN + lane] = src;
              }
              queue.u[4 * Queue::kN + lane] = j;
            }
            __syncwarp();
            q_head = 0;
            q_cnt = got;
            if (got == 0) break;
          }
          const uint32_t take = min(want, q_cnt);
          const uint32_t rank = __popc(dead & ((1u << lane) - 1u));
          if (!alive && rank < take) {
            const uint32_t e = q_head + rank;
            const uint32_t j = queue.u[4 * Queue::kN + e];
            if (j != 0xffffffffu) {
              if (j != job) {
                flush_stats();
                job = j;
              }
              p.x = queue.f[0 * Queue::kN + e];
              p.y = queue.f[1 * Queue::kN + e];
              p.z = queue.f[2 * Queue::kN + e];
              p.dx = queue.f[3 * Queue::kN + e];
              p.dy = queue.f[4 * Queue::kN + e];
              p.dz = queue.f[5 * Queue::kN + e];
              nl = queue.f[6 * Queue::kN + e];
              r.x = ((uint64_t)queue.u[1 * Queue::kN + e] << 32) | queue.u[0 * Queue::kN + e];
              r.a = queue.u[2 * Queue::kN + e];
              const uint32_t lp = queue.u[3 * Queue::kN + e];
              p.label = lp & 0xffu;
              p.weight = queue.u[5 * Queue::kN + e];
              if constexpr (kDirs) src_idx = queue.u[6 * Queue::kN + e];
              p.tof = 0;
              enter_label();
              pst = lp / kQueuePassed;
              /* the weight it started with: only emitting voxels' photons
               * have another weight than the job's */
              absorbed += !(lp & kQueuePassed) ? p.weight : kDirs && __ldg(&job_of()->src_kind) == MCFL_SRC_VOXELS
                                                               ? 0xFFFFFFFFu
                                                               : __ldg(&job_of()->start_weight);
              alive = true;
            }
          }
          q_head += take;
          q_cnt -= take;
          want -= take;
          dead = __ballot_sync(kFull, !alive);
        }
        __syncwarp();
        w.q_head = q_head;
        w.q_cnt = q_cnt;
        __syncwarp();
      } else {
        /* mixed media: the free lanes set up their own photons */
        const bool need = !alive && !(ex0 && ex1);
        const unsigned nm = __ballot_sync(kFull, need);
        if (nm) {
          unsigned long long *ctr = L.ticket_counter;
          uint64_t end = ticket_end_of();
          if (tq ? ex1 : ex0) tq ^= 1u;
          if (tq) {
            ctr = L.ticket_counter2;
            end = L.ticket_end2;
          }
          const int leader = __ffs(nm) - 1;
          unsigned long long base = 0ull;
          if ((int)lane == leader) base = atomicAdd(ctr, (unsigned long long)__popc(nm));
          base = __shfl_sync(kFull, base, leader);
          bool over = false;
          if (need) {
            const uint64_t t = base + (uint64_t)__popc(nm & ((1u << lane) - 1u));
            if (t < end) {
              const uint32_t j = tq ? find_job(L.jobs, L.order2, L.n_jobs2, t) : find_job(L.jobs, L.order, L.n_jobs, t);
              if (j != 0xffffffffu) {
                if (j != job) {
                  flush_stats();
                  job = j;
                  load_med(job_of(), m);
                }
                k = __ldg((const unsigned long long *)&job_of()->photon_base) +
                    (t - __ldg((const unsigned long long *)&job_of()->ticket_begin));
                uint32_t src = 0;
                launch_photon<0, false>(job_of(), m, k, L.mult, p, r, src);
                pst = 0;
                pst0 = 0;
                absorbed += p.weight;
                alive = true;
                enter_label();
                nl = next_depth();
              }
            } else {
              over = true;
            }
          }
          if (__any_sync(kFull, over)) {
            if (tq) ex1 = true;
            else ex0 = true;
          }
        }
      }
    }

    const unsigned live = __ballot_sync(kFull, alive);
    if (live == 0u) {
      if (sliced && ex0 && ex1) break;
      continue;
    }
    uint32_t made = 0;
    if (alive) {
      uint32_t left = w.cap_left;
      if (sliced || tail) left = min(left, w.period_left);
      w.common = left;
      real zn, xn, yn, s, q;
      bool inside, special;
      uint32_t vi, g;
      Rec c;
      real u_hg, cosp, sinp;
      /* Whether a pass is special.  A direction can become NaN (a cosine that
       * rounds beyond 1), and its photon walks on, outside the grid, until
       * the roulette: about one photon in 1e5, for some 1e4 passes, so these
       * passes have to be common where they can.  A NaN position is no reason
       * (fminf passes it over); a NaN direction is one in fast math, where the
       * deflection then starts as from the z axis and gives a number again. */
      auto needs_decisions = [&]() {
        return !(fminf(zn, s) > MCFL_C(0.0)) || (MCFL_EXACT_MATH ? q <= MCFL_C(0.0) : !(q > MCFL_C(0.0))) ||
               zn >= m.esp || p.weight <= w_event || left == 0u;
      };
      /* the hitting density at a point that is not a common pass's end */
      auto tally_at = [&](real x, real y, real z, uint32_t w) {
        if ((kPhd || (!kNoPhd && m.fhd)) && MCFL_FABS(x) < m.hx && MCFL_FABS(y) < m.hy && z < m.esp)
          atomicAdd(&m.fhd[walk_voxel(m, x, y, z)], (unsigned long long)w);
      };
      for (;;) { /* kStay: until a photon ends or the warp has to look up */
      /* ---- common passes, until one is special for some lane ---- */
      for (;;) {
        s = fp_mul(nl, mutr);
        zn = fp_fma(s, p.dz, p.z);
        xn = fp_fma(p.dx, s, p.x);
        yn = fp_fma(p.dy, s, p.y);
        inside = MCFL_FABS(xn) < m.hx && MCFL_FABS(yn) < m.hy;
        const uint32_t ix = MCFL_R2U_RZ(fp_mul(fp_add(xn, m.hx), m.gx)),
                       iy = MCFL_R2U_RZ(fp_mul(fp_add(yn, m.hy), m.gy)), iz = MCFL_R2U_RZ(fp_mul(zn, m.gz));
        const uint8_t *at;
        if (!kUniform || kTime || !kNoPhd) vi = min(ix + m.nx * (iy + m.ny * iz), m.total - 1u);
        if (kUniform)
          at = tiles + min(ix * 16u + (iy * 4u + (iz + (iy >> 2) * tile_y + (iz >> 2) * tile_z)), tile_last);
        else
          at = m.labels + vi;
        /* the end point's label, kept in L1 ahead of other lines (evict-last
         * hint) */
        asm("ld.global.nc.L1::evict_last.u8 %0, [%1];" : "=r"(g) : "l"(at));
        q = fp_one_minus_sq(p.dz);
        special = needs_decisions();
        if (__any_sync(live, special)) break;
        --left;
        walk_draw(r, u_hg, cosp, sinp);
        p.label = inside ? g : 1u;
        c = rec_of_label(p.label);
        p.x = xn;
        p.y = yn;
        p.z = zn;
        if constexpr (kTime) p.tof += tof_fs(fp_mul(s, c.b.w)); /* every label has this index */
        if constexpr (kRuns) {
          const uint32_t w = inside ? p.weight : 0u;
          const bool same = vi == run_at || !inside;
          if (!same) atomicAdd(&m.fhd[run_at], run_w);
          run_w = (same ? run_w : 0ull) + w;
          run_at = same ? run_at : vi;
        } else if ((kPhd || (!kNoPhd && m.fhd)) && inside) {
          atomicAdd(&m.fhd[vi], (unsigned long long)p.weight);
        }
        p.weight -= MCFL_R2U_RU(fp_mul(c.a.y, MCFL_U2R_RN(p.weight)));
        walk_spin<false, kSplit>(p, c, u_hg, cosp, sinp, q);
        mutr = c.a.x;
        nl = walk_depth(r); /* the next pass's draw */
      }

      /* ---- one pass with its decisions: the special lanes run the
       * reference's sequence up to the deflection, which all lanes then make
       * together ---- */
      inside = inside && zn < m.esp;
      special = needs_decisions();
      bool spin_now = true;
      const uint32_t lab = inside ? g : 1u;
      if (special) {
        const real n_old = rec_of_label(p.label).b.w;
        const bool glass = mutr == walk_no_step(); /* a source below the slab */
        const uint32_t w0 = p.weight; /* before an exit takes it */
        uint32_t new_bulk = lab;
        bool stays = s > MCFL_C(0.0) && lab == p.label;
        if (glass) { /* scattering-free: it drew no step length */
          s = MCFL_C(100.0);
          const GlassEnd e = walk_glass<kTime>(p, m, s);
          p.x = e.x;
          p.y = e.y;
          p.z = e.z;
          if constexpr (kTime) p.tof = e.tof;
          new_bulk = e.label;
          stays = false;
        } else {
          if (zn < MCFL_C(0.0) || zn > m.esp) { /* the step reaches a slab face */
            new_bulk = p.label;
            if (zn < MCFL_C(0.0)) {
              new_bulk = 0;
              s = (-p.z) / p.dz;
            }
            if (fp_fma(s, p.dz, p.z) > m.esp) {
              new_bulk = m.last;
              s = fp_add(m.esp, -p.z) / p.dz;
            }
            xn = fp_fma(p.dx, s, p.x);
            yn = fp_fma(p.dy, s, p.y);
            zn = fp_fma(p.dz, s, p.z);
            stays = false;
          }
          p.x = xn;
          p.y = yn;
          p.z = zn;
          if constexpr (kTime) p.tof += tof_fs(fp_mul(s, n_old));
        }
        if (new_bulk != p.label && walk_reflect(p, n_old, rec_of_label(new_bulk).b.w, r)) p.label = new_bulk;
        tally_at(p.x, p.y, p.z, w0);
        spin_now = s > MCFL_C(0.0);
        if (!stays && walk_outside(p.label, m.last)) {
          const bool top = p.label == 0u;
          tally_exit(job_of(), p.x, p.y, p.weight, top, kDirs ? src_idx : 0u);
          if constexpr (kTime) tally_time(job_of(), p.x, p.y, p.weight, p.tof, top);
          ev_add(top ? MCFL_ST_EXIT_TOP : MCFL_ST_EXIT_BOTTOM, p.weight);
          absorbed -= p.weight;
          p.weight = 0u;
          spin_now = false;
        }
        q = fp_one_minus_sq(p.dz);
      } else {
        p.x = xn;
        p.y = yn;
        p.z = zn;
        p.label = lab;
        if constexpr (kTime) p.tof += tof_fs(fp_mul(s, rec_of_label(lab).b.w));
        if ((kPhd || (!kNoPhd && m.fhd)) && inside) atomicAdd(&m.fhd[vi], (unsigned long long)p.weight);
      }
      if (spin_now) {
        walk_draw(r, u_hg, cosp, sinp);
        c = rec_of_label(p.label);
        p.weight -= MCFL_R2U_RU(fp_mul(c.a.y, MCFL_U2R_RN(p.weight)));
        walk_spin<true, kSplit>(p, c, u_hg, cosp, sinp, q);
        mutr = c.a.x;
      }
      /* PhotonSurvive, the pass cap and the photon's end: a common pass
       * leaves a weight above the roulette's */
      if (special) {
        if (p.weight <= kWeightRoulette) {
          if (p.weight == 0u) {
            alive = false;
          } else if (r.co() < kChance) {
            const uint32_t w0 = p.weight;
            p.weight = MCFL_R2U_RN(MCFL_U2R_RN(p.weight) / kChance);
            ev_add(MCFL_ST_R_GAIN, (unsigned long long)(p.weight - w0));
            absorbed += (unsigned long long)(p.weight - w0);
          } else {
            ev_add(MCFL_ST_R_LOSS, p.weight);
            absorbed -= p.weight;
            alive = false;
          }
        }
        const uint32_t passes = pst + (w.common - left) + 1u;
        if (alive && passes >= L.step_cap) {
          ev_add(MCFL_ST_CAPPED, 1ull);
          absorbed -= p.weight;
          alive = false;
        }
        if (!alive) {
          steps += passes - pst0;
          if (!kUniform && L.stop_flag) {
            /* a served slice counts each finished photon at once, and the
             * request's last one raises the stop flag */
            const unsigned long long before =
                atomicAdd((unsigned long long *)__ldg((const unsigned long long *)&job_of()->stats) + MCFL_ST_DONE, 1ull);
            if (before + 1ull == __ldg((const unsigned long long *)&job_of()->photon_base) +
                                     __ldg((const unsigned long long *)&job_of()->photons))
              *(volatile unsigned int *)L.stop_flag = 1u;
          } else {
            ++done;
          }
        } else {
          enter_label();
        }
      }
      if (alive) nl = next_depth();
      if (!kStay || left == 0u || __any_sync(live, !alive)) break;
      --left;
      }
      made = w.common - left + 1u;
      pst += made;
    }
    /* lanes without a photon did not count the passes */
    made = __shfl_sync(kFull, made, __ffs(live) - 1);
    const uint32_t cap_left = w.cap_left, period_left = w.period_left, it = w.it;
    /* past the bound, it is taken anew */
    const uint32_t cap_now = made > cap_left ? __reduce_min_sync(kFull, alive ? pst_event - pst : fresh_left)
                                             : cap_left - made;
    __syncwarp();
    w.cap_left = cap_now;
    if (sliced || tail) w.period_left = period_left - min(made, period_left);
    if (sliced) w.it = it + made;
    __syncwarp();
  }
  if (kRuns && run_w) atomicAdd(&m.fhd[run_at], run_w);
  if (alive) {
    steps += pst - pst0; /* passes of the photon parked by this slice */
    absorbed -= p.weight;
  }
  if (sliced) {
    McflSaved sv;
    sv.alive = alive ? 1u : 0u;
    if (alive) {
      sv.x = (float)p.x; sv.y = (float)p.y; sv.z = (float)p.z;
      sv.dx = (float)p.dx; sv.dy = (float)p.dy; sv.dz = (float)p.dz;
      sv.weight = p.weight;
      sv.label = p.label;
      /* parked before the next pass's step draw: x = lo a + hi with hi < a
       * takes the draw back (a label without scattering made none) */
      const bool drew = mutr != walk_no_step();
      sv.rng_x = drew ? ((r.x % r.a) << 32) | (r.x / r.a) : r.x;
      sv.rng_a = r.a;
      sv.job = job;
      sv.k = k;
      sv.steps = pst;
      sv.src_idx = 0;
      sv.tof = kTime ? p.tof : 0ull;
    }
    L.saved[gtid] = sv;
  }
  flush_stats();
}
