// cellgpu_b200 -- many SPP steps of a small Voronoi system in one launch. Included by system.cu.
//
// A step of the graph path is eight or more dependent launches, two of them behind a conditional
// node. For small systems each launch is a few microseconds of latency around a chain of arithmetic
// that would fit in one: at 300 cells the step took 24 us, of which the chain itself is about 8. Here
// one cooperative launch runs all the steps: the same per-cell code (grp_cell or thread_cell,
// undec_groups, star_one, cc_pair, spp_turn and spp_shift), with barriers between the phases in place
// of kernel boundaries, repair rounds only when the test queued cells, the part of the integration
// that needs no forces done while the blocks meet after the force pass, and the force sums cleared by
// the integrator that read them.
//
// What a step spends (300 cells, 5 blocks): force pass 3.5 us, the rest of the integration 1, two
// barriers; a repair round adds about 9 (star 1.3, commit and check 5, two barriers).
//
// The barrier is a counter in global memory that every block's first thread adds to and polls. All
// blocks are resident (cooperative launch), and a wait gives up after wait_ns (PERSIST_WAIT_NS): the launch
// then ends with CG_ERR_TIMEOUT in the control block, and the system is refused from then on.

namespace cg {

constexpr int PERSIST_WPB = 16;  // warps per block, one block per SM: 128 registers per thread
constexpr unsigned long long PERSIST_WAIT_NS = 20ull * 1000 * 1000 * 1000;

union PersistWarp {
    StarSmem star;
    ThreadWarpSmem t;
    GrpTile<double, VG> g[GPW];
};
// what a step's integration knows before the forces: velocity and next director of the block's first
// blockDim.x cells
struct PersistMove {
    double vx[PERSIST_WPB * 32], vy[PERSIST_WPB * 32], th[PERSIST_WPB * 32];
};
constexpr size_t PERSIST_SMEM = sizeof(PersistWarp) * PERSIST_WPB + sizeof(PersistMove);

struct PersistArgs {
    VoroArgs a;        // a.ctl: the control block; a.ctl[1]: the one of odd steps
    unsigned *bar;     // barrier arrivals, zero at launch
    int cluster;       // the grid is one thread-block cluster: its hardware barrier instead
    int absent;        // arrivals that a barrier waits for and nothing makes (cg_inject_stall), else 0
    unsigned long long wait_ns;  // after which a wait gives up
    int thread_form;   // the force pass in its thread-per-cell form
    const double *noise;  // steps x N normals, or null: drawn
    int steps;
    double dt, mu;
    const int *excl;   // exclusions (null: none) and their external forces
    double2 *ext;
    double *acc;       // null, or per-instance energy sums of the last step (zero between launches),
    double *host_out;  // stored to this page-locked buffer at the end
};

CG_D unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// All threads of the grid. Writes before it are visible after it (the fences also drop the lines that
// the SM's L1 holds). finish() returns false, in every thread of the block, when the wait gave up.
// Work between arrive() and finish() overlaps the wait.
struct GridBarrier {
    unsigned *count;
    unsigned target;
    int *s_ok;
    bool cluster;
    unsigned blocks;  // arrivals per barrier
    unsigned long long wait_ns;
    CG_D void arrive()
    {
        if (cluster) {
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            return;
        }
        target += blocks;
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(count, 1u);
        }
    }
    CG_D bool finish()
    {
        if (cluster) {
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            return true;
        }
        if (threadIdx.x == 0) *s_ok = poll();
        __syncthreads();
        return *s_ok != 0;
    }
    CG_D bool wait()
    {
        arrive();
        return finish();
    }
    // what the block that arrives last (in a cluster: block 0) does with all its threads before any
    // block goes on
    template <typename Last>
    CG_D bool wait_last(Last last)
    {
        if (cluster) {
            wait();
            if (blockIdx.x == 0) last();
            return wait();
        }
        target += blocks + 1;  // one arrival more, when the last block is done
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            *s_ok = atomicAdd(count, 1u) == target - 2;
        }
        __syncthreads();
        const bool am_last = *s_ok != 0;
        if (am_last) {
            __threadfence();
            last();
        }
        __syncthreads();
        if (am_last && threadIdx.x == 0) {
            __threadfence();
            atomicAdd(count, 1u);
        }
        return finish();
    }

private:
    CG_D int poll() const  // one thread
    {
        volatile unsigned *vc = count;
        int ok = 1;
        unsigned long long t0 = 0;
        for (unsigned i = 1; (int)(*vc - target) < 0; ++i) {
            if ((i & 4095u) == 0) {
                const unsigned long long t = now_ns();
                if (t0 == 0) t0 = t;
                else if (t - t0 > wait_ns) {
                    ok = 0;
                    break;
                }
            }
        }
        __threadfence();
        return ok;
    }
};

constexpr int PERSIST_OK = 0, PERSIST_HALT = 1, PERSIST_TIMEOUT = 2;

// The repair of one force evaluation (launch_repair's kernels), after the barrier that ends the force
// pass. Every thread of the grid takes the same decisions, each from words that are constant in the phase
// that reads them: a block that read a word late and left alone would leave the others waiting. A star
// that fails is recorded in `fail`, which the star phases write and the phases after them read; `halt`
// is left to persist_end (the force pass sets it only for rows longer than its slots, which systems of
// 16-slot rows do not have). On PERSIST_OK the rows, forces and counters are those of the repaired
// triangulation.
template <typename R, bool FORCES>
CG_D int persist_repair(const VoroArgs &a, GridBarrier &gb, PersistWarp *wsm, Ctl *sum)
{
    Ctl *ctl = a.ctl;
    volatile Ctl *vc = ctl;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gw = blockIdx.x * PERSIST_WPB + w, nw = gridDim.x * PERSIST_WPB;
    GrpTile<R, VG> *tiles = reinterpret_cast<GrpTile<R, VG> *>(wsm[w].g);
    // the words that decide, in one round trip
    const int halt = vc->halt, undec = vc->n_undec, epoch = vc->epoch;
    int nq = vc->q_count[0];
    if (halt) return PERSIST_HALT;
    const int nu = min(undec, a.N);
    if (nu > 0) {
        for (int base = gw * GPW; base < nu; base += nw * GPW)
            undec_groups<R, VG>(a, ctl, nu, FORCES ? 1 : 0, base, tiles, lane);
        if (!gb.wait()) return PERSIST_TIMEOUT;
        nq = vc->q_count[0];
    }
    int r = 0;
    for (; r < R_MAX && nq > 0; ++r) {
        const int *queue = a.queue + (size_t)r * a.N;
        for (int q = gw; q < nq; q += nw) {
            const int code = star_one(a, r, queue, q, wsm[w].star, lane);
            if (code && lane == 0) atomicExch(&ctl->fail, code);
        }
        if (!gb.wait()) return PERSIST_TIMEOUT;
        if (vc->fail) return PERSIST_HALT;
        if (nq <= a.old_cap) {  // an even warp commits, the next one checks the same two slots
            for (int base = (gw >> 1) * (GPW / 2); base < nq; base += (nw >> 1) * (GPW / 2)) {
                if ((w & 1) == 0)
                    cc_pair<R, FORCES, VG, CC_COMMIT>(a, ctl, r, nq, queue, epoch + r + 1, base, tiles, lane);
                else
                    cc_pair<R, FORCES, VG, CC_CHECK>(a, ctl, r, nq, queue, epoch + r + 1, base, tiles, lane);
            }
        } else {
            for (int base = gw * (GPW / 2); base < nq; base += nw * (GPW / 2))
                cc_pair<R, FORCES, VG, CC_BOTH>(a, ctl, r, nq, queue, epoch + r + 1, base, tiles, lane);
        }
        if (!gb.wait()) return PERSIST_TIMEOUT;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            sum->counters[1] += (unsigned long long)nq;
            sum->counters[3] += 1ull;
        }
        nq = vc->q_count[r + 1];
    }
    if (nq > 0) {  // the local repair did not converge: global rebuild
        if (blockIdx.x == 0 && threadIdx.x == 0) vc->fail = CG_ERR_TOPOLOGY;
        return PERSIST_HALT;
    }
    return PERSIST_OK;
}

// A control block ready for a step with claim epoch `epoch` (counters are kept)
CG_D void ctl_reset(Ctl *c, int epoch)
{
    c->epoch = epoch;
    c->halt = 0;
    c->need_global = 0;
    c->status = 0;
    c->fail = 0;
    c->n_flagged = 0;
    c->n_undec = 0;
    for (int r = 0; r <= R_MAX; ++r) c->q_count[r] = 0;
    c->round = 0;
    c->blocks_done = 0;
}

// The end of a launch. A wait that gave up is an error status (every block's waits give up then).
CG_D void persist_timeout(Ctl *c0, int step)
{
    if (threadIdx.x != 0) return;
    c0->step = step;
    c0->status = CG_ERR_TIMEOUT;
    __threadfence();
    c0->halt = 1;
}

// Otherwise one thread leaves the first control block as the graph's last kernel would: ready for the
// next step, or halted (cur: the block of the halted step; its queues are cleared by the host, since
// other blocks may still be reading them).
CG_D void persist_end(Ctl *c0, Ctl *cur, int st, int step)
{
    Ctl *const c1 = c0 + 1;
    for (int i = 0; i < 8; ++i) {  // the repairs of odd steps counted there
        c0->counters[i] += c1->counters[i];
        c1->counters[i] = 0ull;
    }
    c0->step = step;
    if (st == PERSIST_OK) {
        ctl_reset(c0, c0->epoch > c1->epoch ? c0->epoch : c1->epoch);
        return;
    }
    volatile Ctl *vc = cur;  // (other blocks wrote it)
    const int fail = vc->fail;
    c0->epoch = vc->epoch;
    c0->need_global = fail ? 1 : vc->need_global;
    c0->status = fail ? fail : vc->status;
    __threadfence();
    c0->halt = 1;
}

// The forces of the step are complete: F of cell c (from its fixed-point sums in the deterministic
// mode), exclusions applied, and the sums cleared for the next force pass (clear: F itself too).
template <int FIX>
CG_D double2 take_force(const PersistArgs &p, int c, bool clear)
{
    double2 *F = reinterpret_cast<double2 *>(p.a.F);
    double2 f;
    if (FIX) {
        ulonglong2 *w = reinterpret_cast<ulonglong2 *>(p.a.Ffix) + 4 * (size_t)c;
        const ulonglong2 w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3];
        f = make_double2(fix_force_value(w0, w1), fix_force_value(w2, w3));
        const ulonglong2 z = make_ulonglong2(0ull, 0ull);
        w[0] = z;
        w[1] = z;
        w[2] = z;
        w[3] = z;
    } else {
        f = F[c];
    }
    const bool ex = p.excl && p.excl[c];
    if (ex) {
        p.ext[c] = make_double2(-f.x, -f.y);
        f = make_double2(0.0, 0.0);
    }
    if (FIX || ex || clear) F[c] = (!FIX && clear) ? make_double2(0.0, 0.0) : f;
    return f;
}

// Energies of the configuration whose forces are complete, summed per instance into acc: per warp where
// its cells share an instance, else per cell (the whole grid calls it).
template <typename R>
CG_D void persist_energy(const VoroArgs &a, double *acc, int tid, int nt)
{
    const int i0 = a.cell_inst ? a.cell_inst[0] : 0;
    double sum = 0.0;  // single instance: one addition per warp in all
    for (int c = tid; c - (c & 31) < a.N; c += nt) {  // whole warps
        const bool live = c < a.N;
        const double e = live ? cell_energy<R>(a, c) : 0.0;
        if (a.n_inst == 1) {
            sum += e;
            continue;
        }
        const int inst = live ? a.cell_inst[c] : -1;
        const int first = __shfl_sync(0xffffffffu, inst, 0);
        if (__all_sync(0xffffffffu, inst == first || !live)) {
            double v = e;
            for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
            if ((c & 31) == 0) atomicAdd(&acc[first], v);
        } else if (live) {
            atomicAdd(&acc[inst], e);
        }
    }
    if (a.n_inst == 1) {
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
        if ((threadIdx.x & 31) == 0 && sum != 0.0) atomicAdd(&acc[i0], sum);
    }
}

// the sums to the host buffer, by one block; acc is left zeroed
CG_D void energies_out(const VoroArgs &a, double *acc, double *host_out)
{
    for (int i = threadIdx.x; i < a.n_inst; i += blockDim.x)
        host_out[i] =
            __longlong_as_double((long long)atomicExch(reinterpret_cast<unsigned long long *>(acc + i), 0ull));
    __threadfence_system();
}

// What a step that did not happen (it halted, or an earlier one had) leaves in the host buffer: the
// energies of the stored areas and perimeters, as every other form does. The first block alone sums
// them: no barrier is left to meet at, and halts are rare.
template <typename R>
CG_D void energies_of_halt(const VoroArgs &a, double *acc, double *host_out)
{
    if (blockIdx.x != 0) return;
    persist_energy<R>(a, acc, threadIdx.x, blockDim.x);
    __threadfence();
    __syncthreads();
    energies_out(a, acc, host_out);
}

// The fused force pass with the test over the block's cells [lo, hi): 8 lanes per cell, or a thread per
// cell where a block has more cells than a few passes of its groups cover (FP64 with atomic sums).
template <typename R, int FIX>
CG_D void persist_forces(const VoroArgs &a, PersistWarp *wsm, int lo, int hi, bool thread_form)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gl = lane & (G - 1), gi = lane >> 3;
    if constexpr (std::is_same<R, double>::value && FIX == 0) {
        if (thread_form) {
            for (int base = lo + w * WARP; base < hi; base += PERSIST_WPB * WARP)
                thread_warp<true>(a, base, hi, wsm[w].t, lane);
            return;
        }
    }
    GrpTile<R, VG> *tiles = reinterpret_cast<GrpTile<R, VG> *>(wsm[w].g);
    for (int base = lo + w * GPW; base < hi; base += PERSIST_WPB * GPW)
        grp_cell<R, true, true, VG, FIX>(a, base + gi, base + gi < hi, gl, tiles[gi]);
}

template <typename R, int FIX>
__global__ void __launch_bounds__(PERSIST_WPB * 32, 1) k_voro_steps(PersistArgs p)
{
    extern __shared__ __align__(16) unsigned char persist_smem[];
    __shared__ int s_ok;
    PersistWarp *wsm = reinterpret_cast<PersistWarp *>(persist_smem);
    PersistMove &mv = *reinterpret_cast<PersistMove *>(wsm + PERSIST_WPB);
    VoroArgs a = p.a;
    Ctl *const c0 = p.a.ctl;
    if (c0->halt) {  // uniform across the grid: set by an earlier launch only
        if (p.acc) energies_of_halt<R>(a, p.acc, p.host_out);
        return;
    }
    GridBarrier gb = {p.bar, 0u, &s_ok, p.cluster != 0, gridDim.x + p.absent, p.wait_ns};
    const int step0 = c0->step;
    // a block's cells are contiguous, in whole warps' groups
    const int cpb = (a.N + gridDim.x * GPW - 1) / (gridDim.x * GPW) * GPW;
    const int lo = blockIdx.x * cpb, hi = min(a.N, lo + cpb);
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const bool lead = tid == 0;
    int st = PERSIST_OK, t = 0;
    for (; t < p.steps; ++t) {
        a.ctl = c0 + (t & 1);
        persist_forces<R, FIX>(a, wsm, lo, hi, p.thread_form != 0);
        gb.arrive();
        // while the blocks meet: all of the integration that does not need the forces
        const int first = lo + threadIdx.x;
        if (first < hi) {
            const double xi = p.noise ? p.noise[(size_t)t * a.N + first] : cell_draw(a, first, (uint32_t)(step0 + t));
            double vx, vy;
            mv.th[threadIdx.x] = spp_turn(a, first, xi, p.dt, vx, vy);
            mv.vx[threadIdx.x] = vx;
            mv.vy[threadIdx.x] = vy;
        }
        if (!gb.finish()) {
            st = PERSIST_TIMEOUT;
            break;
        }
        st = persist_repair<R, true>(a, gb, wsm, c0);
        if (st != PERSIST_OK) break;
        // the other control block, last read in the previous step, serves the next one
        if (lead) {
            Ctl *next = c0 + ((t + 1) & 1);
            ctl_reset(next, a.ctl->epoch + R_MAX + 2);
            if (a.ctl->n_flagged) c0->counters[0] += (unsigned long long)a.ctl->n_flagged;
        }
        const bool clear = t + 1 < p.steps;
        if (p.acc && !clear) persist_energy<R>(a, p.acc, tid, nt);
        for (int c = first; c < hi; c += blockDim.x) {
            double vx, vy, th;
            if (c == first) {
                th = mv.th[threadIdx.x];
                vx = mv.vx[threadIdx.x];
                vy = mv.vy[threadIdx.x];
            } else {
                const double xi = p.noise ? p.noise[(size_t)t * a.N + c] : cell_draw(a, c, (uint32_t)(step0 + t));
                th = spp_turn(a, c, xi, p.dt, vx, vy);
            }
            spp_shift(a, c, take_force<FIX>(p, c, clear), vx, vy, p.dt, p.mu);
            a.theta[c] = th;
        }
        if (!gb.wait()) {
            ++t;  // moved, but not every block said so
            st = PERSIST_TIMEOUT;
            break;
        }
    }
    if (st == PERSIST_TIMEOUT) {
        persist_timeout(c0, step0 + t);
        return;
    }
    if (p.acc && st == PERSIST_OK && blockIdx.x == 0) energies_out(a, p.acc, p.host_out);
    if (p.acc && st == PERSIST_HALT) energies_of_halt<R>(a, p.acc, p.host_out);
    if (lead) persist_end(c0, a.ctl, st, step0 + t);
}

// Everything of a step after its force pass, for systems whose force pass fills the GPU as a kernel of its
// own: undecided slots, repair rounds and integration in one cooperative launch, in place of the repair
// start, a conditional node around two kernels per round, the integrator and the step's end. t: the
// step within the call (its parity selects the control block and the barrier counter); last: the call's
// last step, which leaves the first control block ready.
template <typename R, int FIX>
__global__ void __launch_bounds__(PERSIST_WPB * 32, 1) k_voro_tail(PersistArgs p, int t, int last, int move)
{
    extern __shared__ __align__(16) unsigned char persist_smem[];
    __shared__ int s_ok;
    PersistWarp *wsm = reinterpret_cast<PersistWarp *>(persist_smem);
    VoroArgs a = p.a;
    Ctl *const c0 = p.a.ctl, *const c1 = c0 + 1;
    if (c0->halt) {  // uniform across the grid: set by an earlier launch only
        if (p.acc && last) energies_of_halt<R>(a, p.acc, p.host_out);
        return;
    }
    a.ctl = c0 + (t & 1);
    GridBarrier gb = {p.bar + (t & 1), 0u, &s_ok, false, gridDim.x + p.absent, p.wait_ns};
    const int step = c0->step + t;  // (counted at the end of the call)
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const bool lead = tid == 0;
    if (lead) p.bar[(t + 1) & 1] = 0u;  // last used by the previous launch
    int st = persist_repair<R, true>(a, gb, wsm, c0);
    if (st == PERSIST_OK) {
        if (lead) {
            ctl_reset(c0 + ((t + 1) & 1), a.ctl->epoch + R_MAX + 2);  // last read in the previous step
            if (a.ctl->n_flagged) c0->counters[0] += (unsigned long long)a.ctl->n_flagged;
        }
        if (p.acc && last) persist_energy<R>(a, p.acc, tid, nt);
        for (int c = tid; move && c < a.N; c += nt) {
            const double xi = p.noise ? p.noise[(size_t)t * a.N + c] : cell_draw(a, c, (uint32_t)step);
            double vx, vy;
            const double th = spp_turn(a, c, xi, p.dt, vx, vy);
            spp_shift(a, c, take_force<FIX>(p, c, !last), vx, vy, p.dt, p.mu);
            a.theta[c] = th;
        }
        if (!last) return;
        if (!gb.wait()) st = PERSIST_TIMEOUT;
    }
    if (st == PERSIST_TIMEOUT) {
        persist_timeout(c0, step);
        return;
    }
    if (p.acc && st == PERSIST_OK && blockIdx.x == 0) energies_out(a, p.acc, p.host_out);
    if (p.acc && last && st == PERSIST_HALT) energies_of_halt<R>(a, p.acc, p.host_out);
    if (lead) {
        persist_end(c0, a.ctl, st, st == PERSIST_OK ? step + 1 : step);
        if (st == PERSIST_HALT) c1->halt = 1;  // the force passes of the call's odd steps do nothing either
    }
}

// The sums that a launch's first force pass adds to, and the barrier counters, cleared in one kernel.
// cudaMemsetAsync in its place made host-driven steps wait for the copy of the next step's noise, which
// runs beside them: 60000 / 90000 cells 49 / 65 us per host step, 41 / 49 with this (the step graph of
// the time before: 54 / 62); single steps without copies take the same time either way.
__global__ void __launch_bounds__(256) k_persist_clear(ulonglong2 *sums, long long n, unsigned *bar)
{
    const long long nt = (long long)gridDim.x * blockDim.x, tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long long i = tid; i < n; i += nt) sums[i] = make_ulonglong2(0ull, 0ull);
    if (tid < 2) bar[tid] = 0u;
}

// The end of a FIRE iteration (the whole grid): second Verlet half and the sums, per block for a single
// instance, else per warp where it is uniform; then the update of the instances by the block that
// arrives last. complete(i): what the force of dof i still needs. Returns false when a wait gave up.
template <typename Complete>
CG_D bool fire_finish(const FireArgs &f, GridBarrier &gb, double (&s_red)[4][PERSIST_WPB], int *s_running, Ctl *c0,
                      int tid, int nt, Complete complete)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double P = 0, ff = 0, vv = 0, fm = 0;
    for (int i = tid; i - lane < f.ndof; i += nt) {  // whole warps
        double P1 = 0, ff1 = 0, vv1 = 0;
        int inst = -1;
        if (i < f.ndof) {
            complete(i);
            inst = fire_vv2(f, i, P1, ff1, vv1);
        }
        if (f.n_inst == 1) {
            P += P1;
            ff += ff1;
            vv += vv1;
            fm = fmax(fm, ff1);
        } else if (__all_sync(full, inst == __shfl_sync(full, inst, 0))) {
            double fm1 = ff1;
            for (int off = 16; off > 0; off >>= 1) {
                P1 += __shfl_down_sync(full, P1, off);
                ff1 += __shfl_down_sync(full, ff1, off);
                vv1 += __shfl_down_sync(full, vv1, off);
                fm1 = fmax(fm1, __shfl_down_sync(full, fm1, off));
            }
            if (lane == 0 && inst >= 0) fire_add(f.st + inst, P1, ff1, vv1, fm1);
        } else if (inst >= 0) {
            fire_add(f.st + inst, P1, ff1, vv1, ff1);
        }
    }
    if (f.n_inst == 1) {
        for (int off = 16; off > 0; off >>= 1) {
            P += __shfl_down_sync(full, P, off);
            ff += __shfl_down_sync(full, ff, off);
            vv += __shfl_down_sync(full, vv, off);
            fm = fmax(fm, __shfl_down_sync(full, fm, off));
        }
        if (lane == 0) {
            s_red[0][w] = P;
            s_red[1][w] = ff;
            s_red[2][w] = vv;
            s_red[3][w] = fm;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < PERSIST_WPB; ++k) {
                P += s_red[0][k];
                ff += s_red[1][k];
                vv += s_red[2][k];
                fm = fmax(fm, s_red[3][k]);
            }
            fire_add(f.st, P, ff, vv, fm);
        }
    }
    return gb.wait_last([&]() {
        if (threadIdx.x == 0) *s_running = 0;
        __syncthreads();
        bool running = false;
        for (int k = threadIdx.x; k < f.n_inst; k += blockDim.x)
            running = !fire_update(f.st + k, f.prm, f.iter_counter) || running;
        if (running) *s_running = 1;
        __syncthreads();
        if (threadIdx.x == 0) c0->fire_stop = !*s_running;
    });
}

// FIRE on a small Voronoi system: every iteration's phases (fire.cu: the pending mix with the first
// Verlet half, the force pass with test and repair, the second half with the sums, the update) in one
// launch, up to p.steps iterations or until every instance has stopped. The update of the instances is
// done by the block that arrives last at the barrier after the sums. A halt leaves the iteration
// between its move and its forces, as the graph form does, and the host finishes it.
__global__ void __launch_bounds__(PERSIST_WPB * 32, 1) k_fire_voro(PersistArgs p, FireArgs f)
{
    extern __shared__ __align__(16) unsigned char persist_smem[];
    __shared__ int s_ok, s_running;
    __shared__ double s_red[4][PERSIST_WPB];
    PersistWarp *wsm = reinterpret_cast<PersistWarp *>(persist_smem);
    VoroArgs a = p.a;
    Ctl *const c0 = p.a.ctl;
    if (c0->halt) return;  // uniform across the grid: set by an earlier launch only
    GridBarrier gb = {p.bar, 0u, &s_ok, p.cluster != 0, gridDim.x + p.absent, p.wait_ns};
    const int step0 = c0->step;
    const int cpb = (a.N + gridDim.x * GPW - 1) / (gridDim.x * GPW) * GPW;
    const int lo = blockIdx.x * cpb, hi = min(a.N, lo + cpb);
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const bool lead = tid == 0;
    int st = PERSIST_OK, t = 0;
    bool stop = false;
    for (; t < p.steps && !stop; ++t) {
        a.ctl = c0 + (t & 1);
        for (int i = tid; i < a.N; i += nt) fire_mix_vv1(f, i);
        if (!gb.wait()) {
            st = PERSIST_TIMEOUT;
            break;
        }
        persist_forces<double, 0>(a, wsm, lo, hi, p.thread_form != 0);
        if (!gb.wait()) {
            st = PERSIST_TIMEOUT;
            break;
        }
        st = persist_repair<double, true>(a, gb, wsm, c0);
        if (st != PERSIST_OK) break;
        if (lead) {
            Ctl *next = c0 + ((t + 1) & 1);
            ctl_reset(next, a.ctl->epoch + R_MAX + 2);
            if (a.ctl->n_flagged) c0->counters[0] += (unsigned long long)a.ctl->n_flagged;
        }
        if (!fire_finish(f, gb, s_red, &s_running, c0, tid, nt, [&](int i) { take_force<0>(p, i, false); })) {
            st = PERSIST_TIMEOUT;
            break;
        }
        stop = *(volatile int *)&c0->fire_stop != 0;
    }
    if (st == PERSIST_TIMEOUT) {
        persist_timeout(c0, step0);
        return;
    }
    if (lead) {
        c0->fire_iters = st == PERSIST_HALT ? t + 1 : t;
        persist_end(c0, st == PERSIST_OK ? c0 : a.ctl, st, step0);
    }
}

}  // namespace cg

// Largest systems that step in one cooperative launch, with the thread-per-cell force pass / with the
// 8-lane one. Larger systems take two launches per step, the force pass as a kernel of its own occupancy
// and k_voro_tail.
// us per step of a relaxed tissue, one launch / two per step / the graph:
//               FP64                  deterministic         mixed
//   N = 300      8.6 /  -   / 24.1     8.7 /  -   / 22.1     8.5 /  -   / 20.6
//   N = 8192    17.5 / 23.8 / 39.8    17.7 / 21.3 / 37.6    17.4 / 20.2 / 35.5
//   N = 32768   30.8 / 33.6 / 42      34.4 / 34.6 / 46      33.1 / 32.2 / 45
//   N = 65536   36.3 / 37.3 / 47      46.6 / 43.3 / 55      44.1 / 39.2 / 51
//   N = 100000  49.2 / 45.6 / 58      63.5 / 53.6 / 64      57.1 / 47.5 / 58
//   N = 262144  81.1 / 70.0 / 75.0      -  / 96.6 / 101       -  / 81.3 / 87.4
constexpr int PERSIST_MAX_THREAD = 81920, PERSIST_MAX_CELLS = 30000;
// Single steps bring their own clearing of the sums and the host's share of a launch. us per host step (noise
// in, energy out) / step with drawn normals, a tissue in random order, one launch against two; the step
// graph before there were such forms:
//   FP64     N = 16000  27 / 25   34 / 26    40 / 29       tension  N =  9000  27 / 22   28 / 23    35 / 25
//            N = 31000  34 / 28   36 / 28    44 / 32                N = 16000  32 / 26   32 / 25    41 / 28
//            N = 60000  41 / 35   45 / 35    54 / 37                N = 31000  43 / 35   39 / 31    50 / 35
//            N = 90000    -       49 / 40    62 / 44                N = 60000  64 / 50   52 / 44    61 / 49
//   mixed    N = 16000  27 / 25   28 / 23    34 / 25       deterministic 4000  28 / 20   28 / 21    32 / 25
//            N = 31000  38 / 32   35 / 27    42 / 30                N = 31000     -      42 / 32    47 / 33
//            N = 60000  52 / 45   46 / 36    55 / 41                N = 90000     -      63 / 50    72 / 56
constexpr int PERSIST_MAX_SINGLE = 65536;        // FP64, whose force pass has the thread-per-cell form
constexpr int PERSIST_MAX_SINGLE_CELLS = 16384;  // the 8-lane form
constexpr int PERSIST_MAX_SINGLE_FIX = 1024;     // fixed-point sums: 64 bytes per cell, a readout kernel
// Single deterministic steps above this size go through the step graph, which converts the sums and
// integrates at full occupancy. us per host step / drawn step / the same with L2 flushed, two launches
// against the graph: 100000 cells 70 / 58 / 77 and 73 / 62 / 80, 131072 78 / 66 / 85 and 78 / 69 / 88,
// 180000 91 / 82 / 100 and 90 / 83 / 96, 262144 119 / 107 / 129 and 111 / 102 / 117. (Mixed precision takes two
// launches: 262144 94 / 87 / 104 and 99 / 90 / 106.)
constexpr int PERSIST_MAX_TWO_FIX = 131072;

template <typename R, int FIX>
static const void *persist_kernel() { return (const void *)cg::k_voro_steps<R, FIX>; }
template <typename R, int FIX>
static const void *tail_kernel() { return (const void *)cg::k_voro_tail<R, FIX>; }

// whether the force pass has a thread-per-cell form
static bool persist_thread_ok(const cg_system *s)
{
    return s->precision == CG_FP64 && !s->det && s->tension_mode == 0 && s->K == VG;
}

// Systems of up to this many cells minimise in cooperative launches (atomic sums); us per iteration
// against the graph: 1000 cells 16.9 / 48.1, 65536 49.2 / 60.3, 200000 86.2 / 96.3.
constexpr int PERSIST_MAX_FIRE = 200000;
constexpr int PERSIST_FIRE_ITERS = 256;  // iterations per launch

// Grids of up to this many blocks (1024 cells) are one thread-block cluster, whose barrier takes about
// 0.4 us; the counter's takes 1.4 to 1.7.
constexpr int PERSIST_CLUSTER = 16;
// Cells per block above which the force pass takes its thread-per-cell form: one pass of 512 threads
// takes about as long as three of the 64 groups (N = 24576 29.2 us per step either way, 16384 26.7 with
// groups and 29.1 with threads, 65536 43.9 and 35.7).
constexpr int PERSIST_THREAD_CELLS = 192;

// One block per SM at most, and no more blocks than the cells fill. Calls that run at the same time on
// other streams take their share of the SMs, what small ones leave included: grids that fill the GPU would
// take turns. us per step or
// iteration of all of M systems in M threads, full grids / shared ones / graphs:
//   FIRE 16384 cells  M = 2  42 / 31 / 51    4   83 / 44 /  72    8  163 /  58 / 122
//   FIRE 65536        M = 2  55 / 48 / 67    4  108 / 90 /  98    8  219 / 151 / 196
//   SPP  16384        M = 2  38 / 24 / 52    4   74 / 31 /  71    8  147 /  46 / 123
//   SPP  65536        M = 2  58 / 48 / 69    4  116 / 82 /  99    8  233 / 147 / 194
static int persist_grid(const cg_system *s)
{
    const int per_sm = cg::PERSIST_WPB * GPW;
    return std::max(1, std::min(s->in_run ? running_streams.share(s, per_sm) : s->sms, nblk(s->N, per_sm)));
}

// Cells above which k_spp integrates after the tail, at full occupancy (the tail has 16 warps per SM): a
// 963507-cell ensemble 184 -> 167 us per step (the graph: 178), 400000 cells 92.4 -> 90.2, 262144 the same.
// Single steps from 200000: at 262144 cells with L2 flushed 86.0 -> 84.0 (warm 68.7 -> 70.0, host steps
// 81.5 -> 81.1); at 180000 75.8 -> 73.8, 59.1 -> 60.4, 73.4 -> 73.5.
constexpr int SPLIT_MOVE_CELLS = 300000, SPLIT_MOVE_SINGLE = 200000;

// Whether steps can run without the step graph: the device takes the launches, 32-slot rows need the wide
// forms of the repair, and the profiling form unrolls graphs.
static bool persist_any(const cg_system *s)
{
    const char *u = getenv("CG_GRAPH_UNROLLED");
    return !(u && u[0] == '1') && s->K <= VG && !s->coop_refused;
}

enum StepForm { STEP_GRAPH, STEP_ONE, STEP_TWO };  // the step graph, one launch, two launches per step

// The form that n steps take. Single steps beside those of other streams (host-driven systems) go
// through the step graph, whose kernels overlap with theirs; two small systems also fit side by side.
// us per round of single steps of M systems, one launch / graph:
//   300 cells    M = 2  21 / 29    4  40 / 30    8   66 / 37
//   4096 cells   M = 2  24 / 34    4  32 / 37    8   64 / 43
//   16384 cells  M = 2  52 / 44    4 102 / 47    8  195 / 59
static StepForm step_form(const cg_system *s, int n)
{
    if (!persist_any(s)) return STEP_GRAPH;
    if (n == 1) {
        const bool small = s->N <= (s->det                  ? PERSIST_MAX_SINGLE_FIX
                                    : persist_thread_ok(s) ? PERSIST_MAX_SINGLE
                                                           : PERSIST_MAX_SINGLE_CELLS);
        const int others = busy_streams.others(s);
        if (others > 0) return small && others == 1 && 2 * persist_grid(s) <= s->sms ? STEP_ONE : STEP_GRAPH;
        if (small) return STEP_ONE;
        return s->det && s->N > PERSIST_MAX_TWO_FIX ? STEP_GRAPH : STEP_TWO;
    }
    return s->N <= (persist_thread_ok(s) ? PERSIST_MAX_THREAD : PERSIST_MAX_CELLS) ? STEP_ONE : STEP_TWO;
}

// A launch that the device refuses (fewer SMs than the grid for this process, no room for a cluster in any
// GPC): nothing of it ran, and the system's steps go by graphs from then on.
constexpr int PERSIST_REFUSED = 1;

static bool launch_refused(cudaError_t e)
{
    return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources ||
           e == cudaErrorInvalidConfiguration || e == cudaErrorInvalidClusterSize || e == cudaErrorNotSupported;
}

static int persist_refused(cg_system *s)
{
    cudaGetLastError();  // (not sticky)
    s->coop_refused = true;
    return PERSIST_REFUSED;
}

// Whether a launch of this grid is one cluster (whose hardware barrier has no limit to run out).
static bool persist_cluster(const cg_system *s, int grid)
{
    return grid <= PERSIST_CLUSTER && !s->stall_ns && !s->inject_refusal;
}

// A cooperative launch, or one cluster where the grid is small and a GPC has room for it (*cluster, an
// argument of the kernel, is set accordingly).
static int persist_launch(cg_system *s, int grid, int *cluster, const void *kernel, void **args, size_t smem)
{
    *cluster = persist_cluster(s, grid);
    if (s->inject_refusal) grid = 4 * s->sms;  // (a block takes an SM)
    CG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(cg::PERSIST_WPB * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s->stream;
    cudaLaunchAttribute at;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaSuccess;
    if (*cluster) {
        CG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = grid;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        e = cudaLaunchKernelExC(&cfg, kernel, args);
        if (launch_refused(e)) {
            cudaGetLastError();
            *cluster = 0;
            CG_CUDA(cudaMemsetAsync(s->persist_bar, 0, 2 * sizeof(unsigned), s->stream));
        }
    }
    if (!*cluster) {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
        e = cudaLaunchKernelExC(&cfg, kernel, args);
        if (launch_refused(e)) return persist_refused(s);
    }
    CG_CUDA(e);
    enqueued(s);
    s->kernels_enqueued += 1;
    return CG_OK;
}

// Before a launch: force sums (fixed-point ones where fix) and barrier counters at zero. One cluster needs no
// counters, and its few sums are cleared sooner by a memset (400 cells in mixed precision 21.5 against 23.3
// us per host step, 100 cells 23.7 against 24.8).
static int persist_clear(cg_system *s, int grid, const unsigned long long *fix, bool sums = true)
{
    const long long n = sums ? (long long)ndof(s) * (fix ? 2 * FIXF / 2 : 1) : 0;
    void *p = fix ? (void *)s->Ffix : (void *)s->F;
    if (persist_cluster(s, grid)) {
        if (n) CG_CUDA(cudaMemsetAsync(p, 0, sizeof(ulonglong2) * n, s->stream));
        return CG_OK;
    }
    k_persist_clear<<<std::max(1, std::min(8 * s->sms, nblk((int)std::min(n, 1ll << 30), 256))), 256, 0, s->stream>>>(
        reinterpret_cast<ulonglong2 *>(p), n, s->persist_bar);
    s->kernels_enqueued += 1;
    return check_launch();
}

static int persist_args(cg_system *s, int grid, cg::PersistArgs &p)
{
    if (!s->persist_bar) CG_TRY(dalloc(s, &s->persist_bar, 2));
    memset(&p, 0, sizeof(p));
    p.a = sys_args(s);
    p.a.old_cap = std::min(s->N, OLD_ROWS);  // commit and check on two warps
    p.bar = s->persist_bar;
    p.absent = s->stall_ns ? 1 : 0;
    p.wait_ns = s->stall_ns ? s->stall_ns : cg::PERSIST_WAIT_NS;
    p.excl = s->n_excl > 0 ? s->excl : nullptr;
    p.ext = s->ext_force;
    p.thread_form = persist_thread_ok(s) && s->N > PERSIST_THREAD_CELLS * grid;
    return CG_OK;
}

static bool persist_fire_ok(const cg_system *s)
{
    return s->model == CG_MODEL_VORONOI && !s->det && s->N <= PERSIST_MAX_FIRE && persist_any(s);
}

// up to n FIRE iterations, enqueued, or PERSIST_REFUSED (the FIRE state is set up and F holds the current forces)
static int enqueue_fire_persistent(cg_system *s, int n, cg::FireArgs f)
{
    cg::PersistArgs p;
    const int grid = persist_grid(s);
    CG_TRY(persist_args(s, grid, p));
    CG_TRY(persist_clear(s, grid, nullptr, false));
    p.steps = n;
    void *args[] = {&p, &f};
    return persist_launch(s, grid, &p.cluster, (const void *)cg::k_fire_voro, args, cg::PERSIST_SMEM);
}

// the steps of p, each as its force pass and a cooperative launch for the rest (the sums are cleared)
template <typename R>
static int split_steps(cg_system *s, int grid, cg::PersistArgs p)
{
    const void *k = p.a.Ffix ? tail_kernel<R, 1>() : tail_kernel<R, 0>();
    if (s->inject_refusal) grid = 4 * s->sms;
    CG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cg::PERSIST_SMEM));
    const bool own_move = s->N > (p.steps == 1 ? SPLIT_MOVE_SINGLE : SPLIT_MOVE_CELLS) && !p.a.Ffix && !p.excl;
    for (int t = 0; t < p.steps; ++t) {
        VoroArgs a = p.a;
        a.ctl = p.a.ctl + (t & 1);
        launch_groups<R, true, true>(a, s->N, s->stream, s->tune_force);
        int last = t + 1 == p.steps, move = !own_move;
        void *args[] = {&p, &t, &last, &move};
        const cudaError_t e = cudaLaunchCooperativeKernel(k, dim3(grid), dim3(cg::PERSIST_WPB * 32), args,
                                                          cg::PERSIST_SMEM, s->stream);
        if (t == 0 && launch_refused(e)) {  // the force pass has run: take its queues back
            Ctl c;
            persist_refused(s);
            CG_TRY(read_ctl(s, c));
            if (!c.halt) CG_TRY(clear_queues(s));  // (halted before: it did nothing)
            return PERSIST_REFUSED;
        }
        CG_CUDA(e);
        if (own_move)  // (the step is counted at the end of the call, by its last tail)
            k_spp<R><<<nblk((s->N + 1) / 2, SPP_BLOCK), SPP_BLOCK, 0, s->stream>>>(
                p.a, p.noise ? p.noise + (size_t)t * s->N : nullptr, p.dt, p.mu, last ? (uint32_t)-1 : (uint32_t)t, !last);
    }
    enqueued(s);
    s->kernels_enqueued += (own_move ? 3 : 2) * (long long)p.steps;
    return check_launch();
}

// n SPP steps, enqueued, or PERSIST_REFUSED (noise: n x N normals on the device, or null; energy_dst: page-locked host
// memory for the energies of the last step's force evaluation, e2e_acc allocated)
template <typename R>
static int enqueue_persistent(cg_system *s, StepForm form, int n, double dt, double mu, const double *noise,
                              double *energy_dst = nullptr)
{
    cg::PersistArgs p;
    const int grid = persist_grid(s);
    CG_TRY(persist_args(s, grid, p));
    p.noise = noise;
    p.steps = n;
    p.dt = dt;
    p.mu = mu;
    const bool fix_energy = energy_dst && p.a.Ffix;  // fixed-point sums: the separate readout kernel
    if (energy_dst && !fix_energy) {
        p.acc = s->e2e_acc;
        p.host_out = energy_dst;
    }
    const void *k = p.a.Ffix ? persist_kernel<R, 1>() : persist_kernel<R, 0>();
    CG_TRY(persist_clear(s, form == STEP_ONE ? grid : s->sms, p.a.Ffix));
    if (form == STEP_ONE) {
        void *args[] = {&p};
        const int st = persist_launch(s, grid, &p.cluster, k, args, cg::PERSIST_SMEM);
        if (st) return st;
    } else {
        const int st = split_steps<R>(s, grid, p);
        if (st) return st;
    }
    if (fix_energy) {
        k_energy_to_host<R><<<nblk(s->N, 256), 256, 0, s->stream>>>(p.a, s->e2e_acc, s->e2e_done, energy_dst);
        s->kernels_enqueued += 1;
    }
    return CG_OK;
}
