// cellgpu_b200 -- many steps, or FIRE iterations, of a vertex-model system in one launch. Included by
// system.cu after persist.cu, whose barrier and control-block handling it shares.
//
// A step of the graph path is three dependent launches around little work (12 us a step at 100 cells as
// at 1000). Here one cooperative launch runs them with the
// same per-cell and per-vertex code and grid barriers between the phases. The T1 sweep stays one block
// per instance; it runs only when the detection queued an edge: with one instance in the block that
// arrives last at the barrier after the detection, else spread over the blocks behind a barrier of its
// own.

namespace cg {

struct PersistVmArgs {
    VertArgs a;           // a.ctl: the control block; a.ctl[1]: the one of odd steps
    unsigned *bar;        // barrier arrivals, zero at launch
    int cluster;          // the grid is one thread-block cluster
    int absent;           // as in PersistArgs
    unsigned long long wait_ns;
    int kind;             // 0 Brownian, 1 self-propelled
    const double *noise;  // steps x (2 Nv or Nc) normals, or null: drawn
    int steps;
    double dt, mu, T;
};

constexpr int PVM_GPW = 32 / VM_G;
constexpr size_t PVM_TILES = sizeof(VmTile) * PERSIST_WPB * PVM_GPW;
constexpr size_t PVM_SMEM = PVM_TILES > T1_SMEM ? PVM_TILES : T1_SMEM;

// forces of the block's cells (F zero before)
CG_D void pvm_forces(const VertArgs &a, unsigned char *smem)
{
    VmTile *tiles = reinterpret_cast<VmTile *>(smem);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = w * PVM_GPW + lane / VM_G;
    const int cpb = (a.Nc + gridDim.x * PVM_GPW - 1) / (gridDim.x * PVM_GPW) * PVM_GPW;
    const int lo = blockIdx.x * cpb, hi = min(a.Nc, lo + cpb);
    for (int base = lo + w * PVM_GPW; base < hi; base += PERSIST_WPB * PVM_GPW) {  // warp-uniform
        const int c = base + lane / VM_G;
        vm_forces_cell(a, c, c < hi, 1, tiles[g], lane);
        __syncwarp();  // the tile is free for the warp's next cells
    }
}

// T1 detection and sweep on the current positions, after a barrier; ends with a barrier. The number
// of queued edges is counted in the control block's n_flagged.
CG_D int pvm_t1(const VertArgs &a, Ctl *ctl, GridBarrier &gb, unsigned char *smem, int tid, int nt)
{
    volatile Ctl *vc = ctl;
    for (int v = tid; v < a.Nv; v += nt) vm_detect(a, v, &ctl->n_flagged);
    if (a.n_inst == 1) {
        if (!gb.wait_last([&]() {
                if (vc->n_flagged > 0) t1_replay(a, ctl, 0, smem);
            }))
            return PERSIST_TIMEOUT;
    } else {
        if (!gb.wait()) return PERSIST_TIMEOUT;
        if (vc->n_flagged > 0) {
            for (int i = blockIdx.x; i < a.n_inst; i += gridDim.x) {
                t1_replay(a, ctl, i, smem);
                __syncthreads();
            }
            if (!gb.wait()) return PERSIST_TIMEOUT;
        }
    }
    return vc->halt ? PERSIST_HALT : PERSIST_OK;
}

// force of vertex v, once complete; the sums are cleared for the next force pass (clear: F itself too)
CG_D double2 pvm_take_force(const VertArgs &a, int v, bool clear)
{
    double2 f;
    if (a.Ffix) {
        ulonglong2 *w = reinterpret_cast<ulonglong2 *>(a.Ffix) + 4 * (size_t)v;
        const ulonglong2 w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3];
        f = make_double2(fix_force_value(w0, w1), fix_force_value(w2, w3));
        const ulonglong2 z = make_ulonglong2(0ull, 0ull);
        w[0] = z;
        w[1] = z;
        w[2] = z;
        w[3] = z;
        a.F[v] = f;
    } else {
        f = a.F[v];
        if (clear) a.F[v] = make_double2(0.0, 0.0);
    }
    return f;
}

__global__ void __launch_bounds__(PERSIST_WPB * 32, 1) k_vm_steps(const __grid_constant__ PersistVmArgs p)
{
    extern __shared__ __align__(16) unsigned char persist_smem[];
    __shared__ int s_ok;
    const VertArgs &a = p.a;
    Ctl *const c0 = p.a.ctl, *cur = c0;
    if (c0->halt) return;  // uniform across the grid: set by an earlier launch only
    GridBarrier gb = {p.bar, 0u, &s_ok, p.cluster != 0, gridDim.x + p.absent, p.wait_ns};
    const int step0 = c0->step;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const bool lead = tid == 0;
    int st = PERSIST_OK, t = 0;
    for (; t < p.steps; ++t) {
        cur = c0 + (t & 1);
        const uint32_t step = (uint32_t)(step0 + t);
        pvm_forces(a, persist_smem);
        gb.arrive();
        // while the blocks meet: the noise, or the velocity, of the thread's first vertex
        double2 d = make_double2(0.0, 0.0);
        const auto displacement = [&](int v) {
            if (p.kind) return vm_spp_velocity(a, v);
            if (!p.noise) return vm_noise(a, v, step);
            const double *nz = p.noise + 2 * ((size_t)t * a.Nv + v);
            return make_double2(nz[0], nz[1]);
        };
        if (tid < a.Nv) d = displacement(tid);
        if (!gb.finish()) {
            st = PERSIST_TIMEOUT;
            break;
        }
        if (lead) ctl_reset(c0 + ((t + 1) & 1), cur->epoch + R_MAX + 2);  // last read in the previous step
        for (int v = tid; v < a.Nv; v += nt) {
            if (v != tid) d = displacement(v);
            const double2 f = pvm_take_force(a, v, t + 1 < p.steps);
            if (p.kind)
                vm_spp_move(a, v, d, f, p.dt, p.mu);
            else
                vm_brownian_move(a, v, d, f, p.dt, p.mu, p.T);
        }
        if (!gb.wait()) {
            st = PERSIST_TIMEOUT;
            break;
        }
        if (p.kind)  // every vertex has read its cells' directors
            for (int c = tid; c < a.Nc; c += nt)
                vm_spp_director(a, c, p.noise ? p.noise + (size_t)t * a.Nc : nullptr, step, p.dt);
        st = pvm_t1(a, cur, gb, persist_smem, tid, nt);
        if (st != PERSIST_OK) break;
    }
    if (st == PERSIST_TIMEOUT) {
        persist_timeout(c0, step0 + t);
        return;
    }
    if (lead) {
        if (st == PERSIST_HALT) cur->n_flagged = 0;  // the count of queued edges (last read before the sweep)
        persist_end(c0, cur, st, step0 + t);
    }
}

// FIRE iterations (fire.cu): the pending mix with the first Verlet half, T1 detection and sweep, forces,
// the second half with the sums, the update by the block that arrives last. A halt (a full cell row)
// leaves the iteration between its move and its forces, as the graph form does.
__global__ void __launch_bounds__(PERSIST_WPB * 32, 1) k_fire_vm(const __grid_constant__ PersistVmArgs p, FireArgs f)
{
    extern __shared__ __align__(16) unsigned char persist_smem[];
    __shared__ int s_ok, s_running;
    __shared__ double s_red[4][PERSIST_WPB];
    const VertArgs &a = p.a;
    Ctl *const c0 = p.a.ctl, *cur = c0;
    if (c0->halt) return;  // uniform across the grid: set by an earlier launch only
    GridBarrier gb = {p.bar, 0u, &s_ok, p.cluster != 0, gridDim.x + p.absent, p.wait_ns};
    const int step0 = c0->step;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const bool lead = tid == 0;
    int st = PERSIST_OK, t = 0;
    bool stop = false;
    for (; t < p.steps && !stop; ++t) {
        cur = c0 + (t & 1);
        for (int i = tid; i < a.Nv; i += nt) fire_mix_vv1(f, i);
        if (!gb.wait()) {
            st = PERSIST_TIMEOUT;
            break;
        }
        if (lead) ctl_reset(c0 + ((t + 1) & 1), cur->epoch + R_MAX + 2);
        st = pvm_t1(a, cur, gb, persist_smem, tid, nt);
        if (st != PERSIST_OK) break;
        pvm_forces(a, persist_smem);
        if (!gb.wait()) {
            st = PERSIST_TIMEOUT;
            break;
        }
        if (!fire_finish(f, gb, s_red, &s_running, c0, tid, nt, [](int) {})) {
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
        if (st == PERSIST_HALT) cur->n_flagged = 0;
        c0->fire_iters = st == PERSIST_HALT ? t + 1 : t;
        persist_end(c0, st == PERSIST_OK ? c0 : cur, st, step0);
    }
}

}  // namespace cg

// Largest systems that step, or minimise, in one launch. us per Brownian step and per FIRE iteration
// (192 from a random dual), one launch against the graph:
//   Nc = 100    9.2 / 12.1   13.0 / 17.1
//   Nc = 300    9.8 / 12.2   14.9 / 17.7
//   Nc = 1000  10.4 / 12.4   18.9 / 20.9
//   Nc = 4096  15.4 / 13.9   29.5 / 27.4
// Above, the phases fill more SMs than the barriers save, and the sweep runs in fewer registers here.
constexpr int PERSIST_VM_MAX = 2048;

static bool persist_vm_ok(const cg_system *s, bool fire)
{
    return s->model == CG_MODEL_VERTEX && !s->coop_refused && s->vmax <= VM_ROW_G && s->N <= PERSIST_VM_MAX && !(fire && s->det);
}

static int persist_vm_args(cg_system *s, cg::PersistVmArgs &p)
{
    if (!s->persist_bar) CG_TRY(dalloc(s, &s->persist_bar, 2));
    memset(&p, 0, sizeof(p));
    p.a = vm_args(s);
    p.bar = s->persist_bar;
    p.absent = s->stall_ns ? 1 : 0;
    p.wait_ns = s->stall_ns ? s->stall_ns : cg::PERSIST_WAIT_NS;
    return CG_OK;
}

// n steps, enqueued, or PERSIST_REFUSED (noise: n steps' normals on the device, or null)
static int enqueue_vm_persistent(cg_system *s, int kind, int n, double dt, double mu, double T, const double *noise)
{
    cg::PersistVmArgs p;
    CG_TRY(persist_vm_args(s, p));
    p.kind = kind;
    p.noise = noise;
    p.steps = n;
    p.dt = dt;
    p.mu = mu;
    p.T = T;
    const int grid = persist_grid(s);
    CG_TRY(persist_clear(s, grid, p.a.Ffix));
    void *args[] = {&p};
    return persist_launch(s, grid, &p.cluster, (const void *)cg::k_vm_steps, args, cg::PVM_SMEM);
}

// up to n FIRE iterations, enqueued, or PERSIST_REFUSED (the FIRE state is set up and F holds the current forces)
static int enqueue_fire_vm(cg_system *s, int n, cg::FireArgs f)
{
    cg::PersistVmArgs p;
    CG_TRY(persist_vm_args(s, p));
    const int grid = persist_grid(s);
    CG_TRY(persist_clear(s, grid, nullptr, false));
    p.steps = n;
    void *args[] = {&p, &f};
    return persist_launch(s, grid, &p.cluster, (const void *)cg::k_fire_vm, args, cg::PVM_SMEM);
}
