// Solve groups: sets of contacts and constraints that share no dynamic body with the rest of
// the scene, small enough for one CTA to solve alone (k_solve_groups, jg_solver.cu).
//
// The solver's order only matters between rows on one dynamic body, so independent parts of a
// scene need no common schedule: a group runs all substeps and passes of a step by itself, with
// its bodies in shared memory and no grid-wide wait.  In a batch every world is a group; in a
// single world the groups are the connected components of the bodies under the step's contacts
// and constraints.  The order keys (grid and local colour, or remainder colour) are those of the
// schedule, so the results are the same bits whichever solve runs.
//
// The groups are used only when every one of them fits a CTA, and when no contact or
// constraint touches a kinematic body (whose pose changes between substeps without belonging
// to any group), lacks a dynamic one, joins dynamic bodies of two worlds of a batch (its bodies
// would belong to two groups) or names a body beyond the uploaded ones (WorldDev::nb_rows; it has
// no place here), and when the groups are not those that the tasks solve faster (jg_group_dense);
// otherwise k_solve_tasks solves the step.  All of this is decided on the device, as the sizes live there.
#include "jg_sync.cuh"

namespace {

// The root of x; parents only point to smaller indices.  No path is shortened here: a lookup
// may run beside others.
__device__ __forceinline__ int find_root(const int* parent, int x) {
    for (;;) {
        const int p = ((const volatile int*)parent)[x];
        if (p == x) return x;
        x = p;
    }
}
// Joins two components: the larger root goes below the smaller one; a failed swap means that
// another thread moved it first, and the search continues from there.  The paths walked are
// halved on the way (a root never moves by that store, so it cannot undo a link).
__device__ __forceinline__ void join(int* parent, int a, int b) {
    volatile int* p = parent;
    for (;;) {
        for (int q = p[a]; q != a; q = p[a]) { const int r = p[q]; if (r != q) p[a] = r; a = q; }
        for (int q = p[b]; q != b; q = p[b]) { const int r = p[q]; if (r != q) p[b] = r; b = q; }
        if (a == b) return;
        if (a < b) { const int t = a; a = b; b = t; }
        if (atomicCAS(&parent[a], a, b) == a) return;
    }
}

__device__ __forceinline__ bool awake(int4 bi) { return bi.x != JG_MOTION_STATIC && (bi.y & JG_BODY_ACTIVE); }

// What a constraint means for the groups: 0 nothing to solve (asleep), 1 a group member,
// 2 the groups cannot take it.
__device__ __forceinline__ int member_kind(const WorldDev& w, int2 b, int4 i1, int4 i2) {
    if (w.allow_deact && !awake(i1) && !awake(i2)) return 0;
    if (i1.x == JG_MOTION_KINEMATIC || i2.x == JG_MOTION_KINEMATIC || max(b.x, b.y) >= w.nb) return 2;
    const bool d1 = i1.x == JG_MOTION_DYNAMIC, d2 = i2.x == JG_MOTION_DYNAMIC;
    // (a constraint may be added across worlds, and a body with rows moved to another one)
    if (d1 && d2 && w.nworlds > 1 && i1.z != i2.z) return 2;
    return d1 || d2 ? 1 : 2;
}

// Adds up over the lanes at the same counter first.
__device__ __forceinline__ void add_to(int* counter, int v) {
    const unsigned act = __activemask(), same = __match_any_sync(act, (unsigned long long)counter);
    const int sum = __reduce_add_sync(same, v);
    if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(counter, sum);
}
// Lanes at the same counter take consecutive values of it.
__device__ __forceinline__ int take_place(int* counter) {
    const unsigned act = __activemask(), same = __match_any_sync(act, (unsigned long long)counter);
    const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(same));
    return __shfl_sync(act, base, leader) + __popc(same & ((1u << lane) - 1u));
}

// Single worlds: the connected components.
__global__ void k_group_link(WorldDev w) {
    if (w.gr->off) return;
    const ArbStore& A = w.arb[w.cur];
    const int narb = min(w.ctr->narb, w.cap_arb), n = narb + w.nj;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        int2 b;
        if (c < narb) b = A.body[c];
        else { const int4 h = w.joints[c - narb].hdr; b = make_int2(h.y, h.z); }
        const int4 i1 = w.binfo[b.x], i2 = w.binfo[b.y];
        if (i1.x != JG_MOTION_DYNAMIC || i2.x != JG_MOTION_DYNAMIC || member_kind(w, b, i1, i2) != 1) continue;
        join(w.gr_root, b.x, b.y);
    }
}

// Members per group and each member's place in its group; each touched body claims a slot.
__global__ void k_group_count(WorldDev w) {
    if (w.gr->off) return;
    const ArbStore& A = w.arb[w.cur];
    const int narb = min(w.ctr->narb, w.cap_arb), n = narb + w.nj;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        int2 b;
        if (c < narb) b = A.body[c];
        else { const int4 h = w.joints[c - narb].hdr; b = make_int2(h.y, h.z); }
        const int4 i1 = w.binfo[b.x], i2 = w.binfo[b.y];
        const int kind = member_kind(w, b, i1, i2);
        if (kind == 2) w.gr->off = 1;
        if (kind != 1) { w.gr_pos[c] = make_int2(-1, 0); continue; }
        const bool d1 = i1.x == JG_MOTION_DYNAMIC, d2 = i2.x == JG_MOTION_DYNAMIC;
        const int root = w.nworlds > 1 ? (d1 ? i1.z : i2.z) : find_root(w.gr_root, d1 ? b.x : b.y);
        const int pos = take_place((c < narb ? w.gr_narb : w.gr_njoint) + root);
        w.gr_pos[c] = make_int2(root, pos);
        if (c < narb) add_to(w.gr_ncon + root, __popc(A.info[c].x & 15));
        if (d1 && atomicCAS(&w.gr_slot[b.x], -1, -2) == -1) w.gr_slot[b.x] = take_place(w.gr_nbody + root);
        if (d2 && atomicCAS(&w.gr_slot[b.y], -1, -2) == -1) w.gr_slot[b.y] = take_place(w.gr_nbody + root);
    }
}

// Space of each component (or world), and the groups: neighbouring ones (32 keys, one warp) share
// a CTA up to `share` rows, so that a scene of many small parts fills the lanes of a warp with
// rows of one level; a part above that is a group by itself.  `roomy`: groups up to which the step has
// an SM for each; `dense_class`: the smallest CTA whose groups may count as dense.
__global__ void k_group_offsets(WorldDev w, int share_div, int roomy, int dense_class) {
    if (w.gr->off) return;
    int contacts = 0, dense = 0, roomy_dense = 0;
    const int n = w.nworlds > 1 ? w.nworlds : w.nb;
    const int share = max((min(w.ctr->narb, w.cap_arb) + w.nj) / share_div, 1);
    const int lane = threadIdx.x & 31;
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += gridDim.x * blockDim.x) {
        const int i = base + lane;
        const int na = i < n ? w.gr_narb[i] : 0, nj = i < n ? w.gr_njoint[i] : 0, nbody = i < n ? w.gr_nbody[i] : 0,
                  ncon = i < n ? w.gr_ncon[i] : 0;
        const int rows = na + nj, bytes = rows ? jg_group_bytes(nbody, na, nj, ncon) : 0;
        // greedy: the running group of the warp's keys, in order
        int first = lane, run_rows = 0, run_bytes = 0, start = 0;
        for (int k = 0; k < 32; k++) {
            const int r = __shfl_sync(0xffffffffu, rows, k), by = __shfl_sync(0xffffffffu, bytes, k);
            if (r == 0) continue;
            if (run_rows == 0 || run_rows + r > share || run_bytes + by > jg_group_smem(0)) { start = k; run_rows = 0; run_bytes = 0; }
            run_rows += r; run_bytes += by;
            if (lane == k) first = start;
        }
        // prefix sums place the members of a group side by side
        int pa = na, pj = nj, pb = nbody, pc = ncon;
        for (int o = 1; o < 32; o <<= 1) {
            const int xa = __shfl_up_sync(0xffffffffu, pa, o), xj = __shfl_up_sync(0xffffffffu, pj, o), xb = __shfl_up_sync(0xffffffffu, pb, o), xc = __shfl_up_sync(0xffffffffu, pc, o);
            if (lane >= o) { pa += xa; pj += xj; pb += xb; pc += xc; }
        }
        int oa = 0, oj = 0, ob = 0;
        if (lane == 31 && pa + pj) { oa = atomicAdd(&w.gr->arbs, pa); oj = atomicAdd(&w.gr->joints, pj); ob = atomicAdd(&w.gr->bodies, pb); }
        oa = __shfl_sync(0xffffffffu, oa, 31); oj = __shfl_sync(0xffffffffu, oj, 31); ob = __shfl_sync(0xffffffffu, ob, 31);
        GroupRec r;
        r.arb = oa + pa - na; r.joint = oj + pj - nj; r.body = ob + pb - nbody;
        r.narb = na; r.njoint = nj; r.nbody = nbody;
        if (rows) w.gr_part[i] = make_int4(r.arb, r.joint, r.body, 0);
        // the first part of a group sums the others up to the next group's first
        const unsigned heads = __ballot_sync(0xffffffffu, rows > 0 && first == lane);
        const unsigned later = heads & ~((2u << lane) - 1u);
        const int last = later ? __ffs(later) - 2 : 31;
        const int ea = __shfl_sync(0xffffffffu, pa, last), ej = __shfl_sync(0xffffffffu, pj, last), eb = __shfl_sync(0xffffffffu, pb, last);
        const int ec = __shfl_sync(0xffffffffu, pc, last);
        if (rows == 0 || first != lane) continue;
        r.ncon = ec - (pc - ncon);
        r.narb = oa + ea - r.arb; r.njoint = oj + ej - r.joint; r.nbody = ob + eb - r.body;
        const int need = jg_group_bytes(r.nbody, r.narb, r.njoint, r.ncon);
        if (need > jg_group_smem(2) || r.nbody + r.njoint >= 65536 || (w.nworlds <= 1 && r.narb + r.njoint > JG_GROUP_MAXROWS)) {
            w.gr->off = 1;
            continue;
        }
        const int cls = need > jg_group_smem(1) ? 2 : (need > jg_group_smem(0) ? 1 : 0);
        contacts += r.ncon;
        if (cls >= dense_class && 2 * r.ncon >= 5 * (r.narb + r.njoint)) {
            if (r.ncon > jg_group_dense(false, w.nworlds > 1)) dense += r.ncon;
            if (r.ncon > jg_group_dense(true, w.nworlds > 1)) roomy_dense += r.ncon;
        }
        const int k = atomicAdd(&w.gr->count[cls], 1);
        w.gr_rec[cls * (size_t)w.cap_bodies + k] = r;
    }
    // Dense parts (mostly four contacts to a row, and more of them than the L1 holds): one of them decides
    // for a single world, whose time is that of its longest part, more than half of the contacts for a
    // batch.
    contacts = __reduce_add_sync(0xffffffffu, contacts);
    dense = __reduce_add_sync(0xffffffffu, dense);
    roomy_dense = __reduce_add_sync(0xffffffffu, roomy_dense);
    if (lane == 0 && contacts) {
        atomicAdd(&w.gr->contacts, contacts);
        if (dense) atomicAdd(&w.gr->dense, dense);
        if (roomy_dense) atomicAdd(&w.gr->roomy_dense, roomy_dense);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&w.gr->blocks, 1) != (int)gridDim.x - 1) return;
    __threadfence();
    int groups = 0;
    for (int c = 0; c < JG_GROUP_CLASSES; c++) groups += __ldcg(&w.gr->count[c]);
    const int d = groups <= roomy ? __ldcg(&w.gr->roomy_dense) : __ldcg(&w.gr->dense);
    if (d > (w.nworlds > 1 ? __ldcg(&w.gr->contacts) / 2 : 0)) w.gr->off = 1;
}

// Member lists; a body's slot becomes its place among all groups' bodies.
__global__ void k_group_scatter(WorldDev w) {
    if (w.gr->off) return;
    const int narb = min(w.ctr->narb, w.cap_arb), n = narb + w.nj;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    for (int c = tid; c < n; c += nth) {
        const int2 p = w.gr_pos[c];
        if (p.x < 0) continue;
        if (c < narb) w.gr_arb[w.gr_part[p.x].x + p.y] = c;
        else w.gr_joint[w.gr_part[p.x].y + p.y] = c - narb;
    }
    for (int b = tid; b < w.nb; b += nth) {
        const int s = w.gr_slot[b];
        if (s < 0) continue;
        const int root = w.nworlds > 1 ? w.binfo[b].z : find_root(w.gr_root, b);
        const int at = w.gr_part[root].z + s;
        w.gr_body[at] = b;
        w.gr_slot[b] = at;
    }
}

}  // namespace

// After the colour permutation, which has cleared what is counted here: the groups of the arbiters in the
// live store.
void jg_launch_groups(WorldDev& w, cudaStream_t s, int nsm) {
    if (w.nworlds <= 1) k_group_link<<<nsm * 4, 256, 0, s>>>(w);
    k_group_count<<<nsm * 4, 256, 0, s>>>(w);
    const bool batch = w.nworlds > 1;
    k_group_offsets<<<nsm * 2, 256, 0, s>>>(w, nsm * jg_group_ctas(0), !batch || w.nworlds <= nsm ? nsm : 0,
                                            batch && w.nworlds > 2 * nsm ? 1 : 0);
    k_group_scatter<<<nsm * 4, 256, 0, s>>>(w);
}

int jg_group_launches(const WorldDev& w) { return w.nworlds <= 1 ? 4 : 3; }
