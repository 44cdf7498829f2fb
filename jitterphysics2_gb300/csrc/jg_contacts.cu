// Persistent contact cache and solver colouring.
//
// merge:   the contact stream is matched against the live arbiters through an
//          open-addressing hash on the ordered shape-id pair (ArbiterKey, Arbiter.cs:67-103);
//          unknown keys allocate a new arbiter (ContactData.Init, Contact.cs:271-286), then
//          ResetMode and AddContact run per manifold point (World.RegisterContact,
//          World.Detect.cs:294-324; ContactData.AddContact / SortCachedPoints, Contact.cs:329-580).
// colour:  Jones-Plassmann colouring of contacts and joints with per-body colour masks;
//          static and kinematic bodies never conflict because the solver never writes them.
//          It replaces the reference's per-body spin locks (World.Step.cs:924-986).
// permute: arbiters with contacts are moved to the other buffer sorted by colour; arbiters
//          left without contacts are dropped (RemoveBrokenArbiters, World.Step.cs:839-860).
// update:  ContactData.UpdatePosition (Contact.cs:238-264, :762-797) after the solve.
//
// The contact-cache rules follow code the reference derived from the Bullet Physics
// Engine (zlib license, (c) 2003-2006 Erwin Coumans, https://bulletphysics.org): provided
// 'as-is', without any express or implied warranty; altered source versions must be
// plainly marked as such; this notice may not be removed or altered from any source
// distribution.
#include "jg_sync.cuh"

namespace {

constexpr unsigned long long HEMPTY = 0xffffffffffffffffull;
constexpr float BreakThreshold = 0.02f;

__device__ __forceinline__ unsigned long long akey(int2 k) {
    return ((unsigned long long)(unsigned)k.x << 32) | (unsigned)k.y;
}
__device__ __forceinline__ unsigned hash64(unsigned long long k) {
    k ^= k >> 33; k *= 0xff51afd7ed558ccdull; k ^= k >> 33; k *= 0xc4ceb9fe1a85ec53ull; k ^= k >> 33;
    return (unsigned)k;
}

__global__ void k_hash_clear(WorldDev w) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < w.hcap; i += gridDim.x * blockDim.x) {
        w.hkeys[i] = HEMPTY;
        w.hvals[i] = -1;
    }
}

__device__ __forceinline__ int hash_insert(WorldDev& w, unsigned long long key, int val) {
    unsigned mask = (unsigned)w.hcap - 1u;
    unsigned h = hash64(key) & mask;
    for (int probe = 0; probe < w.hcap; probe++) {
        unsigned long long prev = atomicCAS(&w.hkeys[h], HEMPTY, key);
        if (prev == HEMPTY) { w.hvals[h] = val; return val; }
        if (prev == key) return -2;
        h = (h + 1) & mask;
    }
    return -3;
}
__device__ __forceinline__ int hash_find(const WorldDev& w, unsigned long long key) {
    unsigned mask = (unsigned)w.hcap - 1u;
    unsigned h = hash64(key) & mask;
    for (int probe = 0; probe < w.hcap; probe++) {
        unsigned long long k = w.hkeys[h];
        if (k == key) return w.hvals[h];
        if (k == HEMPTY) return -1;
        h = (h + 1) & mask;
    }
    return -1;
}

__global__ void k_hash_build(WorldDev w) {
    const ArbStore& A = w.arb[w.cur];
    int n = w.ctr->narb;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x)
        hash_insert(w, akey(A.key[a]), a);
}

// Contact.Initialize (Contact.cs:703-759)
__device__ void contact_init(const WorldDev& w, const ArbStore& A, int i, int b1, int b2, int mode, float restitution,
                             v3 p1, v3 p2, v3 n, bool is_new) {
    v3 pos1 = mk3(w.pos[b1]), pos2 = mk3(w.pos[b2]);
    q4 q1 = mkq(w.q[b1]), q2 = mkq(w.q[b2]);
    v3 rel1 = p1 - pos1, rel2 = p2 - pos2;
    A.cr1[i] = f4(rel1, A.cr1[i].w);
    A.cr2[i] = f4(rel2, A.cr2[i].w);
    A.cp1[i] = f4(rotate_inv(rel1, q1), 0.f);
    A.cp2[i] = f4(rotate_inv(rel2, q2), 0.f);
    if (!is_new) return;
    SBody B1 = w.body[b1], B2 = w.body[b2];
    v3 v1 = mk3(B1.v), v2 = mk3(B2.v), w1 = mk3(B1.w), w2 = mk3(B2.w);
    v3 dv = v2 - v1;
    if (mode == 0 || (mode & (2 | 8)) != 0) {
        dv = v2 + cross(w2, rel2);
        dv = dv - (v1 + cross(w1, rel1));
    }
    float rnv = dot(dv, n);
    float bias = 0.f;
    if (rnv < -1.0f) bias = -restitution * rnv;
    v3 t1 = dv - n * rnv;
    float num = len2(t1);
    if (num > 1e-12f) {
        num = 1.0f / sqrtf(num);
        t1 = t1 * num;
    } else {
        t1 = create_orthonormal(n);
    }
    v3 t2 = cross(t1, n);
    A.cn[i] = f4(n, bias);
    A.ct1[i] = f4(t1, 0.f);
    A.ct2[i] = f4(t2, __int_as_float(2));   // Flags.NewContact
    A.cacc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ __forceinline__ float area4(v3 p0, v3 p1, v3 p2, v3 p3) {
    v3 a0 = p0 - p1, a1 = p0 - p2, a2 = p0 - p3;
    v3 b0 = p2 - p3, b1 = p1 - p3, b2 = p1 - p2;
    return fmaxf(fmaxf(len2(cross(a0, b0)), len2(cross(a1, b1))), len2(cross(a2, b2)));
}

// ContactData.AddContact + SortCachedPoints (Contact.cs:329-416, :555-580)
__device__ void add_contact(const WorldDev& w, const ArbStore& A, int a, int& usage, int b1, int b2, int mode,
                            float restitution, v3 p1, v3 p2, v3 n, int& created) {
    const int cap = w.cap_arb;
    v3 rp1 = p1 - mk3(w.pos[b1]);
    if ((usage & 15) == 15) {
        v3 c0 = mk3(A.cr1[a]), c1 = mk3(A.cr1[cap + a]), c2 = mk3(A.cr1[2 * cap + a]), c3 = mk3(A.cr1[3 * cap + a]);
        float ar0 = area4(rp1, c1, c2, c3), ar1 = area4(rp1, c0, c2, c3), ar2 = area4(rp1, c0, c1, c3), ar3 = area4(rp1, c0, c1, c2);
        const float eps = -0.0001f;
        float big = 0.f;
        int mask = 0;
        if (ar0 > big + eps) { big = ar0; mask = 1; }
        if (ar1 > big + eps) { big = ar1; mask = 2; }
        if (ar2 > big + eps) { big = ar2; mask = 4; }
        if (ar3 > big + eps) { mask = 8; }
        int k = mask == 2 ? 1 : (mask == 4 ? 2 : (mask == 8 ? 3 : 0));
        contact_init(w, A, k * cap + a, b1, b2, mode, restitution, p1, p2, n, false);
        usage |= mask;
        return;
    }
    int closest = -1;
    float dist = 3.402823466e+38f;
    for (int k = 0; k < 4; k++) {
        if (!(usage & (1 << k))) continue;
        float d = len2(mk3(A.cr1[k * cap + a]) - rp1);
        if (d < dist) { dist = d; closest = k; }
    }
    if (dist < BreakThreshold * BreakThreshold) {
        contact_init(w, A, closest * cap + a, b1, b2, mode, restitution, p1, p2, n, false);
        return;
    }
    for (int k = 0; k < 4; k++) {
        if (!(usage & (1 << k))) {
            contact_init(w, A, k * cap + a, b1, b2, mode, restitution, p1, p2, n, true);
            usage |= 1 << k;
            created++;
            return;
        }
    }
}

__global__ void k_merge(WorldDev w, StepParams sp, int2* ev_created) {
    const ArbStore& A = w.arb[w.cur];
    int ns = min(w.ctr->nstream, w.cap_pairs);
    int created_pts = 0, contacts = 0, spec = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += gridDim.x * blockDim.x) {
        int2 key = w.cs_key[i];
        unsigned long long k64 = akey(key);
        int a = hash_find(w, k64);
        int b1 = w.sinfo[key.x].y, b2 = w.sinfo[key.y].y;
        float4 m1 = w.mat[b1], m2 = w.mat[b2];
        if (a < 0) {
            a = atomicAdd(&w.ctr->narb, 1);
            if (a >= w.cap_arb) { atomicCAS(&w.ctr->status, 0, JG_ERR_CAPACITY); continue; }
            if (w.allow_deact) {  // HandleDeferredArbiters: AddToActiveList on both islands (World.Step.cs:880-914)
                atomicOr(&w.binfo[b1].w, 3);
                atomicOr(&w.binfo[b2].w, 3);
            }
            A.key[a] = key;
            A.body[a] = make_int2(b1, b2);
            A.mat[a] = make_float4(fmaxf(m1.x, m2.x), fmaxf(m1.y, m2.y), sp.spec_relax, 0.f);
            A.info[a] = make_int4(0, 0, -1, 1);
            int e = atomicAdd(&w.ctr->nnew, 1);
            if (e < w.cap_arb) ev_created[e] = key;
        }
        int4 info = A.info[a];
        float restitution = A.mat[a].y;
        int usage = info.x;
        if (!sp.persistent) usage = 0;
        // ContactData.ResetMode (Contact.cs:288-296)
        int mode = (w.binfo[b1].x == JG_MOTION_DYNAMIC ? 3 : 0) | (w.binfo[b2].x == JG_MOTION_DYNAMIC ? 12 : 0);
        float4 nc = w.cs_n[i];
        v3 n = mk3(nc);
        int cnt = __float_as_int(nc.w) & 0xff;
        // a speculative contact updates linear velocities only: ResetMode(SolveMode.Angular)
        // (World.Detect.cs:193-194)
        if (__float_as_int(nc.w) & JG_STREAM_SPECULATIVE) { mode &= ~(2 | 8); spec++; }
        // ResetMode before AddContact: Initialize reads the mode
        for (int k = 0; k < cnt; k++)
            add_contact(w, A, a, usage, b1, b2, mode, restitution, mk3(w.cs_pa[4 * i + k]), mk3(w.cs_pb[4 * i + k]), n, created_pts);
        A.info[a] = make_int4(usage, mode, info.z, info.w);
        contacts += __popc(usage & 15);
    }
    if (created_pts) atomicAdd(&w.ctr->new_contacts, created_pts);
    if (spec) atomicAdd(&w.ctr->nspec_hit, spec);
    (void)contacts;
}

// ---- colouring -----------------------------------------------------------------------------
__device__ __forceinline__ unsigned prio(unsigned long long key) { return hash64(key * 0x9E3779B97F4A7C15ull + 1); }

__device__ __forceinline__ void cons_bodies(const WorldDev& w, const ArbStore& A, int c, int narb, int& b1, int& b2,
                                            unsigned long long& key) {
    if (c < narb) {
        int2 b = A.body[c];
        b1 = b.x; b2 = b.y;
        key = akey(A.key[c]);
    } else {
        int4 h = w.joints[c - narb].hdr;
        b1 = h.y; b2 = h.z;
        key = 0x8000000000000000ull | (unsigned long long)(c - narb);
    }
    if (w.binfo[b1].x != JG_MOTION_DYNAMIC) b1 = -1;
    if (w.binfo[b2].x != JG_MOTION_DYNAMIC) b2 = -1;
}

// Colours of the remainder (arbiters outside the tasks, and all joints), cooperative: adjacency
// build, Jones-Plassmann, colour counts.  A constraint takes the smallest colour free on its
// bodies once every neighbour of higher priority has one (no neighbour of lower priority can
// come before it), so the colours do not depend on the timing, and each thread simply
// looks at its own constraints again until they are coloured: no barrier per round.  Without a
// remainder the kernel only marks the arbiters, with no barrier at all.  (27 boxes: 54 -> 3 us;
// the joints of 1024 chains 197 -> 121.)
__global__ void k_color(WorldDev w) {
    const ArbStore& A = w.arb[w.cur];
    const int narb = w.ctr->narb < w.cap_arb ? w.ctr->narb : w.cap_arb;
    const int nj = w.nj;
    const int ncons = narb + nj;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    int* status = &w.ctr->status;
    const bool tasks = w.sc->ntasks > 0;
    const int first = tasks ? w.sc->narb_task : 0;  // the remainder follows the tasks
    const int lo = w.sc->nrem ? 0 : narb;  // (without a remainder of arbiters, the joints alone)
    for (int c = tid; c < JG_MAX_COLORS; c += nth) w.jorder[w.cap_joints + c] = 0;
    if (nj == 0 && w.sc->nrem == 0) {
        for (int c = tid; c < narb; c += nth) w.cstat[c] = (A.info[c].x & 15) == 0 ? -2 : -4;
        for (int c = tid; c <= JG_MAX_COLORS; c += nth) {
            w.color_start[c] = first;
            w.jcolor_start[c] = 0;
            w.color_cursor[c] = 0;
        }
        if (tid == 0) { w.ctr->ncolors = 0; w.remaining[0] = 0; }
        return;
    }
    for (int b = tid; b < w.nb_rows; b += nth) { w.deg[b] = 0; w.bmask[2 * b] = 0ull; w.bmask[2 * b + 1] = 0ull; }
    for (int c = tid; c < JG_MAX_COLORS + 1; c += nth) { w.color_count[c] = 0; w.color_cursor[c] = 0; }
    if (tid < 2) w.remaining[tid] = 0;
    if (!grid_sync(w.bar_count, w.bar_gen, status)) return;
    for (int c = tid; c < ncons; c += nth) {
        if (c < narb && (A.info[c].x & 15) == 0) { w.cstat[c] = -2; continue; }
        if (c < narb && tasks && w.sc_dst[c] >= 0) { w.cstat[c] = -4; continue; }  // solved in a task
        int b1, b2; unsigned long long key;
        cons_bodies(w, A, c, narb, b1, b2, key);
        w.cstat[c] = -1;
        w.cprio[c] = prio(key);
        if (b1 >= 0) atomicAdd(&w.deg[b1], 1);
        if (b2 >= 0 && b2 != b1) atomicAdd(&w.deg[b2], 1);
    }
    if (!grid_sync(w.bar_count, w.bar_gen, status)) return;
    // space for each body's list, in any order
    for (int base = blockIdx.x * blockDim.x; base < w.nb_rows; base += nth) {
        const int i = base + threadIdx.x, lane = threadIdx.x & 31;
        const int v = i < w.nb_rows ? w.deg[i] : 0;
        int x = v;
        for (int o = 1; o < 32; o <<= 1) { int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
        int off = 0;
        if (lane == 31 && x) off = atomicAdd(&w.remaining[1], x);
        off = __shfl_sync(0xffffffffu, off, 31);
        if (i < w.nb_rows) { w.adj_off[i] = off + x - v; w.deg[i] = 0; }
    }
    if (!grid_sync(w.bar_count, w.bar_gen, status)) return;
    for (int c = lo + tid; c < ncons; c += nth) {
        if (w.cstat[c] < -1) continue;
        int b1, b2; unsigned long long key;
        cons_bodies(w, A, c, narb, b1, b2, key);
        if (b1 >= 0) { int s = atomicAdd(&w.deg[b1], 1); w.adj[w.adj_off[b1] + s] = c; }
        if (b2 >= 0 && b2 != b1) { int s = atomicAdd(&w.deg[b2], 1); w.adj[w.adj_off[b2] + s] = c; }
    }
    if (!grid_sync(w.bar_count, w.bar_gen, status)) return;
    // cstat = colour once coloured; every thread of the launch is resident, and the highest
    // uncoloured priority can always take its colour, so the looking ends
    const unsigned long long t0 = globaltimer_ns();
    unsigned idle = 0;
    for (bool pending = true; pending;) {
        pending = false;
        bool progress = false;
        for (int c = lo + tid; c < ncons; c += nth) {
            if (w.cstat[c] != -1) continue;
            int b1, b2; unsigned long long key;
            cons_bodies(w, A, c, narb, b1, b2, key);
            const unsigned pc = w.cprio[c];
            bool ready = true;
            for (int side = 0; side < 2 && ready; side++) {
                const int b = side == 0 ? b1 : b2;
                if (b < 0) continue;
                const int beg = w.adj_off[b], end = beg + w.deg[b];
                for (int e = beg; e < end; e++) {
                    const int n = w.adj[e];
                    if (n == c || ld_relaxed_int(&w.cstat[n]) != -1) continue;
                    const unsigned pn = w.cprio[n];
                    if (pn > pc || (pn == pc && n > c)) { ready = false; break; }
                }
            }
            if (!ready) { pending = true; continue; }
            __threadfence();  // the neighbours' colours before the masks they set
            unsigned long long m0 = 0, m1 = 0;
            if (b1 >= 0) { m0 |= __ldcg(&w.bmask[2 * b1]); m1 |= __ldcg(&w.bmask[2 * b1 + 1]); }
            if (b2 >= 0) { m0 |= __ldcg(&w.bmask[2 * b2]); m1 |= __ldcg(&w.bmask[2 * b2 + 1]); }
            int color;
            if (~m0) color = __ffsll((long long)~m0) - 1;
            else if (~m1) color = 64 + __ffsll((long long)~m1) - 1;
            else { atomicCAS(status, 0, JG_ERR_CAPACITY); color = JG_MAX_COLORS - 1; }
            unsigned long long* word = &w.bmask[color >> 6];
            const unsigned long long bit = 1ull << (color & 63);
            if (b1 >= 0) atomicOr(word + 2 * b1, bit);
            if (b2 >= 0) atomicOr(word + 2 * b2, bit);
            __threadfence();
            *(volatile int*)&w.cstat[c] = color;
            progress = true;
        }
        if (!pending || progress) continue;
        if ((++idle & 63) == 0) {
            if (ld_relaxed_int(status) == JG_ERR_TIMEOUT) break;
            if (globaltimer_ns() - t0 > 1000000000ull) { atomicCAS(status, 0, JG_ERR_TIMEOUT); break; }
        }
        __nanosleep(40);
    }
    // colour counts (joint counts in the cursor, reset before use); the last block to finish
    // turns them into first places
    for (int c = lo + tid; c < ncons; c += nth) {
        const int col = w.cstat[c];
        if (col < 0) continue;
        int* counter = c < narb ? &w.color_count[col] : &w.color_cursor[col];
        const unsigned act = __activemask(), same = __match_any_sync(act, (unsigned long long)counter);
        if ((int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(counter, __popc(same));
    }
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&w.remaining[0], 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last || threadIdx.x >= 32) return;
    __threadfence();
    int acc = first, jacc = 0, nc = 0;
    for (int base = 0; base < JG_MAX_COLORS; base += 32) {
        const int c = base + threadIdx.x;
        const int t = __ldcg(&w.color_count[c]), jt = __ldcg(&w.color_cursor[c]);
        int x = t, y = jt;
        for (int o = 1; o < 32; o <<= 1) {
            const int px = __shfl_up_sync(0xffffffffu, x, o), py = __shfl_up_sync(0xffffffffu, y, o);
            if ((int)threadIdx.x >= o) { x += px; y += py; }
        }
        const unsigned used = __ballot_sync(0xffffffffu, t || jt);
        if (used) nc = base + 32 - __clz(used);
        w.color_start[c] = acc + x - t;
        w.jcolor_start[c] = jacc + y - jt;
        w.color_cursor[c] = 0;
        acc += __shfl_sync(0xffffffffu, x, 31);
        jacc += __shfl_sync(0xffffffffu, y, 31);
    }
    if (threadIdx.x == 0) {
        w.color_start[JG_MAX_COLORS] = acc;
        w.jcolor_start[JG_MAX_COLORS] = jacc;
        w.color_cursor[JG_MAX_COLORS] = 0;
        w.ctr->ncolors = nc;
        w.remaining[0] = 0;
    }
}

// Moves every arbiter with contacts to the other buffer at its colour slot, four lanes per
// arbiter, one for each contact slot (a lane that copied them one after another waited for
// memory four times: 22 -> 9 us at a thousand arbiters).  Counts the contacts on the way; the
// last block sets the new arbiter count.  With `groups` it also clears what the search for the solve
// groups counts in (jg_groups.cu).
__global__ void k_permute(WorldDev w, int2* ev_removed, int* dst_index, bool groups) {
    const ArbStore& S = w.arb[w.cur];
    const ArbStore& D = w.arb[1 - w.cur];
    const int narb = w.ctr->narb < w.cap_arb ? w.ctr->narb : w.cap_arb;
    const int cap = w.cap_arb;
    const int k = threadIdx.x & 3;
    int contacts = 0;
    for (int base = blockIdx.x * blockDim.x; base < 4 * narb; base += gridDim.x * blockDim.x) {
        const int a = (base + (int)threadIdx.x) >> 2;
        const bool live = a < narb;
        const int st = live ? w.cstat[a] : -2;
        int4 info = make_int4(0, 0, 0, 0);
        int2 bb = make_int2(0, 0);
        if (live) { info = S.info[a]; bb = S.body[a]; }
        int d = -1;
        if (live && k == 0) {
            if (st == -4) d = w.sc_dst[a];
            else if (st >= 0) d = w.color_start[st] + atomicAdd(&w.color_cursor[st], 1);
            else {
                int e = atomicAdd(&w.ctr->nremoved, 1);
                if (e < cap) ev_removed[e] = S.key[a];
                if (w.allow_deact) {  // RemoveBrokenArbiters: AddToActiveList on both islands (World.Step.cs:845-846)
                    atomicOr(&w.binfo[bb.x].w, 3);
                    atomicOr(&w.binfo[bb.y].w, 3);
                }
            }
            dst_index[a] = d;
        }
        d = __shfl_sync(0xffffffffu, d, 0, 4);
        if (d < 0) continue;
        if (info.x & (1 << k)) {
            const int s = k * cap + a, t = k * cap + d;
            const float4 cn = S.cn[s], t1 = S.ct1[s], t2 = S.ct2[s], r1 = S.cr1[s], r2 = S.cr2[s], ac = S.cacc[s], p1 = S.cp1[s],
                         p2 = S.cp2[s];
            D.cn[t] = cn; D.ct1[t] = t1; D.ct2[t] = t2; D.cr1[t] = r1; D.cr2[t] = r2; D.cacc[t] = ac; D.cp1[t] = p1; D.cp2[t] = p2;
            contacts++;
        }
        if (k != 0) continue;
        const int4 i1 = w.binfo[bb.x], i2 = w.binfo[bb.y];
        // a row is solved and updated while one of its bodies is an awake non-static body
        // (memContacts activation follows the bodies, World.Step.cs:1247-1275, :1325-1345)
        const bool asleep = w.allow_deact && !((i1.x != JG_MOTION_STATIC && (i1.y & JG_BODY_ACTIVE)) ||
                                               (i2.x != JG_MOTION_STATIC && (i2.y & JG_BODY_ACTIVE)));
        const float4 mat = S.mat[a];
        D.key[d] = S.key[a];
        D.body[d] = bb;
        D.info[d] = make_int4(info.x, (info.y & 0xffff) | (asleep ? JG_ARB_ASLEEP : 0), st == -4 ? w.sc_lcol[a] : JG_ORDER_REMAINDER + st,
                              info.w);
        // velocities of a non-dynamic body stay constant through the solve
        const int nd = i1.x != JG_MOTION_DYNAMIC ? bb.x : (i2.x != JG_MOTION_DYNAMIC ? bb.y : -1);
        int4 ls = make_int4(-1, -1, 3, 0);
        if (st == -4) {  // task arbiters: body slots, and what the iterations read besides the rows, in one record
            ls = w.sc_ls[a];
            ls.z = (info.x & 15) | ((info.y & 15) << 4) | (nd >= 0 ? 256 : 0) | (asleep ? JG_TASK_ASLEEP : 0);
            ls.w = __float_as_int(mat.x);
        }
        D.lslot[d] = ls;
        D.sv[d] = nd >= 0 ? w.body[nd].v : make_float4(0.f, 0.f, 0.f, 0.f);
        D.sv[cap + d] = nd >= 0 ? w.body[nd].w : make_float4(0.f, 0.f, 0.f, 0.f);
        D.mat[d] = mat;
    }
    const int nj = w.nj;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nj; j += gridDim.x * blockDim.x) {
        const int st = w.cstat[narb + j];
        const int col = st >= 0 ? st : 0;
        int d = w.jcolor_start[col] + atomicAdd(&w.jorder[w.cap_joints + col], 1);
        w.jorder[d] = j;
        w.joints[j].hdr.w = JG_ORDER_REMAINDER + col;
    }
    contacts = __reduce_add_sync(0xffffffffu, contacts);
    if ((threadIdx.x & 31) == 0 && contacts) atomicAdd(&w.ctr->contacts, contacts);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&w.remaining[0], 1) == (int)gridDim.x - 1) {
            const int n = w.color_start[JG_MAX_COLORS];
            w.ctr->narb = n;
            if (groups) {
                GroupCtl c;
                memset(&c, 0, sizeof(c));
                // (arbiters outside the tasks interleave with the constraints' levels; in a step that has run
                // out of colours two rows of a body share a level, and a group would wait for a row that
                // never comes)
                c.off = (w.nworlds <= 1 && n > JG_GROUP_MAXARB) || n > w.ctr->narb_task || __ldcg(&w.ctr->status) != 0 ? 1 : 0;
                *w.gr = c;
            }
        }
    }
    if (!groups) return;
    const int nb = max(w.nb, w.nworlds);
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        if (b < w.nb) { w.gr_root[b] = b; w.gr_slot[b] = -1; }
        w.gr_narb[b] = 0; w.gr_njoint[b] = 0; w.gr_nbody[b] = 0; w.gr_ncon[b] = 0;
    }
}

// ContactData.UpdatePosition (Contact.cs:238-264) / Contact.UpdatePosition (Contact.cs:762-797)
// Four lanes per arbiter, one for each contact slot.
__global__ void k_update_contacts(WorldDev w) {
    const ArbStore& A = w.arb[w.cur];
    const int n = w.ctr->narb, cap = w.cap_arb;
    const int k = threadIdx.x & 3;
    for (int base = blockIdx.x * blockDim.x; base < 4 * n; base += gridDim.x * blockDim.x) {
        const int a = (base + (int)threadIdx.x) >> 2;
        int4 info = make_int4(0, JG_ARB_ASLEEP, 0, 0);
        if (a < n) info = A.info[a];
        const bool awake = !(info.y & JG_ARB_ASLEEP);  // sleeping contacts keep their points
        bool keep = true;
        if (awake && (info.x & (1 << k))) {
            const int i = k * cap + a;
            int2 b = A.body[a];
            v3 pos1 = mk3(w.pos[b.x]), pos2 = mk3(w.pos[b.y]);
            q4 q1 = mkq(w.q[b.x]), q2 = mkq(w.q[b.y]);
            v3 rel1 = rotate(mk3(A.cp1[i]), q1);
            v3 p1 = rel1 + pos1;
            v3 rel2 = rotate(mk3(A.cp2[i]), q2);
            v3 p2 = rel2 + pos2;
            float4 r1 = A.cr1[i], r2 = A.cr2[i];
            A.cr1[i] = f4(rel1, r1.w);
            A.cr2[i] = f4(rel2, r2.w);
            v3 dist = p1 - p2;
            v3 nrm = mk3(A.cn[i]);
            float pen = dot(dist, nrm);
            if (pen < -BreakThreshold * 0.1f) keep = false;
            else {
                dist = dist - pen * nrm;
                if (len2(dist) > BreakThreshold * BreakThreshold) keep = false;
            }
        }
        const unsigned broken = (__ballot_sync(0xffffffffu, !keep) >> (threadIdx.x & 28)) & 15u;
        if (awake && k == 0) {
            const int usage = info.x & 15;
            A.info[a] = make_int4((usage | (usage << 4)) & ~(int)broken, info.y, info.z, 0);
        }
    }
}

}  // namespace

void jg_launch_merge(WorldDev& w, const StepParams& p, cudaStream_t s, int nsm) {
    int blocks = nsm * 4;
    k_hash_clear<<<blocks, 256, 0, s>>>(w);
    k_hash_build<<<blocks, 256, 0, s>>>(w);
    k_merge<<<blocks, 128, 0, s>>>(w, p, w.ev_created);
}

// Returns 0, or -1 when the cooperative colouring launch is refused.
int jg_launch_color(WorldDev& w, cudaStream_t s, int nsm, bool groups) {
    if (w.lc_color_grid == 0) {
        int occ = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_color, 256, 0);
        if (occ < 1) occ = 1;
        w.lc_color_grid = nsm * (occ < 2 ? occ : 2);
    }
    cudaMemsetAsync(w.bar_count, 0, sizeof(unsigned) * 2, s);
    void* args[] = {(void*)&w};
    cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_color, dim3(w.lc_color_grid), dim3(256), args, 0, s);
    if (e != cudaSuccess) return -1;
    k_permute<<<nsm * 4, 256, 0, s>>>(w, w.ev_removed, w.dst_index, groups);
    return 0;
}

void jg_flip_store(WorldDev& w) { w.cur = 1 - w.cur; }

void jg_launch_update_contacts(WorldDev& w, cudaStream_t s, int nsm) {
    k_update_contacts<<<nsm * 4, 256, 0, s>>>(w);
}
