// trace.cu -- sm_103a kernels of the stochastic split ray tracer, as a wavefront pipeline.
//
// Hot path of SplitRayTracer.cast_ray_distributed / End_Trace ("Classes_Complete_Trace -
// TaskAll.cs":335-536).  Octave rays live in a ring queue in HBM; every iteration of the device
// loop runs these kernels on one stream:
//   k_feed       1 warp: retire the last wave, hand the next batch of primaries to phase A while
//                the ring runs low (primaries stream in until the run is done, so no launch tail).
//                In graph mode it runs once before the loop; k_cond then does its step.
//   k_broadband  phase A, one thread per fed primary: emission (Classes_Sources.cs:256-265,
//                390-403), BVH walk, broadband detection (Classes_Receivers.cs:803-829), absorption
//                (Classes_Materials.cs:166-178) and Scatter_Early (4498-4570); the band children of
//                every bounce and the final split are appended to the ring (TaskAll:347-424).  Its last
//                block sizes the wave: as many ring items as leave room for their outputs.
//   k_trace      one thread per wave item: the BVH walk only, a lean kernel that keeps many warps
//                resident to hide L1/L2 latency; writes (triangle, t) per item.
//   k_shade      one thread per wave item: receiver detection into FP64 histograms (837-877),
//                absorption, one Philox draw block, Scatter_Late (phase B, 4629-4701) or
//                Scatter_VeryLate (phase C, 4572-4627), then the surviving ray and a split child are
//                appended to the ring with one atomic per warp (TaskAll:429-536).
//   k_map        with mapping receivers: the wave's receiver-grid walks, beside k_shade.
//   k_bounce     small scenes without mapping receivers, instead of the last three: walk and shade, a ray staying
//                in its lane over up to 32 interactions.
// A run of more than 256 primaries is several such loops, each over a share of them (run_worker_body).
// Random numbers are Philox4x32-10 streams keyed by (seed, primary, stream id, block): the streams
// the CPU oracle draws, so a ray's decisions do not depend on scheduling.
#include "device_common.cuh"

namespace pach {
namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ void ring_store(const DevRun &r, unsigned long long i, const ORayItem &it) {
    store_item(r.ring, i & (r.ring_cap - 1), it);
}

// Item j of the current wave: the sorted copy when the wave was sorted, else the ring in place.
__device__ __forceinline__ const ORayItem *wave_item(const DevRun &r, unsigned long long head, unsigned long long j) {
    return r.wave_buf ? r.wave_buf + j : r.ring + ((head + j) & (r.ring_cap - 1));
}

// All 32 lanes call: lane gets the first of its n ring slots; one atomic per warp.
__device__ __forceinline__ unsigned long long warp_append(unsigned long long *tail, int n) {
    const int lane = threadIdx.x & 31;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    unsigned long long base = 0;
    if (lane == 31 && total) base = atomicAdd(tail, (unsigned long long)total);
    base = __shfl_sync(FULL, base, 31);
    return base + (unsigned long long)(incl - n);
}

// ------------------------------------------------------------------------------------------
// scheduling (one warp)
// ------------------------------------------------------------------------------------------
// Primaries are fed in schedule order.  A plain run's schedule is its primaries in order; a batch's is
// every room's pilot (its first kPilotPrimaries primaries, room by room) and then every room's rest,
// with sched_off / sched_prim (2 n_rooms segments) mapping schedule positions to primaries.
//
// Pilots measure the ring footprint the feed plans batches with: the peak live count per primary (x 3)
// of the hungriest room.  The margin: a pilot fits in one wave, so each wave advances its trees by a
// whole level, while a batch larger than a wave is traced first-in-first-out across two levels at once
// and peaks higher per primary (measured up to 2.7x on 12-receiver shoeboxes at 20k primaries);
// size_wave doubles the figure again when the ring passes three quarters full.
//
// A pilot counts as measured once its live count has fallen an eighth below its peak: split trees grow
// while phase-B rays carry energy and only shrink afterwards, so the peak is over by then.  Waiting for
// the pilot's last ray instead cost a second full chain of waves, each a few launch latencies long
// (1003-primary shoebox 260 waves, now 228; 2500-primary hall with a map 228, now 182).  Rooms of a
// batch are counted separately (room_live), so after the first room's pilot the others run together, as
// many as the plan lets into half the ring: 8 rooms x 500 primaries take 381 waves and 288 ms where one
// pilot after another took about 1100 waves and 445 ms.
//
// Both are forecasts: a later room's trees may be many times the first room's, and a pilot may grow again.  A run
// whose ring is full after all starts over in careful mode: each room's pilot alone in an empty ring and to its
// last ray, one interaction a wave (run_worker_body).

// Pilot footprint of the group in flight, or false while it may still grow.  All 32 lanes call.
__device__ bool pilots_measured(const DevRun &r, WaveCtl *c, unsigned long long live, bool decaying,
                                unsigned long long &pp) {
    const int lane = threadIdx.x & 31;
    if (r.careful && live != 0) return false;
    if (r.n_rooms == 1) {
        if (live != 0 && !(decaying && live <= c->pilot_peak - c->pilot_peak / 8)) return false;
        pp = c->pilot_peak * 3 / (unsigned long long)c->pilot_count + 1;
        return true;
    }
    const int g0 = c->pilot_first, g1 = c->pilot_room;
    bool ok = true;
    unsigned long long best = 0;
    for (int i = g0 + lane; i < g1; i += 32) {
        const unsigned peak = r.room_peak[i], now = r.room_live[i];
        ok = ok && (now == 0 || now <= peak - peak / 8);
        const long long n = g1 - g0 == 1 ? c->pilot_count : r.sched_off[i + 1] - r.sched_off[i];
        const unsigned long long v = (unsigned long long)peak * 3 / (unsigned long long)max(n, 1ll) + 1;
        if (v > best) best = v;
    }
    if (!__all_sync(FULL, ok)) return false;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(FULL, best, o);
        if (v > best) best = v;
    }
    pp = best;
    return true;
}

// First primary of the loop's next n.  Loops that share a room have shares of their own in number only: which
// primaries they are goes by a common cursor, so that whatever a cancelled run has fed is the first of its primaries.
__device__ __forceinline__ long long take_primaries(const DevRun &r, const WaveCtl *c, long long next, long long n) {
    return r.cursor ? c->prim_first + (long long)atomicAdd(r.cursor, (unsigned long long)n) : next;
}

// Retires the last wave and decides what phase A gets next.  All 32 lanes call; lane 0 writes.
__device__ void feed_step(const DevRun &r) {
    WaveCtl *c = r.ctl;
    const int lane = threadIdx.x & 31;
    const unsigned long long head = c->head + c->m;
    const unsigned long long live = c->tail - head;
    const bool decaying = live <= c->last_live;
    const bool done = c->done != 0;
    long long prim_end = c->prim_end;
    const long long next = c->next_prim;
    // cancellation (graph mode): stop feeding; the primaries already fed run to completion
    int cancelled = 0;
    if (lane == 0 && r.cancel && prim_end > next) cancelled = *r.cancel;
    if (__shfl_sync(FULL, cancelled, 0)) prim_end = next;
    unsigned long long pp = 0;
    const bool in_flight = c->pilot_count > 0;
    const bool measured = !done && in_flight && pilots_measured(r, c, live, decaying, pp);
    __syncwarp();
    if (lane != 0) return;
    c->head = head;
    c->m = 0;
    c->pa_count = 0;
    if (done) return;
    c->prim_end = prim_end;
    c->last_live = live;
    if (in_flight) {
        if (!measured) return;
        if (pp < r.feed_bound) pp = r.feed_bound;
        if (pp > c->per_prim) c->per_prim = pp;
        c->pilot_count = 0;
    }
    if (next >= prim_end) return;
    const unsigned long long half = r.ring_cap / 2;
    const unsigned long long per_prim = c->per_prim ? c->per_prim : r.feed_bound;
    // hard limit: the phase-A output of every fed primary must fit
    unsigned long long fit = (r.ring_cap - live) / r.feed_bound;
    if (fit > (unsigned long long)r.feed_batch) fit = (unsigned long long)r.feed_batch;
    if (fit > (unsigned long long)(prim_end - next)) fit = (unsigned long long)(prim_end - next);
    long long lim = prim_end - next;
    // rooms without a primary in this schedule have no pilot
    while (r.n_rooms > 1 && c->pilot_room < r.n_rooms &&
           __ldg(r.sched_off + c->pilot_room + 1) == __ldg(r.sched_off + c->pilot_room))
        ++c->pilot_room;
    if (c->pilot_room < r.n_rooms) {
        // a batch never reaches into a pilot that has not run
        const long long first = r.n_rooms == 1 ? next : __ldg(r.sched_off + c->pilot_room);
        if (next >= first) {
            int k = c->pilot_room;
            unsigned long long n = 0;
            if (r.n_rooms == 1 || c->per_prim == 0 || r.careful) {  // the first pilot runs alone
                if (live != 0) return;
                n = r.n_rooms == 1 ? (unsigned long long)kPilotPrimaries
                                   : (unsigned long long)(__ldg(r.sched_off + k + 1) - next);
                ++k;
            } else {
                unsigned long long plan = live < half ? (half - live) / per_prim : 0;
                if (plan > fit) plan = fit;
                while (k < r.n_rooms) {
                    const unsigned long long q = (unsigned long long)(__ldg(r.sched_off + k + 1) - next);
                    if (q > plan && !(n == 0 && live == 0)) break;
                    n = q;
                    ++k;
                    if (q > plan) break;  // alone and larger than the plan: fed in part
                }
                if (n == 0) return;
            }
            if (n > (unsigned long long)kPilotPrimaries && r.n_rooms == 1) n = kPilotPrimaries;
            if (n > fit) n = fit;
            if (n < 1) n = 1;  // the ring holds the phase-A output of at least 4 primaries: checked at set-up
            c->pa_begin = take_primaries(r, c, next, (long long)n);
            c->pa_count = (long long)n;
            c->next_prim = next + (long long)n;
            c->pilot_count = (long long)n;
            c->pilot_peak = 0;
            c->pilot_first = c->pilot_room;
            c->pilot_room = k;
            c->last_live = 0;
            return;
        }
        if (lim > first - next) lim = first - next;
    }
    // Split trees grow for many waves after phase A, so a batch is fed only once the previous one
    // has peaked: the live count is low and no longer rising (generations of primaries).
    if (live <= r.low_water && (decaying || live == 0)) {
        // soft limit: the new batch's peak keeps the ring at most half full
        const unsigned long long soft = live < half ? (half - live) / per_prim : 0;
        unsigned long long n = fit;
        if (soft < n) n = soft > 0 ? soft : (live == 0 ? 1 : 0);
        if (n > (unsigned long long)lim) n = (unsigned long long)lim;
        if (n > 0) {
            c->pa_begin = take_primaries(r, c, next, (long long)n);
            c->pa_count = (long long)n;
            c->next_prim = next + (long long)n;
            c->pressure = 0;
        }
    }
}

__global__ void k_feed(DevRun r) { feed_step(r); }

// Sizes the wave: as many ring items as leave room for their outputs.  One warp, after every append of
// the phase-A batch (tail is read past L1: other blocks of this kernel have moved it).
__device__ void size_wave(const DevRun &r) {
    WaveCtl *c = r.ctl;
    const int lane = threadIdx.x & 31;
    if (r.n_rooms > 1 && c->pilot_count > 0)
        for (int i = c->pilot_first + lane; i < c->pilot_room; i += 32) {
            const unsigned now = __ldcg(r.room_live + i);
            if (now > r.room_peak[i]) r.room_peak[i] = now;
        }
    if (lane != 0) return;
    if (c->done) { c->m = 0; return; }
    const unsigned long long live = __ldcg(&c->tail) - c->head;
    if (live > c->peak_live) c->peak_live = live;
    c->live_now = live;
    if (c->pilot_count > 0 && live > c->pilot_peak) c->pilot_peak = live;
    // the batches outgrew their plan: plan the next ones with twice the footprint per primary
    if (live > r.ring_cap / 4 * 3 && !c->pressure && c->per_prim) {
        c->pressure = 1;
        c->per_prim *= 2;
    }
    unsigned long long m = (r.ring_cap - live) / 2;  // each item leaves at most two
    if (m > live) m = live;
    if (m > r.max_wave) m = r.max_wave;
    c->m = m;
    // a wave of k interactions leaves its items and at most k children of each phase-B ray in the ring
    const unsigned long long splitting = (unsigned long long)max(__ldcg(&c->live_b), 1ll);
    const unsigned long long per = max((r.ring_cap - live - m) / min(splitting, max(m, 1ull)), 1ull);
    // a wave that does not fill the machine is a matter of latency: its split children should not wait long
    const unsigned long long most = (unsigned long long)(m < r.full_wave ? min(r.max_bounces, kSmallBounces) : r.max_bounces);
    c->bounces = (int)(per < most ? per : most);
    c->trace_next = 0;
    c->map_next = 0;
    if (m) ++c->waves;
    if (live == 0 && c->next_prim >= c->prim_end) c->done = 1;
    if (live > 0 && m == 0) { ++c->overflow; c->done = 1; }  // ring full: cannot make progress
}

// Last node of a graph-mode iteration: decides whether the while loop runs again, and feeds the next
// iteration.  The loop ends when the run is done, and also -- as a failure -- after max_iters
// iterations or 4096 consecutive iterations that neither traced nor fed, so it always terminates.
// Progress goes to mapped host memory for the polling host thread.
__global__ void k_cond(DevRun r, cudaGraphConditionalHandle h) {
    WaveCtl *c = r.ctl;
    int stop = 0;
    if (r.n_loops > 1) {  // the rays that all loops hold now, each as its last wave was sized
        unsigned long long sum = 0;
        if ((int)threadIdx.x < r.n_loops)
            sum = __ldcg(&reinterpret_cast<const WaveCtl *>(reinterpret_cast<const char *>(r.loops) + threadIdx.x * kCtlStride)->live_now);
        for (int o = 1; o < kMaxPipes; o <<= 1) sum += __shfl_xor_sync(FULL, sum, o);
        if (threadIdx.x == 0) atomicMax(&r.cnt->peak_live, sum);
    }
    if (threadIdx.x == 0) {
        ++c->iters;
        if (c->m == 0 && c->pa_count == 0 && !c->done) ++c->idle;
        else c->idle = 0;
        stop = c->done != 0;
        if (!stop && (c->iters >= r.max_iters || c->idle >= 4096)) {
            c->gave_up = 1;
            stop = 1;
        }
        if (!stop && r.cancel && *r.cancel >= 2) {  // abort: the host stops waiting for fed primaries
            c->gave_up = 2;
            stop = 1;
        }
        if (r.mirror) {
            HostMirror *hm = r.mirror;
            hm->next_prim = c->next_prim;
            hm->iters = c->iters;
            hm->segments = r.cnt->seg_broad + r.cnt->seg_b + r.cnt->seg_c;
            hm->end_traces = r.cnt->end_traces;
            hm->gave_up = c->gave_up;
            hm->done = stop;
        }
        cudaGraphSetConditional(h, stop ? 0u : 1u);
    }
    if (__shfl_sync(FULL, stop, 0)) return;
    feed_step(r);
}

// ------------------------------------------------------------------------------------------
// phase A: broadband rays (cast_ray_distributed, TaskAll:347-424)
// ------------------------------------------------------------------------------------------
// SMALL: scenes of at most kFuseMaxTris triangles walk with the plain stack (see stack_push).
template <bool MAP, bool SMALL>
__global__ void __launch_bounds__(128) k_broadband(DevRun r) {
    extern __shared__ float4 s_rec_buf[];
    __shared__ int s_last;
    WaveCtl *c = r.ctl;
    const long long p0 = c->pa_begin, cnt = c->pa_count;
    // most iterations have nothing to emit: all blocks but one leave at once (13 us of empty blocks
    // staging receivers and flushing counters before, 3 us of the same iteration's kernels now)
    if (cnt == 0) {
        if (blockIdx.x == 0 && threadIdx.x < 32) size_wave(r);
        return;
    }
    const long long used = (cnt + blockDim.x - 1) / blockDim.x;  // blocks with work
    if ((long long)blockIdx.x >= used) return;
    const int *s_rid;
    const float4 *s_rec = stage_receivers(r, s_rec_buf, s_rid);
    LocalCounters L;
    const DevScene &S = r.S;
    const bool count_room = r.n_rooms > 1 && c->pilot_count > 0;
    int born = 0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += stride) {
        int room;
        const long long prim = scheduled_primary(r, p0 + i, room);
        const RoomParams &P = r.rooms[room];
        // SourceCluster round robin (Classes_Sources.cs:712-722)
        const int s = P.src_begin + (int)((prim + 1) % P.nsrc);
        const float4 src = r.src[s];
        float w;
        float3 d = primary_dir(r, P.nsrc, (uint32_t)prim, (int)src.w, w);
        float E[kBands], sc[kBands];
#pragma unroll
        for (int o = 0; o < kBands; ++o) {
            E[o] = 1.f;
            sc[o] = r.e0[s * kBands + o] * w;
            L.init += (double)sc[o];
        }
        float3 pos = f3(src);
        double t_sum = 0.0;
        int order = 0, plane = -1;
        bool lost = false;
        float eh;
        do {
            float t;
            int tri;
            TraceWork tw;
            const bool hit = SMALL ? trace_ray<int>(S, P.bvh_root, P.t_eps, pos, d, plane, t, tri, tw)
                                   : trace_ray<int2>(S, P.bvh_root, P.t_eps, pos, d, plane, t, tri, tw);
            L.v[C_RET] += tw.retests;
            ++L.v[C_SEGA];
            if (!hit) {
                if (order > P.is_order) {
                    L.v[C_DET] += detect_broad(r, P, s_rec, s_rid, pos, d, 1e6f, t_sum, E, sc, (uint32_t)prim);
                    if constexpr (MAP) L.v[C_DET] += map_detect_broad(r.map, P, pos, d, 1e6f, t_sum, E, sc);
                }
#pragma unroll
                for (int o = 0; o < kBands; ++o) L.lost += (double)(E[o] * sc[o]);
                lost = true;
                break;
            }
            if (order > P.is_order) {
                L.v[C_DET] += detect_broad(r, P, s_rec, s_rid, pos, d, t, t_sum, E, sc, (uint32_t)prim);
                if constexpr (MAP) L.v[C_DET] += map_detect_broad(r.map, P, pos, d, t, t_sum, E, sc);
            }
            t_sum += (double)t * P.inv_c_d;
            pos = pos + d * t;
            const float4 A = __ldg(S.tri + 3 * tri), B = __ldg(S.tri + 3 * tri + 1);
            plane = __float_as_int(A.w);
            const int poly = __float_as_int(B.w);
            const int k = order++;
            float3 n = f3(__ldg(S.pnormal + poly));
            float cos_t = dot3(d, n);
            float smid[kBands], tau[kBands];
#pragma unroll
            for (int o = 0; o < kBands; ++o) {
                const float4 m = __ldg(S.mat + poly * kBands + o);
                E[o] *= m.x;  // Basic_Material.Absorb
                smid[o] = P.pure_specular ? 0.f : m.z;
                tau[o] = (S.has_trans && !P.pure_specular) ? __ldg(S.trans + poly * kBands + o) : 0.f;
            }
            // Scatter_Early
            if (cos_t > 0.f) { n = n * -1.f; cos_t = -cos_t; }
            int nchild = 0;
#pragma unroll
            for (int o = 0; o < kBands; ++o) nchild += (E[o] != 0.f) ? (tau[o] > 0.f ? 3 : 1) : 0;
            unsigned long long slot = nchild ? atomicAdd(&c->tail, (unsigned long long)nchild) : 0ull;
            if (count_room && nchild) atomicAdd(r.room_live + room, (unsigned)nchild);
            born += nchild;
#pragma unroll
            for (int o = 0; o < kBands; ++o) {
                if (E[o] == 0.f) continue;
                Ray ch = new_ray(pos, d, E[o] * smid[o], sc[o], t_sum, (uint32_t)prim, sid_early(k, o, 0), o, 3, plane,
                                 room);
                E[o] *= (1.f - smid[o]);
                const float4 U = draw(r.seed, (uint32_t)prim, ch.sid, 0u);
                ch.d = lambert(n, U.x, U.y);
                if (tau[o] > 0.f) {
                    const Ray tr = new_ray(pos, d, E[o] * tau[o], sc[o], t_sum, (uint32_t)prim, sid_early(k, o, 1), o, 0,
                                           plane, room);
                    E[o] *= (1.f - tau[o]);
                    Ray td = ch;
                    td.I = ch.I * tau[o];
                    ch.I *= (1.f - tau[o]);
                    td.d = ch.d * -1.f;
                    td.sid = sid_early(k, o, 2);
                    ring_store(r, slot++, to_item(tr));
                    ring_store(r, slot++, to_item(td));
                    L.v[C_OCT] += 2;
                }
                ring_store(r, slot++, to_item(ch));
                ++L.v[C_OCT];
            }
            d = d - n * (2.f * cos_t);
            eh = 0.f;
#pragma unroll
            for (int o = 0; o < kBands; ++o) eh = (o == P.h_oct) ? E[o] : eh;
            if (order >= P.max_broad && eh > kTP1) { ++L.v[C_CAP]; break; }
        } while (eh > kTP1);
        if (!lost) {
            const int nfin = P.oct_hi - P.oct_lo + 1;
            unsigned long long slot = atomicAdd(&c->tail, (unsigned long long)nfin);
            if (count_room) atomicAdd(r.room_live + room, (unsigned)nfin);
            born += nfin;
#pragma unroll
            for (int o = 0; o < kBands; ++o) {
                if (o < P.oct_lo || o > P.oct_hi) continue;
                const Ray it = new_ray(pos, d, E[o], sc[o], t_sum, (uint32_t)prim, sid_final(o), o, 0, plane, room);
                ring_store(r, slot++, to_item(it));
                ++L.v[C_OCT];
            }
        }
        ++L.v[C_PRIM];
    }
    born = (int)__reduce_add_sync(FULL, (unsigned)born);
    if ((threadIdx.x & 31) == 0 && born) atomicAdd(reinterpret_cast<unsigned long long *>(&c->live_b), (unsigned long long)born);
    flush_counters(r, L);
    // the last block with work sizes the wave
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned n = (unsigned)(used < (long long)gridDim.x ? used : (long long)gridDim.x);
        s_last = atomicAdd(&c->bb_blocks, 1u) == n - 1;
        if (s_last) c->bb_blocks = 0;
        __threadfence();
    }
    __syncthreads();
    if (s_last && threadIdx.x < 32) size_wave(r);
}

// ------------------------------------------------------------------------------------------
// wave ordering: counting sort by (direction octant, Morton code of the origin cell) so that the
// rays of a warp start close together heading the same way and walk similar BVH paths
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned spread3(unsigned x) {  // 3 bits -> every third bit
    return (x & 1u) | ((x & 2u) << 2) | ((x & 4u) << 4);
}

__device__ __forceinline__ unsigned sort_key(const DevRun &r, float4 P, float4 D) {
    const int cx = min(max((int)((P.x - r.sort_lo[0]) * r.sort_inv[0]), 0), kSortGrid - 1);
    const int cy = min(max((int)((P.y - r.sort_lo[1]) * r.sort_inv[1]), 0), kSortGrid - 1);
    const int cz = min(max((int)((P.z - r.sort_lo[2]) * r.sort_inv[2]), 0), kSortGrid - 1);
    const unsigned morton = spread3((unsigned)cx) | (spread3((unsigned)cy) << 1) | (spread3((unsigned)cz) << 2);
    const unsigned oct = (D.x < 0.f ? 1u : 0u) | (D.y < 0.f ? 2u : 0u) | (D.z < 0.f ? 4u : 0u);
    return (oct << 9) | morton;
}

__global__ void __launch_bounds__(256) k_sort_count(DevRun r) {
    __shared__ unsigned h[kSortBins];
    for (int i = threadIdx.x; i < kSortBins; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const unsigned long long m = r.ctl->m, head = r.ctl->head;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long j = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; j < m; j += stride) {
        const float4 *q = reinterpret_cast<const float4 *>(r.ring + ((head + j) & (r.ring_cap - 1)));
        atomicAdd(&h[sort_key(r, __ldg(q), __ldg(q + 1))], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSortBins; i += blockDim.x)
        if (h[i]) atomicAdd(&r.bin_count[i], h[i]);
}

// One block of 1024 threads, 4 bins each: exclusive scan into the cursors; clears the counts.
__global__ void __launch_bounds__(1024) k_sort_scan(DevRun r) {
    __shared__ unsigned warp_sum[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned c[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        c[k] = r.bin_count[4 * t + k];
        r.bin_count[4 * t + k] = 0;
        s += c[k];
    }
    unsigned incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        unsigned w = warp_sum[lane], wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(FULL, wi, o);
            if (lane >= o) wi += v;
        }
        warp_sum[lane] = wi - w;  // exclusive warp offsets
    }
    __syncthreads();
    unsigned run = warp_sum[warp] + incl - s;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        r.bin_cursor[4 * t + k] = run;
        run += c[k];
    }
}

__global__ void __launch_bounds__(256) k_sort_scatter(DevRun r) {
    const unsigned long long m = r.ctl->m, head = r.ctl->head;
    const unsigned long long m32 = (m + 31) & ~31ull;
    const int lane = threadIdx.x & 31;
    const unsigned long long warp0 = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long base = warp0; base < m32; base += stride) {
        const unsigned long long j = base + lane;
        const bool act = j < m;
        const unsigned amask = __ballot_sync(FULL, act);
        if (!act) continue;
        const ORayItem it = load_item(r.ring, (head + j) & (r.ring_cap - 1));
        const float4 *f = reinterpret_cast<const float4 *>(&it);
        const unsigned key = sort_key(r, f[0], f[1]);
        const unsigned peers = __match_any_sync(amask, key);
        const int leader = __ffs(peers) - 1;
        unsigned pos = 0;
        if (lane == leader) pos = atomicAdd(&r.bin_cursor[key], (unsigned)__popc(peers));
        pos = __shfl_sync(amask, pos, leader) + __popc(peers & ((1u << lane) - 1u));
        store_item(r.wave_buf, pos, it);
    }
}

// ------------------------------------------------------------------------------------------
// phases B and C, split into the BVH walk and the surface interaction
// ------------------------------------------------------------------------------------------
// The walk's result for wave slot j: the nearest triangle (-1: none), its distance, and the polygon and
// coplanar group the shading pass needs (read from the triangle record, which the walk has just tested).
__device__ __forceinline__ void write_hit(const DevRun &r, const DevScene &S, unsigned j, int tri, float t) {
    int poly = -1, plane = -1;
    if (tri >= 0) {
        plane = __ldg(reinterpret_cast<const int *>(S.tri + 3 * tri) + 3);
        poly = __ldg(reinterpret_cast<const int *>(S.tri + 3 * tri + 1) + 3);
    }
    r.hits[j] = make_int4(tri, __float_as_int(t), poly, plane);
}

// The speculative walk tests the warp's leaves once at most kSpecSlack lanes are still looking for
// their first leaf (and some lane holds one) instead of waiting for the last: leaves tested sooner
// shrink the best hit sooner (fewer nodes and triangles per ray) and the warp idles less.  Measured
// on the arena (500k triangles) for 0 / 2 / 8 / 10 / 12 / 16 / 24 / 31: 1.65 / 1.73 / 1.78 / 1.80 /
// 1.79 / 1.76 / 1.58 / 1.23 G segments/s; on the 20k-triangle hall 0 / 8 / 12: 1.82 / 1.99 / 1.97.
// Lanes whose walk has ended write their hits and take new rays once kTraceRefill of them are there: one at a time
// each cost the warp the loads and three divisions of a ray start.  Device ms of the hall and the arena, refill at
// 1 / 4 / 6 / 8 / 12 / 16 / 20 with slack 10: 140.2 / 136.8 / 135.2 / 134.0 / 133.5 / 135.6 / 140.4 and 87.9 / 87.0 /
// 86.1 / 85.1 / 84.8 / 86.7 / 87.2; at 12 with slack 8 131.8 and 84.7, with 6 131.4 and 85.4.  With the stack of
// 4-byte entries: 12 and 10 127.0 and 79.9, 12 and 8 125.2 and 80.2, 10 and 8 125.3 and 79.6, 10 and 6 124.1 and 79.9.
constexpr int kSpecSlack = 6;
constexpr int kTraceRefill = 10;

// Persistent BVH walk with dynamic ray fetch: every loop iteration a lane descends inner nodes to
// its next leaf and tests it; a lane whose walk has ended writes its hit and takes the next wave
// item (one ticket atomic per warp; the speculative walk: once kTraceRefill lanes wait), so a warp does not idle on
// its slowest lane.
// Values the walk needs only when a ray starts or ends, once per leaf or once per warp iteration live
// in shared memory (each lane's wave index, the plane it leaves and its hit tolerance; each warp's node
// and triangle counts), not in registers: the walk's 40 registers already spill.  The counts are taken
// in kernel-timing runs only (r.count_work): they cost a ballot and a shared-memory update per pass.
template <int MINB, bool SPEC, bool QUANT>
__global__ void __launch_bounds__(256, MINB) k_trace(DevRun r) {
    __shared__ unsigned s_item[256];
    __shared__ int s_skip[256];
    __shared__ float s_teps[256];
    __shared__ unsigned long long s_cnt[8][2];
    WaveCtl *c = r.ctl;
    const unsigned long long m = c->m, head = c->head;
    const DevScene &S = r.S;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) s_cnt[wid][0] = s_cnt[wid][1] = 0;
    __syncwarp();
    TraceWork w;
    bool have = false, exhausted = false, done = false;
    unsigned j = 0;  // index in the wave (a wave holds at most half the ring: < 2^31 items)
    float3 o = make_float3(0.f, 0.f, 0.f), d = o;
    float ix = 0.f, iy = 0.f, iz = 0.f, ox = 0.f, oy = 0.f, oz = 0.f, best = FLT_MAX;
    int skip = -1, node = 0, sp = 0, bi = -1, leaf = 0;
    float teps = S.t_eps;
    // 4-byte entries: a box beyond the best hit is then entered once more and rejected by its children's test, yet the
    // stack is what the walk reads most, and its lines that miss L1: hall 131.8 -> 125.2 ms, arena 83.8 -> 80.2
    // against (id, distance) entries.  (The first 4 to 16 in shared memory 128 and 82, the top in a register 130.5 and
    // 81.8; 5 or 7 blocks an SM 135 and 133.)
    int stack[kBvhStack];
    for (;;) {
        const unsigned need = __ballot_sync(FULL, !have && !exhausted);
        if (need && (!SPEC || __popc(need) >= kTraceRefill || !__any_sync(FULL, have))) {
            if constexpr (SPEC) {
                if (done) write_hit(r, S, s_item[threadIdx.x], bi, best);
                done = false;
            }
            const int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(&c->trace_next, (unsigned long long)__popc(need));
            base = __shfl_sync(FULL, base, leader);
            if (!have && !exhausted) {
                const unsigned long long jj = base + __popc(need & ((1u << lane) - 1u));
                j = (unsigned)jj;
                if (jj < m) {
                    const float4 *q = reinterpret_cast<const float4 *>(wave_item(r, head, j));
                    const float4 P = __ldcs(q), D = __ldcs(q + 1), X = __ldcs(q + 3);
                    o = f3(P);
                    d = f3(D);
                    skip = __float_as_int(X.w);
                    const int room = (int)(__float_as_uint(X.z) >> 6);
                    const float dx = fabsf(d.x) < 1e-20f ? copysignf(1e-20f, d.x) : d.x;
                    const float dy = fabsf(d.y) < 1e-20f ? copysignf(1e-20f, d.y) : d.y;
                    const float dz = fabsf(d.z) < 1e-20f ? copysignf(1e-20f, d.z) : d.z;
                    ix = 1.0f / dx; iy = 1.0f / dy; iz = 1.0f / dz;
                    if constexpr (!QUANT) { ox = o.x * ix; oy = o.y * iy; oz = o.z * iz; }
                    node = r.n_rooms > 1 ? __ldg(&r.rooms[room].bvh_root) : 0;
                    teps = r.n_rooms > 1 ? __ldg(&r.rooms[room].t_eps) : S.t_eps;
                    if constexpr (SPEC) {
                        s_item[threadIdx.x] = j;
                        s_skip[threadIdx.x] = skip;
                        s_teps[threadIdx.x] = teps;
                    }
                    sp = 0; best = FLT_MAX; bi = -1;
                    have = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (!__any_sync(FULL, have)) break;  // every lane is exhausted
        if constexpr (SPEC) {
            // Speculative walk: a lane that has found a leaf keeps descending inner nodes while any
            // lane of the warp is still looking for its first leaf; then the warp tests its leaves
            // together.  node: >= 0 inner node, < 0 leaf, kEmptyChild nothing left; leaf: 0 none.
            if (have && node < 0 && node != kEmptyChild && leaf == 0) {
                leaf = node;
                node = stack_pop(stack, sp, best);
            }
            for (;;) {
                // stop when no lane is still looking for its first leaf, or when at most kSpecSlack are
                // and some lane holds a leaf to test (every pass of this loop advances the lanes still
                // looking, so it ends)
                const int looking = __popc(__ballot_sync(FULL, have && node >= 0 && leaf == 0));
                if (looking == 0 || (looking <= kSpecSlack && __any_sync(FULL, have && leaf != 0))) break;
                if (r.count_work) {
                    const unsigned stepping = __ballot_sync(FULL, have && node >= 0);
                    if (lane == 0) s_cnt[wid][0] += (unsigned)__popc(stepping);
                }
                if (have && node >= 0) {
                    int next;
                    node = (QUANT ? bvh4q_step(S.bvhq, node, ix, iy, iz, o.x, o.y, o.z, best, stack, sp, next)
                                  : bvh4_step(S.bvh, node, ix, iy, iz, ox, oy, oz, best, stack, sp, next))
                               ? next
                               : kEmptyChild;
                    if (node < 0 && node != kEmptyChild && leaf == 0) {
                        leaf = node;
                        node = kEmptyChild;
                    }
                    // one loop for the lanes that met no child and those that just found their leaf: the stack is
                    // two thirds of the walk's L1 requests (hall 140.5 -> 137.7 ms, arena 88.4 -> 86.9 against a
                    // loop for each; the top entry in registers 138.8 and 87.8)
                    while (node == kEmptyChild && sp > 0) {
                        const int e = stack[--sp];
                        if (e < 0 && leaf == 0) leaf = e;
                        else node = e;
                    }
                }
            }
            const bool testing = have && leaf != 0;
            if (r.count_work) {
                const unsigned ntri = __reduce_add_sync(FULL, testing ? (unsigned)(((~leaf) & 15) + 1) : 0u);
                if (lane == 0) s_cnt[wid][1] += ntri;
            }
            if (testing) {
                const int code = ~leaf;
                const int f0 = code >> 4, cnt = (code & 15) + 1;
                const int sk = s_skip[threadIdx.x];
                const float te = s_teps[threadIdx.x];
                for (int k = 0; k < cnt; ++k) test_tri(S, te, f0 + k, o, d, sk, best, bi, w);
                leaf = 0;
            }
            if (have && node == kEmptyChild) {
                done = true;
                have = false;
            }
        } else {
            if (!have) continue;
            while (node >= 0) {
                ++w.nodes;
                int next;
                node = (QUANT ? bvh4q_step(S.bvhq, node, ix, iy, iz, o.x, o.y, o.z, best, stack, sp, next)
                              : bvh4_step(S.bvh, node, ix, iy, iz, ox, oy, oz, best, stack, sp, next))
                           ? next
                           : stack_pop(stack, sp, best);
            }
            const bool fin = node == kEmptyChild;
            if (!fin) {
                const int code = ~node;
                const int f0 = code >> 4, cnt = (code & 15) + 1;
                w.tris += (unsigned)cnt;
                for (int k = 0; k < cnt; ++k) test_tri(S, teps, f0 + k, o, d, skip, best, bi, w);
                node = stack_pop(stack, sp, best);
            }
            if (node == kEmptyChild) {
                write_hit(r, S, j, bi, best);
                have = false;
            }
        }
    }
    if constexpr (SPEC) {
        if (done) write_hit(r, S, s_item[threadIdx.x], bi, best);
    }
    // one atomic per warp for each counter
    unsigned long long a = w.retests, b = w.nodes, c2 = w.tris;
    if constexpr (SPEC) {
        __syncwarp();
        b = lane == 0 ? s_cnt[wid][0] : 0;
        c2 = lane == 0 ? s_cnt[wid][1] : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(FULL, a, o);
        b += __shfl_down_sync(FULL, b, o);
        c2 += __shfl_down_sync(FULL, c2, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (a) atomicAdd(&r.cnt->retests, a);
        if (b) atomicAdd(&r.cnt->bvh_nodes, b);
        if (c2) atomicAdd(&r.cnt->tri_tests, c2);
    }
}

// The part of a split child that differs from its parent.
struct Child {
    float I;
    float3 d;
    unsigned long long sid;
    int mask;
};
__device__ __forceinline__ Ray child_ray(const Ray &R, const Child &C) {
    Ray c = R;
    c.I = C.I; c.d = C.d; c.sid = C.sid; c.mask = C.mask;
    c.nb = 0;
    c.phase = 0;
    return c;
}

// One surface interaction at hit h (triangle, t bits, polygon, coplanar group): the ray moves to the surface, is
// absorbed and scattered.  Returns whether it goes on; split: C is its split child (at the same place).
__device__ __forceinline__ bool surface(const DevRun &r, const DevScene &S, const RoomParams &P, int4 h, Ray &R,
                                        bool &split, Child &C, LocalCounters &L) {
    const float t = __int_as_float(h.y);
    R.t_sum += (double)t * P.inv_c_d;
    R.p = R.p + R.d * t;
    R.plane = h.w;
    const int poly = h.z;
    const float3 n = f3(__ldg(S.pnormal + poly));
    const float cos_t = dot3(n, R.d);
    const float4 mt = __ldg(S.mat + poly * kBands + R.oct);  // (1-alpha, s_lo, s_mid, s_hi)
    R.I *= mt.x;
    const float4 U = draw(r.seed, R.prim, R.sid, 1u + R.nb);
    const uint32_t nb = R.nb++;
    const bool transmit = S.has_trans && !P.pure_specular && U.x < __ldg(S.trans + poly * kBands + R.oct);
    const float3 spec = R.d - n * (2.f * cos_t);
    const float3 nn = cos_t > 0.f ? n * -1.f : n;
    // Scatter_Late (phase B) and Scatter_VeryLate (phase C) end in the same two directions, so that the lanes of both
    // share one Lambert direction: shoebox, 100k primaries 762 -> 733 ms, arena 84.5 -> 83.8.  (The time comparison
    // and the conversion of t on the integer pipe: 730 and 83.8.)
    const bool late = R.phase == 0;
    const bool diffuse = !P.pure_specular && (late ? !(U.y > mt.w) : U.y < mt.z);
    if (late && diffuse && U.y > mt.y) {
        split = true;
        C.I = R.I * (1.f - mt.z);
        R.I *= mt.z;
        C.mask = R.mask & ~1;
        C.d = transmit ? spec * -1.f : spec;
        C.sid = sid_late(R.sid, nb);
        ++L.v[C_OCT];
    }
    R.d = diffuse ? lambert(nn, U.z, U.w) : spec;
    if (transmit) R.d = R.d * -1.f;
    R.mask = diffuse ? R.mask | 3 : R.mask & ~1;
    // phase-B loop test (TaskAll:473): failing it enters End_Trace, which always traces at least one more segment;
    // phase C: TaskAll:534
    const bool on = R.t_sum < P.cotime && R.I > (late ? kTP2 : kTP3);
    if (late && !on) { R.phase = 1; ++L.v[C_END]; }
    bool alive = late || on;
    if (alive && (long long)R.nb >= r.max_seg) { ++L.v[C_CAP]; alive = false; }
    return alive;
}

// FUSED: walk the ray here instead of reading k_trace's hit (small scenes, whose walk is a few
// cached nodes: the separate trace pass would only re-read the ray and round-trip its hit via HBM).
// The shading pass alone takes receivers four at a time through a cheap test, in four 256-thread blocks per SM (64
// registers): on the 64-receiver arena -28 % and -6 % shading time against one at a time in three blocks.  Beside the
// other loops' walks that holds from the fewest receivers on (hall, 10k primaries with 2 / 8 / 16 of them 66.1 / 67.0 /
// 68.1 ms against 66.4 / 68.1 / 69.9; 20k primaries 121.0 against 124.4).  The fused walk: two blocks (128 registers),
// one at a time.
template <bool FUSED>
__global__ void __launch_bounds__(256, FUSED ? 2 : 4) k_shade(DevRun r) {
    extern __shared__ float4 s_rec_buf[];
    const int *s_rid;
    const float4 *s_rec = stage_receivers(r, s_rec_buf, s_rid);
    LocalCounters L;
    const DevScene &S = r.S;
    WaveCtl *c = r.ctl;
    const unsigned long long m = c->m, head = c->head;
    const unsigned long long m32 = (m + 31) & ~31ull;
    const bool count_room = r.n_rooms > 1 && c->pilot_count > 0;
    const int lane = threadIdx.x & 31;
    const unsigned long long warp0 = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long base = warp0; base < m32; base += stride) {
        const unsigned long long j = base + lane;
        int nout = 0;
        Ray R, C;
        if (j < m) {
            R = to_ray(load_item(wave_item(r, head, j), 0));
            int4 h;  // (triangle, t bits, polygon, coplanar group)
            if constexpr (FUSED) {
                float tt;
                int tri;
                TraceWork tw;
                const int root = r.n_rooms > 1 ? __ldg(&r.rooms[R.room].bvh_root) : 0;
                const float teps = r.n_rooms > 1 ? __ldg(&r.rooms[R.room].t_eps) : S.t_eps;
                h = make_int4(-1, 0, -1, -1);
                if (trace_ray<int>(S, root, teps, R.p, R.d, R.plane, tt, tri, tw)) {
                    const float4 A = __ldg(S.tri + 3 * tri), B = __ldg(S.tri + 3 * tri + 1);
                    h = make_int4(tri, __float_as_int(tt), __float_as_int(B.w), __float_as_int(A.w));
                }
                L.v[C_RET] += tw.retests;
                r.hits[j] = h;  // for the map's kernel
            } else {
                h = r.hits[j];
            }
            const bool hit = h.x >= 0;
            const float t = __int_as_float(h.y);
            ++L.v[R.phase == 0 ? C_SEGB : C_SEGC];
            const RoomParams &P = r.rooms[R.room];
            L.v[C_DET] += detect_octave<!FUSED>(r, P, s_rec, s_rid, R.p, R.d, hit ? t : 1e6f, R.t_sum, R.I * R.scale, R.oct,
                                        R.mask, R.prim);
            if (!hit) {
                // lost: no End_Trace after a miss in phase B (TaskAll:437-443), loop exit in phase C (500-505)
                L.lost += (double)(R.I * R.scale);
            } else {
                Child ch;
                bool split = false;
                bool alive = surface(r, S, P, h, R, split, ch, L);
                if (split) C = child_ray(R, ch);
                if (!alive && split) { R = C; split = false; alive = true; }
                nout = (alive ? 1 : 0) + (split ? 1 : 0);
            }
        }
        if (count_room) {  // live count of each ray's room (pilots of a batch)
            const int room = j < m ? (int)R.room : -1;
            const unsigned peers = __match_any_sync(FULL, room);
            const int d = __reduce_add_sync(peers, nout - 1);
            if (room >= 0 && d != 0 && lane == __ffs(peers) - 1) atomicAdd(r.room_live + room, (unsigned)d);
        }
        const unsigned long long slot = warp_append(&c->tail, nout);
        if (nout >= 1) ring_store(r, slot, to_item(R));
        if (nout == 2) ring_store(r, slot + 1, to_item(C));
    }
    flush_counters(r, L);
}

// The map's detections of the wave's octave rays (Map_Receiver.CheckRay, Pach_Map_Receiver.cs:1810-1826): energy
// I 10^(-0.1 m t) / (pi r^2), t = arrival time after the receiver's direct arrival (s).
// Inside the shading kernel each lane walked its segment's cells and their receivers to the end: 8.2 of 32 lanes
// active.  Here a warp takes 32 segments at a time, keeps those that walk the grid, and a lane whose walk is over
// takes the next of them; each step moves every lane by one cell or two receivers, and detections wait in a queue
// until 32 are there.  Bound: latency of the chain cell - entry - receiver (42 % of the issue slots, 20 lanes active;
// one receiver a step 162 us where two take 131 on a wave of 1.7M segments; four blocks an SM no faster), so it runs
// beside the shading kernel, which reads the same wave: 20k-triangle hall, 608 receivers, 2500 primaries 42.2 ->
// 38.7 ms, beside it 36.9.  Any number of idle lanes from 4 to 20 may wait for the next take: the same time.
struct MapHit {
    double t_sum;
    float t, I;       // chord midpoint, absolute energy
    float dx, dy, dz;
    unsigned at;      // receiver << 3 | band
};
constexpr int kMapQueue = 64;
constexpr int kMapHits = 96;   // 31 waiting and two of every lane
constexpr int kMapRefill = 12;

__global__ void __launch_bounds__(256, 3) k_map(DevRun r) {
    __shared__ unsigned s_job[8][kMapQueue];
    __shared__ MapHit s_hit[8][kMapHits];
    WaveCtl *c = r.ctl;
    const MapDev &M = r.map;
    const unsigned long long m = c->m, head = c->head;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    unsigned *jobs = s_job[threadIdx.x >> 5];
    MapHit *queue = s_hit[threadIdx.x >> 5];
    int njobs = 0, queued = 0;
    unsigned long long found = 0;
    bool more = true, walking = false;
    MapCursor K;
    K.e = K.e1 = 0;
    float3 o = make_float3(0.f, 0.f, 0.f), d = o;
    float tseg = 0.f;
    double t_sum = 0;
    float I = 0.f;
    unsigned oct = 0;
    auto segment = [&](unsigned i, float3 &so, float3 &sd, float &st) {
        const float4 *q = reinterpret_cast<const float4 *>(wave_item(r, head, i));
        so = f3(q[0]);
        sd = f3(q[1]);
        const int4 h = r.hits[i];
        st = h.x >= 0 ? __int_as_float(h.y) : 1e6f;
    };
    auto add = [&](int i) {
        const MapHit x = queue[i];
        const int k = (int)(x.at >> 3), oct = (int)(x.at & 7u);
        const double time = x.t_sum + (double)(x.t * r.rooms[0].inv_c) - __ldg(M.direct + k);
        map_add(M, k, oct, time, x.I * exp2f(M.atten_k[oct] * (float)time) * M.size_mod,
                make_float3(x.dx, x.dy, x.dz));
    };
    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !walking);
        if (__popc(idle) >= kMapRefill) {
            const int want = __popc(idle);
            while (more && njobs < want) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(&c->map_next, 32ull);
                base = __shfl_sync(FULL, base, 0);
                if (base >= m) { more = false; break; }
                bool cross = false;
                const unsigned long long i = base + lane;
                if (i < m) {
                    float3 so, sd;
                    float st;
                    segment((unsigned)i, so, sd, st);
                    MapCursor X;
                    cross = X.start(M, so, sd, st);
                }
                const unsigned who = __ballot_sync(FULL, cross);
                if (cross) jobs[njobs + __popc(who & below)] = (unsigned)i;
                njobs += __popc(who);
            }
            __syncwarp();
            if (njobs == 0 && idle == FULL) break;
            const int rank = __popc(idle & below);
            if (!walking && rank < njobs) {
                const unsigned j = jobs[njobs - 1 - rank];
                segment(j, o, d, tseg);
                const Ray R = to_ray(load_item(wave_item(r, head, j), 0));
                t_sum = R.t_sum;
                I = R.I * R.scale;
                oct = (unsigned)R.oct;
                walking = K.start(M, o, d, tseg);
                if (walking) K.enter(M);
            }
            njobs = max(njobs - want, 0);
            __syncwarp();
        }
        if (walking && K.e == K.e1) {
            walking = K.advance(M);
            if (walking) K.enter(M);
        }
        bool hit[2] = {false, false};
        float t[2] = {0.f, 0.f};
        int k[2] = {0, 0};
        if (walking && K.e < K.e1) {
            float half;
            const bool two = K.e + 1 < K.e1;
            const uint2 en = __ldg(M.entry + K.e), en1 = __ldg(M.entry + K.e + two);
            K.e += 1 + two;
            k[0] = (int)en.x;
            k[1] = (int)en1.x;
            const float4 c0 = __ldg(M.rec + k[0]), c1 = __ldg(M.rec + k[1]);
            hit[0] = !(en.y & K.seen) && sphere_hit(c0, o, d, tseg, t[0], half);
            hit[1] = two && !(en1.y & K.seen) && sphere_hit(c1, o, d, tseg, t[1], half);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const unsigned who = __ballot_sync(FULL, hit[q]);
            if (hit[q]) {
                MapHit x;
                x.t_sum = t_sum;
                x.t = t[q];
                x.I = I;
                x.dx = d.x; x.dy = d.y; x.dz = d.z;
                x.at = (unsigned)k[q] << 3 | oct;
                queue[queued + __popc(who & below)] = x;
            }
            queued += __popc(who);
            found += __popc(who);
        }
        while (queued >= 32) {
            __syncwarp();
            queued -= 32;
            add(queued + lane);
            __syncwarp();
        }
    }
    __syncwarp();
    if (lane < queued) add(lane);
    if (lane == 0 && found) atomicAdd(&r.cnt->detections, found);
}

// Small scenes: walk and shade, each lane keeping its ray in registers over up to ctl->bounces interactions, then
// taking the next wave item (a lane whose ray ends takes one at once).  Split children go to the ring as they
// arise; rays that have used up their interactions go back to it.
// Bound: issue (61 % of slots, 19.6 of 32 lanes active: interactions differ) at three blocks an SM; two or four
// blocks 848 and 834 ms where three take 753.  One interaction a
// launch read and wrote every ray (128 bytes) and appended it each time, and a chain of 200 interactions was 200
// waves: a 1003-primary shoebox took 228 waves and 19.1 ms, now 30 and 9.6 ms (in three loops 8.7); 100k primaries 1180
// ms, then 753, now 733.
//
// Detections wait in a queue of the warp until 32 are there, so that a lane's detection (FP64 time and bin, six
// atomics) does not hold the other 31: in a 3-receiver shoebox 3 % of the segments, two of three iterations.
struct Detection {
    double t_sum;
    float t, half, I;      // chord midpoint and half length, absolute energy
    float dx, dy, dz;
    unsigned at;           // receiver slot << 5 | band << 2 | mask
    uint32_t prim;
    unsigned room, pad;
};
constexpr int kQueue = 64;

template <bool PLANES>
__global__ void __launch_bounds__(256, 3) k_bounce(DevRun r) {
    extern __shared__ float4 s_rec_buf[];
    __shared__ Detection s_det[8][kQueue];
    __shared__ float4 s_plane[2 * kMaxPlanes];
    const int *s_rid;
    const float4 *s_rec = stage_receivers(r, s_rec_buf, s_rid);
    LocalCounters L;
    const DevScene &S = r.S;
    WaveCtl *c = r.ctl;
    const unsigned long long m = c->m, head = c->head;
    const int bounces = c->bounces, lane = threadIdx.x & 31;
    const bool count_room = r.n_rooms > 1 && c->pilot_count > 0;
    if constexpr (PLANES) {
        if (r.n_rooms == 1) {
            const int np = 2 * r.rooms[0].n_planes;
            if ((int)threadIdx.x < np) s_plane[threadIdx.x] = S.plane[2 * r.rooms[0].plane_begin + threadIdx.x];
            __syncthreads();
        }
    }
    Detection *queue = s_det[threadIdx.x >> 5];
    int queued = 0;
    auto detect = [&](int i) {
        const Detection e = queue[i];
        const int s = (int)(e.at >> 5);
        detect_octave_one(r, r.rooms[e.room], s_rid, s, s_rec[s], make_float3(e.dx, e.dy, e.dz), e.t, e.half, e.t_sum, e.I,
                          (int)(e.at >> 2) & 7, (int)e.at & 3, e.prim);
    };
    Ray R;
    bool have = false, exhausted = false;
    int left = 0, splitting = 0;  // phase-B rays put into the ring less those taken out
    for (;;) {
        const unsigned need = __ballot_sync(FULL, !have && !exhausted);
        if (need) {
            const int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(&c->trace_next, (unsigned long long)__popc(need));
            base = __shfl_sync(FULL, base, leader);
            if (!have && !exhausted) {
                const unsigned long long j = base + __popc(need & ((1u << lane) - 1u));
                if (j < m) {
                    R = to_ray(load_item(r.ring, (head + j) & (r.ring_cap - 1)));
                    left = bounces;
                    splitting -= R.phase == 0;
                    have = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (!__any_sync(FULL, have)) break;
        float t = 0.f;
        int tri = -1, s0 = 0, s1 = 0;
        bool hit = false;
        if (have) {
            const RoomParams &P = r.rooms[R.room];
            TraceWork tw;
            const int root = r.n_rooms > 1 ? P.bvh_root : 0;
            const float teps = r.n_rooms > 1 ? P.t_eps : S.t_eps;
            if constexpr (PLANES)
                hit = plane_walk(S, r.n_rooms == 1 ? s_plane : S.plane + 2 * P.plane_begin, P.n_planes, P.plane_eps, root,
                                 teps, R.p, R.d, R.plane, t, tri, tw);
            else
                hit = trace_ray<int>(S, root, teps, R.p, R.d, R.plane, t, tri, tw);
            L.v[C_RET] += tw.retests;
            ++L.v[R.phase == 0 ? C_SEGB : C_SEGC];
            s0 = P.rec_begin;
            s1 = s0 + P.R;
        }
        // Spherical_Receiver.CheckRay over the room's receivers
        for (;; ++s0) {
            if (!__any_sync(FULL, s0 < s1)) break;
            float tc = 0.f, half = 0.f;
            const bool found = s0 < s1 && sphere_hit(s_rec[s0], R.p, R.d, hit ? t : 1e6f, tc, half);
            const unsigned who = __ballot_sync(FULL, found);
            if (!who) continue;
            if (found) {
                ++L.v[C_DET];
                Detection e;
                e.t_sum = R.t_sum;
                e.t = tc; e.half = half; e.I = R.I * R.scale;
                e.dx = R.d.x; e.dy = R.d.y; e.dz = R.d.z;
                e.at = (unsigned)s0 << 5 | (unsigned)R.oct << 2 | (unsigned)R.mask;
                e.prim = R.prim;
                e.room = (unsigned)R.room;
                e.pad = 0;
                queue[queued + __popc(who & ((1u << lane) - 1u))] = e;
            }
            queued += __popc(who);
            if (queued >= 32) {
                __syncwarp();
                queued -= 32;
                detect(queued + lane);
                __syncwarp();
            }
        }
        if (have) {
            const RoomParams &P = r.rooms[R.room];
            bool alive = false, split = false;
            Child ch;
            if (!hit) {
                // lost: no End_Trace after a miss in phase B (TaskAll:437-443), loop exit in phase C (500-505)
                L.lost += (double)(R.I * R.scale);
            } else {
                const float4 A = __ldg(S.tri + 3 * tri), B = __ldg(S.tri + 3 * tri + 1);
                alive = surface(r, S, P, make_int4(tri, __float_as_int(t), __float_as_int(B.w), __float_as_int(A.w)), R,
                                split, ch, L);
            }
            if (split) {
                if (alive) {
                    // one atomic for the lanes that are here together
                    const unsigned here = __activemask();
                    const int first = __ffs(here) - 1;
                    unsigned long long slot = 0;
                    if (lane == first) slot = atomicAdd(&c->tail, (unsigned long long)__popc(here));
                    slot = __shfl_sync(here, slot, first) + __popc(here & ((1u << lane) - 1u));
                    ring_store(r, slot, to_item(child_ray(R, ch)));
                    ++splitting;
                    if (count_room) atomicAdd(r.room_live + R.room, 1u);
                } else {
                    R = child_ray(R, ch);  // the child takes the parent's place
                    alive = true;
                }
            }
            if (!alive) {
                have = false;
                if (count_room) atomicSub(r.room_live + R.room, 1u);
            }
            --left;
        }
        const unsigned back = __ballot_sync(FULL, have && left <= 0);
        if (back) {
            const int first = __ffs(back) - 1;
            unsigned long long slot = 0;
            if (lane == first) slot = atomicAdd(&c->tail, (unsigned long long)__popc(back));
            slot = __shfl_sync(FULL, slot, first) + __popc(back & ((1u << lane) - 1u));
            if (have && left <= 0) {
                ring_store(r, slot, to_item(R));
                splitting += R.phase == 0;
                have = false;
            }
        }
    }
    __syncwarp();
    if (lane < queued) detect(lane);
    splitting = (int)__reduce_add_sync(FULL, (unsigned)splitting);
    if (lane == 0 && splitting)
        atomicAdd(reinterpret_cast<unsigned long long *>(&c->live_b), (unsigned long long)(long long)splitting);
    flush_counters(r, L);
}

// ------------------------------------------------------------------------------------------
// pure-specular paths and emission directions (parity probes)
// ------------------------------------------------------------------------------------------
__global__ void k_paths(DevScene S, int n, const double *o, const double *dd, int maxb, int *poly, double *tout,
                        double *pts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float3 p = make_float3((float)o[3 * i], (float)o[3 * i + 1], (float)o[3 * i + 2]);
    float3 d = unit3(make_float3((float)dd[3 * i], (float)dd[3 * i + 1], (float)dd[3 * i + 2]));
    int plane = -1;
    TraceWork rt;
    for (int b = 0; b < maxb; ++b) {
        const size_t k = (size_t)i * maxb + b;
        poly[k] = -1; tout[k] = 0; pts[3 * k] = pts[3 * k + 1] = pts[3 * k + 2] = 0;
    }
    for (int b = 0; b < maxb; ++b) {
        float t;
        int tri;
        if (!trace_ray(S, 0, S.t_eps, p, d, plane, t, tri, rt)) break;
        const size_t k = (size_t)i * maxb + b;
        const float4 A = __ldg(S.tri + 3 * tri), B = __ldg(S.tri + 3 * tri + 1);
        const int pl = __float_as_int(B.w);
        p = p + d * t;
        poly[k] = pl;
        tout[k] = t;
        pts[3 * k] = p.x; pts[3 * k + 1] = p.y; pts[3 * k + 2] = p.z;
        const float3 nrm = f3(__ldg(S.pnormal + pl));
        d = d - nrm * (2.f * dot3(d, nrm));
        plane = __float_as_int(A.w);
    }
}

__global__ void k_emit(DevRun r, long long p0, int n, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long prim = p0 + i;
    const RoomParams &P = r.rooms[0];
    const int s = P.src_begin + (int)((prim + 1) % P.nsrc);
    const float3 d = emit_dir(r, P.nsrc, prim, (int)r.src[s].w);
    out[3 * i] = d.x; out[3 * i + 1] = d.y; out[3 * i + 2] = d.z;
}

// Direct-sound visibility (Direct_Sound.Check_Validity, Classes_Direct.cs:654-685): from each
// source towards each receiver, shoot; a hit before the receiver distance through a transmissive
// polygon multiplies the band transmission and the ray continues from the hit point, comparing its
// next hit with the full source-receiver distance again (as coded); any other hit decides.
__global__ void k_direct(DevScene S, const double *src, int nsrc, const double *rec, int nrec, int max_cross,
                         int *valid, double *transmod) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nsrc * nrec) return;
    const int k = p / nsrc, s = p % nsrc;
    const double dx = rec[3 * k] - src[3 * s], dy = rec[3 * k + 1] - src[3 * s + 1], dz = rec[3 * k + 2] - src[3 * s + 2];
    const double dist = sqrt(dx * dx + dy * dy + dz * dz);
    float3 o = make_float3((float)src[3 * s], (float)src[3 * s + 1], (float)src[3 * s + 2]);
    const float3 d = make_float3((float)(dx / dist), (float)(dy / dist), (float)(dz / dist));
    double tm[kBands];
#pragma unroll
    for (int b = 0; b < kBands; ++b) tm[b] = 1.0;
    int plane = -1, ok = 1;
    for (int c = 0; c < max_cross; ++c) {
        float t;
        int tri;
        TraceWork w;
        if (!trace_ray(S, 0, S.t_eps, o, d, plane, t, tri, w)) { ok = 1; break; }
        ok = (double)t >= dist ? 1 : 0;
        const float4 A = __ldg(S.tri + 3 * tri), B = __ldg(S.tri + 3 * tri + 1);
        const int poly = __float_as_int(B.w);
        bool transmissive = false;
        if (S.has_trans)
            for (int b = 0; b < kBands; ++b) transmissive = transmissive || __ldg(S.trans + poly * kBands + b) > 0.f;
        if (ok || !transmissive) break;
        for (int b = 0; b < kBands; ++b) tm[b] *= (double)__ldg(S.trans + poly * kBands + b);
        o = o + d * t;
        plane = __float_as_int(A.w);
    }
    valid[p] = ok;
#pragma unroll
    for (int b = 0; b < kBands; ++b) transmod[(size_t)p * kBands + b] = tm[b];
}

__global__ void k_prop_sample(DevRun r, long long p0, int n, float *dirs, float *weights) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float w;
    const float3 d = proposal_dir(r, (uint32_t)(p0 + i), w);
    dirs[3 * i] = d.x; dirs[3 * i + 1] = d.y; dirs[3 * i + 2] = d.z;
    weights[i] = w;
}

// Histogram scaling on the way to the host: HBM-bound, n x 16 bytes (the 20 M doubles of the arena's
// histograms in 0.06 ms; the host loop it replaces took 20 ms on one core).
__global__ void __launch_bounds__(256) k_scale(double *dst, const double *src, size_t n, double f, const double *rows,
                                               size_t first, size_t per_row) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        dst[i] = src[i] * (rows ? __ldg(rows + (first + i) / per_row) : f);
}

}  // namespace

// ------------------------------------------------------------------------------------------
// host wrappers
// ------------------------------------------------------------------------------------------
static size_t rec_smem(const DevRun &r) { return (size_t)receiver_smem_bytes(r.R); }

cudaError_t launch_feed(const DevRun &r, cudaStream_t s) {
    k_feed<<<1, 32, 0, s>>>(r);
    return cudaGetLastError();
}

cudaError_t launch_broadband(const DevRun &r, int blocks, int threads, cudaStream_t s, bool map, bool small) {
    if (map) {
        if (small) k_broadband<true, true><<<blocks, threads, rec_smem(r), s>>>(r);
        else k_broadband<true, false><<<blocks, threads, rec_smem(r), s>>>(r);
    } else {
        if (small) k_broadband<false, true><<<blocks, threads, rec_smem(r), s>>>(r);
        else k_broadband<false, false><<<blocks, threads, rec_smem(r), s>>>(r);
    }
    return cudaGetLastError();
}

cudaError_t launch_cond(const DevRun &r, cudaGraphConditionalHandle h, cudaStream_t s) {
    k_cond<<<1, 32, 0, s>>>(r, h);
    return cudaGetLastError();
}

cudaError_t launch_sort(const DevRun &r, int blocks, cudaStream_t s) {
    k_sort_count<<<blocks, 256, 0, s>>>(r);
    k_sort_scan<<<1, 1024, 0, s>>>(r);
    k_sort_scatter<<<blocks, 256, 0, s>>>(r);
    return cudaGetLastError();
}

// variant = blocks per SM (3..6) + 16 x speculative + 32 x quantised nodes
#define PACH_TRACE_VARIANTS(X)                                                                         \
    X(3, false, false) X(4, false, false) X(5, false, false) X(6, false, false) X(4, true, false)    \
    X(6, true, false) X(4, false, true) X(6, false, true) X(4, true, true) X(6, true, true)

cudaError_t launch_trace(const DevRun &r, int variant, int blocks, int threads, cudaStream_t s) {
    switch (variant) {
#define PACH_LAUNCH(M, SP, Q) \
    case M + (SP ? 16 : 0) + (Q ? 32 : 0): k_trace<M, SP, Q><<<blocks, threads, 0, s>>>(r); break;
        PACH_TRACE_VARIANTS(PACH_LAUNCH)
#undef PACH_LAUNCH
        default: k_trace<4, false, false><<<blocks, threads, 0, s>>>(r); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_shade(const DevRun &r, int blocks, int threads, cudaStream_t s, bool fused) {
    if (fused) k_shade<true><<<blocks, threads, rec_smem(r), s>>>(r);
    else k_shade<false><<<blocks, threads, rec_smem(r), s>>>(r);
    return cudaGetLastError();
}

cudaError_t launch_map(const DevRun &r, int blocks, cudaStream_t s) {
    k_map<<<blocks, 256, 0, s>>>(r);
    return cudaGetLastError();
}

cudaError_t launch_bounce(const DevRun &r, int blocks, int threads, cudaStream_t s, bool planes) {
    if (planes) k_bounce<true><<<blocks, threads, rec_smem(r), s>>>(r);
    else k_bounce<false><<<blocks, threads, rec_smem(r), s>>>(r);
    return cudaGetLastError();
}

cudaError_t bounce_occupancy(int threads, int smem, int *blocks_per_sm, bool planes) {
    return planes ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_bounce<true>, threads, smem)
                  : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_bounce<false>, threads, smem);
}

cudaError_t wave_kernel_occupancy(int variant, int threads, int smem_shade, int *bpsm_trace, int *bpsm_shade,
                                  bool fused) {
    cudaError_t e;
    switch (variant) {
#define PACH_OCC(M, SP, Q)                                                                           \
    case M + (SP ? 16 : 0) + (Q ? 32 : 0):                                                           \
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(bpsm_trace, k_trace<M, SP, Q>, threads, 0); \
        break;
        PACH_TRACE_VARIANTS(PACH_OCC)
#undef PACH_OCC
        default: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(bpsm_trace, k_trace<4, false, false>, threads, 0); break;
    }
    if (e != cudaSuccess) return e;
    return fused ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(bpsm_shade, k_shade<true>, threads, smem_shade)
                 : cudaOccupancyMaxActiveBlocksPerMultiprocessor(bpsm_shade, k_shade<false>, threads, smem_shade);
}

cudaError_t launch_scale(double *dst, const double *src, size_t n, double f, const double *rows, size_t first,
                         size_t per_row, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 8192);
    k_scale<<<blocks, 256, 0, s>>>(dst, src, n, f, rows, first, per_row);
    return cudaGetLastError();
}

cudaError_t launch_paths(const DevScene &S, int n, const double *o, const double *d, int max_bounces, int *poly,
                         double *t, double *pts, cudaStream_t s) {
    k_paths<<<(n + 127) / 128, 128, 0, s>>>(S, n, o, d, max_bounces, poly, t, pts);
    return cudaGetLastError();
}

cudaError_t launch_emit(const DevRun &r, long long p0, int n, double *out, cudaStream_t s) {
    k_emit<<<(n + 127) / 128, 128, 0, s>>>(r, p0, n, out);
    return cudaGetLastError();
}

cudaError_t launch_direct(const DevScene &S, const double *src, int nsrc, const double *rec, int nrec, int max_cross,
                          int *valid, double *transmod, cudaStream_t s) {
    const int n = nsrc * nrec;
    k_direct<<<(n + 127) / 128, 128, 0, s>>>(S, src, nsrc, rec, nrec, max_cross, valid, transmod);
    return cudaGetLastError();
}

cudaError_t launch_prop_sample(const DevRun &r, long long p0, int n, float *dirs, float *weights, cudaStream_t s) {
    k_prop_sample<<<(n + 127) / 128, 128, 0, s>>>(r, p0, n, dirs, weights);
    return cudaGetLastError();
}

}  // namespace pach
