// FP32 wavefront path integrator for sm_100a.
//
// The reference runs radiance() (src/integrator.rs:53-135) once per sample on
// CPU threads over Morton-ordered tiles (src/render.rs:116-206).  Here a
// pixel's samples are cut into tasks (the reference's Task with its
// sample_start seeding); a pool of path slots pulls tasks and runs each
// task's samples one after another, so a slot's u64 PCG32 state continues
// the task's reference stream draw for draw.  One bounce of all live paths
// is one iteration of:
//
//   trace<closest> : closest hit of every active slot (BVH2 traversal, FP32)
//   shade          : miss/env, Russian roulette, emitter, NEE sample
//                    generation (env + area light, power-heuristic MIS),
//                    BSDF sample; samples with nothing pending complete here
//   trace<any>     : occlusion of the NEE shadow rays
//   regen          : samples whose shadow rays were pending complete: the
//                    f64 sums (+ Welford for adaptive sampling), then the
//                    next camera ray or the next task
//
// Slots are visited in slot order (an active byte per slot); shadow records
// and pending completions go through queues filled with warp-aggregated
// atomics.  The first iterations are launched from the host; a loop that goes on
// runs in one CUDA graph whose WHILE conditional node is re-armed on the device
// until no slot is active.  Small renders have no loop: k_paths runs their paths
// whole.
#include "fp32_device.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <type_traits>
#include <vector>

namespace tpt {
namespace wf {

// ---- kernels ------------------------------------------------------------------
// A task is the reference's Task restricted to one pixel (src/task.rs:11-27):
// samples [sample_start, sample_end) of that pixel, with the RNG seeded from
// seed_for(x, y, sample_start) ^ seed (src/render.rs:142).  Task t covers
// pixel t % n_pixels and sample chunk t / n_pixels; chunk 0 starts each
// pixel's reference stream.  With one chunk per pixel the schedule is the
// reference's own.
// Batch renders: a slot's task belongs to one job, whose scene view (root,
// camera, env map, lights), parameters and film overlay the batch-wide ones.
struct Film {
    double* acc;
    double* acc_w;
    double* acc_sq;
};
__device__ __forceinline__ void apply_job(const WfJob& J, WfScene& S, WfParams& P, Film& F, long long& base) {
    S.cam = J.cam;
    S.top_root = J.top_root;
    S.env_kind = J.env_kind; S.env_w = J.env_w; S.env_h = J.env_h; S.env_has_cdf = J.env_has_cdf;
    S.env_black = J.env_black;
    S.env_row_guide = S.env_col_guide = nullptr;  // (a batch's maps are searched whole)
    S.env_tex = J.env_tex; S.env_row = J.env_row; S.env_col = J.env_col;
    S.lights = J.lights; S.light_cdf = J.light_cdf; S.lights64 = J.lights64; S.n_lights = J.n_lights;
    P.width = J.width; P.height = J.height; P.spp = J.spp; P.max_bounces = J.max_bounces; P.rr_start = J.rr_start;
    P.seed = J.seed; P.n_pixels = J.n_pixels; P.task_spp = J.task_spp; P.n_chunks = J.n_chunks;
    P.row_begin = J.row_begin; P.row_step = J.row_step;
    P.px_map = nullptr; P.sample_base = 0; P.sample_end = J.spp;
    P.px_div = J.px_div; P.w_div = J.w_div;
    F.acc = J.acc; F.acc_w = J.acc_w; F.acc_sq = nullptr;
    base = J.task_begin;
}
// Job holding a batch-wide task id (tasks are numbered job after job).
__device__ __forceinline__ int find_job(const WfParams& P, long long task) {
    int lo = 0, hi = P.n_jobs;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (P.jobs[mid].task_begin <= task) lo = mid; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ Film film_of(const WfState& st) { return Film{st.acc, st.acc_w, st.acc_sq}; }

// The scene, parameters and film of a job (single renders: of the render).
struct View {
    WfScene S;
    WfParams P;
    Film F;
    long long task_begin;
};
template <bool BATCH>
__device__ __forceinline__ View view_of(const WfScene& S0, const WfParams& P0, const WfState& st, int job) {
    View v{S0, P0, film_of(st), 0};
    if constexpr (BATCH) apply_job(P0.jobs[job], v.S, v.P, v.F, v.task_begin);
    return v;
}

// Where task lt (its index within its job) sits: task-space pixel j = lt %
// n_pixels, sample chunk lt / n_pixels; the film pixel (through px_map in an
// adaptive round), its first sample and its length.
// Task ids are below 2^31 (the host lengthens tasks until they are).
struct TaskPos { int j, pixel, sample_start, len; };
__device__ __forceinline__ TaskPos task_pos(const WfParams& P, long long lt) {
    TaskPos t;
    const uint32_t u = (uint32_t)lt;
    const int chunk = (int)fdiv(P.px_div, u);
    t.j = (int)(u - (uint32_t)chunk * (uint32_t)P.n_pixels);
    t.pixel = P.px_map ? __ldg(P.px_map + t.j) : t.j;
    t.sample_start = P.sample_base + chunk * P.task_spp;
    const int end = P.sample_end > 0 ? P.sample_end : P.spp;
    t.len = min(P.task_spp, end - t.sample_start);
    return t;
}

// The pool's task cursor counts fetch ids from task_first.  Without camera
// culling a fetch id is the task itself.  With it (P.geo_map), the ids of
// the current chunk batch enumerate, chunk by chunk, the tasks of the n_geo
// pixels in geo_map, in film order: the task order of the batch with the
// culled pixels' tasks left out (k_sky_tasks renders those).  A multi-job
// render does the same per job, jobs one after another (WfJob::fetch_begin;
// geo_map then holds batch-wide pixel ids).
__device__ __forceinline__ long long fetch_end(const WfParams& P) {
    if (!P.geo_map) return P.n_tasks;
    if (P.jobs) return P.n_fetch;
    return P.task_first + (P.n_tasks - P.task_first) / P.n_pixels * P.n_geo;
}
// The last job whose begin (a job-ordered id space: fetch ids, sky tasks)
// is at most f; jobs with an empty stretch share the next job's begin.
template <class Begin>
__device__ __forceinline__ int job_at(const WfParams& P, long long f, Begin begin) {
    int lo = 0, hi = P.n_jobs;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (begin(P.jobs[mid]) <= f) lo = mid; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ long long task_of_fetch(const WfParams& P, long long f) {
    if (!P.geo_map) return f;
    if (P.jobs) {
        const WfJob& J = P.jobs[job_at(P, f, [](const WfJob& x) { return x.fetch_begin; })];
        const uint32_t v = (uint32_t)(f - J.fetch_begin);
        const uint32_t c = fdiv(J.geo_div, v);
        const int gp = __ldg(P.geo_map + J.geo_begin + (v - c * (uint32_t)J.n_geo));
        return J.task_begin + (long long)c * J.n_pixels + (gp - J.pixel_begin);
    }
    const uint32_t v = (uint32_t)(f - P.task_first);
    const uint32_t c = fdiv(P.geo_div, v);
    return P.task_first + (long long)c * P.n_pixels + __ldg(P.geo_map + (v - c * (uint32_t)P.n_geo));
}

template <bool BATCH>
__device__ __forceinline__ void start_task(const WfScene& S0, const WfParams& P0, const WfState& st, int slot,
                                           long long task) {
    WfScene S = S0;
    WfParams P = P0;
    Film F = film_of(st);
    long long base = 0;
    if constexpr (BATCH) {
        const int j = find_job(P0, task);
        st.job[slot] = j;
        apply_job(P0.jobs[j], S, P, F, base);
    }
    const TaskPos tp = task_pos(P, task - base);  // task within its job
    const int row = (int)fdiv(P.w_div, (uint32_t)tp.pixel);
    const int x = tp.pixel - row * P.width, y = P.row_begin + row * P.row_step;
    uint64_t rng = task_seed((uint32_t)x, (uint32_t)y, (uint32_t)tp.sample_start, P.seed);
    float3 o, d;
    float time;
    camera_ray(S.cam, x, y, 1.0f / (float)P.width, 1.0f / (float)P.height, rng, o, d, time);
    store_path(st, slot, make_int4(0, 0, 0, (int)task), rng);
    sts(&st.ray_o[slot], make_float4(o.x, o.y, o.z, ifloat(-1)));
    sts(&st.ray_d[slot], make_float4(d.x, d.y, d.z, ifloat(-1)));
    sts(&st.beta[slot], make_float4(1.0f, 1.0f, 1.0f, 0.0f));
    sts(&st.rad[slot], make_float4(0.0f, 0.0f, 0.0f, time));
}

// A task's f64 sums: radiance and count, squares (when wanted), and the
// Welford mean and m2 of one-task adaptive sampling.  They start at zero with
// the task's first sample and go to the slot's records while samples are
// left, so a one-sample task (most renders that do not fill the pool) never
// touches those.
struct Sums {
    double4 a, q;
    double2 w;
};
__device__ __forceinline__ Sums zero_sums() {
    return Sums{make_double4(0.0, 0.0, 0.0, 0.0), make_double4(0.0, 0.0, 0.0, 0.0), make_double2(0.0, 0.0)};
}
__device__ __forceinline__ Sums load_sums(const WfState& st, int slot, bool first) {
    Sums s = zero_sums();
    if (!first && !st.rsamp) {
        s.a = lds(&st.sacc[slot]);
        if (st.ssq) s.q = lds(&st.ssq[slot]);
        if (st.welford) s.w = st.welford[slot];
    }
    return s;
}
__device__ __forceinline__ void store_sums(const WfState& st, int slot, const Sums& s) {
    if (st.rsamp) return;
    sts(&st.sacc[slot], s.a);
    if (st.ssq) sts(&st.ssq[slot], s.q);
    if (st.welford) st.welford[slot] = s.w;
}
__device__ __forceinline__ void add_sample(Sums& s, float3 L, bool squares) {
    s.a.x += (double)L.x; s.a.y += (double)L.y; s.a.z += (double)L.z; s.a.w += 1.0;
    if (squares) {
        s.q.x += (double)L.x * (double)L.x; s.q.y += (double)L.y * (double)L.y; s.q.z += (double)L.z * (double)L.z;
    }
}

template <bool BATCH>
__global__ void k_init(WfScene S, WfParams P, WfState st) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const long long avail = fetch_end(P) - P.task_first;  // tasks of this chunk batch
    const int first = (int)(avail < (long long)P.n_slots ? avail : P.n_slots);
    if (i == 0) {
        st.ctr->n_ext[0] = first;
        st.ctr->next_task = P.task_first + first;
    }
    if (i >= P.n_slots) return;
    st.act[i] = i < first ? 1 : 0;
    if (i < first) {
        st.q_ext[0][i] = i;
        start_task<BATCH>(S, P, st, i, task_of_fetch(P, P.task_first + i));
    }
}

// Adds a thread's trace counters to the render totals (one atomic per warp).
template <bool COUNT>
__device__ __forceinline__ void flush_counts(WfCounters* c, int stage, const TraceCount& t) {
    if (!COUNT) return;
    unsigned long long v[8] = {t.nodes, t.tris, t.spheres, t.inst, t.node_steps, t.leaves, t.leaf_steps, t.fast_steps};
    for (int k = 0; k < 8; ++k)
        for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
    if (lane_id() == 0) {
        atomicAdd(&c->cnt_nodes[stage], v[0]);
        atomicAdd(&c->cnt_tris[stage], v[1]);
        atomicAdd(&c->cnt_spheres[stage], v[2]);
        atomicAdd(&c->cnt_inst[stage], v[3]);
        atomicAdd(&c->cnt_node_steps[stage], v[4]);
        atomicAdd(&c->cnt_leaves[stage], v[5]);
        atomicAdd(&c->cnt_leaf_steps[stage], v[6]);
        atomicAdd(&c->cnt_fast_steps, v[7]);
    }
}

// Persistent trace kernel over the extension queue (ANY = false: closest
// hit) or the shadow records (ANY = true: occlusion).  Each lane traces its
// own ray; every `chunk` leaf visits the warp reconverges and lanes whose
// ray has finished take new rays from the queue (one atomic per warp), so
// short rays (most camera rays miss every box) do not idle their warp
// while long ones traverse.
// Camera-ray misses (src/integrator.rs:71-83 at bounce 0) are the most
// common samples of an open scene: a camera ray that leaves the scene adds
// the env (or sky) radiance and the sample is done.  When such a sample is
// not the last of its task, the closest-hit kernel finishes it in place --
// the f64 task sums, the next camera ray from the pixel's stream
// (src/render.rs:151-158) -- and traces that ray at once, instead of a
// round trip through the shading kernel.  Same arithmetic and draws as
// k_shade + finish_sample; off for adaptive renders (their stopping rule
// runs in finish_sample) and for the adjoint.  Returns false when the slot
// is not such a sample.
template <bool BATCH>
__device__ __forceinline__ bool camera_miss_next(const WfScene& S0, const WfParams& P, const WfState& st, int slot,
                                                 Tracer& T) {
    int4 m;
    uint64_t rng;
    load_path(st, slot, m, rng);
    if (m.y != 0) return false;
    // the render's (or the slot's batch job's) camera, env map and film
    const WfJob* J = BATCH ? P.jobs + st.job[slot] : nullptr;
    const int max_bounces = BATCH ? J->max_bounces : P.max_bounces;
    if (max_bounces <= 0) return false;
    TaskPos tp;
    if constexpr (BATCH) {
        const long long lt = (long long)m.w - J->task_begin;
        const uint32_t chunk = fdiv(J->px_div, (uint32_t)lt);
        tp.j = tp.pixel = (int)((uint32_t)lt - chunk * (uint32_t)J->n_pixels);
        tp.sample_start = (int)chunk * J->task_spp;
        tp.len = min(J->task_spp, J->spp - tp.sample_start);
    } else {
        tp = task_pos(P, (long long)m.w);
    }
    if (m.x + 1 >= tp.len) return false;  // the task's last sample ends in the shading kernel
    WfScene S = S0;
    if constexpr (BATCH) {
        S.env_kind = J->env_kind; S.env_w = J->env_w; S.env_h = J->env_h; S.env_tex = J->env_tex;
    }
    const float3 L = clamp_lum(f3(1.0f, 1.0f, 1.0f) * background(S, T.wd), 50.0f);  // beta = 1 at bounce 0
    if (!BATCH && st.rsamp) {  // adaptive round: the sample itself, for the in-order stopping rule
        sts(&st.rsamp[(size_t)tp.j * P.round_len + (tp.sample_start - P.sample_base) + m.x],
            make_float4(L.x, L.y, L.z, 0.0f));
    } else {
        Sums sums = load_sums(st, slot, m.x == 0);
        add_sample(sums, L, st.ssq != nullptr);
        store_sums(st, slot, sums);
    }
    m.x += 1;
    const int pixel = tp.pixel;
    const int width = BATCH ? J->width : P.width, height = BATCH ? J->height : P.height;
    const int row_begin = BATCH ? J->row_begin : P.row_begin, row_step = BATCH ? J->row_step : P.row_step;
    float3 o, d;
    float ptime;
    const int row = (int)fdiv(BATCH ? J->w_div : P.w_div, (uint32_t)pixel);
    camera_ray(BATCH ? J->cam : S0.cam, pixel - row * width, row_begin + row * row_step, 1.0f / (float)width,
               1.0f / (float)height, rng, o, d, ptime);
    store_path(st, slot, m, rng);
    sts(&st.ray_o[slot], make_float4(o.x, o.y, o.z, ifloat(-1)));
    sts(&st.ray_d[slot], make_float4(d.x, d.y, d.z, ifloat(-1)));
    sts(&st.rad[slot], make_float4(0.0f, 0.0f, 0.0f, ptime));
    tracer_start_at(BATCH ? J->top_root : S0.top_root, T, o, d, kTMax, -1, -1);
    return true;
}

template <bool ANY, bool COUNT, bool SHARED_STACK, bool BATCH>
__global__ void __launch_bounds__(kTraceBlock) k_trace(WfScene S, WfParams P, WfState st, int n_slots, int chunk,
                                                       const WfJob* __restrict__ jobs, int cur) {
    // Extension rays come from a sweep of every slot's act byte in slot
    // order, or, once few paths are live (forward renders, use_ext_queue),
    // from the compacted queue the shading and completion kernels push;
    // shadow rays from the shadow-record queue.
    const bool queue = ANY || (P.ext_queue && (P.ordered_queue || use_ext_queue(st.ctr->n_ext[cur], n_slots, P.queue_div)));
    const int n = ANY ? st.ctr->n_sh : (queue ? st.ctr->n_ext[cur] : n_slots);
    int* fetch = ANY ? &st.ctr->fetch_sh : &st.ctr->fetch_ext;
    const int* __restrict__ q = ANY ? st.q_sh : st.q_ext[cur];
    int* flags = &st.ctr->flags;
    __shared__ int sstack[SHARED_STACK ? kSharedStack * kTraceBlock : 1];
    int lstack[SHARED_STACK ? 1 : kStack];
    using Stack = typename std::conditional<SHARED_STACK, TStack<kTraceBlock, kSharedStack>, TStack<1, kStack>>::type;
    const Stack stack{SHARED_STACK ? sstack + threadIdx.x : lstack};
    Tracer T;
    TraceCount cnt;
    int item = -1;
    bool exhausted = false;
    const unsigned lt_mask = (1u << lane_id()) - 1u;
    unsigned long long fast_done = 0;  // samples finished by camera_miss_next
    for (;;) {
        const bool want = item < 0 && !exhausted;
        const unsigned m = __ballot_sync(0xffffffffu, want);
        if (m) {
            const int leader = __ffs(m) - 1;
            int base = 0;
            if ((int)lane_id() == leader) base = atomicAdd(fetch, __popc(m));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (want) {
                const int k = base + __popc(m & lt_mask);
                if (k < n) {
                    item = queue ? q[k] : (st.act[k] ? k : -1);
                    if (item < 0) {
                        // inactive slot: nothing to trace; refill next round
                    } else if (ANY) {
                        const float4 o4 = lds(&st.sh_o[item]), d4 = lds(&st.sh_d[item]);
                        const int self_inst = fbits(reinterpret_cast<const float*>(st.sh_c + item)[3]);
                        const int root = BATCH ? __ldg(&jobs[st.job[item >> 1]].top_root) : S.top_root;
                        tracer_start_at(root, T, f3(o4), f3(d4), o4.w, fbits(d4.w), self_inst);
                    } else {
                        const float4 o4 = lds(&st.ray_o[item]), d4 = lds(&st.ray_d[item]);
                        const int root = BATCH ? __ldg(&jobs[st.job[item]].top_root) : S.top_root;
                        tracer_start_at(root, T, f3(o4), f3(d4), kTMax, fbits(o4.w), fbits(d4.w));
                    }
                } else {
                    exhausted = true;
                }
            }
        }
        // A window of inactive slots leaves every lane empty but the cursor
        // short of n: the warp keeps fetching until all lanes are exhausted.
        if (!__any_sync(0xffffffffu, item >= 0 || !exhausted)) break;
        if (item >= 0 && tracer_run<COUNT>(S, T, stack, kEps, chunk, flags, cnt, ANY)) {
            if (ANY) {
                reinterpret_cast<float*>(st.sh_c + item)[3] = T.hit_prim >= 0 ? 0.0f : 1.0f;
            } else {
                if (P.camera_fast && T.hit_prim < 0 && camera_miss_next<BATCH>(S, P, st, item, T)) {
                    if (COUNT) count_step(cnt.fast_steps);
                    ++fast_done;
                    continue;  // this lane traces the task's next camera ray
                }
                sts(&st.hit[item], make_float4(T.hit_prim >= 0 ? T.tmax : kTMax, ifloat(T.hit_prim), ifloat(T.hit_inst), 0.0f));
            }
            item = -1;
        }
    }
    flush_counts<COUNT>(st.ctr, ANY ? 1 : 0, cnt);
    if (!ANY) {
        for (int off = 16; off > 0; off >>= 1) fast_done += __shfl_down_sync(0xffffffffu, fast_done, off);
        if (lane_id() == 0 && fast_done) {
            atomicAdd(&st.ctr->samples, fast_done);
            atomicAdd(&st.ctr->rays_closest, fast_done);
            if (COUNT) atomicAdd(&st.ctr->cnt_fast, fast_done);
        }
    }
}


__device__ __forceinline__ float3 take_pending(const WfState& st, int slot, int& fl, float3 L) {
    if (fl & F_PEND_ENV) {
        const float4 c = lds(&st.sh_c[2 * slot]);
        if (c.w > 0.5f) L = L + f3(c);
    }
    if (fl & F_PEND_AREA) {
        const float4 c = lds(&st.sh_c[2 * slot + 1]);
        if (c.w > 0.5f) L = L + f3(c);
    }
    fl &= ~(F_PEND_ENV | F_PEND_AREA);
    return L;
}

// End of one sample of a slot (src/render.rs:143-191): the sample's radiance
// joins the task's f64 sums (and the Welford statistics of adaptive
// sampling).  If the task has samples left, the pixel's next camera ray is
// written and the path state reset (returns true); otherwise the task's sums
// go to the film (one task per pixel) or to the task's partial sums, and
// need_task is set so the slot takes a new task.
// finish_sums does all of that but the camera ray and the slot's records:
// the sums are the caller's, tp is the task's place.
__device__ __forceinline__ bool finish_sums(const WfParams& P, const WfState& st, int4& m, float3 L, bool& need_task,
                                            const Film& F, const TaskPos& tp, Sums& s) {
    const long long task = (long long)m.w;       // batch-wide task id
    m.x += 1;
    const int task_len = tp.len;
    bool stop = m.x >= task_len;
    if (P.adaptive) {  // Welford on luminance (render.rs:160-176)
        const double l = 0.2126 * (double)L.x + 0.7152 * (double)L.y + 0.0722 * (double)L.z;
        const double delta = l - s.w.x;
        s.w.x += delta / (double)m.x;
        s.w.y += delta * (l - s.w.x);
        const int min_spp = min(max(P.adaptive_min_spp, 1), max(task_len, 1));
        if (m.x >= min_spp && m.x > 1) {
            const double var = s.w.y / (double)(m.x - 1);
            if (sqrt(var) / fmax(fabs(s.w.x), 1e-4) < P.adaptive_threshold) stop = true;
        }
    }
    need_task = stop;
    if (st.rsamp) {  // adaptive round: the sample itself, for the in-order stopping rule (k_round_merge adds it)
        sts(&st.rsamp[(size_t)tp.j * P.round_len + (tp.sample_start - P.sample_base) + m.x - 1],
            make_float4(L.x, L.y, L.z, 0.0f));
        return !stop;
    }
    add_sample(s, L, st.acc_sq != nullptr);
    if (stop) {
        if (P.n_chunks == 1) {  // one task per pixel: straight into the film
            const size_t px = (size_t)tp.pixel;
            F.acc[3 * px] = s.a.x; F.acc[3 * px + 1] = s.a.y; F.acc[3 * px + 2] = s.a.z;
            F.acc_w[px] = s.a.w;
            if (F.acc_sq) { F.acc_sq[3 * px] = s.q.x; F.acc_sq[3 * px + 1] = s.q.y; F.acc_sq[3 * px + 2] = s.q.z; }
        } else {  // per-task sums, merged in task order by k_merge
            st.part[task - P.task_first] = s.a;
            if (st.part_sq) st.part_sq[task - P.task_first] = s.q;
        }
    }
    return !stop;
}
__device__ __forceinline__ bool finish_sample(const WfScene& S, const WfParams& P, const WfState& st, int slot,
                                              int4& m, int& fl, float3& L, float3& beta, float& last_pdf,
                                              float& ptime, uint64_t& rng, bool& need_task, const Film& F,
                                              long long base) {
    const TaskPos tp = task_pos(P, (long long)m.w - base);
    Sums sums = load_sums(st, slot, m.x == 0);
    if (!finish_sums(P, st, m, L, need_task, F, tp, sums)) return false;
    store_sums(st, slot, sums);
    float3 o, d;
    const int row = (int)fdiv(P.w_div, (uint32_t)tp.pixel);
    camera_ray(S.cam, tp.pixel - row * P.width, P.row_begin + row * P.row_step, 1.0f / (float)P.width,
               1.0f / (float)P.height, rng, o, d, ptime);
    sts(&st.ray_o[slot], make_float4(o.x, o.y, o.z, ifloat(-1)));
    sts(&st.ray_d[slot], make_float4(d.x, d.y, d.z, ifloat(-1)));
    beta = f3(1.0f, 1.0f, 1.0f);
    last_pdf = 0.0f;
    L = f3(0, 0, 0);
    m.y = 0;
    fl = 0;
    return true;
}

// Slots whose task finished take the next tasks from the pool (one atomic
// per warp); -1 = none left, or not wanted.  Must be called by all lanes of
// a converged warp.
__device__ __forceinline__ long long next_task(const WfParams& P, const WfState& st, bool need_task) {
    const unsigned want = __ballot_sync(0xffffffffu, need_task);
    if (!want) return -1;
    const int leader = __ffs(want) - 1;
    long long t0 = 0;
    if ((int)lane_id() == leader)
        t0 = (long long)atomicAdd((unsigned long long*)&st.ctr->next_task, (unsigned long long)__popc(want));
    t0 = __shfl_sync(0xffffffffu, t0, leader);
    if (!need_task) return -1;
    const long long t = t0 + __popc(want & ((1u << lane_id()) - 1u));
    return t < fetch_end(P) ? task_of_fetch(P, t) : -1;
}
template <bool BATCH>
__device__ __forceinline__ bool take_next_task(const WfScene& S, const WfParams& P, const WfState& st, int slot,
                                               bool need_task) {
    const long long task = next_task(P, st, need_task);
    if (task < 0) return false;
    start_task<BATCH>(S, P, st, slot, task);
    return true;
}

// ---- shading -------------------------------------------------------------------
// Material-sorted shading (TPT_SHADE_SORT=1): one bounce of radiance()
// (src/integrator.rs:67-132), split by what the ray found.  k_shade_pre takes every queued path: misses (env + MIS), Russian
// roulette and emitter hits end the sample in place; surface hits are sorted
// into one queue per material kind with warp-ballot compaction.
// k_shade_surface<KIND> then runs NEE and BSDF sampling for one material
// kind, so each kernel carries only its own BSDF and no warp diverges on the
// material.
constexpr int kKinds = 5;  // TPT_MAT_LAMBERT .. TPT_MAT_SUBSURFACE

// Warp-aggregated count of `pred` lanes added to *counter.
__device__ __forceinline__ void warp_count(int* counter, bool pred) {
    const unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (mask && (int)lane_id() == __ffs(mask) - 1) atomicAdd(counter, __popc(mask));
}

__global__ void __launch_bounds__(128) k_shade_pre(WfScene S, WfParams P, WfState st, int cur) {
    const int live = st.ctr->n_ext[cur];  // the slots the closest-hit kernel traced
    const bool use_q = P.ordered_queue || use_ext_queue(live, P.n_slots, P.queue_div);
    const int n = use_q ? live : P.n_slots;
    const int* __restrict__ qe = st.q_ext[cur];
    const int nxt = cur ^ 1;
    const bool has_env = S.env_kind == TPT_ENV_MAP;
    const int stride = gridDim.x * blockDim.x;
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
        const int i = base + (int)lane_id();
        bool again = false, need_task = false, finished = false, surface = false;
        int kind = 0, slot = 0;
        const bool active = i < n && (use_q || st.act[i]);
        if (active) {
            slot = use_q ? qe[i] : i;
            const float4 o4 = lds(&st.ray_o[slot]), d4 = lds(&st.ray_d[slot]);
            const float3 ro = f3(o4), rd = f3(d4);
            const float4 h4 = lds(&st.hit[slot]);
            const int prim = fbits(h4.y), inst = fbits(h4.z);
            const float4 b4 = lds(&st.beta[slot]);
            float3 beta = f3(b4);
            float last_pdf = b4.w;
            const float4 r4 = lds(&st.rad[slot]);
            float3 L = f3(r4);
            float ptime = r4.w;
            int4 m;
            uint64_t rng;
            load_path(st, slot, m, rng);
            int fl = m.z;
            L = take_pending(st, slot, fl, L);
            bool done = m.y >= P.max_bounces;  // max_bounces = 0: radiance() returns 0
            if (!done && prim < 0) {  // miss (:71-83)
                float3 contrib = beta * background(S, rd);
                if (has_env && (fl & F_LAST_ND)) contrib = contrib * mis(last_pdf, env_pdf(S, rd));
                L = L + clamp_lum(contrib, 50.0f);
                done = true;
            }
            if (!done && m.y >= P.rr_start) {  // Russian roulette (:89-95)
                const float p = fmaxf(fminf(max3(beta), 0.95f), 0.05f);
                if (pcg_f32(rng) > p) done = true;
                else beta = beta / p;
            }
            if (!done) {
                const float3 hp = ro + rd * h4.x;
                float3 ng;
                int mid;
                if (inst < 0) {
                    const float4 cr = __ldg(&S.spheres[prim].cr);
                    ng = (hp - f3(cr)) / cr.w;
                    mid = __ldg(&S.spheres[prim].mat);
                } else {
                    const TriF32* tp = S.tris + (prim - S.n_spheres);
                    const float4 v0 = __ldg(&tp->v0), e1 = __ldg(&tp->e1), e2 = __ldg(&tp->e2);
                    const float3 no = cross(f3(e1), f3(e2));
                    const InstanceF32* I = S.inst + inst;
                    const float4 n0 = __ldg(&I->nrm[0]), n1 = __ldg(&I->nrm[1]), n2 = __ldg(&I->nrm[2]);
                    ng = normalize(f3(n0.x * no.x + n0.y * no.y + n0.z * no.z, n1.x * no.x + n1.y * no.y + n1.z * no.z,
                                      n2.x * no.x + n2.y * no.y + n2.z * no.z));
                    const int ov = fbits(__ldg(&I->wbox_max.w));
                    mid = ov >= 0 ? ov : fbits(v0.w);
                }
                kind = __ldg(&S.mats[mid].kind);
                if (kind == TPT_MAT_DIFFUSE_LIGHT) {  // emitter (:100-104)
                    L = L + clamp_lum(beta * f3(__ldg(&S.mats[mid].c)), 50.0f);
                    done = true;
                } else {
                    st.surf_p[slot] = make_float4(hp.x, hp.y, hp.z, h4.x);
                    st.surf_n[slot] = make_float4(ng.x, ng.y, ng.z, ifloat(mid));
                    surface = true;
                }
            }
            if (done) {  // nothing is pending: the sample ends here
                again = finish_sample(S, P, st, slot, m, fl, L, beta, last_pdf, ptime, rng, need_task, film_of(st), 0);
                finished = true;
            }
            sts(&st.beta[slot], make_float4(beta.x, beta.y, beta.z, last_pdf));
            sts(&st.rad[slot], make_float4(L.x, L.y, L.z, ptime));
            m.z = fl;
            store_path(st, slot, m, rng);
        }
        if (take_next_task<false>(S, P, st, slot, need_task)) again = true;
        if (active) st.act[slot] = (again || surface) ? 1 : 0;
        if (!P.ordered_queue) warp_push(st.q_ext[nxt], &st.ctr->n_ext[nxt], again, slot);
        for (int k = 0; k < kKinds; ++k)
            warp_push(st.q_mat + (size_t)k * P.n_slots, &st.ctr->n_mat[k], surface && kind == k, slot);
        warp_count(&st.ctr->n_done_in_shade, finished);
    }
}

// One bounce of radiance() (src/integrator.rs:67-132) per queued path, all
// material kinds in one kernel (the default; it keeps each path's state in
// registers through the whole bounce).
//
// Bound by the latency of the path-state loads and, before this shape, by
// instruction fetch: 80 to 100 KB of straight code, of which a warp on its own
// waited for every line (7 to 13 "no instruction" cycles per issue), at 14 of
// 32 lanes.  So a block of 256 first orders its slots by what their rays met
// (miss or material kind), its warps go through the stages together (1.2 "no
// instruction" cycles left), each stage appears once -- one evaluation of the
// env map for misses and NEE samples, one camera ray for the next sample and
// the next task -- and the records of its next slots are prefetched.
// Measured on one B200, ms: sphere scene 256x256 x 64 spp 2.82 -> 2.33, built-in
// scene 853x479 x 17 spp 2.92 -> 2.32, mesh scene 960x540 x 64 spp 9.92 ->
// 9.08, the 1080p frame 147 -> 140.  Stages without the ordering, blocks of
// 128: 2.46 / 2.50 / 9.63 / 139; blocks of 512: 2.29 / 2.34 / 9.25 / 143.
constexpr int kShadeBlock = 256;
// A path between two closest-hit rays, in registers.
struct PathRegs {
    float3 o, d;              // the ray
    int self_prim, self_inst; // what it starts on
    float t;                  // what it met
    int prim, inst;
    float3 beta, L;
    float last_pdf, time;
    int4 m;                   // samples done, bounce, (flags in fl), task
    int fl;
    uint64_t rng;
};

// One bounce of radiance() (src/integrator.rs:67-132): what the closest-hit
// ray met, the NEE samples -- `emit(k, origin, tmax, direction, contribution)`
// for each shadow ray, 0 = env, 1 = area light -- and the next ray --
// `next(origin, direction, self primitive, self instance)`.  The callbacks let
// k_shade store the rays at once instead of keeping them in registers (its
// budget: 1080p frame +3% with them kept).  Returns true when the path ends.  STAGED: every thread of the block calls
// it, `active` or not, and the block's warps meet between the stages.
template <bool STAGED, class Emit, class Next>
__device__ __forceinline__ bool bounce(const WfScene& S, const WfParams& P, PathRegs& p, bool active, Emit&& emit,
                                       Next&& next) {
    auto stage = [] {
        if constexpr (STAGED) __syncthreads();
    };
    const bool has_env = active && S.env_kind == TPT_ENV_MAP;
    const float3 rd = p.d;
    const int prim = p.prim, inst = p.inst;
    float3 hp = f3(0, 0, 0), ng = f3(0, 0, 0);
    int mid = 0, kind = 0;
    bool done = active && p.m.y >= P.max_bounces, surface = false;  // max_bounces = 0: radiance() returns 0
    const bool miss = active && !done && prim < 0;
    if (active && !done && !miss) {
        if (p.m.y >= P.rr_start) {  // Russian roulette (:89-95)
            const float q = fmaxf(fminf(max3(p.beta), 0.95f), 0.05f);
            if (pcg_f32(p.rng) > q) done = true;
            else p.beta = p.beta / q;
        }
        if (!done) {
            hp = p.o + rd * p.t;
            if (inst < 0) {
                const SphereF32 sp = S.spheres[prim];
                ng = (hp - f3(sp.cr)) / sp.cr.w;
                mid = sp.mat;
            } else {
                const TriF32* tp = S.tris + (prim - S.n_spheres);
                const float4 v0 = __ldg(&tp->v0), e1 = __ldg(&tp->e1), e2 = __ldg(&tp->e2);
                const float3 no = cross(f3(e1), f3(e2));
                const InstanceF32* I = S.inst + inst;
                const float4 n0 = __ldg(&I->nrm[0]), n1 = __ldg(&I->nrm[1]), n2 = __ldg(&I->nrm[2]);
                ng = normalize(f3(n0.x * no.x + n0.y * no.y + n0.z * no.z, n1.x * no.x + n1.y * no.y + n1.z * no.z,
                                  n2.x * no.x + n2.y * no.y + n2.z * no.z));
                const int ov = fbits(__ldg(&I->wbox_max.w));
                mid = ov >= 0 ? ov : fbits(v0.w);
            }
            kind = S.mats[mid].kind;
            if (kind == TPT_MAT_DIFFUSE_LIGHT) {  // emitter (:100-104)
                p.L = p.L + clamp_lum(p.beta * f3(S.mats[mid].c), 50.0f);
                done = true;
            } else {
                surface = true;
            }
        }
    }
    const bool nee = surface && kind != TPT_MAT_METAL && kind != TPT_MAT_DIELECTRIC;
    const bool entering = dot(ng, rd) < 0.0f;
    const float3 n = entering ? ng : -ng;
    const float3 wo = -rd;
    stage();
    // the env map in the ray's direction (a miss) or the NEE sample's
    float3 wi = rd, li = f3(0, 0, 0);
    float pe = 1.0f / (4.0f * kPi);
    bool want_pdf = (p.fl & F_LAST_ND) != 0;
    // a black map (XML scenes carry one) adds 0 whatever the direction: its
    // samples only take their two draws
    const bool dark = S.env_black && p.beta.x + p.beta.y + p.beta.z < INFINITY;
    if (nee && has_env) {
        if (dark) {
            pcg_f32(p.rng);
            pcg_f32(p.rng);
        } else {
            want_pdf = env_sample_to(S, p.rng, wi);
        }
    }
    stage();
    if (has_env && !dark && (miss || nee)) {
        float pdf = pe;
        li = env_at(S, wi, &pdf);
        if (want_pdf) pe = pdf;
    }
    stage();
    if (miss) {  // (:71-83)
        if (!has_env) li = sky(rd);
        float3 contrib = p.beta * li;
        if (has_env && (p.fl & F_LAST_ND)) contrib = contrib * mis(p.last_pdf, pe);
        p.L = p.L + clamp_lum(contrib, 50.0f);
        done = true;
    }
    if (nee && has_env && !dark) {  // nee_environment (:148-172)
        const float c = fmaxf(dot(n, wi), 0.0f);
        if (c > 0.0f && pe > 0.0f) {
            float3 f;
            float pb;
            mat_eval(S.mats[mid], wo, wi, n, f, pb);
            const float3 contrib = p.beta * f * li * (c * mis(pe, pb) / pe);
            if (contrib.x > 0.0f || contrib.y > 0.0f || contrib.z > 0.0f) emit(0, hp + wi * kEps, kTMax, wi, contrib);
        }
    }
    stage();
    if (nee) {
        float3 lp, le;
        float lpdf;
        int lidx;
        double lud, lvd;
        if (sample_light(S, p.rng, hp, lp, le, lpdf, lidx, lud, lvd)) {  // nee_area_light (:178-213)
            const float3 tl = lp - hp;
            const float dist = length(tl);
            if (dist > 1e-6f) {
                const float3 wl = tl / dist;
                const float c = fmaxf(dot(n, wl), 0.0f);
                if (c > 0.0f && !ref_light_self_occluded(S.lights64, S.spheres64, S.inst64, lidx, p.o, rd, p.t, lud, lvd,
                                                         (double)p.time)) {
                    float3 f;
                    float pb;
                    mat_eval(S.mats[mid], wo, wl, n, f, pb);
                    const float3 contrib = p.beta * f * le * (c * mis(lpdf, pb) / lpdf);
                    // stops 1e-4 short of the light: the light itself is
                    // handled by ref_light_self_occluded
                    if (contrib.x > 0.0f || contrib.y > 0.0f || contrib.z > 0.0f)
                        emit(1, hp + wl * kEps, fmaxf(dist - 2.0f * kEps, kEps), wl, contrib);
                }
            }
        }
    }
    stage();
    if (surface) {  // Material::sample (src/material.rs:76-201)
        const MaterialF32 mt = S.mats[mid];
        const float3 mc = f3(mt.c);
        float3 nd = f3(0, 0, 0), w = f3(0, 0, 0), no = hp;
        float pdf = 0.0f;
        bool delta = false, ok = true, self_ok = true;
        switch (kind) {
            case TPT_MAT_LAMBERT:
            case TPT_MAT_SUBSURFACE: {
                const bool sub = kind == TPT_MAT_SUBSURFACE;
                w = mc;
                if (sub) {
                    const float sc = fmaxf(mt.c.w, 1e-4f);
                    const float u = fmaxf(pcg_f32(p.rng), 1e-12f);
                    const float dist = -__logf(u) * sc;
                    w = mc * __expf(-dist / sc);
                    no = hp - ng * dist;
                    self_ok = false;     // origin moved off the surface
                }
                nd = cos_hemi(sub ? ng : n, p.rng);  // subsurface: unoriented normal (material.rs:187-188)
                pdf = fmaxf(dot(n, nd), 0.0f) / kPi;
                break;
            }
            case TPT_MAT_METAL:
                nd = rd - n * (2.0f * dot(rd, n));
                w = mc;
                delta = true;
                break;
            case TPT_MAT_DIELECTRIC: {
                const float ior = mt.c.w;
                const float eta = entering ? 1.0f / ior : ior;
                const float ci = fmaxf(dot(wo, n), 0.0f);
                const float fq = (ior - 1.0f) / (ior + 1.0f);
                const float f0 = fq * fq;
                const float fr = f0 + (1.0f - f0) * pow5(1.0f - ci);
                float3 bt = f3(1, 1, 1);
                if (!entering) {
                    const float dist = fmaxf(p.t, 0.0f);
                    bt = f3(__expf(-mc.x * dist), __expf(-mc.y * dist), __expf(-mc.z * dist));
                }
                const float cosi = fminf(fmaxf(dot(wo, n), -1.0f), 1.0f);
                const float sin2t = eta * eta * (1.0f - cosi * cosi);
                const bool has_refr = !(sin2t >= 1.0f);
                const bool refl = !has_refr || pcg_f32(p.rng) < fr;
                if (refl) {
                    nd = rd - n * (2.0f * dot(rd, n));
                    bt = bt * (fr / fmaxf(fr, 1e-6f));
                } else {
                    nd = rd * eta + n * (eta * cosi - sqrtf(1.0f - sin2t));
                    bt = bt * ((1.0f - fr) / fmaxf(1.0f - fr, 1e-6f)) * (eta * eta);
                }
                w = bt;
                delta = true;
                break;
            }
            case TPT_MAT_GGX: {
                GgxSample gs;
                if (!ggx_sample(rd, n, mt, p.rng, gs)) { ok = false; break; }
                nd = gs.nd;
                w = gs.w;
                pdf = gs.pdf;
                break;
            }
            default:
                ok = false;
        }
        if (!ok) {
            done = true;
        } else {
            p.beta = p.beta * w;
            p.last_pdf = pdf;
            p.fl = delta ? (p.fl & ~F_LAST_ND) : (p.fl | F_LAST_ND);
            next(no + nd * kEps, nd, self_ok ? prim : -1, self_ok ? inst : -1);
            p.m.y += 1;
            if (p.m.y >= P.max_bounces) done = true;  // bounce loop bound (:67)
        }
    }
    stage();
    return done;
}

// The camera ray of sample m.x of the task at tp (src/render.rs:151-158) and
// the path state it starts with; the first sample seeds the task's stream.
__device__ __forceinline__ void start_sample(const WfScene& S, const WfParams& P, const TaskPos& tp, PathRegs& p) {
    const int row = (int)fdiv(P.w_div, (uint32_t)tp.pixel);
    const int x = tp.pixel - row * P.width, y = P.row_begin + row * P.row_step;
    if (p.m.x == 0) p.rng = task_seed((uint32_t)x, (uint32_t)y, (uint32_t)tp.sample_start, P.seed);
    camera_ray(S.cam, x, y, 1.0f / (float)P.width, 1.0f / (float)P.height, p.rng, p.o, p.d, p.time);
    p.self_prim = p.self_inst = -1;
    p.beta = f3(1.0f, 1.0f, 1.0f);
    p.L = f3(0.0f, 0.0f, 0.0f);
    p.last_pdf = 0.0f;
    p.m.y = 0;
    p.fl = 0;
}

// A slot's path as the last iteration left it, its pending shadow rays'
// results included.
__device__ __forceinline__ PathRegs load_slot(const WfState& st, int slot) {
    PathRegs p;
    const float4 o4 = lds(&st.ray_o[slot]), d4 = lds(&st.ray_d[slot]);
    p.o = f3(o4);
    p.d = f3(d4);
    p.self_prim = fbits(o4.w);
    p.self_inst = fbits(d4.w);
    const float4 b4 = lds(&st.beta[slot]), r4 = lds(&st.rad[slot]);
    p.beta = f3(b4);
    p.last_pdf = b4.w;
    p.time = r4.w;
    load_path(st, slot, p.m, p.rng);
    p.fl = p.m.z;
    p.L = take_pending(st, slot, p.fl, f3(r4));
    p.t = kTMax;
    p.prim = p.inst = -1;
    return p;
}

// What the shading stages do with a live slot: 0 = its ray left the scene, 1 +
// the material kind it hit.
__device__ __forceinline__ int shade_class(const WfScene& S, const WfState& st, int slot) {
    const float4 h4 = __ldg(&st.hit[slot]);
    const int prim = fbits(h4.y), inst = fbits(h4.z);
    if (prim < 0) return 0;
    int mid;
    if (inst < 0) {
        mid = __ldg(&S.spheres[prim].mat);
    } else {
        const int ov = fbits(__ldg(&S.inst[inst].wbox_max.w));
        mid = ov >= 0 ? ov : fbits(__ldg(&S.tris[prim - S.n_spheres].v0.w));
    }
    return 1 + __ldg(&S.mats[mid].kind);
}
// The block's slots ordered by class, stable: thread t gets the t-th.  cls:
// the thread's own class (7 = no slot).
__device__ __forceinline__ int sort_by_class(int slot, int cls, int (*counts)[8], int* order) {
    const int w = threadIdx.x >> 5;
    int rank = 0;
    for (int k = 0; k < 8; ++k) {
        const unsigned m = __ballot_sync(0xffffffffu, cls == k);
        if (cls == k) rank = __popc(m & ((1u << lane_id()) - 1u));
        if (lane_id() == (unsigned)k) counts[w][k] = __popc(m);
    }
    __syncthreads();
    // exclusive prefix over (class, warp), one warp
    constexpr int W = kShadeBlock / 32;
    if (w == 0) {
        int run = 0;
        for (int k = 0; k < 8; ++k) {
            int v = lane_id() < (unsigned)W ? counts[lane_id()][k] : 0, x = v;
            for (int off = 1; off < W; off <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, off);
                if ((int)lane_id() >= off) x += y;
            }
            if (lane_id() < (unsigned)W) counts[lane_id()][k] = run + x - v;
            run += __shfl_sync(0xffffffffu, x, W - 1);
        }
    }
    __syncthreads();
    order[counts[w][cls] + rank] = cls == 7 ? -1 : slot;
    __syncthreads();
    return order[threadIdx.x];
}

// CTAS: blocks of 128 threads' worth of registers per SM (4, 6 or 8).
template <bool BATCH, int CTAS>
__global__ void __launch_bounds__(kShadeBlock, CTAS * 128 / kShadeBlock) k_shade(WfScene S0, WfParams P0, WfState st,
                                                                                int cur) {
    // At 6+ blocks of 128 per SM the kernel spills: ptxas may put the spills
    // in shared memory instead of local memory, which at 1024 threads per SM
    // does not fit in L1 (1080p frame: +1.0% paths/s).
    if constexpr (CTAS >= 6) asm volatile(".pragma \"enable_smem_spilling\";");
    __shared__ int counts[kShadeBlock / 32][8], order[kShadeBlock];
    const int live = st.ctr->n_ext[cur];  // the slots the closest-hit kernel traced
    const bool use_q = P0.ordered_queue || use_ext_queue(live, P0.n_slots, P0.queue_div);
    const int n = use_q ? live : P0.n_slots;
    const int* __restrict__ qe = st.q_ext[cur];
    const int nxt = cur ^ 1;
    const int stride = gridDim.x * blockDim.x;
    for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const int i = base + (int)threadIdx.x;
        bool active = i < n && (use_q || st.act[i]);
        int slot = active ? (use_q ? qe[i] : i) : 0;
        slot = sort_by_class(slot, active ? shade_class(S0, st, slot) : 7, counts, order);
        active = slot >= 0;
        if (use_q && i + stride < n) {  // the records of the block's next slots, on their way to L2
            const int next = __ldg(qe + i + stride);
            auto fetch = [](const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); };
            fetch(st.ray_o + next); fetch(st.ray_d + next); fetch(st.hit + next);
            fetch(st.beta + next); fetch(st.rad + next); fetch(st.path + next);
        }
        PathRegs p{};
        int job = 0;
        if (active) {
            if constexpr (BATCH) job = st.job[slot];
            p = load_slot(st, slot);
            const float4 h4 = lds(&st.hit[slot]);
            p.t = h4.x;
            p.prim = fbits(h4.y);
            p.inst = fbits(h4.z);
        }
        int sh[2] = {0, 0};
        const int prim = p.prim, inst = p.inst;
        const View vb = view_of<BATCH>(S0, P0, st, job);  // (an idle thread: job 0's)
        const bool done = bounce<true>(vb.S, vb.P, p, active, [&](int k, float3 so, float tmax, float3 wi, float3 contrib) {
            sts(&st.sh_o[2 * slot + k], make_float4(so.x, so.y, so.z, tmax));
            sts(&st.sh_d[2 * slot + k], make_float4(wi.x, wi.y, wi.z, ifloat(prim)));
            sts(&st.sh_c[2 * slot + k], make_float4(contrib.x, contrib.y, contrib.z, ifloat(inst)));
            sh[k] = 1;
        }, [&](float3 o, float3 d, int self_prim, int self_inst) {
            sts(&st.ray_o[slot], make_float4(o.x, o.y, o.z, ifloat(self_prim)));
            sts(&st.ray_d[slot], make_float4(d.x, d.y, d.z, ifloat(self_inst)));
        });
        if (active) p.fl |= (sh[0] ? F_PEND_ENV : 0) | (sh[1] ? F_PEND_AREA : 0);
        bool cont = active && !done, need_task = false, camera = false;
        const bool term = active && done && (sh[0] || sh[1]), finished = active && done && !term;
        TaskPos tp{};
        if (finished) {  // nothing pending: the sample ends here instead of in k_regen
            const View v = view_of<BATCH>(S0, P0, st, job);
            tp = task_pos(v.P, (long long)p.m.w - v.task_begin);
            Sums sums = load_sums(st, slot, p.m.x == 0);
            camera = finish_sums(v.P, st, p.m, p.L, need_task, v.F, tp, sums);
            if (camera) store_sums(st, slot, sums);
        }
        const long long task = next_task(P0, st, need_task);
        if (task >= 0) {
            if constexpr (BATCH) {
                job = find_job(P0, task);
                st.job[slot] = job;
            }
            const View v = view_of<BATCH>(S0, P0, st, job);
            tp = task_pos(v.P, task - v.task_begin);
            p.m = make_int4(0, 0, 0, (int)task);
            camera = true;
        }
        if (camera) {
            const View v = view_of<BATCH>(S0, P0, st, job);
            start_sample(v.S, v.P, tp, p);
            sts(&st.ray_o[slot], make_float4(p.o.x, p.o.y, p.o.z, ifloat(-1)));
            sts(&st.ray_d[slot], make_float4(p.d.x, p.d.y, p.d.z, ifloat(-1)));
            cont = true;
        }
        if (cont || term) {
            if (cont) sts(&st.beta[slot], make_float4(p.beta.x, p.beta.y, p.beta.z, p.last_pdf));
            sts(&st.rad[slot], make_float4(p.L.x, p.L.y, p.L.z, p.time));
            p.m.z = p.fl;
            store_path(st, slot, p.m, p.rng);
        }
        if (active) st.act[slot] = cont ? 1 : 0;
        if (!P0.ordered_queue) warp_push(st.q_ext[nxt], &st.ctr->n_ext[nxt], cont, slot);
        warp_push(st.q_term, &st.ctr->n_term, term, slot);
        warp_count(&st.ctr->n_done_in_shade, finished);
        warp_push(st.q_sh, &st.ctr->n_sh, sh[0] != 0, 2 * slot);
        warp_push(st.q_sh, &st.ctr->n_sh, sh[1] != 0, 2 * slot + 1);
    }
}

template <int KIND>
__global__ void __launch_bounds__(128) k_shade_surface(WfScene S, WfParams P, WfState st, int cur) {
    const int n = st.ctr->n_mat[KIND];
    const int* __restrict__ q = st.q_mat + (size_t)KIND * P.n_slots;
    const int nxt = cur ^ 1;
    const bool has_env = S.env_kind == TPT_ENV_MAP;
    const int stride = gridDim.x * blockDim.x;
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
        const int i = base + (int)lane_id();
        bool cont = false, term = false, need_task = false, finished = false;
        int slot = 0;
        int sh_env = 0, sh_area = 0;
        if (i < n) {
            slot = q[i];
            const float3 ro = f3(lds(&st.ray_o[slot])), rd = f3(lds(&st.ray_d[slot]));
            const float4 sp4 = st.surf_p[slot], sn4 = st.surf_n[slot];
            const float3 hp = f3(sp4), ng = f3(sn4);
            const float4 h4 = lds(&st.hit[slot]);
            const int prim = fbits(h4.y), inst = fbits(h4.z);
            const int mid = fbits(sn4.w);
            const float4 b4 = lds(&st.beta[slot]);
            float3 beta = f3(b4);
            float last_pdf = b4.w;
            const float4 r4 = lds(&st.rad[slot]);
            float3 L = f3(r4);
            float ptime = r4.w;
            int4 m;
            uint64_t rng;
            load_path(st, slot, m, rng);
            int fl = m.z;
            const MaterialF32 mt = S.mats[mid];
            const float3 mc = f3(mt.c);
            bool done = false;
            {
                {
                    const bool entering = dot(ng, rd) < 0.0f;
                    const float3 n = entering ? ng : -ng;
                    const float3 wo = -rd;
                    if (KIND != TPT_MAT_METAL && KIND != TPT_MAT_DIELECTRIC) {
                        if (has_env) {  // nee_environment (:148-172)
                            float3 wi, li;
                            float pe;
                            env_sample_dir(S, rng, wi, li, pe);
                            const float c = fmaxf(dot(n, wi), 0.0f);
                            if (c > 0.0f && pe > 0.0f) {
                                float3 f;
                                float pb;
                                mat_eval(mt, wo, wi, n, f, pb);
                                const float3 contrib = beta * f * li * (c * mis(pe, pb) / pe);
                                if (contrib.x > 0.0f || contrib.y > 0.0f || contrib.z > 0.0f) {
                                    const float3 so = hp + wi * kEps;
                                    sts(&st.sh_o[2 * slot], make_float4(so.x, so.y, so.z, kTMax));
                                    sts(&st.sh_d[2 * slot], make_float4(wi.x, wi.y, wi.z, ifloat(prim)));
                                    sts(&st.sh_c[2 * slot], make_float4(contrib.x, contrib.y, contrib.z, ifloat(inst)));
                                    sh_env = 1;
                                    fl |= F_PEND_ENV;
                                }
                            }
                        }
                        float3 lp, le;
                        float lpdf;
                        int lidx;
                        double lud, lvd;
                        if (sample_light(S, rng, hp, lp, le, lpdf, lidx, lud, lvd)) {  // nee_area_light (:178-213)
                            const float3 tl = lp - hp;
                            const float dist = length(tl);
                            if (dist > 1e-6f) {
                                const float3 wi = tl / dist;
                                const float c = fmaxf(dot(n, wi), 0.0f);
                                if (c > 0.0f && !ref_light_self_occluded(S.lights64, S.spheres64, S.inst64, lidx, ro, rd, h4.x, lud, lvd, (double)ptime)) {
                                    float3 f;
                                    float pb;
                                    mat_eval(mt, wo, wi, n, f, pb);
                                    const float3 contrib = beta * f * le * (c * mis(lpdf, pb) / lpdf);
                                    if (contrib.x > 0.0f || contrib.y > 0.0f || contrib.z > 0.0f) {
                                        const float3 so = hp + wi * kEps;
                                        // stops 1e-4 short of the light: the light itself is
                                        // handled by ref_light_self_occluded
                                        sts(&st.sh_o[2 * slot + 1], make_float4(so.x, so.y, so.z, fmaxf(dist - 2.0f * kEps, kEps)));
                                        sts(&st.sh_d[2 * slot + 1], make_float4(wi.x, wi.y, wi.z, ifloat(prim)));
                                        sts(&st.sh_c[2 * slot + 1], make_float4(contrib.x, contrib.y, contrib.z, ifloat(inst)));
                                        sh_area = 1;
                                        fl |= F_PEND_AREA;
                                    }
                                }
                            }
                        }
                    }
                    // Material::sample (src/material.rs:76-201)
                    float3 nd = f3(0, 0, 0), w = f3(0, 0, 0), no = hp;
                    float pdf = 0.0f;
                    bool delta = false, ok = true, self_ok = true;
                    switch (KIND) {
                        case TPT_MAT_LAMBERT:
                            nd = cos_hemi(n, rng);
                            w = mc;
                            pdf = fmaxf(dot(n, nd), 0.0f) / kPi;
                            break;
                        case TPT_MAT_METAL:
                            nd = rd - n * (2.0f * dot(rd, n));
                            w = mc;
                            delta = true;
                            break;
                        case TPT_MAT_DIELECTRIC: {
                            const float ior = mt.c.w;
                            const float eta = entering ? 1.0f / ior : ior;
                            const float ci = fmaxf(dot(wo, n), 0.0f);
                            const float fq = (ior - 1.0f) / (ior + 1.0f);
                            const float f0 = fq * fq;
                            const float fr = f0 + (1.0f - f0) * pow5(1.0f - ci);
                            float3 bt = f3(1, 1, 1);
                            if (!entering) {
                                const float dist = fmaxf(h4.x, 0.0f);
                                bt = f3(__expf(-mc.x * dist), __expf(-mc.y * dist), __expf(-mc.z * dist));
                            }
                            const float cosi = fminf(fmaxf(dot(wo, n), -1.0f), 1.0f);
                            const float sin2t = eta * eta * (1.0f - cosi * cosi);
                            const bool has_refr = !(sin2t >= 1.0f);
                            const bool refl = !has_refr || pcg_f32(rng) < fr;
                            if (refl) {
                                nd = rd - n * (2.0f * dot(rd, n));
                                bt = bt * (fr / fmaxf(fr, 1e-6f));
                            } else {
                                nd = rd * eta + n * (eta * cosi - sqrtf(1.0f - sin2t));
                                bt = bt * ((1.0f - fr) / fmaxf(1.0f - fr, 1e-6f)) * (eta * eta);
                            }
                            w = bt;
                            delta = true;
                            break;
                        }
                        case TPT_MAT_GGX: {
                            GgxSample gs;
                            if (!ggx_sample(rd, n, mt, rng, gs)) { ok = false; break; }
                            nd = gs.nd;
                            w = gs.w;
                            pdf = gs.pdf;
                            break;
                        }
                        case TPT_MAT_SUBSURFACE: {
                            const float sc = fmaxf(mt.c.w, 1e-4f);
                            const float u = fmaxf(pcg_f32(rng), 1e-12f);
                            const float dist = -__logf(u) * sc;
                            nd = cos_hemi(ng, rng);  // unoriented normal (material.rs:187-188)
                            w = mc * __expf(-dist / sc);
                            no = hp - ng * dist;
                            pdf = fmaxf(dot(n, nd), 0.0f) / kPi;
                            self_ok = false;     // origin moved off the surface
                            break;
                        }
                        default:
                            ok = false;
                    }
                    if (!ok) {
                        done = true;
                    } else {
                        beta = beta * w;
                        last_pdf = pdf;
                        fl = delta ? (fl & ~F_LAST_ND) : (fl | F_LAST_ND);
                        const float3 o2 = no + nd * kEps;
                        sts(&st.ray_o[slot], make_float4(o2.x, o2.y, o2.z, ifloat(self_ok ? prim : -1)));
                        sts(&st.ray_d[slot], make_float4(nd.x, nd.y, nd.z, ifloat(self_ok ? inst : -1)));
                        m.y += 1;
                        if (m.y >= P.max_bounces) done = true;  // bounce loop bound (:67)
                    }
                }
            }
            if (done && !sh_env && !sh_area) {
                cont = finish_sample(S, P, st, slot, m, fl, L, beta, last_pdf, ptime, rng, need_task, film_of(st), 0);
                finished = true;
            } else {
                cont = !done;
                term = done;
            }
            sts(&st.beta[slot], make_float4(beta.x, beta.y, beta.z, last_pdf));
            sts(&st.rad[slot], make_float4(L.x, L.y, L.z, ptime));
            m.z = fl;
            store_path(st, slot, m, rng);
        }
        if (take_next_task<false>(S, P, st, slot, need_task)) cont = true;
        if (i < n) st.act[slot] = cont ? 1 : 0;
        if (!P.ordered_queue) warp_push(st.q_ext[nxt], &st.ctr->n_ext[nxt], cont, slot);
        warp_push(st.q_term, &st.ctr->n_term, term, slot);
        warp_push(st.q_sh, &st.ctr->n_sh, sh_env != 0, 2 * slot);
        warp_push(st.q_sh, &st.ctr->n_sh, sh_area != 0, 2 * slot + 1);
        warp_count(&st.ctr->n_done_in_shade, finished);
    }
}

// Samples that ended with shadow rays pending finish here, after k_shadow
// has resolved their visibility.
// The completion kernel's per-slot body (k_regen): a
// path that ended with shadow rays pending takes their results, then
// finish_sample.  Returns whether the slot traces on (the task's next
// camera ray); need_task when its task is done.
template <bool BATCH>
__device__ __forceinline__ bool regen_slot(const WfScene& S0, const WfParams& P0, const WfState& st, int slot,
                                           bool& need_task) {
    bool again = false;
    WfScene S = S0;
    WfParams P = P0;
    Film F = film_of(st);
    long long tbase = 0;
    if constexpr (BATCH) apply_job(P0.jobs[st.job[slot]], S, P, F, tbase);
    int4 m;
    uint64_t rng;
    load_path(st, slot, m, rng);
    int fl = m.z;
    const float4 r4 = lds(&st.rad[slot]);
    float ptime = r4.w;
    float3 L = take_pending(st, slot, fl, f3(r4));
    float3 beta = f3(1.0f, 1.0f, 1.0f);
    float last_pdf = 0.0f;
    again = finish_sample(S, P, st, slot, m, fl, L, beta, last_pdf, ptime, rng, need_task, F, tbase);
    if (again) sts(&st.beta[slot], make_float4(1.0f, 1.0f, 1.0f, 0.0f));
    sts(&st.rad[slot], make_float4(L.x, L.y, L.z, ptime));
    m.z = fl;
    store_path(st, slot, m, rng);
    return again;
}

template <bool BATCH>
__global__ void __launch_bounds__(128) k_regen(WfScene S0, WfParams P0, WfState st, int cur) {
    const int n = st.ctr->n_term;
    const int nxt = cur ^ 1;
    const int stride = gridDim.x * blockDim.x;
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
        const int i = base + (int)lane_id();
        bool again = false, need_task = false;
        int slot = 0;
        if (i < n) {
            slot = st.q_term[i];
            again = regen_slot<BATCH>(S0, P0, st, slot, need_task);
        }
        if (take_next_task<BATCH>(S0, P0, st, slot, need_task)) again = true;
        if (i < n) st.act[slot] = again ? 1 : 0;
        if (!P0.ordered_queue) warp_push(st.q_ext[nxt], &st.ctr->n_ext[nxt], again, slot);
    }
}

// Film of a multi-chunk render: each pixel's task sums added in task order
// (the reference merges task results in task-id order, src/render.rs:226-241).
// A render in chunk batches merges each batch onto the film the previous
// ones left: the same additions in the same order.
// ---- camera culling -------------------------------------------------------------
// A film pixel is "open" when no camera ray through it can reach a leaf of
// the top-level tree (a sphere group or an instance): then each of its
// samples is a camera ray that leaves the scene (src/integrator.rs:71-83 at
// bounce 0), and k_sky_tasks computes it without a trace.  The test is
// conservative: the pixel's footprint, widened by 1% of a pixel on every
// side, spans a pyramid from the pinhole; each side plane is turned outward
// by a bound on the FP32 error of camera_ray's direction (cull_may_hit)
// and every box is padded by 1e-5 of the coordinates' magnitude
// (far above the FP32 error of the trace kernels' slab tests), and a box is
// passed over only when one side plane has it wholly outside.  All in f64.
struct CullFrustum {
    double3 o;
    double3 n[4];  // unit inward side normals
    double sin_m;
    double o_mag;  // largest |o| component
};
__device__ __forceinline__ double3 dd3(float3 a) { return make_double3(a.x, a.y, a.z); }
__device__ __forceinline__ double3 dsub(double3 a, double3 b) { return make_double3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ double ddot(double3 a, double3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ double3 dcross(double3 a, double3 b) {
    return make_double3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
// Unnormalised camera direction at screen position (sx, sy), as camera_ray
// forms it before normalising.
__device__ __forceinline__ double3 cull_dir(const CameraF32& c, double sx, double sy) {
    const double hw = c.half_w, hh = c.half_h;
    return make_double3(-(double)c.w.x + c.u.x * (sx * hw) + c.v.x * (sy * hh),
                        -(double)c.w.y + c.u.y * (sx * hw) + c.v.y * (sy * hh),
                        -(double)c.w.z + c.u.z * (sx * hw) + c.v.z * (sy * hh));
}
// true when the box [lo, hi] lies wholly outside the frustum (padded).
__device__ __forceinline__ bool cull_outside(const CullFrustum& F, double3 lo, double3 hi) {
    const double mag = fmax(fmax(fmax(fabs(lo.x), fabs(hi.x)), fmax(fabs(lo.y), fabs(hi.y))), fmax(fabs(lo.z), fabs(hi.z)));
    const double pad = 1e-5 * (mag + F.o_mag) + 1e-30;
    const double3 c = make_double3(0.5 * (lo.x + hi.x), 0.5 * (lo.y + hi.y), 0.5 * (lo.z + hi.z));
    const double3 h = make_double3(0.5 * (hi.x - lo.x) + pad, 0.5 * (hi.y - lo.y) + pad, 0.5 * (hi.z - lo.z) + pad);
    const double3 co = dsub(c, F.o);
    const double3 far = make_double3(fabs(co.x) + h.x, fabs(co.y) + h.y, fabs(co.z) + h.z);
    const double reach = F.sin_m * sqrt(ddot(far, far));  // the outward turn at the box's farthest point
    for (int k = 0; k < 4; ++k) {
        const double3 n = F.n[k];
        const double s = ddot(n, co) + fabs(n.x) * h.x + fabs(n.y) * h.y + fabs(n.z) * h.z + reach;
        if (s < 0.0) return true;
    }
    return false;
}

// True when a camera ray through pixel (x, y) of a width x height film may
// reach a leaf of the top-level tree rooted at `root` (see above).  Lens
// cameras, and renders whose paths end before their first bounce, are
// never culled.
// What the primitives of a leaf code (not TPT_REF_NONE) leave to the walk
// of cull_may_hit: keep = true when they may be hit (spheres, triangles, a
// transformed instance), else the node to walk on (the mesh tree of an
// identity instance, which the traversal tests with the world ray, so its
// boxes are world boxes under the same slab test) or TPT_REF_NONE (an
// empty leaf or mesh: nothing to hit).
__device__ __forceinline__ int cull_leaf(const WfScene& S, int ref, bool& keep) {
    const uint32_t code = (uint32_t)(~ref), first = code >> 3, count = code & 7u;
    keep = false;
    if (count == 0u) return TPT_REF_NONE;  // an empty leaf (exit markers never sit in nodes)
    keep = true;
    if (count != 7u) return TPT_REF_NONE;  // spheres or triangles
    const int mw = __float_as_int(S.inst[first].wbox_min.w);
    if (!(mw & kInstIdentity)) return TPT_REF_NONE;
    const int mroot = S.meshes[mw & kInstMeshMask].root_ref;
    if (mroot < 0) {  // an empty mesh, or one leaf whose box the instance box was
        keep = mroot != TPT_REF_NONE;
        return TPT_REF_NONE;
    }
    keep = false;
    return mroot;
}

// Most nodes one pixel's walk visits; past them the pixel stays in the path pool.
constexpr int kCullMaxVisits = 1024;

__device__ bool cull_may_hit(const WfScene& S, const CameraF32& c, int root, int x, int y, int width, int height,
                             int max_bounces) {
    if (!(c.lens_radius == 0.0f && c.focus_dist > 0.0f && max_bounces > 0)) return true;
    // camera_ray: sx = (x + jx) * inv_w * 2 - 1, sy = 1 - (y + jy) * inv_h * 2, jx, jy in [0, 1)
    const double iw = (double)(1.0f / (float)width), ih = (double)(1.0f / (float)height);
    const double sx0 = ((double)x - 0.01) * iw * 2.0 - 1.0, sx1 = ((double)x + 1.01) * iw * 2.0 - 1.0;
    const double sy0 = 1.0 - ((double)y + 1.01) * ih * 2.0, sy1 = 1.0 - ((double)y - 0.01) * ih * 2.0;
    const double3 d[4] = {cull_dir(c, sx0, sy0), cull_dir(c, sx1, sy0), cull_dir(c, sx1, sy1), cull_dir(c, sx0, sy1)};
    const double3 mid = cull_dir(c, 0.5 * (sx0 + sx1), 0.5 * (sy0 + sy1));
    CullFrustum F;
    F.o = dd3(c.o);
    F.o_mag = fmax(fmax(fabs(F.o.x), fabs(F.o.y)), fabs(F.o.z));
    // FP32 error bound of camera_ray's direction: a few ulps of the screen
    // basis, and of (o + base * focus_dist) - o relative to focus_dist
    F.sin_m = sin(1e-5 + 4e-6 * (1.0 + F.o_mag / (double)c.focus_dist));
    for (int k = 0; k < 4; ++k) {
        double3 n = dcross(d[k], d[(k + 1) & 3]);
        const double len = sqrt(ddot(n, n));
        if (!(len > 0.0)) return true;  // degenerate footprint: keep the pixel
        n = make_double3(n.x / len, n.y / len, n.z / len);
        if (ddot(n, mid) < 0.0) n = make_double3(-n.x, -n.y, -n.z);
        F.n[k] = n;
    }
    if (root == TPT_REF_NONE) return false;
    int ref = root;
    if (root < 0) {  // a single leaf at the root: the bounds of its instance or spheres
        const uint32_t code = (uint32_t)(~root), first = code >> 3, count = code & 7u;
        double3 lo, hi;
        if (count == 7u) {
            const InstanceF32& I = S.inst[first];
            lo = make_double3(I.wbox_min.x, I.wbox_min.y, I.wbox_min.z);
            hi = make_double3(I.wbox_max.x, I.wbox_max.y, I.wbox_max.z);
            if (!(lo.x <= hi.x)) return false;  // an empty mesh
            if (cull_outside(F, lo, hi)) return false;
            bool keep;
            ref = cull_leaf(S, root, keep);
            if (keep) return true;
            if (ref == TPT_REF_NONE) return false;
        } else {
            lo = make_double3(INFINITY, INFINITY, INFINITY);
            hi = make_double3(-INFINITY, -INFINITY, -INFINITY);
            for (uint32_t k = first; k < first + count; ++k) {
                const float4 cr = S.spheres[k].cr;
                const double r = fabs((double)cr.w);
                lo = make_double3(fmin(lo.x, cr.x - r), fmin(lo.y, cr.y - r), fmin(lo.z, cr.z - r));
                hi = make_double3(fmax(hi.x, cr.x + r), fmax(hi.y, cr.y + r), fmax(hi.z, cr.z + r));
            }
            return !cull_outside(F, lo, hi);
        }
    }
    int stack[64];
    int sp = 0;
    for (int visits = 1;; ++visits) {
        if (visits > kCullMaxVisits) return true;
        const BvhNode2 nd = S.nodes[ref];
        const double3 lo0 = make_double3(fmin(nd.lx.x, nd.lx.y), fmin(nd.lx.z, nd.lx.w), fmin(nd.zz.x, nd.zz.y));
        const double3 hi0 = make_double3(fmax(nd.lx.x, nd.lx.y), fmax(nd.lx.z, nd.lx.w), fmax(nd.zz.x, nd.zz.y));
        const double3 lo1 = make_double3(fmin(nd.rx.x, nd.rx.y), fmin(nd.rx.z, nd.rx.w), fmin(nd.zz.z, nd.zz.w));
        const double3 hi1 = make_double3(fmax(nd.rx.x, nd.rx.y), fmax(nd.rx.z, nd.rx.w), fmax(nd.zz.z, nd.zz.w));
        const int r[2] = {nd.refs.x, nd.refs.y};
        const bool in[2] = {r[0] != TPT_REF_NONE && !cull_outside(F, lo0, hi0),
                            r[1] != TPT_REF_NONE && !cull_outside(F, lo1, hi1)};
        for (int k = 0; k < 2; ++k) {
            if (!in[k]) continue;
            int next = r[k];
            if (next < 0) {  // a leaf's box
                bool keep;
                next = cull_leaf(S, next, keep);
                if (keep) return true;
                if (next == TPT_REF_NONE) continue;
            }
            if (sp == 64) return true;  // deeper than the walk keeps: keep the pixel
            stack[sp++] = next;
        }
        if (sp == 0) return false;
        ref = stack[--sp];
    }
}

// One thread per film pixel (a multi-job render: per pixel of all jobs,
// numbered job after job): may[j] = 1 when a camera ray through pixel j
// may reach a top-level leaf, open[j] = 1 otherwise.
template <bool BATCH>
__global__ void k_cull_classify(WfScene S, WfParams P, uint8_t* __restrict__ may, uint8_t* __restrict__ open) {
    const long long gp = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool hit;
    if constexpr (BATCH) {
        if (gp >= P.total_pixels) return;
        const WfJob& J = P.jobs[job_at(P, gp, [](const WfJob& x) { return x.pixel_begin; })];
        const int j = (int)(gp - J.pixel_begin);
        const int row = (int)fdiv(J.w_div, (uint32_t)j);
        hit = cull_may_hit(S, J.cam, J.top_root, j - row * J.width, J.row_begin + row * J.row_step, J.width, J.height,
                           J.max_bounces);
    } else {
        if (gp >= P.n_pixels) return;
        const int j = (int)gp;
        const int row = (int)fdiv(P.w_div, (uint32_t)j);
        hit = cull_may_hit(S, S.cam, S.top_root, j - row * P.width, P.row_begin + row * P.row_step, P.width, P.height,
                           P.max_bounces);
    }
    may[gp] = hit ? 1 : 0;
    open[gp] = hit ? 0 : 1;
}

// Multi-job renders, one block: each job's stretch of the two compacted
// pixel lists (batch-wide pixel ids, ascending), then, job after job, the
// first pool fetch id and the first sky task of each job.  out[0] / out[1]
// = the fetch ids / sky tasks of the whole batch.
__device__ __forceinline__ int lower_bound_int(const int* __restrict__ a, int n, long long key) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((long long)a[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}
__global__ void __launch_bounds__(1024) k_cull_jobs(WfJob* jobs, int n_jobs, const int* __restrict__ may_list,
                                                    const int* __restrict__ open_list, const int* __restrict__ counts,
                                                    long long* out) {
    const int n_may = counts[0], n_open = counts[1];
    for (int k = threadIdx.x; k < n_jobs; k += blockDim.x) {
        WfJob& J = jobs[k];
        J.geo_begin = lower_bound_int(may_list, n_may, J.pixel_begin);
        J.n_geo = lower_bound_int(may_list, n_may, J.pixel_begin + J.n_pixels) - J.geo_begin;
        J.sky_begin = lower_bound_int(open_list, n_open, J.pixel_begin);
        J.n_sky = lower_bound_int(open_list, n_open, J.pixel_begin + J.n_pixels) - J.sky_begin;
        J.geo_div = make_fastdiv((uint32_t)(J.n_geo > 0 ? J.n_geo : 1));
        J.sky_div = make_fastdiv((uint32_t)(J.n_sky > 0 ? J.n_sky : 1));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        long long f = 0, u = 0;
        for (int k = 0; k < n_jobs; ++k) {
            WfJob& J = jobs[k];
            J.fetch_begin = f;
            J.sky_task_begin = u;
            f += (long long)J.n_chunks * J.n_geo;
            u += (long long)J.n_chunks * J.n_sky;
        }
        out[0] = f;
        out[1] = u;
    }
}

// One thread per task of an open pixel (single renders: in the current
// chunk batch, chunk by chunk, the open pixels in film order; multi-job
// renders: job after job): the task's samples exactly as the pool would
// run them -- the stream from seed_for(x, y, sample_start) ^ seed, per
// sample camera_ray, the background at bounce 0 (beta = 1, no MIS),
// clamp_lum, the f64 sums in sample order -- then the film (one task per
// pixel) or the task's partial sums, like finish_sample.
template <bool BATCH>
__global__ void k_sky_tasks(WfScene S0, WfParams P0, WfState st, const int* __restrict__ open_map, int n_open,
                            FastDiv open_div, long long count) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long done = 0;
    if (v < count) {
        WfScene S = S0;
        WfParams P = P0;
        Film F = film_of(st);
        long long task, base = 0;
        int pixel;
        if constexpr (BATCH) {
            const WfJob& J = P0.jobs[job_at(P0, v, [](const WfJob& x) { return x.sky_task_begin; })];
            apply_job(J, S, P, F, base);
            const uint32_t w = (uint32_t)(v - J.sky_task_begin);
            const uint32_t c = fdiv(J.sky_div, w);
            pixel = (int)(__ldg(open_map + J.sky_begin + (w - c * (uint32_t)J.n_sky)) - J.pixel_begin);
            task = J.task_begin + (long long)c * J.n_pixels + pixel;
        } else {
            const uint32_t c = fdiv(open_div, (uint32_t)v);
            pixel = __ldg(open_map + ((uint32_t)v - c * (uint32_t)n_open));
            task = P.task_first + (long long)c * P.n_pixels + pixel;
        }
        const TaskPos tp = task_pos(P, task - base);
        const int row = (int)fdiv(P.w_div, (uint32_t)pixel);
        const int x = pixel - row * P.width, y = P.row_begin + row * P.row_step;
        uint64_t rng = task_seed((uint32_t)x, (uint32_t)y, (uint32_t)tp.sample_start, P.seed);
        double4 a = make_double4(0.0, 0.0, 0.0, 0.0);
        double4 q = make_double4(0.0, 0.0, 0.0, 0.0);
        for (int k = 0; k < tp.len; ++k) {
            float3 o, d;
            float time;
            camera_ray(S.cam, x, y, 1.0f / (float)P.width, 1.0f / (float)P.height, rng, o, d, time);
            const float3 L = clamp_lum(f3(1.0f, 1.0f, 1.0f) * background(S, d), 50.0f);
            a.x += (double)L.x; a.y += (double)L.y; a.z += (double)L.z; a.w += 1.0;
            q.x += (double)L.x * (double)L.x; q.y += (double)L.y * (double)L.y; q.z += (double)L.z * (double)L.z;
        }
        if (P.n_chunks == 1) {
            const size_t px = (size_t)pixel;
            F.acc[3 * px] = a.x; F.acc[3 * px + 1] = a.y; F.acc[3 * px + 2] = a.z;
            F.acc_w[px] = a.w;
            if (F.acc_sq) { F.acc_sq[3 * px] = q.x; F.acc_sq[3 * px + 1] = q.y; F.acc_sq[3 * px + 2] = q.z; }
        } else {
            st.part[task - P0.task_first] = a;
            if (st.part_sq) st.part_sq[task - P0.task_first] = q;
        }
        done = (unsigned long long)tp.len;
    }
    for (int off = 16; off > 0; off >>= 1) done += __shfl_down_sync(0xffffffffu, done, off);
    if (lane_id() == 0 && done) atomicAdd(&st.ctr->sky_samples, done);  // beside k_step: its own counter
}

// Whole paths in one kernel: every lane carries a path in registers from its
// first camera ray to the end of its task, then takes the next one.  A round
// of the block is: the bounce of the closest hits, in step (bounce<true>),
// finished samples and new ones, then the rays -- the bounce's shadow rays
// and the next closest-hit ray -- until no lane of the warp waits.  The steps
// and their order are the wavefront kernels', so the film is the same.
//
// TASKS: small renders, from the pool's tasks, instead of the bounce loop and
// its launches (wf_render decides).  `open`, when given, flags the film's
// pixels (all jobs') whose camera rays leave the scene: their samples are
// not traced (camera culling, counted in sky_samples).  Otherwise the end of
// a bounce loop, once every task has been taken: the live slots of the queue
// the last iteration left, q_ext[0].
//
// `lanes` lanes of each warp take work.  A task whose path outlives
// P.max_iters rounds is dropped (TPT_FLAG_ITER_LIMIT).
//
// Bound by the latency of each path's chain of rays at these sizes, and by
// instruction fetch (the block's warps share it, as in k_shade).  3 blocks per
// SM: 2 trace larger renders 20% slower, 4 spill 330 B (allocation-free 96x96 x
// 16 spp 0.80 ms at 3, 0.92 at 4).  As the end of a loop it replaces a kernel
// of one thread per slot that kept the path in memory: batch of 10 scenes 36.4
// -> 33.1 ms, adaptive Cornell film 480x270 23.1 -> 22.2 ms.
constexpr int kPathsBlock = 128;
template <bool BATCH, bool TASKS, bool SHARED_STACK>
__global__ void __launch_bounds__(kPathsBlock, 3) k_paths(WfScene S0, WfParams P0, WfState st,
                                                      const uint8_t* __restrict__ open, unsigned lanes) {
    __shared__ int sstack[SHARED_STACK ? kSharedStack * kPathsBlock : 1];
    int lstack[SHARED_STACK ? 1 : kStack];
    using Stack = typename std::conditional<SHARED_STACK, TStack<kPathsBlock, kSharedStack>, TStack<1, kStack>>::type;
    const Stack stack{SHARED_STACK ? sstack + threadIdx.x : lstack};
    int* flags = &st.ctr->flags;
    const long long n_items = TASKS ? fetch_end(P0) - P0.task_first : st.ctr->n_ext[0];
    unsigned long long samples = 0, rays_c = 0, rays_s = 0, sky_samples = 0;
    constexpr int kEnv = 1, kArea = 2, kClosest = 4;
    PathRegs p{};
    Sums sums = zero_sums();
    float3 sh_o[2] = {}, sh_d[2] = {}, sh_c[2] = {};
    float sh_t = 0.0f;
    int sh_prim = -1, sh_inst = -1;
    int job = 0, jobs = 0;
    long long visits = 0;
    bool alive = false, ended = false, sky_task = false, exhausted = lane_id() >= lanes;
    // taken anew at each use, so that no job's fields wait in registers
    auto view = [&](int j) { return view_of<BATCH>(S0, P0, st, j); };
    for (;;) {
        const bool shade = alive && !ended;
        if (shade) {
            sh_prim = p.prim;
            sh_inst = p.inst;
        }
        const View v = view(job);  // (a lane without a task: its last job's, or job 0's)
        const bool done = bounce<true>(v.S, v.P, p, shade, [&](int k, float3 so, float tmax, float3 wi, float3 contrib) {
            if (k == 0) { sh_o[0] = so; sh_d[0] = wi; sh_c[0] = contrib; }
            else { sh_o[1] = so; sh_d[1] = wi; sh_c[1] = contrib; sh_t = tmax; }
            jobs |= k == 0 ? kEnv : kArea;
        }, [&](float3 o, float3 d, int self_prim, int self_inst) {
            p.o = o;
            p.d = d;
            p.self_prim = self_prim;
            p.self_inst = self_inst;
        });
        if (shade) {
            if (done) ended = true;
            else jobs |= kClosest;
            if (++visits >= P0.max_iters) {
                raise_flag(flags, TPT_FLAG_ITER_LIMIT);
                alive = false;
                jobs = 0;
            }
        }
        bool camera = false;
        TaskPos tp{};
        if (alive && ended && jobs == 0) {  // the sample is complete
            const View v = view(job);
            tp = task_pos(v.P, (long long)p.m.w - v.task_begin);
            bool task_done = false;
            camera = finish_sums(v.P, st, p.m, p.L, task_done, v.F, tp, sums);
            if (sky_task) ++sky_samples;
            else ++samples;
            alive = !task_done;
        }
        const bool want = !alive && !exhausted;
        const unsigned wm = __ballot_sync(0xffffffffu, want);
        if (wm) {
            const int leader = __ffs(wm) - 1;
            long long base = 0;
            if ((int)lane_id() == leader)
                base = (long long)atomicAdd((unsigned long long*)&st.ctr->next_item, (unsigned long long)__popc(wm));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (want) {
                const long long k = base + __popc(wm & ((1u << lane_id()) - 1u));
                exhausted = k >= n_items;
                if (!exhausted) {
                    alive = true;
                    visits = 0;
                    if constexpr (TASKS) {
                        const long long task = task_of_fetch(P0, P0.task_first + k);
                        long long pixel0 = 0;
                        if constexpr (BATCH) {
                            job = find_job(P0, task);
                            pixel0 = P0.jobs[job].pixel_begin;
                        }
                        const View v = view(job);
                        tp = task_pos(v.P, task - v.task_begin);
                        p.m = make_int4(0, 0, 0, (int)task);
                        sums = zero_sums();
                        sky_task = open && open[pixel0 + tp.pixel];
                        camera = true;
                    } else {
                        const int slot = st.q_ext[0][k];
                        if constexpr (BATCH) job = st.job[slot];
                        p = load_slot(st, slot);
                        sums = load_sums(st, slot, p.m.x == 0);
                        ended = false;
                        jobs = kClosest;
                    }
                }
            }
        }
        if (camera) {
            const View v = view(job);
            start_sample(v.S, v.P, tp, p);
            p.t = kTMax;
            p.prim = p.inst = -1;
            ended = false;
            if (!sky_task) jobs = kClosest;
        }
        if (!__syncthreads_or(alive || !exhausted)) break;
        while (__any_sync(0xffffffffu, jobs != 0)) {
            if (jobs != 0) {
                const int j = jobs & -jobs;
                const bool any = j != kClosest;
                int root = S0.top_root;
                if constexpr (BATCH) root = __ldg(&P0.jobs[job].top_root);
                Tracer T;
                TraceCount cnt;
                tracer_start_at(root, T, j == kEnv ? sh_o[0] : (j == kArea ? sh_o[1] : p.o),
                                j == kEnv ? sh_d[0] : (j == kArea ? sh_d[1] : p.d), j == kArea ? sh_t : kTMax,
                                any ? sh_prim : p.self_prim, any ? sh_inst : p.self_inst);
                while (!tracer_run<false>(S0, T, stack, kEps, 1 << 30, flags, cnt, any)) {
                }
                if (any) {
                    ++rays_s;
                    if (T.hit_prim < 0) p.L = p.L + (j == kEnv ? sh_c[0] : sh_c[1]);
                } else {
                    ++rays_c;
                    p.t = T.hit_prim >= 0 ? T.tmax : kTMax;
                    p.prim = T.hit_prim;
                    p.inst = T.hit_inst;
                }
                jobs ^= j;
            }
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        samples += __shfl_down_sync(0xffffffffu, samples, off);
        rays_c += __shfl_down_sync(0xffffffffu, rays_c, off);
        rays_s += __shfl_down_sync(0xffffffffu, rays_s, off);
        sky_samples += __shfl_down_sync(0xffffffffu, sky_samples, off);
    }
    if (lane_id() == 0) {
        if (samples) atomicAdd(&st.ctr->samples, samples);
        if (rays_c) atomicAdd(&st.ctr->rays_closest, rays_c);
        if (rays_s) atomicAdd(&st.ctr->rays_shadow, rays_s);
        if (sky_samples) atomicAdd(&st.ctr->sky_samples, sky_samples);
    }
}

__global__ void k_merge(WfParams P, WfState st) {
    const int px = blockIdx.x * blockDim.x + threadIdx.x;
    if (px >= P.n_pixels) return;
    const int c0 = (int)(P.task_first / P.n_pixels), c1 = (int)(P.n_tasks / P.n_pixels);
    double ax = 0.0, ay = 0.0, az = 0.0, aw = 0.0, qx = 0.0, qy = 0.0, qz = 0.0;
    if (c0 > 0) {
        ax = st.acc[3 * (size_t)px]; ay = st.acc[3 * (size_t)px + 1]; az = st.acc[3 * (size_t)px + 2];
        aw = st.acc_w[px];
        if (st.acc_sq) { qx = st.acc_sq[3 * (size_t)px]; qy = st.acc_sq[3 * (size_t)px + 1]; qz = st.acc_sq[3 * (size_t)px + 2]; }
    }
    for (int k = c0; k < c1; ++k) {
        const long long t = (long long)(k - c0) * P.n_pixels + px;
        const double4 a = st.part[t];
        ax += a.x; ay += a.y; az += a.z; aw += a.w;
        if (st.acc_sq) {
            const double4 q = st.part_sq[t];
            qx += q.x; qy += q.y; qz += q.z;
        }
    }
    st.acc[3 * (size_t)px] = ax; st.acc[3 * (size_t)px + 1] = ay; st.acc[3 * (size_t)px + 2] = az;
    st.acc_w[px] = aw;
    if (st.acc_sq) { st.acc_sq[3 * (size_t)px] = qx; st.acc_sq[3 * (size_t)px + 1] = qy; st.acc_sq[3 * (size_t)px + 2] = qz; }
}

// End of an iteration: statistics, queue reset, loop condition.
// Batch films: one thread per pixel of all jobs (pixels numbered job after job).
__global__ void k_merge_batch(WfParams P, WfState st) {
    const long long gp = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gp >= P.total_pixels) return;
    int lo = 0, hi = P.n_jobs;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (P.jobs[mid].pixel_begin <= gp) lo = mid; else hi = mid;
    }
    const WfJob& J = P.jobs[lo];
    const long long px = gp - J.pixel_begin;
    if (J.n_chunks == 1) return;  // one task per pixel: finish_sample wrote the film
    double ax = 0.0, ay = 0.0, az = 0.0, aw = 0.0;
    for (int k = 0; k < J.n_chunks; ++k) {
        const double4 a = st.part[J.task_begin + (long long)k * J.n_pixels + px];
        ax += a.x; ay += a.y; az += a.z; aw += a.w;
    }
    J.acc[3 * px] = ax; J.acc[3 * px + 1] = ay; J.acc[3 * px + 2] = az;
    J.acc_w[px] = aw;
}

// ---- adaptive renders in rounds -------------------------------------------------
// Round r renders samples [sample_base, sample_end) of every film pixel still
// sampling (active list, n of them) as ordinary tasks and stores each
// sample's radiance.  This kernel then runs the reference's per-pixel loop
// (src/render.rs:143-180) over those samples in sample order: each joins the
// f64 film sums, the Welford statistics of its luminance are updated, and
// after min_spp samples the pixel stops once the sample relative standard
// deviation sqrt(m2 / (n - 1)) / max(|mean|, 1e-4) is below the threshold.
// A pixel that has not stopped goes to the next round's active list.  The
// sums, counts and the stopping decision are those of one loop over the
// pixel's samples; only the streams differ from the reference's (each task
// of task_spp samples starts at seed_for(x, y, sample_start) ^ seed).
__global__ void k_round_merge(WfParams P, WfState st, const int* __restrict__ active, int n, double4* wstate,
                              int* next_active, int* n_next, unsigned long long* taken) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    bool keep = false;
    int px = 0;
    unsigned long long used = 0;
    if (j < n) {
        px = active[j];
        double4 w = wstate[px];  // n, mean, m2, (unused)
        double ax = st.acc[3 * (size_t)px], ay = st.acc[3 * (size_t)px + 1], az = st.acc[3 * (size_t)px + 2];
        double aw = st.acc_w[px];
        double qx = 0.0, qy = 0.0, qz = 0.0;
        if (st.acc_sq) { qx = st.acc_sq[3 * (size_t)px]; qy = st.acc_sq[3 * (size_t)px + 1]; qz = st.acc_sq[3 * (size_t)px + 2]; }
        const int min_spp = min(max(P.adaptive_min_spp, 1), max(P.spp, 1));
        const float4* smp = st.rsamp + (size_t)j * P.round_len;
        const int len = P.sample_end - P.sample_base;
        bool stop = false;
        for (int k = 0; k < len && !stop; ++k, ++used) {
            const float4 L = smp[k];
            ax += (double)L.x; ay += (double)L.y; az += (double)L.z; aw += 1.0;
            if (st.acc_sq) {
                qx += (double)L.x * (double)L.x; qy += (double)L.y * (double)L.y; qz += (double)L.z * (double)L.z;
            }
            w.x += 1.0;
            const double l = 0.2126 * (double)L.x + 0.7152 * (double)L.y + 0.0722 * (double)L.z;
            const double delta = l - w.y;
            w.y += delta / w.x;
            w.z += delta * (l - w.y);
            if (w.x >= (double)min_spp && w.x > 1.0) {
                const double var = w.z / (w.x - 1.0);
                if (sqrt(var) / fmax(fabs(w.y), 1e-4) < P.adaptive_threshold) stop = true;
            }
        }
        wstate[px] = w;
        st.acc[3 * (size_t)px] = ax; st.acc[3 * (size_t)px + 1] = ay; st.acc[3 * (size_t)px + 2] = az;
        st.acc_w[px] = aw;
        if (st.acc_sq) { st.acc_sq[3 * (size_t)px] = qx; st.acc_sq[3 * (size_t)px + 1] = qy; st.acc_sq[3 * (size_t)px + 2] = qz; }
        keep = !stop && P.sample_end < P.spp;
    }
    warp_push(next_active, n_next, keep, px);
    for (int off = 16; off > 0; off >>= 1) used += __shfl_down_sync(0xffffffffu, used, off);
    if (lane_id() == 0 && used) atomicAdd(taken, used);
}

// Round 0: every film pixel active, film and statistics zero.
__global__ void k_round_init(int n_pixels, int* active, double4* wstate, double* acc, double* acc_w, double* acc_sq) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pixels) return;
    active[i] = i;
    wstate[i] = make_double4(0.0, 0.0, 0.0, 0.0);
    acc[3 * (size_t)i] = 0.0; acc[3 * (size_t)i + 1] = 0.0; acc[3 * (size_t)i + 2] = 0.0;
    acc_w[i] = 0.0;
    if (acc_sq) { acc_sq[3 * (size_t)i] = 0.0; acc_sq[3 * (size_t)i + 1] = 0.0; acc_sq[3 * (size_t)i + 2] = 0.0; }
}

// ---- ordered extension queue ----------------------------------------------------
// After an iteration the live slots (act byte 1) are compacted, in slot
// order, into the next iteration's extension queue: per 16384-slot span a
// count, one block's exclusive scan of the counts, and a scatter.  The
// kernels then visit only live slots, consecutive lanes on ascending slots.
// A thread covers 64 consecutive act bytes (four 16-byte loads in flight).
constexpr int kCmpBlock = 256, kCmpPerThread = 64, kCmpSpan = kCmpBlock * kCmpPerThread;
constexpr int kCmpScanTiles = 16;  // the scan prefetches up to 16 x 1024 counts (2^28 slots)

// Live-slot bits of slots [t0, t0 + 64) (bit k = slot t0 + k).
__device__ __forceinline__ unsigned long long live_bits(const uint8_t* __restrict__ act, int n, int t0) {
    unsigned long long bits = 0;
    if (t0 + kCmpPerThread <= n) {
        const uint4* a = reinterpret_cast<const uint4*>(act + t0);  // t0 is a multiple of 64
        uint4 v[4];
        for (int k = 0; k < 4; ++k) v[k] = a[k];
        for (int k = 0; k < 4; ++k) {
            const unsigned w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
            for (int q = 0; q < 4; ++q)
                for (int b = 0; b < 4; ++b)
                    if ((w[q] >> (8 * b)) & 0xffu) bits |= 1ull << (16 * k + 4 * q + b);
        }
    } else {
        for (int k = 0; k < kCmpPerThread; ++k)
            if (t0 + k < n && act[t0 + k]) bits |= 1ull << k;
    }
    return bits;
}

// Exclusive prefix of v over the block's threads; *total gets the sum.
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        int ws = lane < nw ? warp_sums[lane] : 0;
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, ws, off);
            if (lane >= off) ws += y;
        }
        if (lane < nw) warp_sums[lane] = ws;  // inclusive per warp
    }
    __syncthreads();
    const int before = w > 0 ? warp_sums[w - 1] : 0;
    if (total) *total = warp_sums[(blockDim.x >> 5) - 1];
    const int excl = before + x - v;
    __syncthreads();  // warp_sums may be reused by the caller
    return excl;
}

__global__ void __launch_bounds__(kCmpBlock) k_cmp_count(const uint8_t* __restrict__ act, int n, int* counts) {
    __shared__ int ws[kCmpBlock / 32];
    const int t0 = blockIdx.x * kCmpSpan + threadIdx.x * kCmpPerThread;
    const int c = __popcll(live_bits(act, n, t0));
    int total = 0;
    block_exclusive_scan(c, ws, &total);
    if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

// One block of 1024: counts[0..nb) -> exclusive offsets in place; *n_out =
// the total.  The first 16 x 1024 counts are loaded at once (coalesced),
// then scanned tile by tile; any further tiles load one after another.
__global__ void __launch_bounds__(1024) k_cmp_scan(int* counts, int nb, int* n_out) {
    __shared__ int ws[32];
    int v[kCmpScanTiles];
#pragma unroll
    for (int k = 0; k < kCmpScanTiles; ++k) {
        const int i = k * 1024 + (int)threadIdx.x;
        v[k] = i < nb ? counts[i] : 0;
    }
    int run = 0;
#pragma unroll
    for (int k = 0; k < kCmpScanTiles; ++k) {
        if (k * 1024 >= nb) break;  // uniform over the block
        int total = 0;
        const int ex = block_exclusive_scan(v[k], ws, &total);
        const int i = k * 1024 + (int)threadIdx.x;
        if (i < nb) counts[i] = run + ex;
        run += total;
    }
    for (int b0 = kCmpScanTiles * 1024; b0 < nb; b0 += 1024) {
        const int i = b0 + (int)threadIdx.x;
        int total = 0;
        const int ex = block_exclusive_scan(i < nb ? counts[i] : 0, ws, &total);
        if (i < nb) counts[i] = run + ex;
        run += total;
    }
    if (threadIdx.x == 0) *n_out = run;
}

// The scatter takes its span in four rounds of 4096 slots (16 per thread,
// one 16-byte load): each round's live slot ids are ranked into shared
// memory, then written out by the whole block in consecutive addresses.
__global__ void __launch_bounds__(kCmpBlock) k_cmp_scatter(const uint8_t* __restrict__ act, int n,
                                                          const int* __restrict__ offsets, int* __restrict__ q) {
    constexpr int kRound = kCmpBlock * 16;
    __shared__ int ws[kCmpBlock / 32];
    __shared__ int stage[kRound];
    int out = offsets[blockIdx.x];
    for (int r = 0; r < kCmpSpan / kRound; ++r) {
        const int t0 = blockIdx.x * kCmpSpan + r * kRound + threadIdx.x * 16;
        unsigned bits = 0;
        if (t0 + 16 <= n) {
            const uint4 v = *reinterpret_cast<const uint4*>(act + t0);  // t0 is a multiple of 16
            const unsigned w[4] = {v.x, v.y, v.z, v.w};
            for (int q4 = 0; q4 < 4; ++q4)
                for (int b = 0; b < 4; ++b)
                    if ((w[q4] >> (8 * b)) & 0xffu) bits |= 1u << (4 * q4 + b);
        } else {
            for (int k = 0; k < 16; ++k)
                if (t0 + k < n && act[t0 + k]) bits |= 1u << k;
        }
        int total = 0;
        int pos = block_exclusive_scan(__popc(bits), ws, &total);  // ends with a barrier
        while (bits) {
            const int k = __ffs(bits) - 1;
            bits &= bits - 1;
            stage[pos++] = t0 + k;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < total; i += kCmpBlock) q[out + i] = stage[i];
        out += total;
        __syncthreads();  // stage is refilled next round
    }
}

__global__ void k_step(WfState st, int cur, long long max_iters, cudaGraphConditionalHandle handle, int use_cond,
                       long long fetch_end = 0, int tail_live = 0) {
    WfCounters* c = st.ctr;
    c->rays_closest += (unsigned long long)c->n_ext[cur];
    c->rays_shadow += (unsigned long long)c->n_sh;
    c->samples += (unsigned long long)c->n_term + (unsigned long long)c->n_done_in_shade;
    c->n_done_in_shade = 0;
    for (int k = 0; k < 5; ++k) c->n_mat[k] = 0;
    c->n_ext[cur] = 0;
    c->n_sh = 0;
    c->n_term = 0;
    c->fetch_ext = 0;
    c->fetch_sh = 0;
    c->iters += 1;
    bool more = c->n_ext[cur ^ 1] > 0;
    if (more && tail_live > 0 && c->n_ext[cur ^ 1] <= tail_live && c->next_task >= fetch_end) {
        c->tail = 1;  // the pool's tasks are all taken: k_paths finishes the few live slots
        more = false;
    }
    if (more && c->iters >= max_iters) {
        c->flags |= TPT_FLAG_ITER_LIMIT;
        more = false;
        c->n_ext[cur ^ 1] = 0;  // iterations a host loop has already enqueued find nothing to do
    }
    if (use_cond) cudaGraphSetConditional(handle, more ? 1u : 0u);
}

}  // namespace wf

// ---- buffers ---------------------------------------------------------------
namespace {
size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }
}

namespace {
// Frees the path-state block only (the adaptive-round arrays stay).
void release_state(WfBuffers& b) {
    if (b.block) cudaFree(b.block);
    b.block = nullptr;
    b.slots = 0;
    b.part_tasks = 0;
}
}  // namespace

cudaError_t wf_reserve(WfBuffers& b, size_t slots, size_t part_tasks) {
    if (b.block && b.slots >= slots && b.part_tasks >= part_tasks) return cudaSuccess;
    release_state(b);
    const size_t S = slots, T = part_tasks;
    // (entry 5 holds the two extension queues)
    size_t sz[] = {S * 16, S * 16, S * 16, S * 16, S * 16, 2 * S * 4, S * 16, 2 * S * 16, 2 * S * 16, 2 * S * 16,
                   S * 16, S * 1, 2 * S * 4, S * 4, sizeof(WfCounters), S * 32, S * 32, T * 32, T * 32,
                   S * 16, S * 16, 5 * S * 4, S * 4, wf_compact_spans(S) * 4};
    size_t total = 0;
    for (size_t s : sz) total += align_up(s);
    char* p = nullptr;
    cudaError_t e = cudaMalloc(&p, total);
    if (e != cudaSuccess) return e;
    b.block = p;
    b.slots = slots;
    b.part_tasks = part_tasks;
    size_t off = 0;
    auto take = [&](size_t bytes) { char* r = p + off; off += align_up(bytes); return (void*)r; };
    WfState& st = b.st;
    st.path = (int4*)take(sz[0]);
    st.ray_o = (float4*)take(sz[1]);
    st.ray_d = (float4*)take(sz[2]);
    st.beta = (float4*)take(sz[3]);
    st.rad = (float4*)take(sz[4]);
    st.q_ext[0] = (int*)take(sz[5]);
    st.q_ext[1] = st.q_ext[0] + S;
    st.hit = (float4*)take(sz[6]);
    st.sh_o = (float4*)take(sz[7]);
    st.sh_d = (float4*)take(sz[8]);
    st.sh_c = (float4*)take(sz[9]);
    st.welford = (double2*)take(sz[10]);
    st.act = (uint8_t*)take(sz[11]);
    st.q_sh = (int*)take(sz[12]);
    st.q_term = (int*)take(sz[13]);
    st.ctr = (WfCounters*)take(sz[14]);
    st.sacc = (double4*)take(sz[15]);
    st.ssq = (double4*)take(sz[16]);
    st.part = T ? (double4*)take(sz[17]) : nullptr;
    st.part_sq = T ? (double4*)take(sz[18]) : nullptr;
    st.surf_p = (float4*)take(sz[19]);
    st.surf_n = (float4*)take(sz[20]);
    st.q_mat = (int*)take(sz[21]);
    st.job = (int*)take(sz[22]);
    st.cmp_counts = (int*)take(sz[23]);
    return cudaSuccess;
}

void wf_release(WfBuffers& b) {
    release_state(b);
    if (b.round_block) cudaFree(b.round_block);
    b.round_block = nullptr;
    b.round_pixels = b.round_samples = 0;
    if (b.cull_block) cudaFree(b.cull_block);
    b.cull_block = nullptr;
    b.cull_pixels = 0;
    if (b.ev_fork) cudaEventDestroy(b.ev_fork);
    if (b.ev_join) cudaEventDestroy(b.ev_join);
    if (b.side) cudaStreamDestroy(b.side);
    b.ev_fork = b.ev_join = nullptr;
    b.side = nullptr;
}

namespace {
// Camera-culling arrays for a film of `pixels`: two flag bytes and two
// compacted lists per pixel, the compaction's span counts, two lengths.
cudaError_t cull_reserve(WfBuffers& b, size_t pixels) {
    if (b.cull_block && b.cull_pixels >= pixels) return cudaSuccess;
    if (b.cull_block) cudaFree(b.cull_block);
    b.cull_block = nullptr;
    b.cull_pixels = 0;
    const size_t spans = wf_compact_spans(pixels);
    const size_t sz[] = {pixels, pixels, pixels * 4, pixels * 4, spans * 4, spans * 4, 256};
    size_t total = 0;
    for (size_t x : sz) total += align_up(x);
    char* p = nullptr;
    const cudaError_t e = cudaMalloc(&p, total);
    if (e != cudaSuccess) return e;
    size_t off = 0;
    auto take = [&](size_t bytes) { char* r = p + off; off += align_up(bytes); return (void*)r; };
    b.cull_block = p;
    b.cull_flag[0] = (uint8_t*)take(sz[0]);
    b.cull_flag[1] = (uint8_t*)take(sz[1]);
    b.cull_map[0] = (int*)take(sz[2]);
    b.cull_map[1] = (int*)take(sz[3]);
    b.cull_counts[0] = (int*)take(sz[4]);
    b.cull_counts[1] = (int*)take(sz[5]);
    b.cull_n = (int*)take(sz[6]);
    b.cull_pixels = pixels;
    return cudaSuccess;
}

// Classifies the film's pixels (a multi-job render: every job's) for
// camera culling and compacts both kinds in pixel order: B.cull_map[0] =
// the n_may pixels a camera ray may reach geometry from, B.cull_map[1] =
// the n_open others.  A multi-job render then also gets each job's
// stretches and first ids in the device job table, and n_fetch / n_sky_tasks
// for the whole batch.  7 launches (8 for multi-job renders), one read-back.
cudaError_t cull_classify(const WfScene& S, const WfParams& P, WfBuffers& B, cudaStream_t s, int& n_may, int& n_open,
                          long long& n_fetch, long long& n_sky_tasks) {
    const long long n_ll = P.jobs ? P.total_pixels : (long long)P.n_pixels;
    cudaError_t e = cull_reserve(B, (size_t)n_ll);
    if (e != cudaSuccess) return e;
    const int n = (int)n_ll;
    if (P.jobs) wf::k_cull_classify<true><<<(n + 255) / 256, 256, 0, s>>>(S, P, B.cull_flag[0], B.cull_flag[1]);
    else wf::k_cull_classify<false><<<(n + 255) / 256, 256, 0, s>>>(S, P, B.cull_flag[0], B.cull_flag[1]);
    const int nb = (int)((n + wf::kCmpSpan - 1) / wf::kCmpSpan);
    for (int k = 0; k < 2; ++k) {
        wf::k_cmp_count<<<nb, wf::kCmpBlock, 0, s>>>(B.cull_flag[k], n, B.cull_counts[k]);
        wf::k_cmp_scan<<<1, 1024, 0, s>>>(B.cull_counts[k], nb, B.cull_n + k);
        wf::k_cmp_scatter<<<nb, wf::kCmpBlock, 0, s>>>(B.cull_flag[k], n, B.cull_counts[k], B.cull_map[k]);
    }
    long long* totals = reinterpret_cast<long long*>(B.cull_n + 2);  // 8-byte aligned: cull_n is 256-byte aligned
    if (P.jobs)
        wf::k_cull_jobs<<<1, 1024, 0, s>>>(const_cast<WfJob*>(P.jobs), P.n_jobs, B.cull_map[0], B.cull_map[1],
                                           B.cull_n, totals);
    struct { int n[2]; long long t[2]; } h{{n, 0}, {0, 0}};
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, B.cull_n, sizeof h, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    n_may = h.n[0];
    n_open = h.n[1];
    n_fetch = P.jobs ? h.t[0] : 0;
    n_sky_tasks = P.jobs ? h.t[1] : 0;
    return e;
}
}  // namespace

cudaError_t wf_cull_pixels(const WfScene& S, const WfParams& P, WfBuffers& B, cudaStream_t s, int* n_may,
                           int* n_open) {
    long long f = 0, u = 0;
    return cull_classify(S, P, B, s, *n_may, *n_open, f, u);
}

namespace {
// Adaptive-round arrays: Welford state (32 B) and two active lists (4 B
// each) per film pixel, a counter, and `samples` float4 sample records.
cudaError_t round_reserve(WfBuffers& b, size_t pixels, size_t samples) {
    if (b.round_block && b.round_pixels >= pixels && b.round_samples >= samples) return cudaSuccess;
    if (b.round_block) cudaFree(b.round_block);
    b.round_block = nullptr;
    b.round_pixels = b.round_samples = 0;
    const size_t sz[] = {pixels * 32, pixels * 4, pixels * 4, 256, samples * 16};
    size_t total = 0;
    for (size_t x : sz) total += align_up(x);
    char* p = nullptr;
    cudaError_t e = cudaMalloc(&p, total);
    if (e != cudaSuccess) return e;
    size_t off = 0;
    auto take = [&](size_t bytes) { char* r = p + off; off += align_up(bytes); return (void*)r; };
    b.round_block = p;
    b.wstate = (double4*)take(sz[0]);
    b.active[0] = (int*)take(sz[1]);
    b.active[1] = (int*)take(sz[2]);
    b.n_active = (int*)take(sz[3]);
    b.rsamp = (float4*)take(sz[4]);
    b.round_pixels = pixels;
    b.round_samples = samples;
    return cudaSuccess;
}
}  // namespace

// ---- host driver -------------------------------------------------------------
namespace {

struct Grids { int extend, shade, shadow, regen, surface[5], shade_all, shade_all4, shade_all6, shade_batch, shade_batch8; };

// Shading: the classify kernel, then one surface kernel per material kind
// (each returns at once when its queue is empty).
void launch_shade(const Grids& g, cudaStream_t s, const WfScene& S, const WfParams& P, const WfState& st, int cur) {
    if (P.jobs) {  // batch renders: fused shading only
        if (P.shade_ctas == 8) wf::k_shade<true, 8><<<g.shade_batch8, wf::kShadeBlock, 0, s>>>(S, P, st, cur);
        else wf::k_shade<true, 4><<<g.shade_batch, wf::kShadeBlock, 0, s>>>(S, P, st, cur);
        return;
    }
    if (!P.shade_sort) {
        if (P.shade_ctas == 4) wf::k_shade<false, 4><<<g.shade_all4, wf::kShadeBlock, 0, s>>>(S, P, st, cur);
        else if (P.shade_ctas == 6) wf::k_shade<false, 6><<<g.shade_all6, wf::kShadeBlock, 0, s>>>(S, P, st, cur);
        else wf::k_shade<false, 8><<<g.shade_all, wf::kShadeBlock, 0, s>>>(S, P, st, cur);
        return;
    }
    wf::k_shade_pre<<<g.shade, 128, 0, s>>>(S, P, st, cur);
    wf::k_shade_surface<TPT_MAT_LAMBERT><<<g.surface[0], 128, 0, s>>>(S, P, st, cur);
    wf::k_shade_surface<TPT_MAT_METAL><<<g.surface[1], 128, 0, s>>>(S, P, st, cur);
    wf::k_shade_surface<TPT_MAT_DIELECTRIC><<<g.surface[2], 128, 0, s>>>(S, P, st, cur);
    wf::k_shade_surface<TPT_MAT_GGX><<<g.surface[3], 128, 0, s>>>(S, P, st, cur);
    wf::k_shade_surface<TPT_MAT_SUBSURFACE><<<g.surface[4], 128, 0, s>>>(S, P, st, cur);
}

// Trace kernels keep their stack in shared memory when the scene's deepest
// path (top level + exit marker + mesh tree) fits kSharedStack entries.
template <bool ANY, bool COUNT>
void launch_trace(int grid, cudaStream_t s, const WfScene& S, const WfParams& P, const WfState& st, int n_slots,
                  int chunk, int cur) {
    const bool shared = S.max_stack <= wf::kSharedStack;
    if (P.jobs) {
        if (shared)
            wf::k_trace<ANY, COUNT, true, true><<<grid, wf::kTraceBlock, 0, s>>>(S, P, st, n_slots, chunk, P.jobs, cur);
        else
            wf::k_trace<ANY, COUNT, false, true><<<grid, wf::kTraceBlock, 0, s>>>(S, P, st, n_slots, chunk, P.jobs, cur);
    } else if (shared) {
        wf::k_trace<ANY, COUNT, true, false><<<grid, wf::kTraceBlock, 0, s>>>(S, P, st, n_slots, chunk, nullptr, cur);
    } else {
        wf::k_trace<ANY, COUNT, false, false><<<grid, wf::kTraceBlock, 0, s>>>(S, P, st, n_slots, chunk, nullptr, cur);
    }
}
void launch_regen(int grid, cudaStream_t s, const WfScene& S, const WfParams& P, const WfState& st, int cur) {
    if (P.jobs) wf::k_regen<true><<<grid, 128, 0, s>>>(S, P, st, cur);
    else wf::k_regen<false><<<grid, 128, 0, s>>>(S, P, st, cur);
}

template <class K>
int grid_for(K kernel, int sm_count, int block = 128) {
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, block, 0);
    return sm_count * (occ > 0 ? occ : 1);
}

Grids pick_grids(int sm_count) {
    Grids g{};
    g.extend = grid_for(wf::k_trace<false, false, true, false>, sm_count);
    g.shadow = grid_for(wf::k_trace<true, false, true, false>, sm_count);
    g.shade = grid_for(wf::k_shade_pre, sm_count);
    g.shade_all = grid_for(wf::k_shade<false, 8>, sm_count, wf::kShadeBlock);
    g.shade_all4 = grid_for(wf::k_shade<false, 4>, sm_count, wf::kShadeBlock);
    g.shade_all6 = grid_for(wf::k_shade<false, 6>, sm_count, wf::kShadeBlock);
    g.shade_batch = grid_for(wf::k_shade<true, 4>, sm_count, wf::kShadeBlock);
    g.shade_batch8 = grid_for(wf::k_shade<true, 8>, sm_count, wf::kShadeBlock);
    g.surface[0] = grid_for(wf::k_shade_surface<TPT_MAT_LAMBERT>, sm_count);
    g.surface[1] = grid_for(wf::k_shade_surface<TPT_MAT_METAL>, sm_count);
    g.surface[2] = grid_for(wf::k_shade_surface<TPT_MAT_DIELECTRIC>, sm_count);
    g.surface[3] = grid_for(wf::k_shade_surface<TPT_MAT_GGX>, sm_count);
    g.surface[4] = grid_for(wf::k_shade_surface<TPT_MAT_SUBSURFACE>, sm_count);
    g.regen = grid_for(wf::k_regen<false>, sm_count);
    return g;
}

// k_paths over n_items tasks (TASKS) or live slots: one wave of blocks.
// Fewer items than lanes spread over the warps, so that a warp diverges less.
template <bool TASKS, bool BATCH, bool SHARED>
void launch_paths_as(const WfScene& S, const WfParams& P, const WfState& st, const uint8_t* open, long long n_items,
                     int sm_count, cudaStream_t s) {
    auto kern = wf::k_paths<BATCH, TASKS, SHARED>;
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, wf::kPathsBlock, 0);
    const long long blocks = (long long)sm_count * std::max(occ, 1), warps = blocks * (wf::kPathsBlock / 32);
    const unsigned lanes = (unsigned)std::min<long long>(32, std::max<long long>(1, (n_items + warps - 1) / warps));
    const long long per_block = (long long)lanes * (wf::kPathsBlock / 32);
    const unsigned grid = (unsigned)std::max<long long>(1, std::min(blocks, (n_items + per_block - 1) / per_block));
    kern<<<grid, wf::kPathsBlock, 0, s>>>(S, P, st, open, lanes);
}
template <bool TASKS>
void launch_paths(const WfScene& S, const WfParams& P, const WfState& st, const uint8_t* open, long long n_items,
                  int sm_count, cudaStream_t s) {
    const bool shared = S.max_stack <= wf::kSharedStack;
    if (P.jobs) {
        if (shared) launch_paths_as<TASKS, true, true>(S, P, st, open, n_items, sm_count, s);
        else launch_paths_as<TASKS, true, false>(S, P, st, open, n_items, sm_count, s);
    } else if (shared) {
        launch_paths_as<TASKS, false, true>(S, P, st, open, n_items, sm_count, s);
    } else {
        launch_paths_as<TASKS, false, false>(S, P, st, open, n_items, sm_count, s);
    }
}

// The pool's end of fetch ids (fetch_end on the device).
long long host_fetch_end(const WfParams& P) {
    if (!P.geo_map) return P.n_tasks;
    if (P.jobs) return P.n_fetch;
    return P.task_first + (P.n_tasks - P.task_first) / P.n_pixels * P.n_geo;
}

void enqueue_iteration(const WfScene& S, const WfParams& P, const WfState& st, const Grids& g, cudaStream_t s,
                       cudaGraphConditionalHandle h, int use_cond) {
    for (int cur = 0; cur < 2; ++cur) {
        launch_trace<false, false>(g.extend, s, S, P, st, P.n_slots, P.trace_chunk, cur);
        launch_shade(g, s, S, P, st, cur);
        launch_trace<true, false>(g.shadow, s, S, P, st, P.n_slots, P.trace_chunk, cur);
        launch_regen(g.regen, s, S, P, st, cur);
        if (P.ordered_queue) wf_launch_compact(s, st, cur, P.n_slots);
        wf::k_step<<<1, 1, 0, s>>>(st, cur, P.max_iters, h, use_cond, P.tail_live > 0 ? host_fetch_end(P) : 0,
                                   P.tail_live);
    }
}

struct Events {
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    Events() { cudaEventCreate(&e0); cudaEventCreate(&e1); }
    ~Events() { cudaEventDestroy(e0); cudaEventDestroy(e1); }
};

struct GraphGuard {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    ~GraphGuard() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
    }
};

// Device-driven loop: one WHILE conditional node whose body is two
// iterations; the last kernel of each iteration re-arms the condition on the
// device.
cudaError_t run_graph_loop(const WfEnqueue& enqueue, cudaStream_t stream, bool* built) {
    GraphGuard gg;
    cudaError_t e = cudaGraphCreate(&gg.graph, 0);
    cudaGraphConditionalHandle handle{};
    if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&handle, gg.graph, 1, cudaGraphCondAssignDefault);
    cudaGraphNode_t node{};
    cudaGraphNodeParams np{};
    if (e == cudaSuccess) {
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = handle;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        e = cudaGraphAddNode(&node, gg.graph, nullptr, 0, &np);
    }
    cudaStream_t cap = nullptr;
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
    if (e == cudaSuccess) {
        cudaGraph_t body = np.conditional.phGraph_out[0];
        e = cudaStreamBeginCaptureToGraph(cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            enqueue(cap, handle, 1);
            e = cudaStreamEndCapture(cap, &body);
        }
    }
    if (cap) cudaStreamDestroy(cap);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&gg.exec, gg.graph, 0);
    if (e != cudaSuccess) {
        // Nothing ran yet: report "not supported" so the caller can use the
        // host-driven loop instead.
        cudaGetLastError();
        *built = false;
        return e;
    }
    *built = true;
    e = cudaGraphLaunch(gg.exec, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    return e;
}

// Host-driven loop: the two-iteration body launched directly on the stream
// (no graph, so every kernel launch is visible to a profiler's launch list),
// with a probe of the counters after each, so the loop ends where the
// device-side loop would.  *done = false: it is not at its end after
// max_bodies bodies.
cudaError_t run_host_loop(const WfEnqueue& enqueue, const WfCounters* ctr, long long max_iters, cudaStream_t stream,
                          long long max_bodies, bool* done) {
    WfCounters probe{};
    cudaError_t e = cudaSuccess;
    *done = false;
    for (long long launched = 2; e == cudaSuccess && launched <= 2 * max_bodies; launched += 2) {
        enqueue(stream, cudaGraphConditionalHandle{}, 0);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(&probe, ctr, sizeof(WfCounters), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) break;
        if ((probe.n_ext[0] == 0 && probe.n_ext[1] == 0) ||
            probe.tail ||  // k_paths finishes the live slots
            (probe.flags & TPT_FLAG_ITER_LIMIT) || launched > max_iters + 16) {
            *done = true;
            break;
        }
    }
    return e;
}

// Profiling loop: plain launches with events around every stage and the
// counting variants of the trace kernels.
cudaError_t run_profile_loop(const WfScene& S, const WfParams& P, const WfState& st, const Grids& g,
                             cudaStream_t s, double* stage_ms, unsigned long long* stage_launches) {
    Events ev[4];
    cudaError_t e = cudaSuccess;
    WfCounters probe{};
    for (long long it = 0; it <= P.max_iters + 1 && e == cudaSuccess; it += 2) {
        for (int cur = 0; cur < 2 && e == cudaSuccess; ++cur) {
            cudaEventRecord(ev[0].e0, s);
            launch_trace<false, true>(g.extend, s, S, P, st, P.n_slots, P.trace_chunk, cur);
            cudaEventRecord(ev[0].e1, s);
            cudaEventRecord(ev[1].e0, s);
            launch_shade(g, s, S, P, st, cur);
            cudaEventRecord(ev[1].e1, s);
            cudaEventRecord(ev[2].e0, s);
            launch_trace<true, true>(g.shadow, s, S, P, st, P.n_slots, P.trace_chunk, cur);
            cudaEventRecord(ev[2].e1, s);
            cudaEventRecord(ev[3].e0, s);
            launch_regen(g.regen, s, S, P, st, cur);
            if (P.ordered_queue) wf_launch_compact(s, st, cur, P.n_slots);
            cudaEventRecord(ev[3].e1, s);
            wf::k_step<<<1, 1, 0, s>>>(st, cur, P.max_iters, cudaGraphConditionalHandle{}, 0);
            e = cudaMemcpyAsync(&probe, st.ctr, sizeof(WfCounters), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) break;
            for (int k = 0; k < 4; ++k) {
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, ev[k].e0, ev[k].e1);
                stage_ms[k] += ms;
                stage_launches[k] += 1;
            }
            if (probe.n_ext[0] == 0 && probe.n_ext[1] == 0) return cudaSuccess;
        }
    }
    return e;
}

}  // namespace

// Most renders are through in a few bodies, and a launch of the body with
// its probe (about 20 us between bodies) costs less than building the graph
// (0.35 to 0.4 ms): the sphere scene, 2 bodies, 2.33 -> 1.94 ms, the 1080p
// frame, 9 bodies, 138.6 -> 138.2.  Longer loops go on in the graph, which has no gaps.
constexpr long long kHostBodies = 12;

cudaError_t wf_run_loop(const WfEnqueue& enqueue, const WfCounters* ctr, long long max_iters, cudaStream_t stream,
                        bool use_graph_loop) {
    bool done = false;
    if (use_graph_loop) {
        cudaError_t e = run_host_loop(enqueue, ctr, max_iters, stream, kHostBodies, &done);
        if (e != cudaSuccess || done) return e;
        bool built = false;
        e = run_graph_loop(enqueue, stream, &built);
        if (e == cudaSuccess || built) return e;
    }
    return run_host_loop(enqueue, ctr, max_iters, stream, LLONG_MAX / 2, &done);
}

void wf_trace_grids(int sm_count, int* extend, int* shadow) {
    *extend = grid_for(wf::k_trace<false, false, true, false>, sm_count);
    *shadow = grid_for(wf::k_trace<true, false, true, false>, sm_count);
}

void wf_launch_trace(bool any, int grid, cudaStream_t s, const WfScene& S, const WfParams& P, const WfState& st,
                     int cur) {
    if (any) launch_trace<true, false>(grid, s, S, P, st, P.n_slots, P.trace_chunk, cur);
    else launch_trace<false, false>(grid, s, S, P, st, P.n_slots, P.trace_chunk, cur);
}

void wf_launch_step(cudaStream_t s, const WfState& st, int cur, long long max_iters, cudaGraphConditionalHandle h,
                    int use_cond) {
    wf::k_step<<<1, 1, 0, s>>>(st, cur, max_iters, h, use_cond);
}

size_t wf_compact_spans(size_t n_slots) { return (n_slots + wf::kCmpSpan - 1) / wf::kCmpSpan + 1; }

void wf_launch_compact(cudaStream_t s, const WfState& st, int cur, int n_slots) {
    const int nb = (int)((n_slots + wf::kCmpSpan - 1) / wf::kCmpSpan);
    const int nxt = cur ^ 1;
    wf::k_cmp_count<<<nb, wf::kCmpBlock, 0, s>>>(st.act, n_slots, st.cmp_counts);
    wf::k_cmp_scan<<<1, 1024, 0, s>>>(st.cmp_counts, nb, &st.ctr->n_ext[nxt]);
    wf::k_cmp_scatter<<<nb, wf::kCmpBlock, 0, s>>>(st.act, n_slots, st.cmp_counts, st.q_ext[nxt]);
}

namespace {
void add_counters(WfCounters& a, const WfCounters& b) {
    a.iters += b.iters;
    a.flags |= b.flags;
    a.rays_closest += b.rays_closest;
    a.rays_shadow += b.rays_shadow;
    a.samples += b.samples;
    for (int k = 0; k < 2; ++k) {
        a.cnt_nodes[k] += b.cnt_nodes[k];
        a.cnt_tris[k] += b.cnt_tris[k];
        a.cnt_spheres[k] += b.cnt_spheres[k];
        a.cnt_inst[k] += b.cnt_inst[k];
        a.cnt_node_steps[k] += b.cnt_node_steps[k];
        a.cnt_leaves[k] += b.cnt_leaves[k];
        a.cnt_leaf_steps[k] += b.cnt_leaf_steps[k];
    }
    a.cnt_fast += b.cnt_fast;
    a.cnt_fast_steps += b.cnt_fast_steps;
    a.sky_samples += b.sky_samples;
}

// Kernels one iteration of the bounce loop launches (enqueue_iteration).
long long launches_per_iteration(const WfParams& P) {
    return 3 + (P.shade_sort && !P.jobs ? 6 : 1) + (P.ordered_queue ? 3 : 0) + 1;
}
}  // namespace

namespace {
// Reserves the path state of P.n_slots slots, halving the pool (down to 2^20
// slots) while the device has no room for it; the iteration bound grows to
// match.  A render does not depend on the pool size: each task's samples run
// in one slot and task sums merge in task order.
cudaError_t reserve_pool(WfBuffers& B, WfParams& P, size_t part_tasks) {
    for (;;) {
        const cudaError_t e = wf_reserve(B, (size_t)P.n_slots, part_tasks);
        if (e != cudaErrorMemoryAllocation || P.n_slots <= (1 << 20)) return e;
        cudaGetLastError();
        P.n_slots /= 2;
        P.max_iters *= 2;
    }
}
}  // namespace

// Whether a render of n_tasks tasks of up to task_spp samples runs in k_paths
// alone.  Its divergent lanes trace 2 to 4 times slower than the loop's kernels
// at full size, but the loop's some 25 launches and waits cost 0.3 to 1 ms, and
// once more per sample of a task.  So the line is one of tasks: some 390,000,
// three times as many of one sample, which pay the loop once.  Measured on one
// B200, loop / direct, ms, sphere scene; mesh scene of 81,920 triangles; Cornell box
// with glass:
//   1-sample tasks    36,864   0.44 / 0.14   0.98 / 0.32   1.19 / 0.34
//                  1,179,648   0.84 / 0.60   1.86 / 1.41   2.55 / 2.85  (last direct)
//                  2,097,152   1.09 / 0.97   2.12 / 2.18   3.45 / 4.80
//   8-sample         131,072   2.89 / 0.82   6.33 / 2.23   7.49 / 3.15
//                    491,520   3.84 / 2.23   7.51 / 5.70   10.4 / 9.69  (last direct)
//                  1,048,576   5.05 / 3.98   9.01 / 9.67   15.5 / 19.5
//   64-sample        360,000   19.8 / 10.0   48.3 / 27.7   64.4 / 53.1
//   256-sample       262,144   70.5 / 28.7    180 / 88.5    226 / 156
// Batches of 64 small scenes, 8-sample tasks, two sets: 2.0 M samples 8.6 / 5.4 and
// 8.7 / 6.4, 3.7 M 10.7 / 8.7 and 10.4 / 8.7, 6.5 M 13.4 / 13.4.
// A caller that sets the drain's handover (TPT_TAIL_SLOTS) asks for the loop.
bool wf_one_kernel(long long n_tasks, int task_spp) {
    return n_tasks * std::max(task_spp, 1) <= (task_spp + 2) * 393216LL;
}

namespace {
bool direct_render(const WfParams& P) { return P.tail_live < 0 && wf_one_kernel(P.n_tasks, P.task_spp); }

// A render whose tasks all go to k_paths: no path state, no loop.  With camera
// culling on, one thread per pixel classifies the film first (k_paths reads
// the flags; nothing is compacted or read back).
cudaError_t render_direct(const WfScene& S, const WfParams& P, WfBuffers& B, double* acc, double* acc_w, double* acc_sq,
                          size_t part_tasks, cudaStream_t stream, int sm_count, WfCounters* hc, float* ms) {
    cudaError_t e = wf_reserve(B, std::max<size_t>(B.slots, 1), std::max(B.part_tasks, part_tasks));
    if (e == cudaErrorMemoryAllocation) {  // no room beside the slots of an earlier render
        cudaGetLastError();
        e = wf_reserve(B, 1, part_tasks);
    }
    if (e != cudaSuccess) return e;
    WfState st = B.st;
    st.acc = acc;
    st.acc_w = acc_w;
    st.acc_sq = acc_sq;
    st.welford = nullptr;
    st.ssq = nullptr;
    if (!acc_sq) st.part_sq = nullptr;
    Events total;
    cudaEventRecord(total.e0, stream);
    e = cudaMemsetAsync(st.ctr, 0, sizeof(WfCounters), stream);
    long long launches = 1;
    const uint8_t* open = nullptr;
    const long long pixels = P.jobs ? P.total_pixels : (long long)P.n_pixels;
    const bool pinhole = P.jobs || (P.max_bounces > 0 && S.cam.lens_radius == 0.0f && S.cam.focus_dist > 0.0f);
    if (e == cudaSuccess && P.sky_cull && !P.adaptive && pinhole && pixels < (1ll << 31)) {
        e = cull_reserve(B, (size_t)pixels);
        const unsigned grid = (unsigned)((pixels + 255) / 256);
        if (e == cudaSuccess) {
            if (P.jobs) wf::k_cull_classify<true><<<grid, 256, 0, stream>>>(S, P, B.cull_flag[0], B.cull_flag[1]);
            else wf::k_cull_classify<false><<<grid, 256, 0, stream>>>(S, P, B.cull_flag[0], B.cull_flag[1]);
            open = B.cull_flag[1];
            ++launches;
        }
    }
    if (e == cudaSuccess) {
        launch_paths<true>(S, P, st, open, P.n_tasks, sm_count, stream);
        if (P.n_chunks > 1) {
            if (P.jobs) wf::k_merge_batch<<<(unsigned)((pixels + 255) / 256), 256, 0, stream>>>(P, st);
            else wf::k_merge<<<(P.n_pixels + 255) / 256, 256, 0, stream>>>(P, st);
            ++launches;
        }
        e = cudaGetLastError();
    }
    cudaEventRecord(total.e1, stream);
    WfCounters c{};
    if (e == cudaSuccess) e = cudaMemcpyAsync(&c, st.ctr, sizeof(WfCounters), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e;
    }
    c.samples += c.sky_samples;  // counted apart, as by k_sky_tasks
    c.rays_closest += c.sky_samples;
    c.pool_slots = P.n_slots;
    c.launches = launches;
    *hc = c;
    if (ms) cudaEventElapsedTime(ms, total.e0, total.e1);
    return e;
}
}  // namespace

// A single render whose per-task sums would exceed P.max_part_tasks runs its
// sample chunks in batches (chunks [c0, c1) of every pixel, then the next
// batch), merging each onto the film in task order: device memory for the
// sums stays bounded however many samples a pixel takes.
cudaError_t wf_render(const WfScene& S, const WfParams& P_in, WfBuffers& B, double* acc, double* acc_w, double* acc_sq,
                      cudaStream_t stream, int sm_count, bool use_graph_loop, WfCounters* hc, float* ms, bool profile,
                      double* stage_ms, unsigned long long* stage_launches) {
    WfParams P = P_in;
    long long batch_chunks = P.n_chunks;
    if (!P.jobs && P.n_chunks > 1 && P.max_part_tasks > 0 && P.n_tasks > P.max_part_tasks)
        batch_chunks = std::max<long long>(1, P.max_part_tasks / P.n_pixels);
    // per-task sums of one chunk batch (single renders) or of all tasks (a
    // multi-job render, whose P.n_pixels is 0: every job has its own)
    size_t part_tasks = 0;
    if (P.n_chunks > 1)
        part_tasks = P.jobs ? (size_t)P.n_tasks : (size_t)std::min<long long>(P.n_tasks, batch_chunks * P.n_pixels);
    const bool direct = !profile && use_graph_loop && batch_chunks >= P.n_chunks && direct_render(P);
    if (direct) return render_direct(S, P, B, acc, acc_w, acc_sq, part_tasks, stream, sm_count, hc, ms);
    cudaError_t e = reserve_pool(B, P, part_tasks);
    if (e != cudaSuccess) return e;
    WfState st = B.st;
    st.acc = acc;
    st.acc_w = acc_w;
    st.acc_sq = acc_sq;
    if (!P.adaptive) st.welford = nullptr;
    if (!acc_sq) { st.ssq = nullptr; st.part_sq = nullptr; }
    const Grids g = pick_grids(sm_count);

    Events total;
    cudaEventRecord(total.e0, stream);
    if (profile)
        for (int k = 0; k < 4; ++k) { stage_ms[k] = 0.0; stage_launches[k] = 0; }
    // Camera culling: forward renders (single or multi-job) through pinhole
    // cameras (cull_may_hit keeps every pixel of a lens camera).
    long long launches = 0;
    int n_may = P.n_pixels, n_open = 0;
    long long n_fetch = 0, n_sky_tasks = 0;
    const bool cull_single = !P.jobs && P.max_bounces > 0 && P.n_pixels > 0 && S.cam.lens_radius == 0.0f &&
                             S.cam.focus_dist > 0.0f;
    const bool cull_batch = P.jobs && P.total_pixels > 0 && P.total_pixels < (1ll << 31);
    if (P.sky_cull && !P.adaptive && (cull_single || cull_batch)) {
        e = cull_classify(S, P, B, stream, n_may, n_open, n_fetch, n_sky_tasks);
        launches += P.jobs ? 8 : 7;
        if (e != cudaSuccess) {
            cudaGetLastError();
            return e;
        }
    }
    // With the open pixels culled, the camera rays left that miss are few:
    // the fast path then costs the closest-hit kernel more than it saves
    // (1080p frame: 2.76 -> 2.80 G paths/s without it).
    if (P.camera_fast == 2) P.camera_fast = n_open > 0 ? 0 : 1;
    WfCounters sum{};
    for (long long c0 = 0; c0 < P.n_chunks && e == cudaSuccess; c0 += batch_chunks) {
        WfParams Pb = P;
        if (!P.jobs) {
            Pb.task_first = c0 * P.n_pixels;
            Pb.n_tasks = std::min<long long>(c0 + batch_chunks, P.n_chunks) * P.n_pixels;
        }
        const long long batch_chunk_count = P.jobs ? 0 : (Pb.n_tasks - Pb.task_first) / P.n_pixels;
        if (n_open > 0) {
            // the pool takes the other pixels' tasks; no more slots than those
            Pb.geo_map = B.cull_map[0];
            Pb.n_geo = n_may;
            Pb.geo_div = make_fastdiv((uint32_t)std::max(n_may, 1));
            Pb.n_fetch = n_fetch;
            const long long pooled = P.jobs ? n_fetch : batch_chunk_count * n_may;
            if (pooled > 0 && pooled < Pb.n_slots) Pb.n_slots = (int)pooled;
        }
        // the drain's handover to k_paths (1080p frame, 64 Mi slots: 2.838 -> 2.931 G paths/s at
        // 262,144; 2.921 at 65,536, 2.930 at 1 Mi, 2.781 at 4 Mi)
        if (Pb.tail_live < 0) Pb.tail_live = std::min(262144, Pb.n_slots / 16);
        cudaMemsetAsync(st.ctr, 0, sizeof(WfCounters), stream);
        // The culled tasks run on a side stream beside the bounce loop: they
        // write other tasks' sums, read only the classification, and count
        // into sky_samples alone; the merge waits for them.
        bool sky_side = false;
        if (n_open > 0) {
            const long long count = P.jobs ? n_sky_tasks : batch_chunk_count * n_open;
            const unsigned grid = (unsigned)((count + 255) / 256);
            const FastDiv od = make_fastdiv((uint32_t)n_open);
            if (!B.side) {
                if (cudaStreamCreateWithFlags(&B.side, cudaStreamNonBlocking) != cudaSuccess ||
                    cudaEventCreateWithFlags(&B.ev_fork, cudaEventDisableTiming) != cudaSuccess ||
                    cudaEventCreateWithFlags(&B.ev_join, cudaEventDisableTiming) != cudaSuccess) {
                    cudaGetLastError();
                    if (B.side) cudaStreamDestroy(B.side);
                    B.side = nullptr;
                }
            }
            cudaStream_t ss = stream;
            if (B.side && B.ev_fork && B.ev_join) {
                cudaEventRecord(B.ev_fork, stream);
                cudaStreamWaitEvent(B.side, B.ev_fork, 0);
                ss = B.side;
                sky_side = true;
            }
            if (P.jobs) wf::k_sky_tasks<true><<<grid, 256, 0, ss>>>(S, Pb, st, B.cull_map[1], n_open, od, count);
            else wf::k_sky_tasks<false><<<grid, 256, 0, ss>>>(S, Pb, st, B.cull_map[1], n_open, od, count);
            if (sky_side) cudaEventRecord(B.ev_join, B.side);
            ++launches;
        }
        if (P.jobs) wf::k_init<true><<<(Pb.n_slots + 255) / 256, 256, 0, stream>>>(S, Pb, st);
        else wf::k_init<false><<<(Pb.n_slots + 255) / 256, 256, 0, stream>>>(S, Pb, st);
        ++launches;
        e = cudaGetLastError();
        if (e == cudaSuccess) {
            if (profile) {
                e = run_profile_loop(S, Pb, st, g, stream, stage_ms, stage_launches);
            } else {
                e = wf_run_loop([&](cudaStream_t s, cudaGraphConditionalHandle h, int use_cond) {
                    enqueue_iteration(S, Pb, st, g, s, h, use_cond);
                }, st.ctr, P.max_iters, stream, use_graph_loop);
                if (e == cudaSuccess && Pb.tail_live > 0) {
                    // the slots the loop left (none when it drained the pool)
                    launch_paths<false>(S, Pb, st, nullptr, Pb.tail_live, sm_count, stream);
                    ++launches;
                    e = cudaGetLastError();
                }
            }
        }
        if (sky_side) cudaStreamWaitEvent(stream, B.ev_join, 0);
        if (e == cudaSuccess && P.n_chunks > 1) {
            if (P.jobs)
                wf::k_merge_batch<<<(unsigned)((P.total_pixels + 255) / 256), 256, 0, stream>>>(Pb, st);
            else
                wf::k_merge<<<(P.n_pixels + 255) / 256, 256, 0, stream>>>(Pb, st);
            ++launches;
            e = cudaGetLastError();
        }
        WfCounters part{};
        if (e == cudaSuccess) e = cudaMemcpyAsync(&part, st.ctr, sizeof(WfCounters), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e == cudaSuccess) {
            part.samples += part.sky_samples;  // counted apart by k_sky_tasks
            part.rays_closest += part.sky_samples;
            add_counters(sum, part);
            launches += part.iters * launches_per_iteration(Pb);
        }
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e;
    }
    cudaEventRecord(total.e1, stream);
    e = cudaEventSynchronize(total.e1);
    sum.pool_slots = P.n_slots;
    sum.launches = launches;
    *hc = sum;
    if (e == cudaSuccess && ms) cudaEventElapsedTime(ms, total.e0, total.e1);
    return e;
}

cudaError_t wf_render_adaptive(const WfScene& S, const WfParams& P_in, WfBuffers& B, double* acc, double* acc_w,
                               double* acc_sq, cudaStream_t stream, int sm_count, bool use_graph_loop, WfCounters* hc,
                               float* ms, size_t round_bytes, int* rounds_out) {
    WfParams P0 = P_in;
    const int n_film = P0.n_pixels, tspp = P0.task_spp;
    // round 0 takes the first min_spp samples (whole tasks): no pixel can stop before them
    const int min_spp = std::min(std::max(P0.adaptive_min_spp, 1), std::max(P0.spp, 1));
    const int first_len = std::min(P0.spp, (min_spp + tspp - 1) / tspp * tspp);
    // never more than the render's samples: round_bytes follows the free memory,
    // and a buffer sized by it was allocated anew whenever that grew
    const size_t cap = std::min(std::max(round_bytes / 16, (size_t)n_film * (size_t)first_len),
                                (size_t)n_film * (size_t)std::max(P0.spp, first_len));
    cudaError_t e = round_reserve(B, (size_t)n_film, cap);
    if (e == cudaSuccess) e = reserve_pool(B, P0, 0);
    if (e != cudaSuccess) return e;
    WfState st = B.st;
    st.acc = acc;
    st.acc_w = acc_w;
    st.acc_sq = acc_sq;
    st.welford = nullptr;
    st.ssq = nullptr;
    st.part = nullptr;
    st.part_sq = nullptr;
    st.rsamp = B.rsamp;
    unsigned long long* taken = reinterpret_cast<unsigned long long*>(B.n_active + 2);
    const Grids g = pick_grids(sm_count);
    Events total;
    cudaEventRecord(total.e0, stream);
    wf::k_round_init<<<(n_film + 255) / 256, 256, 0, stream>>>(n_film, B.active[0], B.wstate, acc, acc_w, acc_sq);
    e = cudaMemsetAsync(B.n_active, 0, 256, stream);
    WfCounters sum{};
    int n_active = n_film, cur = 0, base = 0, rounds = 0;
    while (e == cudaSuccess && n_active > 0 && base < P0.spp) {
        int len = first_len;
        if (rounds > 0) {
            // as many samples as the buffer holds for every active pixel, whole tasks, and a task count that
            // fits the path state's 32-bit task ids
            long long fit = (long long)(cap / (size_t)n_active) / tspp * tspp;
            const long long id_fit = (0x7fffffffLL / n_active) * tspp;
            fit = std::min(fit, id_fit);
            len = (int)std::min<long long>(P0.spp - base, std::max<long long>(fit, tspp));
        }
        WfParams Pb = P0;
        Pb.adaptive = 0;  // the stopping rule runs in k_round_merge
        Pb.n_pixels = n_active;
        wf_set_divisors(Pb);
        Pb.px_map = B.active[cur];
        Pb.sample_base = base;
        Pb.sample_end = base + len;
        Pb.round_len = len;
        Pb.n_chunks = (len + tspp - 1) / tspp;
        Pb.n_tasks = (long long)n_active * Pb.n_chunks;
        Pb.task_first = 0;
        Pb.n_slots = (int)std::min<long long>(P0.n_slots, Pb.n_tasks);
        Pb.max_iters = (long long)tspp * (long long)(P0.max_bounces + 1) * ((Pb.n_tasks + Pb.n_slots - 1) / Pb.n_slots + 1) + 16;
        cudaMemsetAsync(st.ctr, 0, sizeof(WfCounters), stream);
        Pb.tail_live = P0.tail_live;
        const bool direct = use_graph_loop && direct_render(Pb);
        if (Pb.tail_live < 0) Pb.tail_live = std::min(262144, Pb.n_slots / 16);  // each round's drain
        if (direct) launch_paths<true>(S, Pb, st, nullptr, Pb.n_tasks, sm_count, stream);
        else wf::k_init<false><<<(Pb.n_slots + 255) / 256, 256, 0, stream>>>(S, Pb, st);
        e = cudaGetLastError();
        if (e == cudaSuccess && !direct)
            e = wf_run_loop([&](cudaStream_t s, cudaGraphConditionalHandle h, int use_cond) {
                enqueue_iteration(S, Pb, st, g, s, h, use_cond);
            }, st.ctr, Pb.max_iters, stream, use_graph_loop);
        if (e == cudaSuccess && !direct && Pb.tail_live > 0) {
            launch_paths<false>(S, Pb, st, nullptr, Pb.tail_live, sm_count, stream);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemsetAsync(B.n_active, 0, sizeof(int), stream);
        if (e == cudaSuccess) {
            wf::k_round_merge<<<(n_active + 255) / 256, 256, 0, stream>>>(Pb, st, B.active[cur], n_active, B.wstate,
                                                                         B.active[cur ^ 1], B.n_active, taken);
            e = cudaGetLastError();
        }
        WfCounters part{};
        int next = 0;
        if (e == cudaSuccess) e = cudaMemcpyAsync(&part, st.ctr, sizeof(WfCounters), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&next, B.n_active, sizeof(int), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) break;
        add_counters(sum, part);
        n_active = next;
        cur ^= 1;
        base += len;
        ++rounds;
    }
    unsigned long long used = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&used, taken, sizeof(used), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e;
    }
    cudaEventRecord(total.e1, stream);
    e = cudaEventSynchronize(total.e1);
    sum.samples = used;  // samples that joined the film; later samples of a round that stopped are dropped
    sum.pool_slots = P0.n_slots;
    *hc = sum;
    if (rounds_out) *rounds_out = rounds;
    if (e == cudaSuccess && ms) cudaEventElapsedTime(ms, total.e0, total.e1);
    return e;
}

}  // namespace tpt

// ---- allocation-free variant ---------------------------------------------------
// Some callers cannot allocate device memory while they render: a process
// that reserves the whole GPU for its own allocator at start-up, or one that
// cannot afford the device-wide synchronisation cudaMalloc/cudaFree imply in
// the middle of a frame loop.  wf_render_noalloc runs k_paths, which carries
// its paths in registers, so all it needs in device memory is the counters,
// a file-scope device variable; it launches it directly (no graph or event
// objects are created) and allocates nothing.
//
// Limits: films of at most kNoAllocMaxSlots pixels.  Every call shares the
// counters: calls that overlap on the GPU (other streams or host threads)
// race on them, and each call clears them.
static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(tpt::WfCounters)];

namespace tpt {
namespace {

constexpr size_t kNoAllocMaxSlots = 16384;  // e.g. 128 x 128

std::mutex g_noalloc_mu;
void* g_noalloc_addr[256] = {};

// Device address of g_noalloc_scratch on the current device, looked up once
// per device (the host-side name of the array is not a device address).
cudaError_t noalloc_scratch(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 256) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_addr[dev] = p;
    }
    *out = g_noalloc_addr[dev];
    return cudaSuccess;
}

}  // namespace

size_t wf_noalloc_max_slots() { return kNoAllocMaxSlots; }

cudaError_t wf_render_noalloc(const WfScene& S, const WfParams& P, double* acc, double* acc_w, cudaStream_t stream,
                              int sm_count, WfCounters* hc) {
    if (P.n_slots <= 0 || (size_t)P.n_slots > kNoAllocMaxSlots || P.n_chunks != 1 || P.n_tasks != P.n_slots)
        return cudaErrorInvalidValue;
    void* base = nullptr;
    cudaError_t e = noalloc_scratch(&base);
    if (e != cudaSuccess) return e;
    WfState st{};
    st.ctr = static_cast<WfCounters*>(base);
    st.acc = acc;
    st.acc_w = acc_w;
    e = cudaMemsetAsync(st.ctr, 0, sizeof(WfCounters), stream);
    if (e != cudaSuccess) return e;
    launch_paths<true>(S, P, st, nullptr, P.n_tasks, sm_count, stream);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(hc, st.ctr, sizeof(WfCounters), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    return e;
}

}  // namespace tpt
