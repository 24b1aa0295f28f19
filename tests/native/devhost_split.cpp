// devhost_split.cpp - the split shadow DDA (GridWalk, grid_task, brick_task in device.cuh)
// run on the host, one ray at a time, tasks in visiting order, as the tracer's queues keep
// them; the first-voxel trace over cell masks; and the one-call area-light candidate. Test infrastructure only.
#include "devhost.cpp"

extern "C" {

// As dh_shadow (the resumable walker): 1 when the visibility test passes. deferred: every
// task is finished after the walk has ended (as when a warp's queue is emptied late), else
// at once. stats[4]: uber cells entered, grid cells visited, tasks, bricks walked.
int dh_shadow_split(const uint32_t* grid, const uint32_t* bricks, const uint32_t* bbox, const uint32_t* ucell,
                    const uint32_t* bmask, const float* O, const float* D, uint32_t pos, uint32_t size, int steps, int deferred, int* stats,
                    float* dist, uint32_t* side) {
    World w = make_world(grid, nullptr, bricks);
    w.bmask = bmask;
    struct Task { float t; uint32_t cell, last; };
    static Task tasks[4096];
    int n = 0, done = 0;
    GridWalk k;
    ShadowRay g;
    const auto* masks = reinterpret_cast<const unsigned long long*>(ucell);
    int st = gw_init(k, g, masks, O[0], O[1], O[2], D[0], D[1], D[2], steps) ? GW_UBER : GW_END;
    bool hit = false;
    float d2 = 0.0f;
    uint32_t s2 = 0;
    auto finish = [&]() {
        for (; done < n && !hit; done++) {
            const Task& q = tasks[done];
            const uint32_t o = grid[q.cell & 0x1FFFFFu];
            float out;
            const int kind = bbox ? grid_task<true>(o, (o & 1u) ? bbox[o >> 1] : 0u, q.cell, g, &out)
                                  : grid_task<false>(o, 0u, q.cell, g, &out);
            s2 = q.last;
            if (kind == 1) { hit = true; d2 = q.t * 8.0f; }
            if (kind == 2) {
                stats[3]++;
                const auto walk = bmask ? brick_task<true> : brick_task<false>;
                hit = walk(w, o >> 1, q.cell, q.t, out, q.last, g, &d2, &s2);
            }
        }
    };
    while (st != GW_END && !hit) {
        if (st == GW_UBER) {
            st = gw_enter(k, g, masks);
            if (st == GW_GRID) stats[0]++;
            continue;
        }
        bool task = false;
        if (!gw_visit(k, &task)) { st = GW_END; continue; }
        stats[1]++;
        if (task) {
            stats[2]++;
            tasks[n++] = Task{k.t, k.p & 0x1FFFFFu, k.last};
            if (!deferred) finish();
        }
        if (!gw_step(k)) st = GW_UBER;
    }
    finish();
    d2 = hit ? d2 + g.to : 0.0f;
    s2 = hit ? s2 : 0u;
    *dist = d2;
    *side = hit ? s2 : 3u;
    const float3 L = f3(D[0], D[1], D[2]);
    const float ns = side_sign(s2, L);
    const float hx = L.x * d2 + O[0], hy = L.y * d2 + O[1], hz = L.z * d2 + O[2];
    const uint32_t vx = f2u(hx - (s2 == 0 ? ns * 0.1f : 0.0f));
    const uint32_t vy = f2u(hy - (s2 == 1 ? ns * 0.1f : 0.0f));
    const uint32_t vz = f2u(hz - (s2 == 2 ? ns * 0.1f : 0.0f));
    const uint32_t ey = pos / (1024u * 1024u), ez = (pos / 1024u) % 1024u, ex = pos % 1024u;
    return ex <= vx && ex + size > vx && ey <= vy && ey + size > vy && ez <= vz && ez + size > vz;
}

int dh_can_reach(const uint8_t* uber, const float* O, const float* D, uint32_t pos, uint32_t size, int steps) {
    return shadow_can_reach(uber, f3(O[0], O[1], O[2]), f3(D[0], D[1], D[2]), pos,
                            size, steps);
}

// trace_first with a budget, or a primary ray (boxes: gbox0 given; masks of the bricks' non-zero
// voxels: bmask0 given)
uint32_t dh_trace_first(const uint32_t* grid, const uint8_t* uber, const uint32_t* bricks, const uint32_t* ucell0, const uint32_t* gbox0,
                        const uint32_t* bmask0, const float* O, const float* D, int budget, int steps, float* dist, uint32_t* side) {
    World w = make_world(grid, uber, bricks);
    w.ucell0 = reinterpret_cast<const uint4*>(ucell0);
    w.gbox0 = reinterpret_cast<const uint2*>(gbox0);
    w.bmask0 = bmask0;
    *dist = 0.0f;
    *side = 0;
    if (!budget)
        return (bmask0 ? trace_primary<true> : trace_primary<false>)(w, f3(O[0], O[1], O[2]), f3(D[0], D[1], D[2]), dist, side);
    const auto f = !gbox0 ? trace_first<0, true, false> : bmask0 ? trace_first<1, true, true> : trace_first<1, true, false>;
    return f(w, O[0], O[1], O[2], D[0], D[1], D[2], steps, dist, side);
}

// trace<1> over cell masks
uint32_t dh_trace_opaque(const uint32_t* grid, const uint8_t* uber, const uint32_t* bricks, const uint32_t* ucell, const uint32_t* gbox,
                         const uint32_t* bmask, const float* O, const float* D, int steps, float* dist, uint32_t* side) {
    World w = make_world(grid, uber, bricks);
    w.ucell = reinterpret_cast<const unsigned long long*>(ucell);
    w.gbox = reinterpret_cast<const uint2*>(gbox);
    w.bmask = bmask;
    *dist = 0.0f;
    *side = 0;
    return trace_first<1, true, true, true>(w, O[0], O[1], O[2], D[0], D[1], D[2], steps, dist, side);
}

// An area-light candidate: one call (area_candidate) and the two functions it stands for.
// in: light centre, size, emission rgb, shading point, offset point, normal sign, albedo/pi rgb;
// out[which]: ph, seed bits, point xyz, weight, face bits. Returns area_candidate's answer.
int dh_area_candidate(const float* in, uint32_t side, uint32_t seed, float* out) {
    const float4 g = make_float4(in[0], in[1], in[2], in[3]), em = make_float4(in[4], in[5], in[6], 0.0f);
    const float3 sp = f3(in[7], in[8], in[9]), spo = f3(in[10], in[11], in[12]), brdf = f3(in[14], in[15], in[16]);
    int ok = 0;
    for (int which = 0; which < 2; which++) {
        uint32_t s = seed, face = 9;
        float3 pos = f3(0.0f, 0.0f, 0.0f);
        float ph = 0.0f, inv = 0.0f;
        if (which == 0) {
            ok = area_candidate(g, em, sp, spo, side, in[13], brdf, s, &ph, &pos, &inv, &face);
        } else {
            pos = sample_area_light(g, spo, s, &inv, &face);
            ph = phat<false>(pos, face, sp, side, in[13], brdf, em, g.w) * inv;
        }
        float* o = out + 7 * which;
        o[0] = ph; o[2] = pos.x; o[3] = pos.y; o[4] = pos.z; o[5] = inv;
        std::memcpy(o + 1, &s, 4);
        std::memcpy(o + 6, &face, 4);
    }
    return ok;
}

}  // extern "C"
