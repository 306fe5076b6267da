// Adjoint of the fused step: forward with checkpoints, backward with recomputation.
// Included by visg_api.cu (member functions of Engine).
//
// visg_forward starts from the simulator's current state, runs the differentiable
// trajectory in FP64 (launch_step_f64: the same algorithm as the float step, in
// double) and keeps its state (x, x_old, contact normal) every `ckpt` steps; at the
// end the simulator's float state is set to the FP64 final state rounded to float.
// visg_backward walks the segments from the last to the first: it replays a segment's
// steps from its checkpoint (deterministic, so the contact set is the forward pass's),
// recording every intermediate state, then runs the two adjoint kernels per step in
// reverse.  The forward pass writes its last segment's states straight into that
// record, so the backward pass after it starts with no replay.

int Engine::forward(int nsteps, int ckpt) {
    if (!finalized) return fail(VISG_ERR_STATE, "not finalized");
    if (G != 1) return fail(VISG_ERR_UNSUPPORTED, "the adjoint runs on a single-garment simulator");
    if (nsteps < 1 || ckpt < 1) return fail(VISG_ERR_INVALID_ARG, "nsteps and checkpoint_every must be >= 1");
    if (!adj.rev) {
        // reverse entry of every directed spring (same list, k-th duplicate to k-th)
        std::vector<uint32_t> hrev(E > 0 ? E : 1, 0xffffffffu);
        std::vector<uint2> ent(E > 0 ? E : 1);
        CU(cudaMemcpy(ent.data(), d_ent, E * sizeof(uint2), cudaMemcpyDeviceToHost));
        for (int64_t i = 0; i < N; ++i) {
            const uint32_t rp = h_rowp[i] & ROW_MASK, re = h_rowp[i + 1] & ROW_MASK;
            for (uint32_t e = rp; e < re; ++e) {
                if (hrev[e] != 0xffffffffu) continue;
                const uint32_t j = ent[e].x & END_MASK, l = ent[e].x >> LIST_SHIFT;
                const uint32_t jp = h_rowp[j] & ROW_MASK, je = h_rowp[j + 1] & ROW_MASK;
                bool found = false;
                for (uint32_t f = jp; f < je && !found; ++f)
                    if (f != e && (ent[f].x & END_MASK) == (uint32_t)i && (ent[f].x >> LIST_SHIFT) == l &&
                        hrev[f] == 0xffffffffu) {
                        hrev[e] = f;
                        hrev[f] = e;
                        found = true;
                    }
                if (!found)
                    return fail(VISG_ERR_UNSUPPORTED,
                                "the adjoint needs a symmetric spring graph (i->j and j->i in the same list)");
            }
        }
        const size_t eb = (size_t)std::max<int64_t>(E, 1) * 4;
        std::vector<uint32_t> hsrc(eb / 4, 0u), hpos(eb / 4, 0u);
        for (int64_t i = 0; i < N; ++i)
            for (uint32_t e = h_rowp[i] & ROW_MASK; e < (h_rowp[i + 1] & ROW_MASK); ++e) hsrc[e] = (uint32_t)i;
        for (int64_t e = 0; e < E; ++e) hpos[e] = (uint32_t)merged_pos[e];
        if (!adj.src) CU(cudaMalloc((void**)&adj.src, eb));
        if (!adj.pos) CU(cudaMalloc((void**)&adj.pos, eb));
        CU(cudaMemcpy(adj.src, hsrc.data(), eb, cudaMemcpyHostToDevice));
        CU(cudaMemcpy(adj.pos, hpos.data(), eb, cudaMemcpyHostToDevice));
        if (!adj.rest64) CU(cudaMalloc((void**)&adj.rest64, (perk ? 4 : 2) * eb));
        CU(launch_entries_f64(d_ent, d_k, adj.rest64, perk ? adj.rest64 + eb / 4 : nullptr, E, stream));
        uint32_t* rev = nullptr;
        CU(cudaMalloc((void**)&rev, eb));
        adj.rev = rev;
        CU(cudaMemcpy(adj.rev, hrev.data(), eb, cudaMemcpyHostToDevice));
    }
    const size_t n3 = 3 * (size_t)N, st = 9 * (size_t)N, e1 = (size_t)std::max<int64_t>(E, 1);
    const int nck = (nsteps + ckpt - 1) / ckpt;
    adj.ready = false;
    adj.rec_seg = -1;
    while ((int)adj.ck.size() > nck) {
        cudaFree(adj.ck.back());
        adj.ck.pop_back();
    }
    while ((int)adj.ck.size() < nck) {
        double* q = nullptr;
        CU(cudaMalloc((void**)&q, st * sizeof(double)));
        adj.ck.push_back(q);
    }
    const size_t rec_states = (size_t)std::min(ckpt, nsteps) + 1;
    if (adj.rec_states != rec_states) {
        cudaFree(adj.rec);
        adj.rec = nullptr;
        adj.rec_states = 0;
        CU(cudaMalloc((void**)&adj.rec, rec_states * st * sizeof(double)));
        adj.rec_states = rec_states;
    }
    if (!adj.tmp) CU(cudaMalloc((void**)&adj.tmp, 2 * st * sizeof(double)));
    if (!adj.vel) CU(cudaMalloc((void**)&adj.vel, 2 * n3 * sizeof(double)));
    if (!adj.lam) CU(cudaMalloc((void**)&adj.lam, 2 * n3 * sizeof(double)));
    if (!adj.G) CU(cudaMalloc((void**)&adj.G, n3 * sizeof(double)));
    if (!adj.gx) CU(cudaMalloc((void**)&adj.gx, 6 * e1 * sizeof(double)));
    if (damped_springs() && !adj.gxo) CU(cudaMalloc((void**)&adj.gxo, 6 * e1 * sizeof(double)));
    if (!adj.dk) CU(cudaMalloc((void**)&adj.dk, (2 * e1 + 2 * n3) * sizeof(double)));
    if (!adj.out) CU(cudaMalloc((void**)&adj.out, e1 * sizeof(float)));
    if (!adj.dsc) CU(cudaMalloc((void**)&adj.dsc, 4 * sizeof(double)));
    if (!adj.wild) CU(cudaMalloc((void**)&adj.wild, sizeof(uint32_t)));
    if (adj.contacts_cap < nsteps) {
        cudaFree(adj.contacts);
        adj.contacts = nullptr;
        adj.contacts_cap = 0;
        CU(cudaMalloc((void**)&adj.contacts, (size_t)nsteps * sizeof(unsigned)));
        adj.contacts_cap = nsteps;
    }
    CU(cudaMemsetAsync(adj.contacts, 0, (size_t)nsteps * sizeof(unsigned), stream));
    CU(cudaMemsetAsync(adj.wild, 0, sizeof(uint32_t), stream));
    adj.ckpt = ckpt;
    adj.nsteps = nsteps;
    // State t lives in its checkpoint, or, inside the last segment, in that segment's
    // record (the backward pass starts there, so it need not replay it), or in one of two
    // buffers; each step reads one of them and writes the next, nothing is copied.
    const int last = nck - 1;
    auto place = [&](int t) -> double* {
        if (t % ckpt == 0 && t < nsteps) return adj.ck[t / ckpt];
        if (t > last * ckpt) return adj.rec + (size_t)(t - last * ckpt) * st;
        return adj.tmp + (size_t)(t & 1) * st;
    };
    double* first = place(0);
    CU(launch_unpack_state(d_state[cur], d_state[cur ^ 1], d_normal, 0, N, d_stage, d_stage + n3, d_stage + 2 * n3,
                           stream));
    CU(launch_widen(d_stage, first, (int64_t)st, stream));
    CU(launch_vel_f64(first, first + n3, damped_springs() ? adj.vel : nullptr, p.dt, adj.wild, (int64_t)n3, stream));
    for (int s = 0; s < nsteps; ++s) CU(step64(place(s), place(s + 1), s, adj.contacts + s));
    // the simulator continues from the FP64 final state, rounded to float
    CU(launch_narrow(place(nsteps), d_stage, (int64_t)st, stream));
    CU(launch_pack_state(d_state[cur], d_state[cur ^ 1], d_normal, 0, N, d_stage, d_stage + n3, d_stage + 2 * n3, p.dt,
                         step_params().drec, step_params().dmax, d_wild, stream));
    CU(cudaMemcpyAsync(h_status + 3, adj.wild, 4, cudaMemcpyDeviceToHost, stream));
    if (int r = sync()) return r;
    adj.was_wild = h_status[3] != 0;
    adj.changed = false;
    adj.rec_seg = last;
    adj.ready = true;
    return VISG_OK;
}

// one FP64 step from state `from` to state `to` ([x | x_old | normal] each), the k-th of its
// run (velocities alternate between two buffers); with `contacts`, the step's projected
// vertices are counted there
cudaError_t Engine::step64(const double* from, double* to, int k, unsigned* contacts) {
    const size_t n3 = 3 * (size_t)N;
    const bool coll = p.collide && any_body;
    Step64Args a;
    a.x = from;
    a.xo = from + n3;
    a.n_in = from + 2 * n3;
    a.xn = to;
    a.xon = to + n3;
    a.n_out = to + 2 * n3;
    a.v = damped_springs() ? adj.vel + (size_t)(k & 1) * n3 : nullptr;
    a.vn = damped_springs() ? adj.vel + (size_t)((k & 1) ^ 1) * n3 : nullptr;
    a.rowp = d_rowp;
    a.ent = d_ent;
    a.src = adj.src;
    a.rest64 = adj.rest64;
    a.k64 = perk ? adj.rest64 + std::max<int64_t>(E, 1) : nullptr;
    for (int l = 0; l < VISG_MAX_LISTS; ++l) a.list_k[l] = (double)p.list_k[l];
    a.bodies = d_views;
    a.body_verts = coll ? bvh[0].verts : nullptr;
    a.body_tris = coll ? bvh[0].tris : nullptr;
    a.p = step_params();
    a.refv = (variant() & SV_REFV) ? 1 : 0;
    a.collide = coll ? 1 : 0;
    a.n = (int)N;
    a.err = d_err;
    a.contacts = contacts;
    a.wild = adj.wild;
    return launch_step_f64(a, stream);
}

// vertices projected in each step of the last forward pass
int Engine::forward_contacts(int64_t* counts, int n) {
    if (!adj.ready) return fail(VISG_ERR_STATE, "visg_forward_contacts needs a visg_forward first");
    if (!counts || n < 0 || n > adj.nsteps) return fail(VISG_ERR_INVALID_ARG, "counts NULL or n out of range");
    std::vector<unsigned> h((size_t)std::max(n, 1));
    if (n > 0) CU(cudaMemcpyAsync(h.data(), adj.contacts, (size_t)n * sizeof(unsigned), cudaMemcpyDeviceToHost, stream));
    if (int r = sync()) return r;
    for (int k = 0; k < n; ++k) counts[k] = (int64_t)h[k];
    return VISG_OK;
}

int Engine::backward(const float* dL_dx, const float* dL_dxo, float* dL_dk, float* dL_dscalar) {
    if (!adj.ready) return fail(VISG_ERR_STATE, "visg_backward needs a visg_forward first");
    if (!dL_dx) return fail(VISG_ERR_INVALID_ARG, "dL_dx is NULL");
    const size_t n3 = 3 * (size_t)N, st = 9 * (size_t)N, e1 = (size_t)std::max<int64_t>(E, 1);
    // The springs' part in x_old: with spring damping, and where a state sets `wild`, which a
    // replay of the forward pass does only where that did.  48 of an entry's 136 bytes.
    if (!adj.gxo && (adj.was_wild || adj.changed)) CU(cudaMalloc((void**)&adj.gxo, 6 * e1 * sizeof(double)));
    CU(cudaMemcpyAsync(d_stage, dL_dx, n3 * sizeof(float), cudaMemcpyHostToDevice, stream));
    if (dL_dxo)
        CU(cudaMemcpyAsync(d_stage + n3, dL_dxo, n3 * sizeof(float), cudaMemcpyHostToDevice, stream));
    else
        CU(cudaMemsetAsync(d_stage + n3, 0, n3 * sizeof(float), stream));
    CU(launch_widen(d_stage, adj.lam, 2 * (int64_t)n3, stream));
    CU(cudaMemsetAsync(adj.dk, 0, (2 * e1 + 2 * n3) * sizeof(double), stream));
    CU(cudaMemsetAsync(adj.dsc, 0, 4 * sizeof(double), stream));
    AdjArgs a;
    a.rowp = d_rowp;
    a.ent = d_ent;
    a.src = adj.src;
    a.rev = adj.rev;
    a.rest64 = adj.rest64;
    a.k64 = perk ? adj.rest64 + e1 : nullptr;
    for (int l = 0; l < VISG_MAX_LISTS; ++l) a.list_k[l] = (double)p.list_k[l];
    a.kd = (double)p.spring_damping;
    a.lx = adj.lam;
    a.lxo = adj.lam + n3;
    a.G = adj.G;
    a.v = adj.vel;  // the replay of a segment is done with it when its reverse sweep starts
    a.gx = adj.gx;
    a.gxo = adj.gxo;
    a.dk = adj.dk;
    a.dkd = adj.dk + e1;
    a.dgc = adj.dk + 2 * e1;
    a.wild = adj.wild;
    a.gather = 0;
    a.n = (int)N;
    a.E = E;
    a.p = step_params();
    a.inv_dt = 1.0 / (double)p.dt;
    a.dt2_mass = (double)p.dt * (double)p.dt / (double)p.mass;
    a.damp_dt = (double)p.force_damping / (double)p.dt;
    for (int seg = (int)adj.ck.size() - 1; seg >= 0; --seg) {
        const int s0 = seg * adj.ckpt, s1 = std::min(s0 + adj.ckpt, adj.nsteps);
        auto state = [&](int t) { return t == s0 ? adj.ck[seg] : adj.rec + (size_t)(t - s0) * st; };
        if (adj.rec_seg != seg) {
            adj.rec_seg = -1;
            if (damped_springs())
                CU(launch_vel_f64(state(s0), state(s0) + n3, adj.vel, p.dt, adj.wild, (int64_t)n3, stream));
            for (int t = s0; t < s1; ++t) CU(step64(state(t), state(t + 1), t - s0));
            adj.rec_seg = seg;
        }
        for (int t = s1 - 1; t >= s0; --t) {
            const double* r = state(t);
            a.x = r;
            a.xo = r + n3;
            a.n_in = r + 2 * n3;  // the normals entering step t
            a.n_out = state(t + 1) + 2 * n3;
            CU(launch_adjoint_step(a, stream));
            a.gather = 1;
        }
    }
    unsigned* bad = reinterpret_cast<unsigned*>(adj.dsc + 3);
    CU(launch_adj_scalars(a.dgc, (int64_t)n3, a.dkd, E, adj.dsc, stream));
    CU(launch_adj_result(adj.dk, adj.pos, adj.out, bad, E, stream));
    double dsc[4];
    CU(cudaMemcpyAsync(dsc, adj.dsc, sizeof dsc, cudaMemcpyDeviceToHost, stream));
    if (dL_dk && E > 0)
        CU(cudaMemcpyAsync(dL_dk, adj.out, (size_t)E * sizeof(float), cudaMemcpyDeviceToHost, stream));
    if (int r = sync()) return r;
    unsigned nbad = 0;
    std::memcpy(&nbad, &dsc[3], sizeof nbad);
    const bool finite = nbad == 0 && std::isfinite((float)dsc[0]) && std::isfinite((float)dsc[1]) &&
                        std::isfinite((float)dsc[2]);
    if (dL_dscalar)
        for (int k = 0; k < 3; ++k) dL_dscalar[k] = (float)dsc[k];
    if (!finite)
        return fail(VISG_ERR_DIVERGED,
                    "the gradient is not finite in float: the trajectory's sensitivity overflowed (an unstable "
                    "forward, or a long stretch of sustained contact at a step size where a projected vertex's "
                    "update amplifies perturbations); the values were written as computed");
    return VISG_OK;
}
