// charge_kernel.inl -- the batched charge kernel, included by charges_batched.cu once per form:
//   CHARGE_DEFER 0: a step's event (Luke emission, intervalley scatter, trap) is drawn at once;
//   CHARGE_DEFER 1: it waits until a quarter of the warp's carriers wait for theirs, while the
//                   others go on stepping.
// A carrier that differs in one bit takes another path, and which form runs depends on the size of
// the batch, so both have to round alike. One text for both makes that likely (a template's two
// instances were contracted into different multiply-adds), not certain: tests/test_gpu_charge_forms.py
// compares them over fields, masks, released energies and parked carriers. With open trapping
// channels they differ in a trapped carrier's energy, and such crystals keep the first form
// (charges_wait).
//
// A carrier is one serial chain of ~19,000 steps, so a step's instruction count is its latency
// (few carriers) as well as its throughput (many). A step without an event (nine of ten) does
// only what the next one reads: |k| once, the velocity of the rates only where a trapping
// channel is open, no kinetic energy (the intervalley threshold is decided by |k|), and no
// exit point for a carrier far from every wall. 4,000 carriers (the first form) 101 -> 66 ms, the
// carriers and phonons of 64 light recoils 117 -> 88 ms; 100,000 carriers 182 -> 134 ms in the first
// form, 99 ms in the waiting one that runs at that size.
// (128, 5): 96 registers, five blocks per SM (with the step as it was, pair drift of 200,000
// events 467 -> 431 ms against (128, 4) at 104 registers; (128, 6) at 80 registers 432 ms)
__global__ void __launch_bounds__(128, 5) CHARGE_KERNEL(const __grid_constant__ FCLat Lp,
                                                         const __grid_constant__ FCDet D,
                                                         const __grid_constant__ RunArgs a,
                                                         const __grid_constant__ ChargeArgs ca) {
    // the crystal constants (the Herring-Vogt valley rotations and mass tensor among them) in
    // shared memory: the step reads the rotation of each carrier's own valley, an index that
    // differs between the lanes of a warp, which the constant bank of the kernel parameters
    // serves one distinct address at a time
    __shared__ alignas(16) FCLat sL;
    static_assert(sizeof(FCLat) % 4 == 0, "FCLat is copied in 4-byte words");
    for (int i = threadIdx.x; i < static_cast<int>(sizeof(FCLat) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&sL)[i] = reinterpret_cast<const uint32_t*>(&Lp)[i];
    __syncthreads();
    if (!lane_active(a.lanes)) return;
#if CHARGE_DEFER
    const unsigned warp_mask = 0xffffffffu >> (32u - a.lanes);
#endif
    const FCLat& L = sL;
    Carrier k;
    CStats st{};
    QCharge knock[kKnockCap];
    int n_knock_stk = 0;
    uint64_t q_next = 0, q_end = 0;  // queue slots reserved by this thread
    unsigned err = 0;
    bool live = false, stop = false, dirty = false;
    const bool track_luke = D.luke_prob > 0.0f;
    const double e_gap = L.bandgap_d;
    F3 E_last = f3(kInfF, 0.0f, 0.0f);
    float iv_last = 0.0f, dk_last = 0.0f;  // of E_last: intervalley rate, |dk/dt| of a unit mass factor
    // c.ekin follows c.p only where it is read: a step without an event (nine of ten) leaves it,
    // and the next step compares |k| with the intervalley threshold instead
    bool ek_known = true;
#if CHARGE_DEFER
    bool done = false;
    FRates R{};            // rates of the step that ended in the pending event
    bool pending = false;  // the carrier's step ended in an event that has not been drawn yet
#endif
    for (;;) {
#if CHARGE_DEFER
        if (!live && !done) {
#else
        if (!live) {
#endif
            if (dirty) {
                sink_charge(a, k.ev, st);
                st = CStats{};
                dirty = false;
            }
            if (n_knock_stk > 0) {
                k = unpark(knock[--n_knock_stk]);
#if CHARGE_DEFER
                live = true;
#endif
            } else if (stop) {
                CHARGE_DONE;
            } else {
                const unsigned long long r = (ca.n_resume_in > 0) ? atomicAdd(ca.resume_next, 1ull) : ~0ull;
                if (r < ca.n_resume_in) {
                    k = unpark(ca.resume_in[r]);
#if CHARGE_DEFER
                    live = true;
                } else if (const unsigned long long at = atomicAdd(ca.next_carrier, 1ull); at >= ca.n_carriers) {
                    done = true;
                } else {
                    const uint32_t i = ca.order[at];
#else
                } else {
                    const unsigned long long i = atomicAdd(ca.next_carrier, 1ull);
                    if (i >= ca.n_carriers) break;
#endif
                    const uint32_t ev = ca.carrier_event[i];
                    const uint64_t j = i - a.ch_off[ev];
                    const cmpmc_charge_track& in = a.ch[i];
                    k.c.pos = f3(static_cast<float>(in.pos[0]), static_cast<float>(in.pos[1]),
                                 static_cast<float>(in.pos[2]));
                    k.c.p = f3(static_cast<float>(in.p_eV[0]), static_cast<float>(in.p_eV[1]),
                               static_cast<float>(in.p_eV[2]));
                    k.c.ekin = static_cast<float>(in.ekin);
                    k.c.t = in.time;
                    k.c.w = static_cast<float>(in.weight);
                    k.c.valley = in.valley;
                    k.c.type = in.type;
                    k.ckey = mix64(ca.carrier_seed ^ mix64(((a.first_event + ev) << 20) | j));
                    k.g.seed(k.ckey);
                    k.ev = ev;
                    k.luke_idx = 0;
                    k.n_knock = 0;
                    k.steps = 0;
                    k.hint = -1;
#if CHARGE_DEFER
                    live = true;
#endif
                }
            }
#if !CHARGE_DEFER
            live = true;
#endif
            ek_known = true;
        }
#if CHARGE_DEFER
        if (!__any_sync(warp_mask, live)) break;
        if (live && !pending) do {
#endif
        // one step may queue one Luke phonon: hold a free slot before drawing anything
        if (track_luke && q_next == q_end) {
            const unsigned long long base = atomicAdd(ca.q_tail, static_cast<unsigned long long>(kQBlock));
            if (base + kQBlock > ca.q_cap) {
                // queue full: park this carrier and every pending knock-on, stop the thread
                const unsigned long long slot = atomicAdd(ca.n_resume_out, 1ull);
                if (!ek_known) k.c.ekin = ekin_of(L, k.c);
                if (slot < ca.resume_cap) ca.resume_out[slot] = park(k);
                else err |= kErrResume;
                while (n_knock_stk > 0) {
                    const unsigned long long s2 = atomicAdd(ca.n_resume_out, 1ull);
                    if (s2 < ca.resume_cap) ca.resume_out[s2] = knock[--n_knock_stk];
                    else { err |= kErrResume; --n_knock_stk; }
                }
                live = false;
                stop = true;
                CHARGE_NEXT;
            }
            q_next = base;
            q_end = base + kQBlock;
        }
        if (k.steps >= 20000000u) {  // the reference's step bound per carrier (engine.hpp:208)
            live = false;
            CHARGE_NEXT;
        }
        FCharge& c = k.c;
        ++k.steps;
        ++st.steps;
        dirty = true;
        const float q_sign = (c.type == 1) ? -1.0f : 1.0f;
        const F3 E = D.mesh.tet ? mesh_field_f(D.mesh, c.pos, k.hint)
                                : (D.mesh2.tri ? mesh2_field_f(D.mesh2, c.pos, k.hint) : D.e_field);
        if (E.x != E_last.x || E.y != E_last.y || E.z != E_last.z) {
            E_last = E;
            iv_last = iv_rate_of_field(L, E);
            dk_last = fnorm(E) * (kCLightF / kHbarCF);
        }
        const bool is_e = (c.type == 1);
        const float kmag = kmag_of(L, c);
        float iv = 0.0f;
        if (is_e && L.n_valleys >= 2) {
            // outside the threshold's band |k| decides as the energy would
            const bool above = ek_known ? c.ekin >= L.iv_min
                               : (kmag < L.k_iv_lo || kmag > L.k_iv_hi) ? kmag > L.k_iv_hi
                                                                        : ekin_e(L, c.valley, c.p) >= L.iv_min;
            iv = above ? iv_last : 0.0f;
        }
        const FRates R0 = rates_at(L, c, kmag, iv);
#if CHARGE_DEFER
        R = R0;
#else
        FRates R = R0;
#endif
        float dt_max = D.dt_cap;
        if (D.dk_frac > 0.0f) {
            const float ks = is_e ? L.ks_e : L.ks_h;
            const float dk_rate = dk_last * (is_e ? L.hv_max : 1.0f);
            if (dk_rate > 0.0f) dt_max = fminf(dt_max, D.dk_frac * fmaxf(ks, kmag) / dk_rate);
        }
        float dt_phys;
        if (D.second) {
            // Leman second-order stepping (engine.hpp:235-254): rate linear in time
            FCharge trial = c;
            trial.p = trial.p + E * (q_sign * kCLightF * dt_max);
            trial.ekin = ekin_of(L, trial);
            const float a0 = R0.tot;
            const float a1 = (rates_of(L, trial, iv_last).tot - a0) / dt_max;
            const float lnu = __logf(k.g.u());
            if (fabsf(a1) * dt_max <= 1e-6f * fmaxf(a0, 1e-30f)) {
                dt_phys = (a0 > 0.0f) ? (-lnu / a0) : kInfF;
            } else {
                const float disc = a0 * a0 - 2.0f * a1 * lnu;
                const float den = sqrtf(fmaxf(disc, 0.0f)) + a0;  // (sqrt(disc) - a0) / a1, cancellation-free
                dt_phys = (disc < 0.0f || !(den > 0.0f)) ? kInfF : (-2.0f * lnu / den);
                if (!(dt_phys >= 0.0f)) dt_phys = kInfF;
            }
        } else {
            dt_phys = (R0.tot > 1.0f) ? (-__logf(k.g.u()) / R0.tot) : kInfF;
        }
        const float dt = fminf(dt_phys, dt_max);
        const F3 dp = E * (q_sign * kCLightF * dt);
        const F3 p_mid = c.p + dp * 0.5f;
        const F3 v_mid = vel_of(L, c.type, c.valley, p_mid);
        const float v_mag = fnorm(v_mid);
        const float d_step = v_mag * dt;
        const bool inside = clear_of_walls(D.R, D.H, D.edge, c.pos.x, c.pos.y, c.pos.z, d_step);
        if (!inside && v_mag > 1e-6f) {
            const F3 v_dir = v_mid * (1.0f / v_mag);
            const FBHit bh = fexit(D.R, D.H, c.pos, v_dir);
            if (bh.d <= d_step) {
                const float dt_b = bh.d / v_mag;
                c.pos = c.pos + v_dir * bh.d;
                c.t += static_cast<double>(dt_b);
                c.p = c.p + E * (q_sign * kCLightF * dt_b);
                c.ekin = ekin_of(L, c);
                ek_known = true;
                const FCSurf& s = D.surf[bh.surf];
                // electrode mask (engine.hpp:284-289), then ChargePhysics::should_absorb_boundary
                // (charge_transport.hpp:187-199)
                int ch_id = -1;
                bool absorb = true;
                if (s.n_pads > 0) {
                    // the out-of-line call gets a copy: only it has its address taken, so
                    // the carrier state stays in registers
                    R128 g_c = k.g;
                    ch_id = mask_call(s.pads, s.n_pads, c.pos.x, c.pos.y, &g_c);
                    k.g = g_c;
                    absorb = ch_id >= 0;
                }
                const float k_perp = -fdot(c.p * (1.0f / kHbarCF), bh.n);
                if (absorb) absorb = k_perp > ((c.type == 1) ? s.min_k_e : s.min_k_h) && k.g.u() < s.prob_abs;
                if (!absorb) {
                    ++st.crefl;
                    c.pos = c.pos + bh.n * kNudge;
                    // ChargePhysics::reflect_at_boundary (charge_transport.hpp:203-241)
                    bool mirrored = false;
                    if (k.g.u() < s.prob_spec) {
                        const F3 kd = funit(c.p);
                        const F3 kr = funit(kd - bh.n * (2.0f * fdot(kd, bh.n)));
                        if (c.type == 2) {
                            c.p = kr * fnorm(c.p);
                            mirrored = true;
                        } else {
                            const F3 pt = ekin_to_p_e(L, c.valley, kr, c.ekin);
                            if (fdot(vel_of(L, 1, c.valley, pt), bh.n) > 1e-6f) {
                                c.p = pt;
                                mirrored = true;
                            }
                        }
                    }
                    if (!mirrored) {
                        const F3 e1 = forth(bh.n);
                        const F3 e2 = fcross(bh.n, e1);
                        if (c.type == 2) {
                            const float phi = kTwoPiF * k.g.u();
                            const float st_ = sqrtf(k.g.u());
                            const float ct = sqrtf(fmaxf(0.0f, 1.0f - st_ * st_));
                            float sp, cp;
                            __sincosf(phi, &sp, &cp);
                            c.p = funit(e1 * (st_ * cp) + e2 * (st_ * sp) + bh.n * ct) * fnorm(c.p);
                        } else {
                            int trial = 0;
                            for (; trial < 16; ++trial) {
                                const float phi = kTwoPiF * k.g.u();
                                const float st_ = sqrtf(k.g.u());
                                const float ct = sqrtf(fmaxf(0.0f, 1.0f - st_ * st_));
                                float sp, cp;
                                __sincosf(phi, &sp, &cp);
                                const F3 dir = funit(e1 * (st_ * cp) + e2 * (st_ * sp) + bh.n * ct);
                                const F3 pt = ekin_to_p_e(L, c.valley, dir, c.ekin);
                                if (fdot(vel_of(L, 1, c.valley, pt), bh.n) > 1e-6f) {
                                    c.p = pt;
                                    break;
                                }
                            }
                            if (trial == 16) c.p = ekin_to_p_e(L, c.valley, bh.n, c.ekin);
                        }
                    }
                    CHARGE_NEXT;
                }
                // collection_release_energy (engine.hpp:889-893)
                const double e_rel = static_cast<double>(c.ekin) + ((c.type == 1) ? (e_gap - D.muF) : D.muF);
                ++st.collected;
                if (s.release) {
                    // BulkDebye / ElectrodeFilm (engine.hpp:302-313): the release kernel emits
                    // the phonons, runs the film cascades and records the hit
                    const unsigned long long slot = atomicAdd(ca.rel_tail, 1ull);
                    if (slot < ca.rel_cap) {
                        ReleaseRec r;
                        r.px = c.pos.x; r.py = c.pos.y; r.pz = c.pos.z;
                        r.w = c.w;
                        r.e_rel = e_rel;
                        r.t = c.t;
                        const uint64_t hi = k.g.next();
                        r.key = (hi << 32) | k.g.next();
                        r.ev = k.ev;
                        r.ch_id = ch_id;
                        r.surf = static_cast<uint8_t>(bh.surf);
                        r.type = static_cast<uint8_t>(c.type);
                        r.pad0 = r.pad1 = 0;
                        r.pad2 = 0;
                        ca.rel[slot] = r;
                    } else {
                        err |= kErrRelease;
                    }
                    live = false;
                    CHARGE_NEXT;
                }
                // ChargeRelease::RecordOnly
                const double recomb = e_rel * static_cast<double>(c.w);
                st.recomb_eV += recomb;
                st.dep += recomb;
                if (a.keep_hits) {
                    atomicAdd(reinterpret_cast<unsigned long long*>(a.ev_nhits + k.ev), 1ull);
                    const unsigned long long idx = atomicAdd(a.hit_count, 1ull);
                    if (idx < a.hit_cap) {
                        cmpmc_sensor_hit h;
                        h.pos[0] = c.pos.x; h.pos[1] = c.pos.y; h.pos[2] = c.pos.z;
                        h.time = c.t;
                        h.edep = recomb;
                        h.incident_energy = e_rel;
                        h.surface_id = static_cast<uint8_t>(bh.surf);
                        h.excitation = static_cast<uint8_t>(c.type);
                        h.mode = 0;
                        h._pad = 0;
                        h.channel_id = ch_id;
                        a.hit_stage[idx] = h;
                        a.hit_key[idx] = k.ev;
                    }
                }
                live = false;
                CHARGE_NEXT;
            }
        }
        c.pos = c.pos + v_mid * dt;
        c.t += static_cast<double>(dt);
        c.p = c.p + dp;
        ek_known = dt_phys <= dt_max;
#if CHARGE_DEFER
        pending = ek_known;
        } while (false);
        // both votes are taken by every lane of the mask, whatever it holds
        const unsigned ready = __ballot_sync(warp_mask, pending);
        const unsigned alive = __ballot_sync(warp_mask, live);
        if (ready && __popc(ready) * kDeferShare >= __popc(alive) && pending) do {
            pending = false;
            FCharge& c = k.c;
            const bool is_e = (c.type == 1);
            c.ekin = ekin_of(L, c);
#else
        if (dt_phys <= dt_max) {
            c.ekin = ekin_of(L, c);
#endif
            if (D.second) {
                R = rates_of(L, c, iv_last);
                if (R.tot <= 0.0f) CHARGE_NEXT;
            }
            const float u_proc = k.g.u() * R.tot;
            if (u_proc < R.trap) {
                ++st.trapped;
                st.esc += (static_cast<double>(c.ekin) + 0.5 * e_gap) * static_cast<double>(c.w);
                live = false;
                CHARGE_NEXT;
            } else if (u_proc < R.trap + R.ion_e + R.ion_h) {
                ++st.ion;
                const bool lib_e = (u_proc < R.trap + R.ion_e);
                const uint32_t nv = (L.n_valleys > 1) ? static_cast<uint32_t>(L.n_valleys) : 1u;
                const int kv = lib_e ? static_cast<int>(k.g.next() % nv) : 0;
                const float u1 = k.g.u(), u2 = k.g.u();
                const float ct = 2.0f * u1 - 1.0f, sn = sqrtf(fmaxf(0.0f, 1.0f - ct * ct));
                float sp, cp;
                __sincosf(kTwoPiF * u2, &sp, &cp);
                Carrier kn;
                kn.c = make_charge_f(L, lib_e ? 1 : 2, c.pos, f3(sn * cp, sn * sp, ct), 1.0e-6f, kv, c.t, c.w);
                kn.ckey = mix64(k.ckey ^ (0xd6e8feb86659fd93ULL * (static_cast<uint64_t>(++k.n_knock))));
                kn.g.seed(kn.ckey);
                kn.ev = k.ev;
                kn.luke_idx = 0;
                kn.n_knock = 0;
                kn.steps = 0;
                kn.hint = k.hint;
                if (n_knock_stk < kKnockCap) knock[n_knock_stk++] = park(kn);
                else err |= kErrChargeStack;
            } else if (u_proc < R.trap + R.ion_e + R.ion_h + R.iv) {
                // ChargePhysics::scatter_intervalley (charge_transport.hpp:169-184)
                const int nv = L.n_valleys;
                if (c.type == 1 && nv >= 2) {
                    const F3 kv = mulr(L.rot[c.valley], c.p * (1.0f / kHbarCF));
                    const int off = 1 + min(static_cast<int>(k.g.u() * static_cast<float>(nv - 1)), nv - 2);
                    const int nvl = (c.valley + off) % nv;
                    const F3 kn = mulrt(L.rot[nvl], kv);
                    c.valley = nvl;
                    c.p = ekin_to_p_e(L, nvl, kn * kHbarCF, c.ekin);
                }
                ++st.iv;
            } else if (R.luke > 0.0f) {
                // ChargePhysics::emit_luke_phonon (charge_transport.hpp:109-166)
                const F3 kt = is_e ? e2s(L, c.valley, c.p * (1.0f / kHbarCF)) : c.p * (1.0f / kHbarCF);
                const float ks = is_e ? L.ks_e : L.ks_h;
                const float km = fnorm(kt);
                if (km > ks * 1.0001f) {
                    const F3 kdir = kt * (1.0f / km);
                    const float v = ks / km;
                    const float u = k.g.u();
                    const float cth = fminf(fmaxf(v + (1.0f - v) * cbrtf(1.0f - u), v), 1.0f);
                    const float sth = sqrtf(fmaxf(0.0f, 1.0f - cth * cth));
                    const float phi = kTwoPiF * k.g.u();
                    const float q = 2.0f * (km * cth - ks);
                    if (q > 0.0f) {
                        float sp, cp;
                        __sincosf(phi, &sp, &cp);
                        const F3 perp = forth(kdir);
                        const F3 qv = frotate(frotate(kdir * q, perp, cth, sth), kdir, cp, sp);
                        const F3 krec = kt - qv;
                        const float e_ph = fnorm(qv) * L.vs_hbar;
                        if (e_ph < c.ekin && e_ph > 0.0f) {
                            F3 qdir;
                            if (!is_e) {
                                c.p = krec * kHbarCF;
                                c.ekin = ekin_h(L, c.p);
                                qdir = funit(qv);
                            } else {
                                qdir = funit(s2e(L, c.valley, qv));
                                const float e_rec = c.ekin - e_ph;
                                c.p = ekin_to_p_e(L, c.valley, s2e(L, c.valley, krec) * kHbarCF, e_rec);
                                c.ekin = e_rec;
                            }
                            ++st.luke;
                            st.luke_eV += static_cast<double>(e_ph) * static_cast<double>(c.w);
                            if (track_luke && (D.luke_prob >= 1.0f || k.g.u() < D.luke_prob)) {
                                const float um = k.g.u();
                                QPhonon qp;
                                qp.px = c.pos.x; qp.py = c.pos.y; qp.pz = c.pos.z;
                                qp.kx = qdir.x; qp.ky = qdir.y; qp.kz = qdir.z;
                                qp.w = c.w * D.luke_wt;
                                qp.mode = static_cast<uint32_t>((um < L.fL) ? 0 : ((um < L.fLST) ? 2 : 1));
                                qp.E = static_cast<double>(e_ph);
                                qp.t = c.t;
                                qp.key = luke_key(k.ckey, k.luke_idx++);
                                qp.ev = k.ev;
                                qp.pad = 0;
                                ca.queue[q_next++] = qp;
                            }
                        }
                    }
                }
            }
#if CHARGE_DEFER
        } while (false);
#else
        }
#endif
    }
    if (dirty) sink_charge(a, k.ev, st);
    if (err) atomicOr(a.err, err);
}
