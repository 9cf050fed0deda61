// charges_batched.cu -- the batched FP32 form of the charge transport
// (SimulationEngine::transport_charges, transport/engine.hpp:192-380): one device thread per
// carrier, drift steps in FP32, per-carrier time of flight and the energy ledger in FP64.
//
// Every carrier owns a random substream keyed by (run seed, event, index within the event),
// so carriers run concurrently in any order. A carrier that emits a tracked
// Neganov-Trofimov-Luke phonon appends it to a device queue instead of a per-event stack;
// the phonon kernel (k_queue_fp32) drains the queue between charge phases. Each queued
// phonon carries its own substream key (the carrier's lineage key mixed with the emission
// index), so a phonon's history does not depend on when or where it is transported.
//
// Queue room is reserved in blocks of kQBlock slots per thread, before the step that may
// need it. When the queue is full the carrier is parked with its generator state
// (QCharge) and the thread stops; the host drains the queue and resumes the parked
// carriers. Nothing waits on another thread, so no phase can stall.
//
// The field is the detector's uniform field or the tetrahedral mesh (DetectorModel::
// electric_field_at, engine.hpp:151-155), walked in FP32 from a per-carrier hint.
//
// FP32 care: kinetic energies are formed as p^2 / (sqrt(p^2 + m^2) + m), not
// sqrt(p^2 + m^2) - m (the rest energies are ~60 keV, the kinetic energies meV), and the
// second-order step solves its quadratic in the cancellation-free form.
#define CMPMC_DEVICE_FAST_MATH 1
#include <algorithm>

#include "charge_shortcuts.cuh"
#include "device.cuh"
#include "fp32.cuh"

namespace cmpmc_gpu {

namespace {

constexpr uint32_t kWaitLanes = 8;  // carriers per warp from which event draws wait
constexpr int kDeferShare = 4;  // of a warp's carriers, the part that waits for an event's draw
constexpr int kQBlock = 32;     // queue slots reserved per thread at a time
constexpr int kKnockCap = 8;    // knock-on carriers (trap ionization) pending per thread
constexpr float kHbarCF = static_cast<float>(kHbarC);
constexpr float kCLightF = static_cast<float>(kCLight);
constexpr float kInfF = __builtin_huge_valf();
constexpr float kMeshTol = -2e-6f;  // FP32 barycentric tolerance (rounding of p - x3 ~ 1e-6)
constexpr int kMeshMaxSteps = 4096;

// FP32 crystal constants of the charge transport (crystal_lattice.hpp:239-293, 322-331;
// charge_kernels.hpp:82-126)
struct FCLat {
    float rot[CMPMC_MAX_VALLEYS][9];
    F3 hv_sqrt, hv_sqrt_inv, inv_mass_ratio;
    float m_e, m_h;          // e_cond_mass, h_mass (eV)
    float ks_e, ks_h;        // k_sound (1/m)
    float tstep_e, tstep_h;  // 3 l0 / v_sound (s)
    float vs_hbar;           // v_sound * hbar (eV m)
    float hv_max;
    int n_valleys;
    int iv_model;
    int traps;               // some trapping or trap-ionisation mean free path is finite
    float k_iv_lo, k_iv_hi;  // |k| surely below / surely above the intervalley threshold iv_min
    float iv_min, iv_qrate, iv_qfield, iv_qpow_half, iv_lrate0, iv_lrate1, iv_lpow;
    float inv_trap_e, inv_trap_h, inv_ion_e_d0, inv_ion_e_a, inv_ion_h_d, inv_ion_h_a0;
    float fL, fLST;
    float bandgap;
    double bandgap_d;
};

struct FCSurf {
    float prob_abs, prob_spec, min_k_e, min_k_h;
    int n_pads;
    const Pad* pads;  // electrode mask
    int release;      // the collected energy goes to the release kernel (BulkDebye, or
                      // ElectrodeFilm on a surface with a film)
};

struct FCDet {
    float R, H;
    F3 e_field;
    FCSurf surf[3];
    float edge;              // distance to the walls below which a step tests its exit point
    float dt_cap, dk_frac;
    int second;              // Leman second-order stepping
    float luke_prob, luke_wt;
    double muF;
    MeshView32 mesh;
    MeshView2_32 mesh2;
};

struct FCharge {
    F3 pos, p;
    float ekin;
    double t;
    float w;
    int valley, type;  // type 1 electron, 2 hole
};

struct CStats {
    uint32_t steps, luke, iv, trapped, ion, crefl, collected;
    double luke_eV, recomb_eV, dep, esc;
};

__device__ __forceinline__ F3 mulr(const float* m, F3 v) {
    return f3(m[0] * v.x + m[1] * v.y + m[2] * v.z, m[3] * v.x + m[4] * v.y + m[5] * v.z,
              m[6] * v.x + m[7] * v.y + m[8] * v.z);
}
__device__ __forceinline__ F3 mulrt(const float* m, F3 v) {
    return f3(m[0] * v.x + m[3] * v.y + m[6] * v.z, m[1] * v.x + m[4] * v.y + m[7] * v.z,
              m[2] * v.x + m[5] * v.y + m[8] * v.z);
}
__device__ __forceinline__ F3 hmul(F3 a, F3 b) { return f3(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ float fnorm(F3 a) { return sqrtf(fdot(a, a)); }

// Herring-Vogt maps (crystal_lattice.hpp:239-293)
__device__ __forceinline__ F3 e2s(const FCLat& L, int iv, F3 v) { return hmul(mulr(L.rot[iv], v), L.hv_sqrt_inv); }
__device__ __forceinline__ F3 s2e(const FCLat& L, int iv, F3 v) { return mulrt(L.rot[iv], hmul(v, L.hv_sqrt)); }
__device__ __forceinline__ float kin_from_p2(float p2, float m) { return p2 / (sqrtf(p2 + m * m) + m); }
__device__ __forceinline__ float ekin_e(const FCLat& L, int iv, F3 p) {
    const F3 ph = e2s(L, iv, p);
    return kin_from_p2(fdot(ph, ph), L.m_e);
}
__device__ __forceinline__ float ekin_h(const FCLat& L, F3 p) { return kin_from_p2(fdot(p, p), L.m_h); }
__device__ __forceinline__ float ekin_of(const FCLat& L, const FCharge& c) {
    return (c.type == 1) ? ekin_e(L, c.valley, c.p) : ekin_h(L, c.p);
}
__device__ __forceinline__ F3 vel_of(const FCLat& L, int type, int iv, F3 p) {
    if (type == 1) {
        const float ek = ekin_e(L, iv, p);
        return mulrt(L.rot[iv], hmul(mulr(L.rot[iv], p), L.inv_mass_ratio)) * (kCLightF / (ek + L.m_e));
    }
    return p * (kCLightF / (ekin_h(L, p) + L.m_h));
}
__device__ __forceinline__ F3 ekin_to_p_e(const FCLat& L, int iv, F3 dir, float ek) {
    const F3 u = funit(dir);
    const F3 uh = e2s(L, iv, u);
    const float band = fdot(uh, uh);
    if (band <= 0.0f || ek <= 0.0f) return f3(0.0f, 0.0f, 0.0f);
    return u * sqrtf((ek * ek + 2.0f * ek * L.m_e) / band);
}
__device__ __forceinline__ float kmag_of(const FCLat& L, const FCharge& c) {
    return (c.type == 1) ? fnorm(e2s(L, c.valley, c.p * (1.0f / kHbarCF))) : fnorm(c.p) * (1.0f / kHbarCF);
}

// ChargePhysics::make_charge (charge_transport.hpp:49-70)
__device__ FCharge make_charge_f(const FCLat& L, int type, F3 pos, F3 dir, float ek, int valley, double t, float w) {
    FCharge c;
    const F3 u = funit(dir);
    c.p = (type == 1) ? ekin_to_p_e(L, valley, u, ek) : u * sqrtf(fmaxf(0.0f, ek * ek + 2.0f * ek * L.m_h));
    c.pos = pos;
    c.ekin = ek;
    c.t = t;
    c.w = w;
    c.valley = valley;
    c.type = type;
    return c;
}

// electrode mask lookup out of line (keeps atan2 out of the step loop)
__device__ __noinline__ int mask_call(const Pad* pads, int n_pads, float x, float y, R128* g) {
    return find_channel(pads, n_pads, static_cast<double>(x), static_cast<double>(y), *g);
}

struct FRates {
    float luke, iv, trap, ion_e, ion_h, tot;
};

// SimulationEngine::charge_rates (engine.hpp:876-886) with luke_emission_rate
// (charge_transport.hpp:82-106) and the Quadratic / Linear intervalley rates
// (charge_kernels.hpp:82-99); `iv` is the field-dependent intervalley rate where the carrier
// has it, `k` its |k|. The velocity is needed by the trapping rates only.
__device__ __forceinline__ FRates rates_at(const FCLat& L, const FCharge& c, float k, float iv) {
    const bool e = (c.type == 1);
    FRates r;
    const float ks = e ? L.ks_e : L.ks_h;
    if (k > ks) {
        const float mach = k / ks;
        const float dm = mach - 1.0f;
        r.luke = (dm * dm * dm) / ((e ? L.tstep_e : L.tstep_h) * mach);
    } else {
        r.luke = 0.0f;
    }
    r.iv = iv;
    if (L.traps) {
        const float v = fnorm(vel_of(L, c.type, c.valley, c.p));
        r.trap = v * (e ? L.inv_trap_e : L.inv_trap_h);
        r.ion_e = v * (e ? L.inv_ion_e_d0 : L.inv_ion_h_d);
        r.ion_h = v * (e ? L.inv_ion_e_a : L.inv_ion_h_a0);
        r.tot = r.luke + r.iv + r.trap + r.ion_e + r.ion_h;
    } else {
        r.trap = r.ion_e = r.ion_h = 0.0f;
        r.tot = r.luke + r.iv;
    }
    return r;
}
// the same for a carrier whose kinetic energy is up to date
__device__ __forceinline__ FRates rates_of(const FCLat& L, const FCharge& c, float iv_field) {
    const float iv = (c.type == 1 && L.n_valleys >= 2 && c.ekin >= L.iv_min) ? iv_field : 0.0f;
    return rates_at(L, c, kmag_of(L, c), iv);
}

__device__ __forceinline__ float iv_rate_of_field(const FCLat& L, F3 E) {
    if (L.iv_model == 0) return L.iv_qrate * __powf(L.iv_qfield * L.iv_qfield + fdot(E, E), L.iv_qpow_half);
    return L.iv_lrate0 + L.iv_lrate1 * __powf(fnorm(E) * 0.01f, L.iv_lpow);
}

// FP32 facet walk (TriLinearMesh3D::find_tetrahedron, mesh_field.hpp:66-100) with a
// tolerance above FP32 rounding; zero field outside the mesh
__device__ __forceinline__ F3 mesh_field_f(const MeshView32& m, F3 p, int32_t& hint) {
    if (hint < 0 || hint >= m.n_tets) hint = m.n_tets / 2;
    for (int step = 0; step < kMeshMaxSteps; ++step) {
        const MeshTet32& t = m.tet[hint];
        const float4 a = __ldg(reinterpret_cast<const float4*>(&t) + 0);  // tinv 0-3
        const float4 b = __ldg(reinterpret_cast<const float4*>(&t) + 1);  // tinv 4-7
        const float4 c = __ldg(reinterpret_cast<const float4*>(&t) + 2);  // tinv 8, x3
        const float dx = p.x - c.y, dy = p.y - c.z, dz = p.z - c.w;
        const float b0 = a.x * dx + a.y * dy + a.z * dz;
        const float b1 = a.w * dx + b.x * dy + b.y * dz;
        const float b2 = b.z * dx + b.w * dy + c.x * dz;
        const float b3 = 1.0f - b0 - b1 - b2;
        float mn = b0;
        int mi = 0;
        if (b1 < mn) { mn = b1; mi = 1; }
        if (b2 < mn) { mn = b2; mi = 2; }
        if (b3 < mn) { mn = b3; mi = 3; }
        if (mn >= kMeshTol) {
            const float4 e = __ldg(reinterpret_cast<const float4*>(&t) + 3);  // e, nb0
            return f3(e.x, e.y, e.z);
        }
        const int32_t next = __ldg(&t.nb[mi]);
        if (next < 0) break;
        hint = next;
    }
    return f3(0.0f, 0.0f, 0.0f);
}

// FP32 edge walk (BiLinearMesh2D::find_triangle / field_at, mesh_field.hpp:376-430) with
// the same FP32 tolerance; the axisymmetric field is rotated back around the z axis
__device__ __forceinline__ F3 mesh2_field_f(const MeshView2_32& m, F3 p, int32_t& hint) {
    float u = p.x, v = p.y;
    if (m.axisym) {
        u = sqrtf(p.x * p.x + p.y * p.y);
        v = p.z;
    }
    if (hint < 0 || hint >= m.n_tris) hint = m.n_tris / 2;
    for (int step = 0; step < kMeshMaxSteps; ++step) {
        const MeshTri32& t = m.tri[hint];
        const float4 a = __ldg(reinterpret_cast<const float4*>(&t) + 0);  // tinv
        const float4 b = __ldg(reinterpret_cast<const float4*>(&t) + 1);  // x2, e
        const float du = u - b.x, dv = v - b.y;
        const float b0 = a.x * du + a.y * dv;
        const float b1 = a.z * du + a.w * dv;
        const float b2 = 1.0f - b0 - b1;
        float mn = b0;
        int mi = 0;
        if (b1 < mn) { mn = b1; mi = 1; }
        if (b2 < mn) { mn = b2; mi = 2; }
        if (mn >= kMeshTol) {
            if (!m.axisym) return f3(b.z, b.w, 0.0f);
            if (u > 1e-15f) return f3(b.z * (p.x / u), b.z * (p.y / u), b.w);
            return f3(0.0f, 0.0f, b.w);
        }
        const int32_t next = __ldg(&t.nb[mi]);
        if (next < 0) break;
        hint = next;
    }
    return f3(0.0f, 0.0f, 0.0f);
}

__device__ __forceinline__ void sink_charge(const RunArgs& a, uint32_t ev, const CStats& st) {
    cmpmc_sim_stats& o = a.ev_stats[ev];
    auto add = [](uint64_t* p, uint32_t v) {
        if (v) atomicAdd(reinterpret_cast<unsigned long long*>(p), static_cast<unsigned long long>(v));
    };
    auto addd = [](double* p, double v) {
        if (v != 0.0) atomicAdd(p, v);
    };
    add(&o.charge_steps, st.steps);
    add(&o.luke_phonons_emitted, st.luke);
    add(&o.intervalley_scatters, st.iv);
    add(&o.charges_trapped, st.trapped);
    add(&o.trap_ionizations, st.ion);
    add(&o.charge_surface_refls, st.crefl);
    add(&o.charges_collected, st.collected);
    addd(&o.total_luke_phonon_eV, st.luke_eV);
    addd(&o.charge_recomb_edep_eV, st.recomb_eV);
    addd(&o.total_deposited_eV, st.dep);
    addd(&o.escaped_or_killed_eV, st.esc);
}

// a carrier and the bookkeeping that travels with it between phases
struct Carrier {
    FCharge c;
    R128 g;
    uint64_t ckey;
    uint32_t ev, luke_idx, n_knock, steps;
    int32_t hint;
};

__device__ __forceinline__ QCharge park(const Carrier& k) {
    QCharge q;
    q.px = k.c.pos.x; q.py = k.c.pos.y; q.pz = k.c.pos.z;
    q.qx = k.c.p.x; q.qy = k.c.p.y; q.qz = k.c.p.z;
    q.ekin = k.c.ekin;
    q.w = k.c.w;
    q.t = k.c.t;
    q.ckey = k.ckey;
    q.rng[0] = k.g.s0; q.rng[1] = k.g.s1; q.rng[2] = k.g.s2; q.rng[3] = k.g.s3;
    q.ev = k.ev;
    q.luke_idx = k.luke_idx;
    q.n_knock = k.n_knock;
    q.hint = k.hint;
    q.valley_type = static_cast<uint32_t>(k.c.valley) | (static_cast<uint32_t>(k.c.type) << 16);
    q.pad[0] = k.steps;
    q.pad[1] = q.pad[2] = 0;
    return q;
}
__device__ __forceinline__ Carrier unpark(const QCharge& q) {
    Carrier k;
    k.c.pos = f3(q.px, q.py, q.pz);
    k.c.p = f3(q.qx, q.qy, q.qz);
    k.c.ekin = q.ekin;
    k.c.w = q.w;
    k.c.t = q.t;
    k.c.valley = static_cast<int>(q.valley_type & 0xffffu);
    k.c.type = static_cast<int>(q.valley_type >> 16);
    k.ckey = q.ckey;
    k.g.s0 = q.rng[0]; k.g.s1 = q.rng[1]; k.g.s2 = q.rng[2]; k.g.s3 = q.rng[3];
    k.ev = q.ev;
    k.luke_idx = q.luke_idx;
    k.n_knock = q.n_knock;
    k.hint = q.hint;
    k.steps = q.pad[0];
    return k;
}

__device__ __forceinline__ uint64_t luke_key(uint64_t ckey, uint32_t idx) {
    return mix64(ckey ^ (0x9e3779b97f4a7c15ULL * (static_cast<uint64_t>(idx) + 1)));
}

// The kernel in its two forms (charge_kernel.inl). An event's code runs for the lanes that have
// one, about three of a full warp in every iteration; waiting fills it with eight, and costs the
// votes and a few idle lanes.
#define CHARGE_KERNEL k_charges_fp32
#define CHARGE_DEFER 0
#define CHARGE_NEXT continue
#define CHARGE_DONE break
#include "charge_kernel.inl"
#undef CHARGE_KERNEL
#undef CHARGE_DEFER
#undef CHARGE_NEXT
#undef CHARGE_DONE
#define CHARGE_KERNEL k_charges_defer_fp32
#define CHARGE_DEFER 1
#define CHARGE_NEXT break
#define CHARGE_DONE done = true
#include "charge_kernel.inl"
#undef CHARGE_KERNEL
#undef CHARGE_DEFER
#undef CHARGE_NEXT
#undef CHARGE_DONE

__global__ void k_carrier_event(const uint64_t* __restrict__ ch_off, uint64_t n_events,
                                uint32_t* __restrict__ carrier_event) {
    for (uint64_t ev = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; ev < n_events;
         ev += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        for (uint64_t j = ch_off[ev]; j < ch_off[ev + 1]; ++j) carrier_event[j] = static_cast<uint32_t>(ev);
}

// ---- the order in which the waiting form starts its carriers ---------------------------------
// Electrons and holes run different branches of every step, and a carrier's steps go with the
// distance it drifts. So the carriers start by type, the longest drift first: a counting sort by
// (type, distance to the exit along the force in a uniform field; type alone in a mesh field).
// Each carrier owns its substream, so the order changes no carrier; it is free within a key.
constexpr int kOrderBins = 64;
constexpr int kOrderKeys = 2 * kOrderBins;
static_assert(kOrderKeys <= 256, "a key is kept in one byte");

__device__ __forceinline__ int order_key(const FCDet& D, const cmpmc_charge_track& c) {
    const bool e = c.type == 1;
    int bin = 0;
    const float e2 = fdot(D.e_field, D.e_field);
    if (!D.mesh.tet && !D.mesh2.tri && e2 > 0.0f) {
        const F3 p = f3(static_cast<float>(c.pos[0]), static_cast<float>(c.pos[1]), static_cast<float>(c.pos[2]));
        const float d = fexit_d(D.R, D.H, p, D.e_field * ((e ? -1.0f : 1.0f) * rsqrtf(e2))).d;
        const float span = 2.0f * fmaxf(D.R, D.H);
        bin = kOrderBins - 1 - min(max(static_cast<int>(d / span * kOrderBins), 0), kOrderBins - 1);
    }
    return (e ? 0 : kOrderBins) + bin;
}

// bins[k]: carriers with key k; k_order_start turns the counts into first places. The key is
// computed once and kept (one byte a carrier): were the second kernel to round a distance on the
// edge of a bin the other way, one place of the order would be written twice and one never.
__global__ void __launch_bounds__(256) k_order_count(const __grid_constant__ FCDet D,
                                                     const cmpmc_charge_track* __restrict__ ch, uint64_t n,
                                                     uint32_t* __restrict__ bins, uint8_t* __restrict__ keys) {
    __shared__ uint32_t cnt[kOrderKeys];
    if (threadIdx.x < kOrderKeys) cnt[threadIdx.x] = 0;
    __syncthreads();
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const int key = order_key(D, ch[i]);
        keys[i] = static_cast<uint8_t>(key);
        atomicAdd(&cnt[key], 1u);
    }
    __syncthreads();
    if (threadIdx.x < kOrderKeys && cnt[threadIdx.x]) atomicAdd(bins + threadIdx.x, cnt[threadIdx.x]);
}
__global__ void __launch_bounds__(kOrderKeys) k_order_start(uint32_t* __restrict__ bins) {
    __shared__ uint32_t part[kOrderKeys];
    const int t = threadIdx.x;
    const uint32_t own = bins[t];
    part[t] = own;
    __syncthreads();
    for (int d = 1; d < kOrderKeys; d <<= 1) {
        const uint32_t v = (t >= d) ? part[t - d] : 0u;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    bins[t] = part[t] - own;
}
__global__ void __launch_bounds__(256) k_order_place(const uint8_t* __restrict__ keys, uint64_t n,
                                                     uint32_t* __restrict__ bins, uint32_t* __restrict__ order) {
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        order[atomicAdd(bins + keys[i], 1u)] = static_cast<uint32_t>(i);
}

// The release phase of the batched charge form (engine.hpp:302-313, 894-925): one collected
// carrier per thread, from its own substream. BulkDebye emits round(E_rel / E_Debye) (at
// least one) Debye phonons; ElectrodeFilm sends the energy into the electrode's film as
// quanta of at most max(4, electrode_seed_max_gap) Delta (photon seeds): the absorbed part
// is the hit, the escaping phonons re-enter the crystal, the rest is lost. The phonons go,
// inward Lambertian with a DOS mode and their own substreams, into the phonon queue of
// the round; the hit and the ledger go to the carrier's event.
template <int kKin>
__global__ void __launch_bounds__(128, 8) k_release_fp32(const __grid_constant__ FLat L,
                                                         const __grid_constant__ Detector D,
                                                         const __grid_constant__ RunArgs a,
                                                         const __grid_constant__ ChargeArgs ca,
                                                         const ReleaseRec* __restrict__ rel, uint64_t n_rel,
                                                         double debye_energy) {
    double refl_buf[kKaplanCap];
    double kwork[4 * kKaplanCap];
    unsigned err = 0;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n_rel;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const ReleaseRec r = rel[i];
        R128 g;
        g.seed(r.key);
        const F3 hp = f3(r.px, r.py, r.pz);
        const F3 n_in = fnormal(r.surf, hp);
        const F3 p0 = hp + n_in * kNudge;
        uint32_t n_ph = 0;  // phonons queued so far (substream index)
        auto emit = [&](double e, unsigned long long slot) {
            const int mode = fdos(L, g.u());
            FKin kin;
            const F3 kd = finward<kKin>(L, mode, n_in, g, kin);
            QPhonon q;
            q.px = p0.x; q.py = p0.y; q.pz = p0.z;
            q.kx = kd.x; q.ky = kd.y; q.kz = kd.z;
            q.w = r.w;
            q.mode = static_cast<uint32_t>(mode);
            q.E = e;
            q.t = r.t;
            q.key = mix64(r.key ^ (0x9e3779b97f4a7c15ULL * (static_cast<uint64_t>(n_ph++) + 1)));
            q.ev = r.ev;
            q.pad = 0;
            ca.queue[slot] = q;
        };
        double hit_eV = 0.0, lost = 0.0;
        if (D.charge_release == 1) {
            const int k = static_cast<int>(round(r.e_rel / debye_energy));
            const int n = (k < 1) ? 1 : k;
            const unsigned long long base = atomicAdd(ca.q_tail, static_cast<unsigned long long>(n));
            if (base + n > ca.q_cap) {
                err |= kErrRelease;
            } else {
                for (int j = 0; j < n; ++j) emit(r.e_rel / n, base + j);
            }
        } else {
            const Film& film = D.surf[r.surf].film;
            const double qmax = dmax(4.0, D.electrode_seed_max_gap) * film.gap_energy;
            const int k = static_cast<int>(ceil(r.e_rel / qmax));
            const int n = (k < 1) ? 1 : k;
            const double q = r.e_rel / n;
            double absorbed = 0.0, emitted = 0.0;
            KBuf refl{refl_buf, 0};
            for (int j = 0; j < n; ++j) {
                absorbed += film_absorb_quantum(film, q, refl, kwork, g, true);
                if (refl.n == 0) continue;
                const unsigned long long base = atomicAdd(ca.q_tail, static_cast<unsigned long long>(refl.n));
                if (base + refl.n > ca.q_cap) {
                    err |= kErrRelease;
                    continue;
                }
                for (int m = 0; m < refl.n; ++m) {
                    emit(refl_buf[m], base + m);
                    emitted += refl_buf[m];
                }
            }
            lost = dmax(0.0, r.e_rel - absorbed - emitted);
            hit_eV = absorbed;
        }
        const double recomb = hit_eV * static_cast<double>(r.w);
        cmpmc_sim_stats& o = a.ev_stats[r.ev];
        if (recomb != 0.0) {
            atomicAdd(&o.charge_recomb_edep_eV, recomb);
            atomicAdd(&o.total_deposited_eV, recomb);
        }
        if (lost != 0.0) atomicAdd(&o.escaped_or_killed_eV, lost * static_cast<double>(r.w));
        if (a.keep_hits) {
            atomicAdd(reinterpret_cast<unsigned long long*>(a.ev_nhits + r.ev), 1ull);
            const unsigned long long idx = atomicAdd(a.hit_count, 1ull);
            if (idx < a.hit_cap) {
                cmpmc_sensor_hit h;
                h.pos[0] = r.px; h.pos[1] = r.py; h.pos[2] = r.pz;
                h.time = r.t;
                h.edep = recomb;
                h.incident_energy = r.e_rel;
                h.surface_id = r.surf;
                h.excitation = r.type;
                h.mode = 0;
                h._pad = 0;
                h.channel_id = r.ch_id;
                a.hit_stage[idx] = h;
                a.hit_key[idx] = r.ev;
            }
        }
    }
    if (err) atomicOr(a.err, err);
}

FCLat make_fclat(const Lattice& L, const float* cdf_f, const Detector& D) {
    FCLat f{};
    for (int v = 0; v < CMPMC_MAX_VALLEYS && v < L.n_valleys; ++v)
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) f.rot[v][3 * i + j] = static_cast<float>(L.valley_rot[v].m[i][j]);
    f.hv_sqrt = F3{static_cast<float>(L.hv_sqrt.x), static_cast<float>(L.hv_sqrt.y), static_cast<float>(L.hv_sqrt.z)};
    f.hv_sqrt_inv = F3{static_cast<float>(L.hv_sqrt_inv.x), static_cast<float>(L.hv_sqrt_inv.y),
                       static_cast<float>(L.hv_sqrt_inv.z)};
    f.inv_mass_ratio = F3{static_cast<float>(1.0 / L.mass_ratio.x), static_cast<float>(1.0 / L.mass_ratio.y),
                          static_cast<float>(1.0 / L.mass_ratio.z)};
    f.m_e = static_cast<float>(L.e_cond_mass);
    f.m_h = static_cast<float>(L.h_mass);
    f.ks_e = static_cast<float>(L.k_sound_e);
    f.ks_h = static_cast<float>(L.k_sound_h);
    f.tstep_e = static_cast<float>((3.0 * L.l0_e) / L.v_sound);
    f.tstep_h = static_cast<float>((3.0 * L.l0_h) / L.v_sound);
    f.vs_hbar = static_cast<float>(L.v_sound * kHbar);
    f.hv_max = static_cast<float>(hv_max_scale(L));
    f.n_valleys = L.n_valleys;
    f.iv_model = L.iv_model;
    f.iv_min = static_cast<float>(L.iv_min_energy);
    const KBand band = k_band(L.iv_min_energy, L.e_cond_mass);
    f.k_iv_lo = band.lo;
    f.k_iv_hi = band.hi;
    f.iv_qrate = static_cast<float>(L.iv_quad_rate);
    f.iv_qfield = static_cast<float>(L.iv_quad_field);
    f.iv_qpow_half = static_cast<float>(0.5 * L.iv_quad_power);
    f.iv_lrate0 = static_cast<float>(L.iv_lin_rate0);
    f.iv_lrate1 = static_cast<float>(L.iv_lin_rate1);
    f.iv_lpow = static_cast<float>(L.iv_lin_power);
    auto inv = [](double mfp) { return (mfp > 0.0 && mfp < 1e20) ? static_cast<float>(1.0 / mfp) : 0.0f; };
    f.inv_trap_e = inv(L.e_trap_mfp);
    f.inv_trap_h = inv(L.h_trap_mfp);
    f.inv_ion_e_d0 = inv(L.e_ion_d0_mfp);
    f.inv_ion_e_a = inv(L.e_ion_a_mfp);
    f.inv_ion_h_d = inv(L.h_ion_d_mfp);
    f.inv_ion_h_a0 = inv(L.h_ion_a0_mfp);
    f.traps = f.inv_trap_e != 0.0f || f.inv_trap_h != 0.0f || f.inv_ion_e_d0 != 0.0f || f.inv_ion_e_a != 0.0f ||
              f.inv_ion_h_d != 0.0f || f.inv_ion_h_a0 != 0.0f;
    f.fL = static_cast<float>(L.fLDOS);
    f.fLST = static_cast<float>(L.fLDOS + L.fSTDOS);
    f.bandgap = static_cast<float>(L.bandgap);
    f.bandgap_d = L.bandgap;
    (void)cdf_f;
    (void)D;
    return f;
}

FCDet make_fcdet(const Detector& D, const MeshView32& mesh, const Lattice& L) {
    FCDet f{};
    f.R = static_cast<float>(D.radius);
    f.H = static_cast<float>(D.half_z);
    f.e_field = F3{static_cast<float>(D.e_field.x), static_cast<float>(D.e_field.y), static_cast<float>(D.e_field.z)};
    for (int i = 0; i < 3; ++i) {
        f.surf[i].prob_abs = static_cast<float>(D.surf[i].prob_charge_abs);
        f.surf[i].prob_spec = static_cast<float>(D.surf[i].prob_charge_spec);
        f.surf[i].min_k_e = static_cast<float>(D.surf[i].min_k_elec);
        f.surf[i].min_k_h = static_cast<float>(D.surf[i].min_k_hole);
        f.surf[i].n_pads = D.surf[i].n_pads;
        f.surf[i].pads = D.surf[i].pads;
        f.surf[i].release = (D.charge_release == 1 || (D.charge_release == 2 && D.surf[i].has_film)) ? 1 : 0;
    }
    f.edge = wall_edge(f.R, f.H);
    f.dt_cap = static_cast<float>(D.charge_dt_cap_s);
    const bool second = (D.charge_stepping == 1);
    f.dk_frac = static_cast<float>(second ? D.charge_sampling_dk_frac : D.charge_max_dk_frac);
    f.second = second ? 1 : 0;
    const double lp = dclamp(D.luke_sample_fraction, 0.0, 1.0);
    f.luke_prob = static_cast<float>(lp);
    f.luke_wt = (lp > 0.0) ? static_cast<float>(1.0 / lp) : 0.0f;
    f.muF = (D.fermi_level_above_Ev_eV >= 0.0) ? D.fermi_level_above_Ev_eV : 0.5 * L.bandgap;
    f.mesh = mesh;
    f.mesh2 = D.mesh2_32;
    return f;
}

}  // namespace

// Waiting pays once a warp holds many carriers. Events of n pairs, ms at once / waiting in order:
// 2,000 (two lanes) 64 / 71, 8,000 (six) 85 / 88, 12,000 (nine) 94 / 92, 20,000 (14) 105 / 95,
// 50,000 (32) 127 / 99 (109 in the caller's order). With open trapping channels the two forms
// round a trapped carrier's energy differently in its last bit, so those crystals keep the first.
bool charges_wait(const Lattice& L, uint32_t lanes) {
    auto open = [](double mfp) { return mfp > 0.0 && mfp < 1e20; };
    const bool traps = open(L.e_trap_mfp) || open(L.h_trap_mfp) || open(L.e_ion_d0_mfp) || open(L.e_ion_a_mfp) ||
                       open(L.h_ion_d_mfp) || open(L.h_ion_a0_mfp);
    return lanes >= kWaitLanes && !traps;
}

// order[n], bins[kOrderKeys], keys[n]
size_t carrier_order_bytes(uint64_t n) { return (n + kOrderKeys) * sizeof(uint32_t) + n; }

cudaError_t launch_carrier_order(const Lattice& L, const Detector& D, const cmpmc_charge_track* ch, uint64_t n,
                                 uint32_t* order, cudaStream_t s, int* launches) {
    const FCDet d = make_fcdet(D, D.mesh32, L);
    uint32_t* bins = order + n;
    uint8_t* keys = reinterpret_cast<uint8_t*>(bins + kOrderKeys);
    const cudaError_t e = cudaMemsetAsync(bins, 0, kOrderKeys * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    const int grid = static_cast<int>(std::min<uint64_t>((n + 255) / 256, 4 * 148));
    k_order_count<<<grid, 256, 0, s>>>(d, ch, n, bins, keys);
    k_order_start<<<1, kOrderKeys, 0, s>>>(bins);
    k_order_place<<<grid, 256, 0, s>>>(keys, n, bins, order);
    *launches += 3;
    return cudaGetLastError();
}

cudaError_t launch_charges_fp32(const Lattice& L, const float* cdf_f, const Detector& D, const RunArgs& a,
                                const ChargeArgs& c, int grid, int block, cudaStream_t s) {
    const FCLat f = make_fclat(L, cdf_f, D);
    const FCDet d = make_fcdet(D, D.mesh32, L);
    if (charges_wait(L, a.lanes)) k_charges_defer_fp32<<<grid, block, 0, s>>>(f, d, a, c);
    else k_charges_fp32<<<grid, block, 0, s>>>(f, d, a, c);
    return cudaGetLastError();
}

cudaError_t charges_fp32_occupancy(int block, int* blocks_per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_charges_fp32, block, 0);
}

cudaError_t launch_release_fp32(const Lattice& L, const float* cdf_f, const Detector& D, const RunArgs& a,
                                const ChargeArgs& c, uint64_t n_rel, int grid, int block, cudaStream_t s) {
    const FLat f = make_flat(L, cdf_f, D);
    if (L.kin_mode != kKinOctahedral)
        k_release_fp32<1><<<grid, block, 0, s>>>(f, D, a, c, c.rel, n_rel, L.debye_energy);
    else
        k_release_fp32<0><<<grid, block, 0, s>>>(f, D, a, c, c.rel, n_rel, L.debye_energy);
    return cudaGetLastError();
}

cudaError_t launch_carrier_event(const uint64_t* ch_off, uint64_t n_events, uint32_t* carrier_event,
                                 cudaStream_t s) {
    k_carrier_event<<<4 * 148, 128, 0, s>>>(ch_off, n_events, carrier_event);
    return cudaGetLastError();
}

}  // namespace cmpmc_gpu
