// Host-side State / fixes: parameter tables, upload/download, run
// preparation (State::prepareForRun, State.cpp:562-647; Integrator::
// basicPrepare / prepareFixes / prepareFinal, Integrator.cu:142-219).
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <limits>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "engine.hpp"

namespace mdx {

uint64_t g_launches = 0;

int high_priority() {
    static int prio = 1;  // not yet read
    if (prio == 1) {
        int least = 0, greatest = 0;
        if (cudaDeviceGetStreamPriorityRange(&least, &greatest) != cudaSuccess) greatest = 0;
        prio = greatest;
    }
    return prio;
}

static thread_local char g_err[1024] = "";
void set_error(int code, const char *fmt, ...) {
    (void)code;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}
const char *last_error() { return g_err; }

// ---------------------------------------------------------------- State
int num_sms() {
    static int cache[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!cache[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
        cache[dev] = n;
    }
    return cache[dev];
}

// Host arrays cross in pieces through pinned and device memory that all states
// of a device share: kStageMost doubles at most, in kSlots slots of which a
// call takes a free one (a state takes one of its own when there is none),
// given back with the process's last state.
// Pinned memory for each state, 72 bytes an atom taken by its first getAtoms,
// made the first pass of 64 new replicas 50 ms; it takes 34 so.
constexpr size_t kStageMost = size_t(1) << 21;
// a call that a program may make but once asks for no more than this, 1.5 MB:
// above 2 MB pinned and device memory take milliseconds to get (first getAtoms
// of a process's only state, 32,000 atoms: 0.9 ms so, 2.5 with 2.3 MB)
constexpr size_t kStageOnce = size_t(3) << 16;
struct StagingSlot {
    std::mutex mu;
    double *h = nullptr, *d = nullptr;
    cudaEvent_t done[3] = {nullptr, nullptr, nullptr};  // of the pieces under way
    size_t size = 0;  // doubles
    int reserve(size_t want) {
        for (cudaEvent_t &e : done)
            if (!e) MDX_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        want = std::min((want + 0x3fff) & ~size_t(0x3fff), kStageMost);
        if (want <= size) return 0;
        drop();
        MDX_CUDA_TRY(cudaMallocHost(&h, want * sizeof(double)));
        MDX_CUDA_TRY(cudaMalloc(&d, want * sizeof(double)));
        size = want;
        return 0;
    }
    void drop() {
        if (h) cudaFreeHost(h);
        if (d) cudaFree(d);
        h = d = nullptr;
        size = 0;
    }
    ~StagingSlot() {
        drop();
        for (cudaEvent_t e : done)
            if (e) cudaEventDestroy(e);
    }
};

namespace {
struct Staging {
    static constexpr int kSlots = 4;
    std::mutex mu;
    int states = 0;
    std::map<int, StagingSlot[kSlots]> devices;  // (entries stay where they are)
    static Staging &all() {
        static Staging *const s = new Staging;  // outlives every state
        return *s;
    }
    void arrive() {
        std::lock_guard<std::mutex> l(mu);
        states++;
    }
    void leave() {
        std::lock_guard<std::mutex> l(mu);
        if (--states == 0) devices.clear();
    }
    StagingSlot *slots(int device) {
        std::lock_guard<std::mutex> l(mu);
        return devices[device];
    }
};
}  // namespace

int StagingUse::take(size_t want) {
    int cur = 0;
    MDX_CUDA_TRY(cudaGetDevice(&cur));
    if (s.device >= 0 && cur != s.device) {
        MDX_CUDA_TRY(cudaSetDevice(s.device));
        back = cur;
    }
    StagingSlot *const all = Staging::all().slots(s.device);
    for (int k = 0; k < Staging::kSlots && !slot; k++)
        if (all[k].mu.try_lock()) slot = all + k;
    if (!slot) {
        if (!s.stage_own) s.stage_own = std::make_shared<StagingSlot>();
        StagingSlot *const own = static_cast<StagingSlot *>(s.stage_own.get());
        own->mu.lock();
        slot = own;
    }
    return slot->reserve(want);
}

StagingUse::~StagingUse() {
    if (busy) cudaStreamSynchronize(s.stream);  // left early
    if (slot) slot->mu.unlock();
    if (back >= 0) cudaSetDevice(back);
}

State::State() {
    units.setLJ();
    Staging::all().arrive();
}

State::~State() {
    Staging::all().leave();
    if (h_status) cudaFreeHost(h_status);
    for (int k = 0; k < 3; k++) {
        if (side[k]) cudaStreamDestroy(side[k]);
        if (ev_join[k]) cudaEventDestroy(ev_join[k]);
    }
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_sorted) cudaEventDestroy(ev_sorted);
    if (stream && own_stream) cudaStreamDestroy(stream);
}

int State::typeFromHandle(const std::string &h) const {
    for (size_t i = 0; i < species.size(); i++)
        if (species[i].handle == h) return (int)i;
    return -1;
}

void State::setBox() {
    box.lod = make_double3(lo[0], lo[1], lo[2]);
    box.Ld = make_double3(hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]);
    box.invLd = make_double3(1.0 / box.Ld.x, 1.0 / box.Ld.y, 1.0 / box.Ld.z);
    box.lo = make_float3((float)lo[0], (float)lo[1], (float)lo[2]);
    box.L = make_float3((float)box.Ld.x, (float)box.Ld.y, (float)box.Ld.z);
    box.invL = make_float3(1.0f / box.L.x, 1.0f / box.L.y, 1.0f / box.L.z);
}

double State::maxRCut() {
    // State::getMaxRCut (State.cpp:502-511), a float max over fixes' cutoffs
    float m = (float)rCut;
    for (Fix *f : fixes)
        for (double x : f->getRCuts()) m = std::fmax(m, (float)x);
    return m;
}

FixPair *State::pairFix() {
    for (Fix *f : fixes)
        if (f->kind == FixKind::Pair) return static_cast<FixPair *>(f);
    return nullptr;
}
FixChargeEwald *State::ewaldFix() {
    for (Fix *f : fixes)
        if (f->kind == FixKind::ChargeEwald) return static_cast<FixChargeEwald *>(f);
    return nullptr;
}
FixChargePairDSF *State::dsfFix() {
    for (Fix *f : fixes)
        if (f->kind == FixKind::ChargeDSF) return static_cast<FixChargePairDSF *>(f);
    return nullptr;
}
FixE3B *State::e3bFix() {
    for (Fix *f : fixes)
        if (f->kind == FixKind::E3B) return static_cast<FixE3B *>(f);
    return nullptr;
}
FixRigid *State::rigidFix() {
    for (Fix *f : fixes)
        if (f->kind == FixKind::Rigid) return static_cast<FixRigid *>(f);
    return nullptr;
}
FixPressureBerendsen *State::barostatFix() {
    for (Fix *f : fixes)
        if (f->kind == FixKind::Barostat) return static_cast<FixPressureBerendsen *>(f);
    return nullptr;
}
FixNoseHoover *State::nhFix() {
    for (Fix *f : fixes)
        if (f->kind == FixKind::NoseHoover) return static_cast<FixNoseHoover *>(f);
    return nullptr;
}

// State::copyAtomDataToGPU (State.cpp:529-610): type bits in xs.w, 1/m in
// vs.w (INVMASSLESS for massless sites), group tag bits in fs.w
int State::upload() {
    const int n = (int)atoms.size();
    if (device < 0) MDX_CUDA_TRY(cudaGetDevice(&device));
    if (!stream) {
        MDX_CUDA_TRY(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        own_stream = true;
    }
    for (int k = 0; k < 3; k++) {
        if (!side[k]) MDX_CUDA_TRY(cudaStreamCreateWithFlags(&side[k], cudaStreamNonBlocking));
        if (!ev_join[k]) MDX_CUDA_TRY(cudaEventCreateWithFlags(&ev_join[k], cudaEventDisableTiming));
    }
    if (!ev_fork) MDX_CUDA_TRY(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
    if (!ev_sorted) MDX_CUDA_TRY(cudaEventCreateWithFlags(&ev_sorted, cudaEventDisableTiming));
    if (!h_status) MDX_CUDA_TRY(cudaMallocHost(&h_status, sizeof(DeviceStatus)));
    if (int e = d_status.alloc(1)) return e;
    MDX_CUDA_TRY(cudaMemset(d_status.p, 0, sizeof(DeviceStatus)));
    DeviceStatus init{};
    init.turn = turn;
    MDX_CUDA_TRY(cudaMemcpy(d_status.p, &init, sizeof(init), cudaMemcpyHostToDevice));
    GPUData &d = gpd;
    d.n = n;
    for (DBuf<float4> *b : {&d.xs, &d.vs, &d.fs, &d.xs_alt, &d.vs_alt, &d.fs_alt, &d.xs_last_build})
        if (int e = b->alloc(n)) return e;
    if (int e = d.qs.alloc(n)) return e;
    if (int e = d.qs_alt.alloc(n)) return e;
    if (int e = d.ids.alloc(n)) return e;
    if (int e = d.ids_alt.alloc(n)) return e;
    if (int e = d.idToIdx.alloc(n)) return e;
    if (int e = d.virials.alloc(6 * (size_t)n)) return e;
    if (int e = red_out.alloc(4)) return e;
    if (int e = e_site.alloc(n)) return e;
    if (int e = sumsAlloc()) return e;
    MDX_CUDA_TRY(cudaMemset(d.virials.p, 0, 6 * (size_t)n * sizeof(float)));
    std::vector<float4> xs(n), vs(n), fs(n);
    std::vector<float> qs(n);
    std::vector<uint32_t> ids(n);
    std::vector<int> idx(n);
    for (int i = 0; i < n; i++) {
        const HostAtom &a = atoms[i];
        float tbits;
        std::memcpy(&tbits, &a.type, sizeof(float));
        xs[i] = make_float4((float)a.pos[0], (float)a.pos[1], (float)a.pos[2], tbits);
        float im = a.mass == 0.0 ? kInvMassless : (float)(1.0 / a.mass);
        vs[i] = make_float4((float)a.vel[0], (float)a.vel[1], (float)a.vel[2], im);
        float gbits;
        std::memcpy(&gbits, &a.groupTag, sizeof(float));
        fs[i] = make_float4((float)a.force[0], (float)a.force[1], (float)a.force[2], gbits);
        qs[i] = (float)a.q;
        ids[i] = (uint32_t)i;
        idx[i] = i;
    }
    MDX_CUDA_TRY(cudaMemcpy(d.xs.p, xs.data(), n * sizeof(float4), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(d.vs.p, vs.data(), n * sizeof(float4), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(d.fs.p, fs.data(), n * sizeof(float4), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(d.xs_last_build.p, xs.data(), n * sizeof(float4), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(d.qs.p, qs.data(), n * sizeof(float), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(d.ids.p, ids.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice));
    MDX_CUDA_TRY(cudaMemcpy(d.idToIdx.p, idx.data(), n * sizeof(int), cudaMemcpyHostToDevice));
    uploaded = true;
    return 0;
}

void host_copy(void *dst, const void *src, size_t bytes) {
    // one core copies about 10 GB/s (less into pages it touches first); a
    // thread costs some 20 us to start: worth it from 2 MB
    const size_t parts = std::min<size_t>(4, bytes >> 20);
    if (parts < 2) {
        std::memcpy(dst, src, bytes);
        return;
    }
    const size_t chunk = (bytes / parts + 4095) / 4096 * 4096;
    std::vector<std::thread> th;
    size_t at = chunk;  // the first chunk is this thread's
    try {
        th.reserve(parts);
        for (; at < bytes; at += chunk)
            th.emplace_back([=] {
                std::memcpy((char *)dst + at, (const char *)src + at, std::min(chunk, bytes - at));
            });
    } catch (...) {
        // no more threads, or no memory for one: the rest here (an exception
        // that left with threads running would end the process)
        std::memcpy((char *)dst + at, (const char *)src + at, bytes - at);
    }
    std::memcpy(dst, src, std::min(chunk, bytes));
    for (std::thread &t : th) t.join();
}

namespace {
// atoms first, first + 1, ... by id (idToIdx from the first on): rounded to
// FP32 here (the host cast's round-to-nearest) into the sorted streams, .w
// kept, and widened back out
__global__ void k_put_by_id(int m, const double *__restrict__ in, const int *__restrict__ idToIdx,
                            float4 *__restrict__ dst) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m) return;
    const int i = idToIdx[j];
    const float w = dst[i].w;
    const double *v = in + 3 * (size_t)j;
    dst[i] = make_float4((float)v[0], (float)v[1], (float)v[2], w);
}
// streams a, b, c after one another (blockIdx.y)
__global__ void k_get_by_id(int m, const int *__restrict__ idToIdx, const float4 *__restrict__ a,
                            const float4 *__restrict__ b, const float4 *__restrict__ c, double *__restrict__ out) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m) return;
    const int i = idToIdx[j];
    const float4 v = blockIdx.y == 0 ? a[i] : (blockIdx.y == 1 ? b[i] : c[i]);
    double *o = out + 3 * ((size_t)blockIdx.y * m + j);
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
}

// runs pieces 0 .. n-1 through a slot, up to `ways` of them under way: send
// queues one, read takes it in once it has arrived
template <class Send, class Read>
int in_pieces(State &s, StagingSlot &g, int n, int ways, Send send, Read read) {
    const size_t part = g.size / ways;
    for (int p = 0; p < n + ways - 1; p++) {
        if (p < n) {
            const size_t at = p % ways * part;
            const size_t doubles = send(p, g.d + at);
            MDX_LAUNCHED();
            MDX_CUDA_TRY(
                cudaMemcpyAsync(g.h + at, g.d + at, doubles * sizeof(double), cudaMemcpyDeviceToHost, s.stream));
            MDX_CUDA_TRY(cudaEventRecord(g.done[p % ways], s.stream));
        }
        const int q = p - (ways - 1);
        if (q < 0 || q >= n) continue;
        MDX_CUDA_TRY(cudaEventSynchronize(g.done[q % ways]));
        read(q, g.h + q % ways * part);
    }
    MDX_CUDA_TRY(cudaGetLastError());
    return 0;
}
}  // namespace

int StagingUse::put(int k, const double *src) {
    StagingSlot &g = *slot;
    const size_t half = g.size / 2;
    const int n = s.gpd.n, most = (int)(half / 3);
    busy = true;
    for (int first = 0; first < n; first += most, pieces++) {
        const int m = std::min(most, n - first);
        const size_t bytes = 3 * (size_t)m * sizeof(double);
        double *const d = g.d + (pieces & 1) * half, *const h = g.h + (pieces & 1) * half;
        if (pieces >= 2) MDX_CUDA_TRY(cudaEventSynchronize(g.done[pieces & 1]));
        host_copy(h, src + 3 * (size_t)first, bytes);
        MDX_CUDA_TRY(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s.stream));
        k_put_by_id<<<(m + 255) / 256, 256, 0, s.stream>>>(m, d, s.gpd.idToIdx.p + first,
                                                           k == 0 ? s.gpd.xs.p : s.gpd.vs.p);
        MDX_LAUNCHED();
        MDX_CUDA_TRY(cudaEventRecord(g.done[pieces & 1], s.stream));
    }
    return 0;
}

int StagingUse::get(double *const out[3]) {
    StagingSlot &g = *slot;
    const GPUData &d = s.gpd;
    // all three arrays on their way at once, or pieces two at a time
    const int n = d.n, ways = 9 * (size_t)n <= g.size ? 3 : 2;
    const int most = (int)(g.size / ways / 3), per = (n + most - 1) / most;
    const float4 *src[3];
    double *dst[3];
    int na = 0;
    for (int k = 0; k < 3; k++) {
        if (!out[k]) continue;
        src[na] = k == 0 ? d.xs.p : (k == 1 ? d.vs.p : d.fs.p);
        dst[na++] = out[k];
    }
    busy = true;
    // array by array, so that each is copied out in long stretches
    const int e = in_pieces(
        s, g, na * per, ways,
        [&](int p, double *buf) {
            const int first = p % per * most, m = std::min(most, n - first);
            const float4 *const a = src[p / per];
            k_get_by_id<<<(m + 255) / 256, 256, 0, s.stream>>>(m, d.idToIdx.p + first, a, a, a, buf);
            return 3 * (size_t)m;
        },
        [&](int p, const double *buf) {
            const int first = p % per * most, m = std::min(most, n - first);
            host_copy(dst[p / per] + 3 * (size_t)first, buf, 3 * (size_t)m * sizeof(double));
        });
    if (e) return e;
    if (na) busy = false;  // all that was queued before has completed too
    return 0;
}

int State::download(double *const *out) {
    if (!uploaded) return 0;
    const int n = gpd.n;
    StagingUse use(*this);
    if (int e = use.take(std::min(9 * (size_t)n, kStageOnce))) return e;
    use.busy = true;
    MDX_CUDA_TRY(cudaMemcpyAsync(h_status, d_status.p, sizeof(DeviceStatus), cudaMemcpyDeviceToHost, stream));
    // all three arrays of some atoms to a piece: a host atom is touched once
    const size_t size = use.slot->size;
    const int ways = 9 * (size_t)n <= size ? 1 : 2, most = (int)(size / ways / 9);
    const int e = in_pieces(
        *this, *use.slot, (n + most - 1) / most, ways,
        [&](int p, double *buf) {
            const int first = p * most, m = std::min(most, n - first);
            k_get_by_id<<<dim3((m + 255) / 256, 3), 256, 0, stream>>>(m, gpd.idToIdx.p + first, gpd.xs.p, gpd.vs.p,
                                                                      gpd.fs.p, buf);
            return 9 * (size_t)m;
        },
        [&](int p, const double *x) {
            const int first = p * most, m = std::min(most, n - first);
            const double *v = x + 3 * (size_t)m, *f = v + 3 * (size_t)m;
            for (int k = 0; k < 3; k++)
                if (out && out[k])
                    host_copy(out[k] + 3 * (size_t)first, x + 3 * (size_t)k * m, 3 * (size_t)m * sizeof(double));
            for (int i = first; i < first + m; i++, x += 3, v += 3, f += 3) {
                HostAtom &a = atoms[i];
                for (int c = 0; c < 3; c++) {
                    a.pos[c] = x[c];
                    a.vel[c] = v[c];
                    a.force[c] = f[c];
                }
            }
        });
    if (e) return e;
    use.busy = false;
    turn = h_status->turn;
    return 0;
}

int State::put(const double *pos, const double *vel) {
    const int n = gpd.n;
    StagingUse use(*this);
    if (int e = use.take(std::min(6 * (size_t)n, kStageOnce))) return e;
    if (pos)
        if (int e = use.put(0, pos)) return e;
    if (vel)
        if (int e = use.put(1, vel)) return e;
    for (int i = 0; i < n; i++)
        for (int d = 0; d < 3; d++) {
            if (pos) atoms[i].pos[d] = pos[3 * (size_t)i + d];
            if (vel) atoms[i].vel[d] = vel[3 * (size_t)i + d];
        }
    MDX_CUDA_TRY(cudaStreamSynchronize(stream));
    use.busy = false;
    return 0;
}

int State::checkStatus() {
    MDX_CUDA_TRY(cudaMemcpyAsync(h_status, d_status.p, sizeof(DeviceStatus), cudaMemcpyDeviceToHost, stream));
    MDX_CUDA_TRY(cudaStreamSynchronize(stream));
    const uint32_t b = h_status->bits;
    if (b & kStatusNlistOverflow) {
        if (mf.on)
            set_error(MDX_ERR_OVERFLOW, "molecule-pair list capacity %d exceeded (max count %u)", mf.cap,
                      h_status->max_mol_neighbors);
        else
            set_error(MDX_ERR_OVERFLOW, "neighbour list capacity %d exceeded (max count %u)", grid.cap,
                      h_status->max_neighbors);
        return MDX_ERR_OVERFLOW;
    }
    if (b & kStatusMolOverflow) {
        set_error(MDX_ERR_OVERFLOW, "E3B molecule list capacity exceeded (max count %u)", h_status->max_mol_neighbors);
        return MDX_ERR_OVERFLOW;
    }
    if (b & kStatusSettleFail) {
        set_error(MDX_ERR_NUMERIC, "SETTLE failed: cos^2 <= 0 (degenerate water triangle)");
        return MDX_ERR_NUMERIC;
    }
    if (b & kStatusConstraint) {
        set_error(MDX_ERR_NUMERIC, "rigid-water bond length drifted beyond 1e-3 A (validateConstraints)");
        return MDX_ERR_NUMERIC;
    }
    return 0;
}

int State::buildNeighborList(bool force) { return nlist_rebuild(*this, force, false); }

// IntegratorUtil::force (IntegratorUtil.cpp:15-30): zero forces, then every
// fix's compute in fix order (pair fixes first, orderPreference -1)
int State::computeForces(int virialMode) {
    if (int e = zero_forces(*this)) return e;
    std::vector<Fix *> order(fixes.begin(), fixes.end());
    std::stable_sort(order.begin(), order.end(),
                     [](Fix *a, Fix *b) { return a->orderPreference < b->orderPreference; });
    for (Fix *f : order)
        if (int e = f->compute(virialMode)) return e;
    MDX_CUDA_TRY(cudaGetLastError());
    return 0;
}

// run preparation in the reference order (IntegratorVerlet::run, :649-684)
int State::prepare() {
    if (!bounds_set) {
        set_error(MDX_ERR_STATE, "state.bounds not set");
        return MDX_ERR_STATE;
    }
    if (atoms.empty()) {
        set_error(MDX_ERR_STATE, "no atoms");
        return MDX_ERR_STATE;
    }
    if (dt <= 0) {
        set_error(MDX_ERR_STATE, "dt must be positive");
        return MDX_ERR_STATE;
    }
    setBox();
    // charge offload (State::handleChargeOffloading, State.cpp:648-660)
    requiresCharges = false;
    FixPair *pf = pairFix();
    FixChargeEwald *ew = ewaldFix();
    FixChargePairDSF *dsf = dsfFix();
    if (ew && dsf) {
        set_error(MDX_ERR_UNSUPPORTED, "one charge fix per state: FixChargeEwald or FixChargePairDSF");
        return MDX_ERR_UNSUPPORTED;
    }
    if (ew) {
        requiresCharges = true;
        if (ew->r_cut < 0) ew->r_cut = rCut;
    }
    if (dsf) requiresCharges = true;
    if (pf) {
        pf->chargeFix = ew;
        pf->dsfFix = dsf;
        pf->chargeRCut = ew ? ew->r_cut : (dsf ? dsf->r_cut : 0.0);
        if (ew) ew->offloaded = true;
    }
    // reset NDF (Atom ndf 3, FixRigid::assignNDF sets 2 / 0)
    for (auto &a : atoms) a.ndf = 3;
    if (FixRigid *r = rigidFix()) {
        if (int e = r->setConsts()) return e;
        for (auto &m : r->mol_ids) {
            atoms[m.x].ndf = atoms[m.y].ndf = atoms[m.z].ndf = 2;
            if (m.w >= 0) atoms[m.w].ndf = 0;
        }
    }
    if (int e = upload()) return e;
    if (int e = nlist_init(*this)) return e;
    {
        // reduction partials for the per-step kinetic sums (allocated here, never
        // while a graph is being captured)
        const int ab = (gpd.n + 255) / 256;
        const int mb = rigidFix() ? ((int)rigidFix()->mol_ids.size() + kMolBlock - 1) / kMolBlock : 0;
        if (int e = red_partials.alloc(ab + mb + 8)) return e;
        if (int e = rigid_flags_prepare(*this)) return e;
    }
    // prepareFixes(false): pair, charge, E3B
    for (Fix *f : fixes) {
        if (f->kind == FixKind::Rigid || f->kind == FixKind::NoseHoover) continue;
        if (int e = f->prepareForRun()) return e;
    }
    if (FixRigid *r = rigidFix()) {
        if (int e = r->prepareForRun()) return e;  // device molecule arrays
    }
    if (int e = nlist_set_interactions(*this)) return e;
    if (int e = molform_init(*this)) return e;
    // first build (GridGPU::periodicBoundaryConditions(-1, true), Integrator.cu:216)
    if (int e = nlist_rebuild(*this, true, false)) return e;
    if (int e = computeForces(0)) return e;  // forceInitial
    if (FixRigid *r = rigidFix()) {
        // prepareFixes(true): SETTLE the initial configuration, M sites,
        // velocity constraints, COM velocity removal.  As in the reference
        // (FixRigid.cu:1825-1834 distributes M-site virials only), the initial
        // M-site force is not moved onto O/H before the first half kick.
        if (int e = rigid_prepare(*this, *r)) return e;
    }
    if (FixNoseHoover *nh = nhFix()) {
        if (int e = nh_prepare(*this, *nh)) return e;
    }
    if (int e = step_turn_prepare(*this)) return e;
    MDX_CUDA_TRY(cudaStreamSynchronize(stream));
    MDX_CUDA_TRY(cudaGetLastError());
    if (int e = checkStatus()) return e;
    prepared = true;
    return 0;
}

// ---------------------------------------------------------------- FixPair
static const char *pair_type_name(int kind) {
    switch (kind) {
        case 1: return "LJCut";
        case 2: return "LJCutWCA";
        case 3: return "LJCutFS";
        case 4: return "LJCHARMM";
        default: return "TICG";
    }
}

FixPair::FixPair(State *s, std::string h, int kind, std::string mix)
    : Fix(s, h, "all", pair_type_name(kind), FixKind::Pair), lj_kind(kind), mixing(mix) {
    orderPreference = -1;  // FixPair.h:34
    // the parameter handles each style's constructor initializes
    if (kind == 5) {
        params["C"] = {};
    } else {
        params["eps"] = {};
        params["sig"] = {};
    }
    if (kind == 4) {
        params["eps14"] = {};
        params["sig14"] = {};
    }
    params["rCut"] = {};
}

bool FixPair::pairActive(int a, int b) const {
    const int nt = (int)state->species.size();
    const size_t nt2 = (size_t)nt * nt, k = (size_t)a * nt + b;
    if (h_params.size() != (size_t)nparam() * nt2) return true;
    if (h_params[nt2 + k] != 0.f) return true;  // 24 eps, or C (TICG)
    return lj_kind == 4 && h_params[3 * nt2 + k] != 0.f;  // 24 eps14
}

// ---------------------------------------------------------------- FixChargePairDSF
FixChargePairDSF::FixChargePairDSF(State *s, std::string h, std::string g)
    : Fix(s, h, g, "ChargePairDSF", FixKind::ChargeDSF) {
    requiresCharges = true;
    setParameters(0.25, 9.0);  // the constructor's defaults (FixChargePairDSF.cu)
}

// FixChargePairDSF::setParameters: A = 2 alpha / sqrt(pi),
// shift = erfc(alpha rc) / rc^2 + A exp(-alpha^2 rc^2) / rc
void FixChargePairDSF::setParameters(double alpha_, double r_cut_) {
    alpha = alpha_;
    r_cut = r_cut_;
    A = 2.0 / std::sqrt(M_PI) * alpha;
    shift = std::erfc(alpha * r_cut) / (r_cut * r_cut) + A * std::exp(-alpha * alpha * r_cut * r_cut) / r_cut;
}

int FixChargePairDSF::prepareForRun() {
    if (!state->pairFix()) {
        set_error(MDX_ERR_UNSUPPORTED, "FixChargePairDSF is evaluated inside a pair fix's kernel: add a pair fix");
        return MDX_ERR_UNSUPPORTED;
    }
    prepared = true;
    return 0;
}

void FixPair::ensureSize() {
    const size_t nt = state->species.size();
    for (auto &kv : params) {
        std::vector<double> &v = kv.second;
        const size_t old = (size_t)std::llround(std::sqrt((double)v.size()));
        if (old == nt && v.size() == nt * nt) continue;
        std::vector<double> nv(nt * nt, std::numeric_limits<double>::quiet_NaN());
        for (size_t i = 0; i < old && i < nt; i++)
            for (size_t j = 0; j < old && j < nt; j++) nv[i * nt + j] = v[i * old + j];
        v.swap(nv);
    }
}

int FixPair::setParameter(const std::string &param, int a, int b, double v) {
    if (params.find(param) == params.end()) {
        set_error(MDX_ERR_ARG, "unknown pair parameter '%s'", param.c_str());
        return MDX_ERR_ARG;
    }
    const int nt = (int)state->species.size();
    if (a < 0 || b < 0 || a >= nt || b >= nt) {
        set_error(MDX_ERR_ARG, "invalid atom types for setParameter");
        return MDX_ERR_ARG;
    }
    ensureSize();
    params[param][a * nt + b] = v;
    params[param][b * nt + a] = v;
    return 0;
}

// prepareParameters (FixPair.cpp:13-63) with each style's lambdas: FixLJCut
// (FixLJCut.cu:83-122), FixWCA (FixWCA.cu:60-106), FixLJCutFS
// (FixLJCutFS.cu:84-130), FixLJCHARMM (FixLJCHARMM.cu:113-180), FixTICG
// (FixTICG.cu:68-83).  Off-diagonal entries left unset are mixed from the
// diagonal ones (eps geometric, sig geometric or arithmetic, rCut the larger
// one, the diagonal rCut defaulting to state.rCut); TICG mixes nothing
// (check_populate: every entry must be set).
int FixPair::prepareForRun() {
    State &s = *state;
    ensureSize();
    const int nt = (int)s.species.size();
    const size_t nt2 = (size_t)nt * nt;
    auto fill = [&](std::vector<double> v, bool geo, bool fillDiag, double diag) {
        if (fillDiag)
            for (int i = 0; i < nt; i++)
                if (std::isnan(v[i * nt + i])) v[i * nt + i] = diag;
        for (int i = 0; i < nt; i++)
            for (int j = 0; j < nt; j++)
                if (std::isnan(v[i * nt + j])) {
                    double a = v[i * nt + i], b = v[j * nt + j];
                    v[i * nt + j] = geo ? std::sqrt((float)a * (float)b) : ((float)a + (float)b) / 2.0;
                }
        return v;
    };
    auto fill_rcut = [&]() {
        // fillRCut = fmax(a, b), diagonal default state->rCut
        std::vector<double> rc = params["rCut"];
        for (int i = 0; i < nt; i++)
            if (std::isnan(rc[i * nt + i])) rc[i * nt + i] = (float)s.rCut;
        for (int i = 0; i < nt; i++)
            for (int j = 0; j < nt; j++)
                if (std::isnan(rc[i * nt + j])) rc[i * nt + j] = std::fmax((float)rc[i * nt + i], (float)rc[j * nt + j]);
        return rc;
    };
    auto all_set = [&](const std::vector<double> &v, const char *what) {
        for (size_t k = 0; k < nt2; k++)
            if (std::isnan(v[k])) {
                set_error(MDX_ERR_STATE, "pair parameter %s not set for every pair of species", what);
                return false;
            }
        return true;
    };
    h_params.assign((size_t)nparam() * nt2, 0.f);
    if (lj_kind == 5) {
        // TICG: {rCut^2, C}, no mixing
        const std::vector<double> &C = params["C"], &rc = params["rCut"];
        if (!all_set(C, "C") || !all_set(rc, "rCut")) return MDX_ERR_STATE;
        for (size_t k = 0; k < nt2; k++) {
            const float r = (float)rc[k];
            h_params[k] = r * r;
            h_params[nt2 + k] = (float)C[k];
        }
    } else {
        const double c14 = s.specialNeighborCoefs[2];
        if (lj_kind == 4) {
            // an unset 1-4 diagonal entry is the ordinary one times the 1-4
            // coefficient, for eps14 and for sig14 (FixLJCHARMM.cu:147-155)
            for (const char *h : {"eps14", "sig14"}) {
                std::vector<double> &v14 = params[h];
                const std::vector<double> &v = params[h[0] == 'e' ? "eps" : "sig"];
                for (int i = 0; i < nt; i++)
                    if (std::isnan(v14[i * nt + i])) v14[i * nt + i] = (float)v[i * nt + i] * (float)c14;
            }
        }
        std::vector<double> eps = fill(params["eps"], true, false, 0);
        std::vector<double> sig = fill(params["sig"], mixing != "arithmetic", false, 0);
        if (!all_set(eps, "eps") || !all_set(sig, "sig")) return MDX_ERR_STATE;
        std::vector<double> rc;
        if (lj_kind == 2) {
            rc.resize(nt2);
            for (size_t k = 0; k < nt2; k++) rc[k] = (float)sig[k] * (float)std::pow(2.0, 1.0 / 6.0);
        } else {
            rc = fill_rcut();
        }
        for (size_t k = 0; k < nt2; k++) {
            const float r = (float)rc[k];
            h_params[k] = r * r;                                    // processRCut
            h_params[nt2 + k] = 24.0f * (float)eps[k];              // processEps
            h_params[2 * nt2 + k] = (float)std::pow((float)sig[k], 6);  // processSig
        }
        if (lj_kind == 3) {
            // F(rCut): the unshifted LJ force magnitude at the pair's cutoff,
            // from its processed parameters (the table EvaluatorLJFS::force
            // reads as params[3]; see EvaluatorLJFS::forcePy, PairEvaluatorLJFS.cu)
            for (size_t k = 0; k < nt2; k++) {
                const float rc2 = h_params[k], eps24 = h_params[nt2 + k], sig6 = h_params[2 * nt2 + k];
                const float p1 = eps24 * 2.0f * sig6 * sig6, p2 = eps24 * sig6;
                const float r2inv = 1.0f / rc2, rinv = std::sqrt(r2inv);
                const float r6inv = r2inv * r2inv * r2inv;
                h_params[3 * nt2 + k] = r6inv * rinv * (p1 * r6inv - p2);
            }
        }
        if (lj_kind == 4) {
            std::vector<double> eps14 = fill(params["eps14"], true, false, 0);
            std::vector<double> sig14 = fill(params["sig14"], mixing != "arithmetic", false, 0);
            if (!all_set(eps14, "eps14") || !all_set(sig14, "sig14")) return MDX_ERR_STATE;
            for (size_t k = 0; k < nt2; k++) {
                h_params[3 * nt2 + k] = 24.0f * (float)eps14[k];
                h_params[4 * nt2 + k] = (float)std::pow((float)sig14[k], 6);
            }
        }
    }
    if (int e = d_params.alloc(h_params.size())) return e;
    MDX_CUDA_TRY(cudaMemcpy(d_params.p, h_params.data(), h_params.size() * sizeof(float), cudaMemcpyHostToDevice));
    prepared = true;
    return 0;
}

std::vector<double> FixPair::getRCuts() {
    // FixPair::getRCuts: the largest pair cutoff
    State &s = *state;
    const int nt = (int)s.species.size();
    double m = s.rCut;
    if (lj_kind == 2) {
        ensureSize();
        for (int k = 0; k < nt * nt; k++) {
            double sg = params["sig"][k];
            if (!std::isnan(sg)) m = std::max(m, sg * std::pow(2.0, 1.0 / 6.0));
        }
        return {m};
    }
    (void)nt;
    ensureSize();
    for (double v : params["rCut"])
        if (!std::isnan(v)) m = std::max(m, v);
    return {m};
}

int FixPair::compute(int virialMode) { return pair_launch(*state, *this, virialMode, true); }

// ---------------------------------------------------------------- FixRigid
FixRigid::FixRigid(State *s, std::string h, std::string st) : Fix(s, h, "all", "Rigid", FixKind::Rigid), style(st) {}

int FixRigid::createRigid(int o, int h1, int h2, int m) {
    State &s = *state;
    const int n = (int)s.atoms.size();
    if (o < 0 || h1 < 0 || h2 < 0 || o >= n || h1 >= n || h2 >= n || m >= n) {
        set_error(MDX_ERR_ARG, "createRigid: atom id out of range");
        return MDX_ERR_ARG;
    }
    // mass ordering check (FixRigid.cu:1580-1594)
    const double mo = s.atoms[o].mass, mh1 = s.atoms[h1].mass, mh2 = s.atoms[h2].mass;
    bool ordered = mo > mh1 && mo > mh2 && mh1 == mh2;
    if (m >= 0) ordered = ordered && mh1 > s.atoms[m].mass;
    if (!ordered) {
        set_error(MDX_ERR_ARG, "Ids in FixRigid::createRigid must be as O, H1, H2, M");
        return MDX_ERR_ARG;
    }
    if (m >= 0) foursite = true;
    else threesite = true;
    mol_ids.push_back(make_int4(o, h1, h2, m));
    return 0;
}

void FixRigid::getBonds(std::vector<std::pair<int, int>> &out) {
    for (auto &m : mol_ids) {
        out.push_back({m.x, m.y});
        out.push_back({m.x, m.z});
        out.push_back({m.y, m.z});
        if (m.w >= 0) out.push_back({m.x, m.w});
    }
}

// setStyleBondLengths, set_fixed_sides, populateRigidData (FixRigid.cu:1137-1436)
int FixRigid::setConsts() {
    State &s = *state;
    if (mol_ids.empty()) {
        set_error(MDX_ERR_STATE, "There needs to be at least one water in FixRigid");
        return MDX_ERR_STATE;
    }
    if (foursite && threesite) {
        set_error(MDX_ERR_UNSUPPORTED, "both 3-site and 4-site models in one FixRigid");
        return MDX_ERR_UNSUPPORTED;
    }
    if (s.units.type != MDX_UNITS_REAL) {
        set_error(MDX_ERR_UNSUPPORTED, "real units must be used for rigid water (FixRigid.cu:1425)");
        return MDX_ERR_UNSUPPORTED;
    }
    double r_OH, r_HH, r_OM = 0, gamma = 0;
    if (style == "TIP4P/2005") { r_OH = 0.9572; r_HH = 1.5139; r_OM = 0.1546; gamma = 0.73612446364836; }
    else if (style == "TIP4P") { r_OH = 0.9572; r_HH = 1.5139; r_OM = 0.15; gamma = 0.74397533; }
    else if (style == "TIP3P") { r_OH = 0.9572; r_HH = 1.5139; }
    else if (style == "SPC" || style == "SPC/E") { r_OH = 1.0; r_HH = 1.633; }
    else {
        set_error(MDX_ERR_ARG, "unsupported FixRigid style '%s'", style.c_str());
        return MDX_ERR_ARG;
    }
    if (foursite && r_OM == 0) {
        set_error(MDX_ERR_ARG, "style '%s' is a 3-site model but M sites were given", style.c_str());
        return MDX_ERR_ARG;
    }
    const double mO = s.atoms[mol_ids[0].x].mass, mH = s.atoms[mol_ids[0].y].mass;
    const double mW = mO + 2.0 * mH;
    rc.wO = mO / mW;
    rc.wH = mH / mW;
    rc.mO = mO;
    rc.mH = mH;
    rc.invmO = 1.0 / mO;
    rc.invmH = 1.0 / mH;
    rc.r_OH = r_OH;
    rc.r_HH = r_HH;
    rc.r_OM = r_OM;
    rc.gamma = gamma;
    rc.invOH = 1.0 / r_OH;
    rc.invHH = 1.0 / r_HH;
    rc.foursite = foursite ? 1 : 0;
    const double half_hh = 0.5 * r_HH;
    const double rab = std::sqrt(r_OH * r_OH - half_hh * half_hh);
    const double ht = std::atan(half_hh / rab);
    const double h1 = 1.5 * M_PI + ht, h2 = 1.5 * M_PI - ht;
    const double comy = (std::sin(h1) + std::sin(h2)) * r_OH * rc.wH;
    rc.ra = -comy;
    rc.rb = rab - rc.ra;
    rc.rc = half_hh;
    rc.inv2Rc = 1.0 / r_HH;
    // constraint matrix (populateRigidData) and its inverse times mO
    const double inv = mO / mH;
    double M[9];
    M[0] = 1.0 + inv;
    M[1] = 1.0 - 0.5 * r_HH * r_HH / (r_OH * r_OH);
    M[2] = inv * 0.5 * r_HH / r_OH;
    M[3] = M[1];
    M[4] = M[0];
    M[5] = M[2];
    M[6] = M[2];
    M[7] = M[5];
    M[8] = 2.0 * inv;
    const double det = M[0] * (M[4] * M[8] - M[5] * M[7]) - M[1] * (M[3] * M[8] - M[5] * M[6]) +
                       M[2] * (M[3] * M[7] - M[4] * M[6]);
    double I[9];
    I[0] = (M[4] * M[8] - M[5] * M[7]) / det;
    I[1] = (M[2] * M[7] - M[1] * M[8]) / det;
    I[2] = (M[1] * M[5] - M[2] * M[4]) / det;
    I[3] = (M[5] * M[6] - M[3] * M[8]) / det;
    I[4] = (M[0] * M[8] - M[2] * M[6]) / det;
    I[5] = (M[2] * M[3] - M[0] * M[5]) / det;
    I[6] = (M[3] * M[7] - M[4] * M[6]) / det;
    I[7] = (M[1] * M[6] - M[0] * M[7]) / det;
    I[8] = (M[0] * M[4] - M[1] * M[3]) / det;
    for (int k = 0; k < 9; k++) rc.Minv[k] = I[k] * mO;
    return 0;
}

int FixRigid::prepareForRun() {
    const int nmol = (int)mol_ids.size();
    if (int e = d_mol_ids.alloc(nmol)) return e;
    if (int e = d_mol_idx.alloc(nmol)) return e;
    MDX_CUDA_TRY(cudaMemcpy(d_mol_ids.p, mol_ids.data(), nmol * sizeof(int4), cudaMemcpyHostToDevice));
    prepared = true;
    return 0;
}

// ---------------------------------------------------------------- FixNoseHoover
FixNoseHoover::FixNoseHoover(State *s, std::string h, std::string g)
    : Fix(s, h, g, "NoseHoover", FixKind::NoseHoover) {
    orderPreference = 50;
}

int FixNoseHoover::setTemperature(double T_, double tau_) {
    if (T_ <= 0 || tau_ <= 0) {
        set_error(MDX_ERR_ARG, "temperature and time constant must be positive");
        return MDX_ERR_ARG;
    }
    T = T_;
    tau = tau_;
    return 0;
}

int FixNoseHoover::setPressure(const std::string &mode, double P, double tau_) {
    if (mode != "ISO") {
        set_error(MDX_ERR_UNSUPPORTED, "FixNoseHoover::setPressure: mode '%s' (this library implements ISO)",
                  mode.c_str());
        return MDX_ERR_UNSUPPORTED;
    }
    if (tau_ <= 0) {
        set_error(MDX_ERR_ARG, "pressure time constant must be positive");
        return MDX_ERR_ARG;
    }
    barostatting = true;
    pressure = P;
    ptau = tau_;
    return 0;
}

int FixNoseHoover::prepareFinal() { return nh_prepare(*state, *this); }

}  // namespace mdx
