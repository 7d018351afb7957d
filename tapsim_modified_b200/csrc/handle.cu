// tg_handle: device state of one mesh and the C-ABI entry points that drive
// the kernels (include/tapsim_gpu.h).  Host code only; kernels live in
// relax.cu, surface.cu and flight.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <deque>
#include <limits>
#include <mutex>
#include <thread>

#include <stdlib.h>
#include <exception>
#include <string>
#include <vector>

#include "../../include/tapsim_gpu.h"
#include "host/amg.h"
#include "kernels.cuh"
#include "learn.h"

using namespace tgd;

static_assert(sizeof(ImpactOut) == sizeof(tg_impact), "impact layout");
static_assert(sizeof(tg_path_point) == 8 * sizeof(float), "path point layout");

namespace {

thread_local std::string g_error;

template <typename T>
struct DBuf {
    T* p = nullptr;
    size_t n = 0;
    cudaError_t alloc(size_t count) {
        release();
        n = count;
        if (count == 0) return cudaSuccess;
        return cudaMalloc(&p, count * sizeof(T));
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
};

}  // namespace

namespace tgapi {
void set_process_error(const std::string& msg) { g_error = msg; }
}  // namespace tgapi

namespace tgd {
static std::atomic<long long> g_launches(0);
// while a thread captures a CUDA graph, its launches are counted here (they
// run when the graph is replayed, which counts them then)
static thread_local long long* t_captured = nullptr;
void count_launch() {
    if (t_captured) ++*t_captured;
    else g_launches.fetch_add(1, std::memory_order_relaxed);
}
long long launches_so_far() { return g_launches.load(std::memory_order_relaxed); }
}  // namespace tgd

struct tg_handle {
    int n = 0, nnz = 0, ntets = 0, ncol = 0;
    // the device that was current at tg_create: the handle's buffers,
    // streams and events live there, and every entry point makes it current
    int device = -1;
    cudaStream_t stream = nullptr;
    std::string err;
    float top_z = 0.0f;
    double snap = 1.0;
    std::vector<tg_type> types;          // by id, id < 0 means absent
    // update_coordination only changes cells whose id is >= 10; without such
    // a type in the table no cell ever has one
    bool coordinationActive = false;
    std::vector<int32_t> segStart;       // host mirror
    std::vector<int32_t> countV, countN;  // host mirrors
    int32_t countAllV = 0, countAllN = 0;
    int32_t surfSlots = 0;
    int32_t surfMinNode = 0, surfMaxNode = -1;  // surface node range of the last selection
    std::vector<int32_t> h_node_tet;
    std::vector<float> h_xyz;
    std::vector<int8_t> h_type;           // host mirror of the type ids

    // device arrays
    DBuf<float> xyz;
    DBuf<int8_t> type, typeScratch;
    DBuf<uint8_t> flags, area_pos;
    DBuf<int32_t> row_ptr, col, rev, colour, tet_v, tet_n, node_tet;
    DBuf<double> geom, volume, c64, ceff64, diag64, q64, phi64;
    DBuf<float> ceff32, diag32;
    DBuf<DType> dtypes;
    DBuf<int> status;
    DBuf<int32_t> rowsV, rowsN, allV, allN, segStartD, countVD, countND, countAllD;
    DBuf<int32_t> surfList, surfSlot, surfCount;
    DBuf<float> surfRatio, surfScore;
    DBuf<float> cgbuf;  // 5 vectors of n floats
    DBuf<double> scalN;
    int maxInnerAlloc = 0;
    DBuf<double> acc;
    DBuf<unsigned long long> keys;
    DBuf<int32_t> result;
    DBuf<int32_t> local, localCount, localScratch;
    // staging for per-call inputs/outputs
    DBuf<int32_t> stageI;
    DBuf<double> stageD;
    DBuf<float> stageF;
    DBuf<ImpactOut> stageImpact;
    // flight paths (tg_trace_path, tg_event_opts.path_cap): 8 words a point
    DBuf<float> pathBuf, pathErr;

    cudaEvent_t evStart = nullptr, evStop = nullptr;
    // error flags of the flights of tg_run_events; potentials of the
    // flights of tg_trace
    DBuf<int> statusTrace;
    DBuf<double> phiTrace;
    // tg_run_events: a ring of flight slots, each with its own stream and
    // snapshots (potentials, vertex fields), so that the flights of
    // successive events run side by side and overlap the relaxations; the
    // main stream only copies the potentials into the next free slot.  A
    // flight takes 9-13 ms beside the relaxations on the 7.3M-cell tip
    // (vertex fields at low priority, then the walk), so eight slots keep
    // the event's stream from waiting for a slot at 4-5 ms per event
    static constexpr int kRing = 8;
    cudaStream_t ringStream[kRing] = {};
    cudaEvent_t ringPhi[kRing] = {}, ringDone[kRing] = {};
    DBuf<double> ringPhiBuf[kRing], ringField[kRing];
    int ringNext = 0;
    bool ringReady = false;
    // the flights' vertex fields are recomputed only for the cells that are
    // free or have a free neighbour (fieldCells, grown by removals on the
    // host); a slot whose field array has not been filled for every cell
    // since the potentials were last written takes the full pass
    bool ringFull[kRing] = {};
    DBuf<int32_t> fieldCells;
    int fieldCount = 0;
    bool fieldAll = false;             // a removal's list was cut short: all cells from then on
    std::vector<uint8_t> h_fieldActive;
    DBuf<uint8_t> cnz;
    std::vector<int32_t> h_row_ptr;
    std::vector<int32_t> h_col;  // the Delaunay neighbours never change

    // non-Neumann free rows in slot order, SELL-32 (cg.cu)
    DBuf<int32_t> vSlotOf, vNodeOf, vSliceStart, vSliceWidth, vCol, vPos, vCount;
    DBuf<float> vVal, vVec;  // vVec: d, x, r, u, w, p, sv, hist, each capacity+1
    DBuf<__nv_bfloat16> vVal16;  // vVal rounded to bf16 (multigrid smoothing pass)
    DBuf<float> vG;              // row sums of the V rows (capacity+1)
    // launch times [ms] of each level's operator and restriction (amg_tune),
    // 0 where a level has none
    float amgTunedA[tgd::kAmgMaxLevels] = {}, amgTunedR[tgd::kAmgMaxLevels] = {};
    float amgTunedFine = 0.0f;  // and of the level-0 pass
    // FP64 inner iterations: couplings at the SELL positions and the vectors
    // d64, x64, r64, p64, s64, w64 (each capacity+1), allocated at the first
    // solve with inner_precision 1
    DBuf<double> vVal64, vVec64;
    DBuf<double> vScal;
    DBuf<double> vfield;     // vertex fields of the current flight call
    DBuf<float> tetpack;     // packed tetrahedra for the flights
    int vCapacity = 0;       // slots incl. the append reserve
    int vActive = 0;         // slots in use (host mirror of vCount)
    double vEntries = 0.0;   // stored (non-padding) couplings

    // pinned host staging of the event loop's small copies, so that they
    // queue without blocking and a sync only waits for the device
    static constexpr int kMaxColours = 4096;
    struct Pinned {
        unsigned long long keys[8];
        double sums[4];
        double r2[4];
        double sb[4 * 17];
        double before[4];     // phi and field_o1 of the removed cell before removal
        double after[4];      // and after
        float normal[4];
        int32_t node[4];
        int32_t misc[4];      // V and N row counts, surface slots
        int32_t result[1024];
        int32_t flipped[1024];
        int32_t counts[2 * kMaxColours];
        int32_t pending[4096];  // cells flipped since the last solve
        int32_t activated[4096];  // cells a removal adds to fieldCells
        int32_t status[4];        // the device status word, read with each sync
        int32_t loopIters[4];     // the looped solve's iterations, read with the next sync
    };
    Pinned* pin = nullptr;
    int vNext = 0;            // host mirror of the V system's slot counter
    // the surface normal of an event's candidate runs on its own stream from
    // snapshots of the cell flags and types, beside the removal and solve
    cudaStream_t auxStream = nullptr;
    cudaEvent_t evSnap = nullptr, evNormal = nullptr;
    DBuf<uint8_t> snapFlags;
    DBuf<int8_t> snapType;
    DBuf<float> normalBuf;
    // One CG iteration of the multigrid solve (update, V-cycle, SpMV and the
    // step of the device iteration counter) captured as a CUDA graph and
    // replayed once per iteration: its kernels take the iteration index and
    // target from device memory (VSys::iter, rel2).  Captured again when the
    // V system's or the hierarchy's device state (pointers, schedules) or
    // the slots in use differ from the ones it was captured with.
    int launchMode = 2;                  // 2: the replayed graph in a device-side loop; 1: replay; 0: launch each kernel
    cudaStream_t captureStream = nullptr;
    cudaGraphExec_t iterExec = nullptr;
    DBuf<int32_t> iterDev;               // [1] the replayed iterations' counter
    DBuf<double> rel2Dev;                // [2] their relative target and iteration cap
    // launch mode 2: the replayed iteration inside a device-side loop (a
    // while-conditional graph node), one launch per inner solve; its count
    // of iterations reaches the host with the solve's next read
    cudaGraphExec_t loopExec = nullptr;
    std::vector<uint64_t> loopKey;
    DBuf<int32_t> loopDone;              // [1] iterations of the last looped solve
    long long loopNodes = 0;             // kernels per iteration of the loop
    long long loopStartNodes = 0;        // and of the solve's start before it
    std::vector<uint64_t> iterKey;       // the device state it was captured with
    long long iterNodes = 0;             // kernels in one replay
    // the same for the node-space CG iterations of the Neumann rows (run_cg)
    cudaGraphExec_t cgExec = nullptr;
    std::vector<uint64_t> cgKey;
    long long cgNodes = 0;
    DBuf<int32_t> cgDone;                // [1] iterations of the last one-launch node-space solve
    DBuf<int32_t> cgIterDev;             // [1] their counter
    DBuf<double> cgTgtDev;               // [2] their targets rel2, abs2
    int lastItersJacobi = 16, lastItersAmg = 4;  // iterations of the last inner solves
    int lastItersCg = 16;

    // multigrid preconditioner of the V system (amg.cu): hierarchy built on
    // the host from the V system as it is, uploaded as CSR levels
    bool amgReady = false;
    int amgSlots = 0;                       // V slots its prolongator covers
    tgd::AmgDev amg{};
    std::vector<DBuf<int32_t>> amgI;
    std::vector<DBuf<float>> amgF;
    void amg_release() {
        for (auto& b : amgI) b.release();
        for (auto& b : amgF) b.release();
        amgI.clear();
        amgF.clear();
        amgReady = false;
        amgSlots = 0;
    }

    VSys vs() {
        VSys v{};
        v.slot_of = vSlotOf.p;
        v.node_of = vNodeOf.p;
        v.slice_start = vSliceStart.p;
        v.slice_width = vSliceWidth.p;
        v.col = vCol.p;
        v.val = vVal.p;
        v.val16 = vVal16.p;
        v.g = vG.p;
        v.vpos = vPos.p;
        const size_t stride = (size_t)vCapacity + 1;
        v.d = vVec.p;
        v.x = vVec.p + stride;
        v.r = vVec.p + 2 * stride;
        v.u = vVec.p + 3 * stride;
        v.w = vVec.p + 4 * stride;
        v.p = vVec.p + 5 * stride;
        v.sv = vVec.p + 6 * stride;
        v.hist = vVec.p + 7 * stride;
        v.scal = vScal.p;
        v.count = vCount.p;
        v.capacity = vCapacity;
        v.val64 = vVal64.p;
        v.d64 = v.x64 = v.r64 = v.p64 = v.s64 = v.w64 = nullptr;
        if (vVec64.p) {
            v.d64 = vVec64.p;
            v.x64 = vVec64.p + stride;
            v.r64 = vVec64.p + 2 * stride;
            v.p64 = vVec64.p + 3 * stride;
            v.s64 = vVec64.p + 4 * stride;
            v.w64 = vVec64.p + 5 * stride;
        }
        v.iter = nullptr;
        v.rel2 = nullptr;
        return v;
    }

    bool bnormValid = false;
    double bnorm2 = 0.0;
    // residuals kept between solves: the last full pass of a converged solve
    // leaves every free row's FP64 residual and Dirichlet part (resid, by
    // node: r, then b) and their sums of squares (rsum: V rows, Neumann rows,
    // b).  Removals list the cells they flip, and the next solve's first
    // residual recomputes only those cells' rows and their neighbours'
    // (launch_residual_rows) instead of every row.  Anything else that
    // changes potentials, couplings or types clears residValid.
    DBuf<double> resid;
    DBuf<double> rsum;
    DBuf<int32_t> resStamp;
    DBuf<int32_t> pendingDev;
    int resEpoch = 0;
    bool residValid = false;
    int nPending = 0;
    bool pendingOverflow = false;
    // warm start bookkeeping: the correction of a solve is recorded (VSys
    // hist) when the solve starts from a converged state changed only by
    // removals; it seeds the next such solve
    bool converged = false;
    int removalsSinceSolve = 0;
    bool histValid = false;
    int lastSite = -1;                 // cell of the last removal
    // Monte-Carlo choice: a stream drawing like rand() after srand(seed)
    struct random_data rng {};
    char rngState[128] = {};
    bool rngSeeded = false;
    tg_learner* learner = nullptr;     // learned near-field start (learn.cu)
    int learnMode = 0;                 // bit 0 collect samples, bit 1 predict
    bool selValid = false;
    tg_select_info sel{};
    int vacuumId = -1;

    DevMesh dm() {
        DevMesh m;
        m.n = n;
        m.nnz = nnz;
        m.ntets = ntets;
        m.xyz = xyz.p;
        m.type = type.p;
        m.flags = flags.p;
        m.row_ptr = row_ptr.p;
        m.col = col.p;
        m.rev = rev.p;
        m.geom = geom.p;
        m.area_pos = area_pos.p;
        m.volume = volume.p;
        m.c64 = c64.p;
        m.cnz = cnz.p;
        m.ceff64 = ceff64.p;
        m.ceff32 = ceff32.p;
        m.diag64 = diag64.p;
        m.diag32 = diag32.p;
        m.q64 = q64.p;
        m.phi64 = phi64.p;
        m.colour = colour.p;
        m.tet_v = tet_v.p;
        m.tet_n = tet_n.p;
        m.node_tet = node_tet.p;
        m.types = dtypes.p;
        m.status = status.p;
        m.snap = snap;
        m.vfield = vfield.p;
        m.phiTrace = phiTrace.p;
        m.tetpack = tetpack.p;
        return m;
    }
    RowLists rl() {
        RowLists r;
        r.rowsV = rowsV.p;
        r.rowsN = rowsN.p;
        r.segStart = segStartD.p;
        r.countV = countVD.p;
        r.countN = countND.p;
        r.allV = allV.p;
        r.allN = allN.p;
        r.countAll = countAllD.p;
        r.ncolours = ncol;
        return r;
    }
    Surface sf() {
        Surface s;
        s.list = surfList.p;
        s.slot = surfSlot.p;
        s.count = surfCount.p;
        s.ratio = surfRatio.p;
        s.score = surfScore.p;
        s.capacity = n;
        return s;
    }
    CGVectors cg() {
        CGVectors v{};
        float* base = cgbuf.p;
        v.x = base;
        v.r = base + (size_t)n;
        v.z = base + 2 * (size_t)n;
        v.p = base + 3 * (size_t)n;
        v.ap = base + 4 * (size_t)n;
        v.scal = scalN.p;
        return v;
    }
};

namespace {

// The handle's device, current for the length of an entry point.
struct DeviceScope : ScopedDevice {
    explicit DeviceScope(const tg_handle* h) : ScopedDevice(h ? h->device : -1) {}
};

int fail(tg_handle* h, int code, const std::string& msg) {
    if (h) h->err = msg;
    g_error = msg;
    return code;
}

int cuda_check(tg_handle* h, cudaError_t e, const char* where) {
    if (e == cudaSuccess) return TG_OK;
    return fail(h, TG_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

#define CK(expr)                                              \
    do {                                                      \
        const int _rc = cuda_check(h, (expr), #expr);         \
        if (_rc != TG_OK) return _rc;                         \
    } while (0)

// Synchronises the stream and maps the device status word to a code.
int status_code(tg_handle* h, int st, const char* where);

// The status word comes back in the same stream-ordered copy as the
// sync, into pinned memory: one round trip per check.
int sync_status(tg_handle* h, const char* where) {
    CK(cudaGetLastError());
    int st = 0;
    if (h->pin) {
        CK(cudaMemcpyAsync(&h->pin->status[0], h->status.p, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
        st = h->pin->status[0];
    } else {
        CK(cudaStreamSynchronize(h->stream));
        CK(cudaMemcpy(&st, h->status.p, sizeof(int), cudaMemcpyDeviceToHost));
    }
    if (st == 0) return TG_OK;
    CK(cudaMemsetAsync(h->status.p, 0, sizeof(int), h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return status_code(h, st, where);
}

// Maps a device status word to a code and message.
int status_code(tg_handle* h, int st, const char* where) {
    std::string what = where;
    if (st & S_NAN) return fail(h, TG_ERR_NAN, what + ": NaN");
    if (st & S_SINGULAR) return fail(h, TG_ERR_SINGULAR, what + ": singular field_o1 system");
    if (st & S_NOT_SURFACE) return fail(h, TG_ERR_NOT_SURFACE, what + ": node is not a surface cell");
    if (st & S_WALK_LIMIT) return fail(h, TG_ERR_WALK_LIMIT, what + ": tetrahedron walk limit");
    if (st & S_UNKNOWN_TYPE) return fail(h, TG_ERR_UNKNOWN_TYPE, what + ": unknown cell type");
    if (st & S_TIMEOUT) return fail(h, TG_ERR_TIMEOUT, what + ": a bounded device wait ran out");
    return fail(h, TG_ERR_CUDA, what + ": device status");
}

template <typename T>
int stage(tg_handle* h, DBuf<T>& b, size_t count) {
    if (b.n >= count) return TG_OK;
    return cuda_check(h, b.alloc(std::max<size_t>(count, 1024)), "staging alloc");
}

int refresh_counts(tg_handle* h) {
    CK(cudaMemcpyAsync(h->countV.data(), h->countVD.p, sizeof(int32_t) * h->ncol, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(h->countN.data(), h->countND.p, sizeof(int32_t) * h->ncol, cudaMemcpyDeviceToHost, h->stream));
    int32_t ca[2];
    CK(cudaMemcpyAsync(ca, h->countAllD.p, sizeof(ca), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(&h->surfSlots, h->surfCount.p, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->countAllV = ca[0];
    h->countAllN = ca[1];
    h->surfSlots = std::min(h->surfSlots, h->n);
    return TG_OK;
}

// n coloured sweeps over all free rows; devAcc receives max |delta| of the
// last.  All but the first launch are links of a chain: none of them writes
// what the next loads before it waits
void sweep_all(tg_handle* h, int32_t n, double* devAcc) {
    DevMesh m = h->dm();
    bool first = true;
    for (int32_t it = 0; it < n; it++)
        for (int c = 0; c < h->ncol; c++) {
            if (h->countV[c] + h->countN[c] <= 0) continue;
            auto go = [&] {
                launch_sweep64(m, h->rowsV.p + h->segStart[c], h->countV[c], h->rowsN.p + h->segStart[c], h->countN[c],
                               it == n - 1 ? devAcc : nullptr, h->stream);
            };
            if (first) {
                go();
            } else {
                ChainScope chained;
                go();
            }
            first = false;
        }
}

// regression slope of the deviation queue as Grid_3d::Table::relax computes
// it (grid_3d.cpp:628-654)
bool stagnated(const std::deque<double>& queue, unsigned queueSize, unsigned cycleSize) {
    if (queueSize == 0 || queue.size() != queueSize) return false;
    const double xMean = (queueSize - 1) / 2.0;
    double yMean = 0.0;
    for (double v : queue) yMean += v;
    yMean /= queueSize;
    double num = 0.0;
    int x = 0;
    for (double v : queue) num += (x++ - xMean) * (v - yMean);
    double den = queueSize;
    den *= queueSize;
    den -= 1;
    den *= queueSize;
    den *= cycleSize;
    den /= 12.0;
    return num / den == 0.0;
}

}  // namespace

extern "C" {

const char* tg_last_error(const tg_handle* h) { return h ? h->err.c_str() : g_error.c_str(); }
int tg_num_nodes(const tg_handle* h) { return h ? h->n : 0; }

int tg_create(const tg_mesh_desc* d, tg_handle** out) {
    if (!d || !out || d->num_nodes <= 0 || !d->xyz || !d->type_id || !d->row_ptr || !d->col || !d->coupling ||
        !d->types || d->num_types <= 0)
        return fail(nullptr, TG_ERR_ARGUMENT, "tg_create: incomplete mesh description");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        return fail(nullptr, TG_ERR_CUDA, "tg_create: no CUDA device");
    tg_handle* h = new tg_handle();
    if (cudaGetDevice(&h->device) != cudaSuccess) {
        delete h;
        return fail(nullptr, TG_ERR_CUDA, "tg_create: no current CUDA device");
    }
    const int n = d->num_nodes;
    const int nnz = d->row_ptr[n];
    h->n = n;
    h->nnz = nnz;
    h->ntets = d->num_tets;
    h->types.assign(128, tg_type{});
    for (auto& t : h->types) t.id = -1;
    for (int k = 0; k < d->num_types; k++) {
        const tg_type& t = d->types[k];
        if (t.id < 0 || t.id > 127) {
            delete h;
            return fail(nullptr, TG_ERR_ARGUMENT, "tg_create: type id out of range");
        }
        h->types[t.id] = t;
        if (t.id >= 10) h->coordinationActive = true;
    }
    // every index the device walks and gathers through must stay inside its
    // array: vertices in [0, N), neighbours and node_tet in [-1, T)
    if (d->num_tets < 0 || (d->num_tets > 0 && (!d->tet_v || !d->tet_n))) {
        delete h;
        return fail(nullptr, TG_ERR_ARGUMENT, "tg_create: tetrahedra arrays missing");
    }
    for (size_t k = 0; k < 4 * (size_t)d->num_tets; k++)
        if (d->tet_v[k] < 0 || d->tet_v[k] >= n || d->tet_n[k] < -1 || d->tet_n[k] >= d->num_tets) {
            delete h;
            return fail(nullptr, TG_ERR_ARGUMENT, "tg_create: tetrahedron vertex or neighbour index out of range");
        }
    if (d->node_tet && d->num_tets > 0)
        for (int i = 0; i < n; i++)
            if (d->node_tet[i] < -1 || d->node_tet[i] >= d->num_tets) {
                delete h;
                return fail(nullptr, TG_ERR_ARGUMENT, "tg_create: node_tet index out of range");
            }
    std::vector<DType> dt(128);
    for (int k = 0; k < 128; k++) {
        const tg_type& t = h->types[k];
        DType& o = dt[k];
        o.present = t.id >= 0;
        o.epsilon = t.epsilon;
        o.evap_field = t.evap_field;
        o.evap_energy = t.evap_energy;
        o.charge_density = t.charge_density;
        o.phi = t.phi;
        o.removable = t.removable != 0;
        o.neumann = t.neumann != 0;
        o.dirichlet = t.dirichlet != 0;
    }
    h->h_type.assign(d->type_id, d->type_id + n);
    std::vector<uint8_t> flags(n, 0);
    for (int i = 0; i < n; i++) {
        const int t = d->type_id[i];
        if (t < 0 || !dt[t].present) {
            delete h;
            return fail(nullptr, TG_ERR_UNKNOWN_TYPE, "tg_create: node with unknown type id");
        }
        if (d->hull && d->hull[i]) flags[i] |= F_HULL;
        if (dt[t].dirichlet) flags[i] |= F_DIRICHLET;
        if (dt[t].neumann) flags[i] |= F_NEUMANN;
    }
    // reverse index, geometric factor, positive-area flag
    std::vector<int32_t> rev(nnz);
    std::vector<double> geom(nnz);
    std::vector<uint8_t> apos(nnz);
    for (int i = 0; i < n; i++)
        for (int q = d->row_ptr[i]; q < d->row_ptr[i + 1]; q++) {
            const int j = d->col[q];
            if (j < 0 || j >= n) {
                delete h;
                return fail(nullptr, TG_ERR_ARGUMENT, "tg_create: neighbour index out of range");
            }
            const int32_t* b = d->col + d->row_ptr[j];
            const int32_t* e = d->col + d->row_ptr[j + 1];
            const int32_t* f = std::lower_bound(b, e, (int32_t)i);
            if (f == e || *f != i) {
                delete h;
                return fail(nullptr, TG_ERR_ARGUMENT, "tg_create: adjacency is not symmetric or not sorted");
            }
            rev[q] = (int32_t)(f - d->col);
            if (d->geom) {
                geom[q] = d->geom[q];
            } else {
                const double e1 = dt[d->type_id[i]].epsilon, e2 = dt[d->type_id[j]].epsilon;
                geom[q] = d->coupling[q] / (2.0 * e1 * e2 / (e1 + e2));
            }
            apos[q] = d->area_pos ? d->area_pos[q] : (geom[q] != 0.0);
        }
    // greedy colouring of the whole Delaunay graph
    std::vector<int32_t> colour(n, -1);
    int ncol = 0;
    {
        std::vector<int> mark(128, -1);
        for (int i = 0; i < n; i++) {
            for (int q = d->row_ptr[i]; q < d->row_ptr[i + 1]; q++) {
                const int c = colour[d->col[q]];
                if (c >= 0 && c < 128) mark[c] = i;
            }
            int c = 0;
            while (c < 128 && mark[c] == i) c++;
            colour[i] = c;
            ncol = std::max(ncol, c + 1);
        }
    }
    if (ncol > 64) {
        delete h;
        return fail(nullptr, TG_ERR_ARGUMENT, "tg_create: more than 64 colours");
    }
    h->ncol = ncol;
    std::vector<int32_t> csize(ncol, 0);
    for (int i = 0; i < n; i++) csize[colour[i]]++;
    h->segStart.assign(ncol, 0);
    for (int c = 1; c < ncol; c++) h->segStart[c] = h->segStart[c - 1] + csize[c - 1];
    h->countV.assign(ncol, 0);
    h->countN.assign(ncol, 0);
    std::vector<int32_t> rowsV(n, -1), rowsN(n, -1), allV, allN;
    for (int i = 0; i < n; i++) {
        if (flags[i] & F_DIRICHLET) continue;
        const int c = colour[i];
        if (flags[i] & F_NEUMANN) {
            rowsN[h->segStart[c] + h->countN[c]++] = i;
            allN.push_back(i);
        } else {
            rowsV[h->segStart[c] + h->countV[c]++] = i;
            allV.push_back(i);
        }
        flags[i] |= F_FREE;
    }
    h->countAllV = (int32_t)allV.size();
    h->countAllN = (int32_t)allN.size();
    allV.resize(n, -1);
    allN.resize(n, -1);
    std::vector<double> phi(n), q(n, 0.0);
    for (int i = 0; i < n; i++) {
        phi[i] = d->phi ? (double)d->phi[i] : (double)dt[d->type_id[i]].phi;
        if (d->volume) q[i] = d->volume[i] * (double)dt[d->type_id[i]].charge_density / kEpsilon0;
    }
    h->top_z = -1e30f;
    double amax = 0.0;
    for (int i = 0; i < n; i++) {
        h->top_z = std::max(h->top_z, d->xyz[3 * i + 2]);
        for (int k = 0; k < 3; k++) amax = std::max(amax, std::fabs((double)d->xyz[3 * i + k]));
    }
    // the integer grid of the host Delaunay builder (delaunay.cpp): |x| <= 2^40
    h->snap = amax > 0.0 ? std::ldexp(1.0, (int)std::floor(std::log2(std::ldexp(1.0, 40) / amax))) : 1.0;
    h->h_xyz.assign(d->xyz, d->xyz + 3 * (size_t)n);
    h->h_row_ptr.assign(d->row_ptr, d->row_ptr + n + 1);
    h->h_col.assign(d->col, d->col + d->row_ptr[n]);
    if (d->node_tet) h->h_node_tet.assign(d->node_tet, d->node_tet + n);

    // ---- V system: slots, SELL-32 couplings, append reserve ----
    auto keepInV = [&](int j) {
        return !(flags[j] & F_NEUMANN) && (!(flags[j] & F_DIRICHLET) || dt[d->type_id[j]].removable);
    };
    const int nV0 = h->countAllV;
    std::vector<int32_t> vlen(nV0);
    int maxRow = 1;
    for (int i = 0; i < n; i++) maxRow = std::max(maxRow, d->row_ptr[i + 1] - d->row_ptr[i]);
    for (int r = 0; r < nV0; r++) {
        const int i = allV[r];
        int c = 0;
        for (int qq = d->row_ptr[i]; qq < d->row_ptr[i + 1]; qq++) c += keepInV(d->col[qq]);
        vlen[r] = c;
    }
    // rows sorted by stored length within windows of 1024 (locality kept,
    // slices nearly full)
    std::vector<int32_t> vorder(nV0);
    for (int r = 0; r < nV0; r++) vorder[r] = r;
    for (int w0 = 0; w0 < nV0; w0 += 1024) {
        const int w1 = std::min(nV0, w0 + 1024);
        std::stable_sort(vorder.begin() + w0, vorder.begin() + w1,
                         [&](int a, int b) { return vlen[a] > vlen[b]; });
    }
    int removableAtoms = 0;
    for (int i = 0; i < n; i++) removableAtoms += (flags[i] & F_DIRICHLET) && dt[d->type_id[i]].removable;
    const int E0 = (nV0 + 31) / 32 * 32;
    const int reserve = ((std::min(65536, std::max(1024, removableAtoms)) + 31) / 32) * 32;
    h->vCapacity = E0 + reserve;
    const int nSlices = h->vCapacity / 32;
    std::vector<int32_t> sliceStart(nSlices + 1, 0), sliceWidth(nSlices, 0);
    for (int s = 0; s < E0 / 32; s++) {
        int wmax = 0;
        for (int k = 0; k < 32; k++) {
            const int r = s * 32 + k;
            if (r < nV0) wmax = std::max(wmax, vlen[vorder[r]]);
        }
        sliceWidth[s] = wmax;
    }
    for (int s = E0 / 32; s < nSlices; s++) sliceWidth[s] = maxRow;
    for (int s = 0; s < nSlices; s++) sliceStart[s + 1] = sliceStart[s] + 32 * sliceWidth[s];
    const size_t vStore = (size_t)sliceStart[nSlices];
    const int zeroSlot = h->vCapacity;
    std::vector<int32_t> vSlotOf(n, -1), vNodeOf(h->vCapacity, -1), vCol(vStore, zeroSlot), vPos(nnz, -1);
    std::vector<float> vVal(vStore, 0.0f), vD(h->vCapacity + 1, 1.0f);
    for (int s = 0; s < nV0; s++) {
        vNodeOf[s] = allV[vorder[s]];
        vSlotOf[vNodeOf[s]] = s;
    }
    for (int s = 0; s < nV0; s++) {
        const int i = vNodeOf[s];
        const int base = sliceStart[s / 32] + (s & 31);
        double diag = 0.0;
        int k = 0;
        for (int qq = d->row_ptr[i]; qq < d->row_ptr[i + 1]; qq++) {
            const int j = d->col[qq];
            const double c = (flags[j] & F_NEUMANN) ? 0.0 : d->coupling[qq];
            diag += c;
            if (!keepInV(j)) continue;
            vCol[base + 32 * k] = vSlotOf[j] >= 0 ? vSlotOf[j] : zeroSlot;
            vVal[base + 32 * k] = (float)c;
            vPos[qq] = base + 32 * k;
            k++;
        }
        vD[s] = (float)diag;
    }
    h->vActive = E0;
    for (int r = 0; r < nV0; r++) h->vEntries += vlen[r];

    auto up = [&](auto& buf, const auto* src, size_t count) -> cudaError_t {
        cudaError_t e = buf.alloc(count);
        if (e != cudaSuccess) return e;
        if (count && src) return cudaMemcpy(buf.p, src, count * sizeof(*src), cudaMemcpyHostToDevice);
        return cudaSuccess;
    };
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    // the event's own work runs at the highest stream priority, so that its
    // kernels take SMs ahead of the blocks of the flight slots
    int leastPriority = 0, greatestPriority = 0;
    chk(cudaDeviceGetStreamPriorityRange(&leastPriority, &greatestPriority));
    chk(cudaStreamCreateWithPriority(&h->stream, cudaStreamNonBlocking, greatestPriority));
    chk(cudaStreamCreateWithPriority(&h->auxStream, cudaStreamNonBlocking, greatestPriority));
    chk(cudaEventCreateWithFlags(&h->evSnap, cudaEventDisableTiming));
    chk(cudaEventCreateWithFlags(&h->evNormal, cudaEventDisableTiming));
    chk(cudaEventCreate(&h->evStart));
    chk(cudaEventCreate(&h->evStop));
    chk(up(h->xyz, d->xyz, 3 * (size_t)n));
    chk(up(h->type, d->type_id, n));
    chk(h->typeScratch.alloc(n));
    chk(up(h->flags, flags.data(), n));
    chk(up(h->area_pos, apos.data(), nnz));
    chk(up(h->row_ptr, d->row_ptr, n + 1));
    chk(up(h->col, d->col, nnz));
    chk(up(h->rev, rev.data(), nnz));
    chk(up(h->colour, colour.data(), n));
    chk(up(h->geom, geom.data(), nnz));
    if (d->volume) chk(up(h->volume, d->volume, n));
    chk(up(h->c64, d->coupling, nnz));
    {
        std::vector<uint8_t> nzv(nnz);
        for (size_t q = 0; q < (size_t)nnz; q++) nzv[q] = d->coupling[q] != 0.0;
        chk(up(h->cnz, nzv.data(), nnz));
        // cells whose vertex field can change: free, or with a free neighbour
        h->h_fieldActive.assign(n, 0);
        std::vector<int32_t> cells;
        for (int i = 0; i < n; i++) {
            bool act = !(flags[i] & F_DIRICHLET);
            for (int q = d->row_ptr[i]; q < d->row_ptr[i + 1] && !act; q++) act = !(flags[d->col[q]] & F_DIRICHLET);
            if (act) {
                h->h_fieldActive[i] = 1;
                cells.push_back(i);
            }
        }
        chk(h->fieldCells.alloc(n));
        if (e == cudaSuccess && !cells.empty())
            chk(cudaMemcpy(h->fieldCells.p, cells.data(), sizeof(int32_t) * cells.size(), cudaMemcpyHostToDevice));
        h->fieldCount = (int)cells.size();
    }
    chk(h->ceff64.alloc(nnz));
    chk(h->ceff32.alloc(nnz));
    chk(h->diag64.alloc(n));
    chk(h->diag32.alloc(n));
    chk(up(h->q64, q.data(), n));
    chk(up(h->phi64, phi.data(), n));
    if (d->num_tets > 0 && d->tet_v && d->tet_n) {
        chk(up(h->tet_v, d->tet_v, 4 * (size_t)d->num_tets));
        chk(up(h->tet_n, d->tet_n, 4 * (size_t)d->num_tets));
    }
    if (d->node_tet) chk(up(h->node_tet, d->node_tet, n));
    chk(up(h->dtypes, dt.data(), 128));
    chk(h->status.alloc(1));
    if (e == cudaSuccess) chk(cudaMemset(h->status.p, 0, sizeof(int)));
    chk(up(h->rowsV, rowsV.data(), n));
    chk(up(h->rowsN, rowsN.data(), n));
    chk(up(h->allV, allV.data(), n));
    chk(up(h->allN, allN.data(), n));
    chk(up(h->segStartD, h->segStart.data(), ncol));
    chk(up(h->countVD, h->countV.data(), ncol));
    chk(up(h->countND, h->countN.data(), ncol));
    int32_t ca[2] = {h->countAllV, h->countAllN};
    chk(up(h->countAllD, ca, 2));
    chk(h->surfList.alloc(n));
    chk(h->surfSlot.alloc(n));
    chk(h->surfCount.alloc(1));
    chk(h->surfRatio.alloc(n));
    chk(h->surfScore.alloc(n));
    chk(h->cgbuf.alloc(5 * (size_t)n));
    if (e == cudaSuccess) chk(cudaMemset(h->cgbuf.p, 0, 5 * (size_t)n * sizeof(float)));
    chk(h->acc.alloc(16));
    chk(h->resid.alloc(2 * (size_t)n));
    if (e == cudaSuccess) chk(cudaMemset(h->resid.p, 0, 2 * (size_t)n * sizeof(double)));
    chk(h->rsum.alloc(4));
    if (e == cudaSuccess) chk(cudaMemset(h->rsum.p, 0, 4 * sizeof(double)));
    chk(h->resStamp.alloc(n));
    if (e == cudaSuccess) chk(cudaMemset(h->resStamp.p, 0, (size_t)n * sizeof(int32_t)));
    chk(h->pendingDev.alloc(4096));
    chk(h->keys.alloc(8));
    chk(h->result.alloc(1024));
    chk(h->local.alloc(1 << 16));
    chk(h->localCount.alloc(66));
    chk(h->localScratch.alloc(1 << 16));
    chk(h->vfield.alloc(3 * (size_t)n));
    chk(h->phiTrace.alloc(n));
    chk(h->statusTrace.alloc(1));
    if (e == cudaSuccess) chk(cudaMemset(h->statusTrace.p, 0, sizeof(int)));
    chk(up(h->vSlotOf, vSlotOf.data(), n));
    chk(up(h->vNodeOf, vNodeOf.data(), h->vCapacity));
    chk(up(h->vSliceStart, sliceStart.data(), nSlices + 1));
    chk(up(h->vSliceWidth, sliceWidth.data(), nSlices));
    chk(up(h->vCol, vCol.data(), vStore));
    chk(up(h->vVal, vVal.data(), vStore));
    chk(h->vVal16.alloc(vStore));
    chk(h->vG.alloc((size_t)h->vCapacity + 1));
    chk(up(h->vPos, vPos.data(), nnz));
    {
        const int32_t next = E0;
        chk(up(h->vCount, &next, 1));
        h->vNext = E0;
    }
    if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void**>(&h->pin), sizeof(tg_handle::Pinned));
    chk(h->snapFlags.alloc(n));
    chk(h->snapType.alloc(n));
    chk(h->normalBuf.alloc(4));
    chk(h->stageI.alloc(1024));
    chk(h->stageD.alloc(1024));
    chk(h->stageF.alloc(1024));
    chk(h->vVec.alloc(8 * ((size_t)h->vCapacity + 1)));
    if (e == cudaSuccess) chk(cudaMemset(h->vVec.p, 0, 8 * ((size_t)h->vCapacity + 1) * sizeof(float)));
    if (e == cudaSuccess) chk(cudaMemcpy(h->vVec.p, vD.data(), vD.size() * sizeof(float), cudaMemcpyHostToDevice));
    if (h->ntets > 0) chk(h->tetpack.alloc(32 * (size_t)h->ntets));
    if (e != cudaSuccess) {
        const std::string msg = std::string("tg_create: ") + cudaGetErrorString(e);
        tg_destroy(h);
        return fail(nullptr, TG_ERR_CUDA, msg);
    }
    launch_rebuild_rows(h->dm(), h->stream);
    launch_vsys_derive(h->vs(), h->vVal.n, h->stream);
    if (h->ntets > 0) launch_pack_tets(h->dm(), h->tetpack.p, h->stream);
    const int rc = sync_status(h, "tg_create");
    if (rc != TG_OK) {
        const std::string msg = h->err;
        tg_destroy(h);
        return fail(nullptr, rc, msg);
    }
    *out = h;
    return TG_OK;
}

void tg_destroy(tg_handle* h) {
    DeviceScope dev_scope(h);
    if (!h) return;
    if (h->stream) cudaStreamSynchronize(h->stream);
    h->xyz.release(); h->type.release(); h->typeScratch.release(); h->flags.release(); h->area_pos.release();
    h->row_ptr.release(); h->col.release(); h->rev.release(); h->colour.release(); h->tet_v.release();
    h->tet_n.release(); h->node_tet.release(); h->geom.release(); h->volume.release(); h->c64.release();
    h->cnz.release(); h->fieldCells.release();
    h->ceff64.release(); h->diag64.release(); h->q64.release(); h->phi64.release(); h->ceff32.release();
    h->diag32.release(); h->dtypes.release(); h->status.release(); h->rowsV.release(); h->rowsN.release();
    h->allV.release(); h->allN.release(); h->segStartD.release(); h->countVD.release(); h->countND.release();
    h->countAllD.release(); h->surfList.release(); h->surfSlot.release(); h->surfCount.release();
    h->surfRatio.release(); h->surfScore.release(); h->cgbuf.release(); h->scalN.release(); h->acc.release();
    h->resid.release(); h->rsum.release(); h->resStamp.release(); h->pendingDev.release();
    h->keys.release(); h->result.release(); h->local.release(); h->localCount.release();
    h->localScratch.release(); h->stageI.release(); h->stageD.release(); h->stageF.release();
    h->stageImpact.release(); h->pathBuf.release(); h->pathErr.release();
    h->amg_release();
    if (h->pin) cudaFreeHost(h->pin);
    h->pin = nullptr;
    if (h->auxStream) {
        cudaStreamSynchronize(h->auxStream);
        cudaStreamDestroy(h->auxStream);
    }
    if (h->iterExec) cudaGraphExecDestroy(h->iterExec);
    if (h->loopExec) cudaGraphExecDestroy(h->loopExec);
    h->loopDone.release();
    if (h->cgExec) cudaGraphExecDestroy(h->cgExec);
    h->cgDone.release();
    h->cgIterDev.release();
    h->cgTgtDev.release();
    if (h->captureStream) cudaStreamDestroy(h->captureStream);
    h->iterDev.release();
    h->rel2Dev.release();
    if (h->evSnap) cudaEventDestroy(h->evSnap);
    if (h->evNormal) cudaEventDestroy(h->evNormal);
    h->snapFlags.release();
    h->snapType.release();
    h->normalBuf.release();
    h->vSlotOf.release(); h->vNodeOf.release(); h->vSliceStart.release(); h->vSliceWidth.release();
    h->vCol.release(); h->vPos.release(); h->vCount.release(); h->vVal.release(); h->vVec.release();
    h->vVal16.release(); h->vG.release(); h->vVal64.release(); h->vVec64.release();
    h->vScal.release(); h->vfield.release(); h->tetpack.release();
    for (int r = 0; r < tg_handle::kRing; r++) {
        if (h->ringStream[r]) {
            cudaStreamSynchronize(h->ringStream[r]);
            cudaStreamDestroy(h->ringStream[r]);
        }
        if (h->ringPhi[r]) cudaEventDestroy(h->ringPhi[r]);
        if (h->ringDone[r]) cudaEventDestroy(h->ringDone[r]);
        h->ringPhiBuf[r].release();
        h->ringField[r].release();
    }
    h->phiTrace.release(); h->statusTrace.release();
    if (h->evStart) cudaEventDestroy(h->evStart);
    if (h->evStop) cudaEventDestroy(h->evStop);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

int tg_timer_start(tg_handle* h) {
    DeviceScope dev_scope(h);
    if (!h) return fail(h, TG_ERR_ARGUMENT, "tg_timer_start: null handle");
    CK(cudaEventRecord(h->evStart, h->stream));
    return TG_OK;
}

int tg_timer_stop(tg_handle* h, float* ms) {
    DeviceScope dev_scope(h);
    if (!h || !ms) return fail(h, TG_ERR_ARGUMENT, "tg_timer_stop: null argument");
    CK(cudaEventRecord(h->evStop, h->stream));
    CK(cudaEventSynchronize(h->evStop));
    CK(cudaEventElapsedTime(ms, h->evStart, h->evStop));
    return TG_OK;
}

int64_t tg_launch_count(const tg_handle*) { return (int64_t)launches_so_far(); }

int tg_set_launch_mode(tg_handle* h, int32_t mode) {
    if (!h || mode < 0 || mode > 2) return fail(h, TG_ERR_ARGUMENT, "tg_set_launch_mode: mode 0, 1 or 2");
    h->launchMode = mode;
    return TG_OK;
}

int tg_bench_kernel(tg_handle* h, int32_t which, int32_t iters, float* avg_ms, double* bytes) {
    DeviceScope dev_scope(h);
    if (!h || iters < 1 || !avg_ms || !bytes) return fail(h, TG_ERR_ARGUMENT, "tg_bench_kernel: bad argument");
    DevMesh m = h->dm();
    // rows of the timed kernel and their neighbour entries
    std::vector<int32_t> rowsV(h->countAllV), rowsN(h->countAllN);
    if (h->countAllV) CK(cudaMemcpy(rowsV.data(), h->allV.p, sizeof(int32_t) * rowsV.size(), cudaMemcpyDeviceToHost));
    if (h->countAllN) CK(cudaMemcpy(rowsN.data(), h->allN.p, sizeof(int32_t) * rowsN.size(), cudaMemcpyDeviceToHost));
    auto entries = [&](const std::vector<int32_t>& rows) {
        double e = 0.0;
        for (int32_t i : rows) e += h->h_row_ptr[i + 1] - h->h_row_ptr[i];
        return e;
    };
    if (which == 0) {
        // k_vcg_spmv over the V system (SELL-32): col + val per stored entry
        // (padding excluded), u (one compulsory read per row, the gathers
        // hit the same vector), d, and the w write per row
        const double rows = (double)h->vActive, stored = h->vEntries;
        *bytes = rows * (4 + 4 + 4) + stored * (4 + 4);
        if (h->vScal.n < 8) CK(h->vScal.alloc(8));
        VSys v = h->vs();
        CK(cudaMemsetAsync(h->vScal.p, 0, 8 * sizeof(double), h->stream));
        launch_vcg_spmv(v, h->vActive, 0, -1.0, false, h->stream);  // warm
        CK(cudaEventRecord(h->evStart, h->stream));
        for (int k = 0; k < iters; k++) launch_vcg_spmv(v, h->vActive, 0, -1.0, false, h->stream);
        CK(cudaEventRecord(h->evStop, h->stream));
    } else if (which == 1) {
        // k_residual over all free rows: row index, two row pointers, col +
        // ceff64 per entry, phi64 (once per row), diag64, q64
        const double rows = (double)(rowsV.size() + rowsN.size()), nnz = entries(rowsV) + entries(rowsN);
        *bytes = rows * (4 + 8 + 8 + 8 + 8) + nnz * (4 + 8);
        launch_residual(m, h->allV.p, h->countAllV, nullptr, h->acc.p, h->stream);
        CK(cudaEventRecord(h->evStart, h->stream));
        for (int k = 0; k < iters; k++) {
            launch_residual(m, h->allV.p, h->countAllV, nullptr, h->acc.p, h->stream);
            launch_residual(m, h->allN.p, h->countAllN, nullptr, h->acc.p, h->stream);
        }
        CK(cudaEventRecord(h->evStop, h->stream));
    } else if (which == 2) {
        // k_amg_fine (the multigrid's level-0 smoothing pass, t = b - A y
        // over SELL-32): col + bf16 val per stored entry, and per row b, y
        // (the gathers hit the same vector), the row sum g and the t write
        if (!h->amgReady) return fail(h, TG_ERR_ARGUMENT, "tg_bench_kernel: no multigrid hierarchy yet");
        const double rows = (double)h->vActive, stored = h->vEntries;
        *bytes = rows * (4 + 4 + 4 + 4) + stored * (4 + 2);
        if (h->vScal.n < 8) CK(h->vScal.alloc(8));
        VSys v = h->vs();
        launch_amg_fine_residual(v, h->vActive, h->amg, h->stream);  // warm
        CK(cudaEventRecord(h->evStart, h->stream));
        for (int k = 0; k < iters; k++) launch_amg_fine_residual(v, h->vActive, h->amg, h->stream);
        CK(cudaEventRecord(h->evStop, h->stream));
    } else {
        return fail(h, TG_ERR_ARGUMENT, "tg_bench_kernel: unknown kernel");
    }
    CK(cudaEventSynchronize(h->evStop));
    float ms = 0.0f;
    CK(cudaEventElapsedTime(&ms, h->evStart, h->evStop));
    *avg_ms = ms / iters;
    return sync_status(h, "tg_bench_kernel");
}

int tg_get_phi(tg_handle* h, double* phi) {
    DeviceScope dev_scope(h);
    if (!h || !phi) return fail(h, TG_ERR_ARGUMENT, "tg_get_phi: null argument");
    CK(cudaMemcpyAsync(phi, h->phi64.p, sizeof(double) * h->n, cudaMemcpyDeviceToHost, h->stream));
    return sync_status(h, "tg_get_phi");
}

int tg_set_phi(tg_handle* h, const double* phi) {
    DeviceScope dev_scope(h);
    if (!h || !phi) return fail(h, TG_ERR_ARGUMENT, "tg_set_phi: null argument");
    CK(cudaMemcpyAsync(h->phi64.p, phi, sizeof(double) * h->n, cudaMemcpyHostToDevice, h->stream));
    for (int r = 0; r < tg_handle::kRing; r++) h->ringFull[r] = true;  // Dirichlet potentials may have changed
    h->bnormValid = false;
    h->selValid = false;
    h->converged = h->histValid = h->residValid = false;
    return sync_status(h, "tg_set_phi");
}

int tg_get_couplings(tg_handle* h, double* out) {
    DeviceScope dev_scope(h);
    if (!h || !out) return fail(h, TG_ERR_ARGUMENT, "tg_get_couplings: null argument");
    CK(cudaMemcpyAsync(out, h->c64.p, sizeof(double) * h->nnz, cudaMemcpyDeviceToHost, h->stream));
    return sync_status(h, "tg_get_couplings");
}

int tg_get_types(tg_handle* h, int8_t* out) {
    DeviceScope dev_scope(h);
    if (!h || !out) return fail(h, TG_ERR_ARGUMENT, "tg_get_types: null argument");
    CK(cudaMemcpyAsync(out, h->type.p, h->n, cudaMemcpyDeviceToHost, h->stream));
    return sync_status(h, "tg_get_types");
}

int tg_relax_cycles(tg_handle* h, int32_t n, double* deviation) {
    DeviceScope dev_scope(h);
    if (!h || n < 1) return fail(h, TG_ERR_ARGUMENT, "tg_relax_cycles: bad argument");
    CK(cudaMemsetAsync(h->acc.p, 0, sizeof(double), h->stream));
    sweep_all(h, n, h->acc.p);
    CK(cudaMemcpyAsync(&h->pin->sums[2], h->acc.p, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    const int rc = sync_status(h, "tg_relax_cycles");
    if (deviation) *deviation = h->pin->sums[2];
    h->selValid = false;
    h->converged = h->histValid = h->residValid = false;
    return rc;
}

int tg_relax_threshold(tg_handle* h, double threshold, int32_t cycle, int32_t queueSize, int64_t maxSweeps,
                       int64_t* iterations, double* deviation) {
    DeviceScope dev_scope(h);
    if (!h || cycle < 1) return fail(h, TG_ERR_ARGUMENT, "tg_relax_threshold: bad argument");
    std::deque<double> queue;
    int64_t iter = 0;
    double dev = 0.0;
    int rc = TG_OK;
    do {
        rc = tg_relax_cycles(h, cycle, &dev);
        if (rc != TG_OK) break;
        queue.push_back(dev);
        while ((int)queue.size() > queueSize) queue.pop_front();
        if (stagnated(queue, (unsigned)queueSize, (unsigned)cycle)) {
            rc = fail(h, TG_ERR_RELAX_FAULT, "tg_relax_threshold: stagnation");
            break;
        }
        iter += cycle;
        if (maxSweeps > 0 && iter >= maxSweeps && dev > threshold) {
            rc = fail(h, TG_ERR_ITERATION_CAP, "tg_relax_threshold: sweep cap reached");
            break;
        }
    } while (dev > threshold);
    if (iterations) *iterations = iter;
    if (deviation) *deviation = dev;
    return rc;
}

int tg_local_relax(tg_handle* h, int32_t node, int32_t shell, double threshold, int32_t cycle, int32_t queueSize,
                   int64_t* iterations, double* deviation) {
    DeviceScope dev_scope(h);
    if (!h || node < 0 || node >= h->n || cycle < 1) return fail(h, TG_ERR_ARGUMENT, "tg_local_relax: bad argument");
    h->converged = h->histValid = h->residValid = false;
    DevMesh m = h->dm();
    launch_local_set(m, node, shell, h->local.p, h->localCount.p, (int)h->local.n, h->localScratch.p,
                     (int)h->localScratch.n, h->ncol, h->stream);
    int rc = TG_OK;
    std::deque<double> queue;
    int64_t iter = 0;
    double dev = 0.0;
    do {
        launch_local_sweeps(m, h->local.p, h->localCount.p, h->ncol, cycle, h->acc.p, h->stream);
        CK(cudaMemcpyAsync(&h->pin->sums[2], h->acc.p, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
        rc = sync_status(h, "tg_local_relax");
        if (rc != TG_OK) break;
        dev = h->pin->sums[2];
        queue.push_back(dev);
        while ((int)queue.size() > queueSize) queue.pop_front();
        if (stagnated(queue, (unsigned)queueSize, (unsigned)cycle)) {
            rc = fail(h, TG_ERR_RELAX_FAULT, "tg_local_relax: stagnation");
            break;
        }
        iter += cycle;
        if (iter > 1000000) {
            rc = fail(h, TG_ERR_ITERATION_CAP, "tg_local_relax: sweep cap reached");
            break;
        }
    } while (dev > threshold);
    if (iterations) *iterations = iter;
    if (deviation) *deviation = dev;
    h->selValid = false;
    return rc;
}

int tg_residual(tg_handle* h, double* rel) {
    DeviceScope dev_scope(h);
    if (!h || !rel) return fail(h, TG_ERR_ARGUMENT, "tg_residual: null argument");
    // ||b||^2 comes with the residual's pass when it is not known
    DevMesh m = h->dm();
    double* bacc = h->bnormValid ? nullptr : h->acc.p + 1;
    CK(cudaMemsetAsync(h->acc.p, 0, 2 * sizeof(double), h->stream));
    launch_residual(m, h->allV.p, h->countAllV, nullptr, h->acc.p, h->stream, bacc);
    launch_residual(m, h->allN.p, h->countAllN, nullptr, h->acc.p, h->stream, bacc);
    CK(cudaMemcpyAsync(h->pin->sums + 2, h->acc.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    const int rc = sync_status(h, "tg_residual");
    if (rc != TG_OK) return rc;
    const double r2 = h->pin->sums[2];
    if (bacc) {
        h->bnorm2 = h->pin->sums[3];
        h->bnormValid = true;
    }
    *rel = h->bnorm2 > 0.0 ? std::sqrt(r2 / h->bnorm2) : std::sqrt(r2);
    return rc;
}

// FP32 conjugate gradients on one row list until r.z falls below
// rtol^2 of its start value or maxIter is reached; returns iterations.
// absTarget2: a floor under the target of r.r (0: none), for a system whose
// part of the global residual only has to fall below a share of the outer
// tolerance
}  // extern "C"

// Every pointer, size and schedule that the replayed iteration's kernels
// take as parameters, field by field.
static std::vector<uint64_t> iteration_key(const VSys& v, const AmgDev& g, int slots) {
    std::vector<uint64_t> k;
    auto p = [&](const void* q) { k.push_back((uint64_t)(uintptr_t)q); };
    auto i = [&](long long x) { k.push_back((uint64_t)x); };
    p(v.slot_of); p(v.node_of); p(v.slice_start); p(v.slice_width); p(v.col); p(v.val); p(v.val16); p(v.g);
    p(v.vpos); p(v.d); p(v.x); p(v.r); p(v.u); p(v.w); p(v.p); p(v.sv); p(v.hist); p(v.scal); p(v.count);
    p(v.iter); p(v.rel2); i(v.capacity); i(slots);
    i(g.levels); p(g.y0); p(g.t0); p(g.coarse_inv); i(g.fine_unroll);
    for (int l = 0; l < g.levels && l < kAmgMaxLevels; l++) {
        const AmgDevLevel& L = g.lev[l];
        i(L.n); i(L.a_lanes); i(L.r_lanes);
        p(L.a_ptr); p(L.a_col); p(L.a_val); p(L.diag); p(L.p_ptr); p(L.p_col); p(L.p_val);
        p(L.r_ptr); p(L.r_col); p(L.r_val); p(L.b); p(L.y); p(L.x); p(L.t);
    }
    return k;
}

// Captures body(stream) into *exec (replacing the one there) on the
// handle's capture stream; *nodes gets the kernels it launched.
template <class F>
static cudaError_t capture_graph(tg_handle* h, F body, cudaGraphExec_t* exec, long long* nodes) {
    if (*exec) {
        cudaError_t e = cudaGraphExecDestroy(*exec);
        *exec = nullptr;
        if (e != cudaSuccess) return e;
    }
    if (!h->captureStream) {
        cudaError_t e = cudaStreamCreateWithFlags(&h->captureStream, cudaStreamNonBlocking);
        if (e != cudaSuccess) return e;
    }
    long long count = 0;
    t_captured = &count;
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(h->captureStream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        body(h->captureStream);
        e = cudaStreamEndCapture(h->captureStream, &graph);
    }
    t_captured = nullptr;
    if (e == cudaSuccess) e = cudaGraphInstantiate(exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (e != cudaSuccess) *exec = nullptr;
    *nodes = count;
    return e;
}

// The replayed CG iteration of the multigrid solve for the V system as it
// is now: captured anew when its device state or its slots in use changed
// (removals append rows, a new slice of 32 every 32 rows); vg: the VSys
// whose kernels read the iteration index and target on the device.
static int iteration_graph(tg_handle* h, const VSys& vg) {
    std::vector<uint64_t> key = iteration_key(vg, h->amg, h->vActive);
    if (h->iterExec && key == h->iterKey) return TG_OK;
    const int slots = h->vActive;
    const cudaError_t e = capture_graph(
        h,
        [&](cudaStream_t cs) {
            launch_vcg_update(vg, slots, 0, -1.0, false, cs, h->amg.y0);
            launch_amg_vcycle(vg, slots, h->amg, 1, -1.0, cs, true);
            launch_vcg_spmv(vg, slots, 1, -1.0, true, cs);
            launch_vcg_replay_step(h->iterDev.p, cs);
        },
        &h->iterExec, &h->iterNodes);
    if (e != cudaSuccess) return cuda_check(h, e, "tg_solve: CG iteration graph");
    h->iterKey.swap(key);
    return TG_OK;
}

// Launch mode 2: the whole inner solve as one graph, its start (init, V-cycle,
// SpMV) and then the replayed iteration inside a while-conditional node.  The
// loop's body is the iteration (update, V-cycle, SpMV) and k_vcg_loop_cond,
// which steps the device counter and sets the node's condition from it and
// rho; the counter steps once per body, so the loop ends by the iteration
// cap.  The kernels are chained (launch_chain): on a 307k-cell tip an
// iteration is twelve kernels of a few us each, whose starts overlap the ends
// of the ones before.  v: the VSys of the start (no counter); vg: the loop's.
// slots: those in use, rounded up to kGraphSlots (the slots beyond hold
// nothing, and their rows only zeros), so that removals seldom make it be
// captured anew, which takes about 1.2 ms.
constexpr int kGraphSlots = 1024;
static int iteration_loop_graph(tg_handle* h, const VSys& v, const VSys& vg) {
    const int slots = std::min(h->vCapacity, (h->vActive + kGraphSlots - 1) / kGraphSlots * kGraphSlots);
    std::vector<uint64_t> key = iteration_key(vg, h->amg, slots);
    key.push_back((uint64_t)(uintptr_t)h->loopDone.p);
    if (h->loopExec && key == h->loopKey) return TG_OK;
    if (h->loopExec) {
        CK(cudaGraphExecDestroy(h->loopExec));
        h->loopExec = nullptr;
    }
    if (!h->captureStream) CK(cudaStreamCreateWithFlags(&h->captureStream, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    long long nodes = 0;
    ChainScope chained;
    t_captured = &nodes;
    cudaError_t e = cudaStreamBeginCapture(h->captureStream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        cudaStream_t cs = h->captureStream;
        launch_vcg_init(v, slots, false, cs, h->amg.y0);
        launch_amg_vcycle(v, slots, h->amg, 0, -1.0, cs, true);
        launch_vcg_spmv(v, slots, 0, -1.0, true, cs);
        e = cudaStreamEndCapture(cs, &graph);
    }
    t_captured = nullptr;
    h->loopStartNodes = nodes;  // kernels of the solve's start
    nodes = 0;
    // the loop follows the start's last kernel
    cudaGraphNode_t last = nullptr;
    if (e == cudaSuccess) {
        size_t count = 0;
        e = cudaGraphGetNodes(graph, nullptr, &count);
        std::vector<cudaGraphNode_t> all(count);
        if (e == cudaSuccess) e = cudaGraphGetNodes(graph, all.data(), &count);
        for (size_t k = 0; e == cudaSuccess && k < count; k++) {
            size_t followers = 0;
            e = cudaGraphNodeGetDependentNodes_v2(all[k], nullptr, nullptr, &followers);
            if (followers == 0) last = all[k];
        }
    }
    cudaGraphConditionalHandle loop{};
    if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&loop, graph, 1, cudaGraphCondAssignDefault);
    cudaGraphNodeParams params{};
    cudaGraphNode_t node = nullptr;
    if (e == cudaSuccess) {
        params.type = cudaGraphNodeTypeConditional;
        params.conditional.handle = loop;
        params.conditional.type = cudaGraphCondTypeWhile;
        params.conditional.size = 1;
        e = cudaGraphAddNode(&node, graph, &last, 1, &params);
    }
    if (e == cudaSuccess) {
        cudaGraph_t body = params.conditional.phGraph_out[0];
        t_captured = &nodes;
        e = cudaStreamBeginCaptureToGraph(h->captureStream, body, nullptr, nullptr, 0,
                                          cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            cudaStream_t cs = h->captureStream;
            launch_vcg_update(vg, slots, 0, -1.0, false, cs, h->amg.y0);
            launch_amg_vcycle(vg, slots, h->amg, 1, -1.0, cs, true);
            launch_vcg_spmv(vg, slots, 1, -1.0, true, cs);
            launch_vcg_loop_cond(loop, h->iterDev.p, vg.scal, h->rel2Dev.p, h->loopDone.p, cs);  // steps the counter
            cudaGraph_t captured = nullptr;
            e = cudaStreamEndCapture(cs, &captured);
        }
        t_captured = nullptr;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&h->loopExec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
        h->loopExec = nullptr;
        return cuda_check(h, e, "tg_solve: CG iteration loop graph");
    }
    h->loopNodes = nodes;  // kernels per iteration of the loop
    h->loopKey.swap(key);
    return TG_OK;
}

// The replayed iteration of the node-space CG on the Neumann rows, captured
// anew when its rows or vectors changed.
static int cg_iteration_graph(tg_handle* h, const DevMesh& m, const int32_t* rows, int count,
                              const CGVectors& vg) {
    std::vector<uint64_t> key;
    for (const void* q : {(const void*)m.row_ptr, (const void*)m.col, (const void*)m.ceff32, (const void*)m.diag32,
                          (const void*)rows, (const void*)vg.x, (const void*)vg.r, (const void*)vg.z,
                          (const void*)vg.p, (const void*)vg.ap, (const void*)vg.scal, (const void*)vg.iter,
                          (const void*)vg.tgt})
        key.push_back((uint64_t)(uintptr_t)q);
    key.push_back((uint64_t)count);
    if (h->cgExec && key == h->cgKey) return TG_OK;
    const cudaError_t e = capture_graph(
        h,
        [&](cudaStream_t cs) {
            launch_cg_iter(m, rows, count, vg, 0, -1.0, -1.0, cs);
            launch_cg_replay_step(h->cgIterDev.p, cs);
        },
        &h->cgExec, &h->cgNodes);
    if (e != cudaSuccess) return cuda_check(h, e, "tg_solve: node-space CG iteration graph");
    h->cgKey.swap(key);
    return TG_OK;
}

extern "C" {

static int run_cg(tg_handle* h, const int32_t* rows, int count, double rtol, int maxIter, int* itersOut,
                  double absTarget2 = 0.0) {
    DevMesh m = h->dm();
    CGVectors v = h->cg();
    DBuf<double>& scal = h->scalN;
    const size_t need = 3 * (size_t)(maxIter + 2);
    if (scal.n < need) {
        CK(scal.alloc(need));
        v = h->cg();
    }
    CK(cudaMemsetAsync(scal.p, 0, sizeof(double) * need, h->stream));
    launch_cg_init(m, rows, count, v, h->stream);
    // stop on the 2-norm of the residual (r.r at scal[3it+2]), the norm the
    // outer FP64 test uses: r.r <= max(rtol^2 r.r_0, absTarget2), tested by
    // the kernels themselves, so the iterations queue before r.r_0 is read
    const double rel2 = rtol * rtol;
    // the iterations replay one captured iteration
    const bool replay = h->launchMode >= 1 && count > 0;
    if (replay) {
        if (!h->cgIterDev.p) CK(h->cgIterDev.alloc(1));
        if (!h->cgTgtDev.p) CK(h->cgTgtDev.alloc(2));
        CGVectors vg = v;
        vg.iter = h->cgIterDev.p;
        vg.tgt = h->cgTgtDev.p;
        const int rc = cg_iteration_graph(h, m, rows, count, vg);
        if (rc != TG_OK) return rc;
        launch_cg_replay_begin(h->cgIterDev.p, h->cgTgtDev.p, rel2, absTarget2, h->stream);
    }
    int it = 0;
    // iterations queued before the first read: one more than the last solve
    // of this system took, then small batches
    int& last = h->lastItersCg;
    int batch = std::min(16, std::max(2, last + 1));
    double sb[3 * 16], s0[3];
    while (it < maxIter) {
        const int start = it;
        const int end = std::min(maxIter, it + batch);
        for (; it < end; it++) {
            if (replay) {
                CK(cudaGraphLaunch(h->cgExec, h->stream));
                g_launches.fetch_add(h->cgNodes, std::memory_order_relaxed);
                continue;
            }
            launch_cg_iter(m, rows, count, v, it, rel2, absTarget2, h->stream);
        }
        // r.r after j iterations sits at scal[3j+2]; the kernels of later
        // iterations of the batch returned early once it met the target
        CK(cudaMemcpyAsync(s0, scal.p, sizeof(double) * 3, cudaMemcpyDeviceToHost, h->stream));
        CK(cudaMemcpyAsync(sb, scal.p + 3 * (size_t)(start + 1), sizeof(double) * 3 * (end - start),
                           cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
        const double target = std::max(s0[2] * rel2, absTarget2);
        if (!(s0[2] > target)) {
            // nothing to do: every queued iteration returned at once
            it = 0;
            break;
        }
        bool done = false;
        for (int j = start + 1; j <= end && !done; j++)
            if (sb[3 * (j - start - 1) + 2] <= target) {
                it = j;
                done = true;
            }
        if (done) break;
        batch = 4;
    }
    last = it;
    *itersOut = it;
    return TG_OK;
}

// Builds the multigrid hierarchy of the V system as it is now (its slots in
// use, their couplings and diagonals read back from the device) and
// uploads it.
static int amg_setup_impl(tg_handle* h, double* seconds) {
    const auto t0 = std::chrono::steady_clock::now();
    h->amg_release();
    const int slots = h->vActive;
    const int slices = (slots + 31) / 32;
    std::vector<int32_t> sliceStart(slices + 1), sliceWidth(slices);
    CK(cudaStreamSynchronize(h->stream));
    CK(cudaMemcpy(sliceStart.data(), h->vSliceStart.p, sizeof(int32_t) * (slices + 1), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(sliceWidth.data(), h->vSliceWidth.p, sizeof(int32_t) * slices, cudaMemcpyDeviceToHost));
    const size_t used = (size_t)sliceStart[slices];
    std::vector<int32_t> col(used);
    std::vector<float> val(used), d(slots);
    CK(cudaMemcpy(col.data(), h->vCol.p, sizeof(int32_t) * used, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(val.data(), h->vVal.p, sizeof(float) * used, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(d.data(), h->vs().d, sizeof(float) * slots, cudaMemcpyDeviceToHost));
    // A = D - C in CSR, slot order
    tg_host::AmgCsr A;
    A.rows = A.cols = slots;
    A.ptr.reserve(slots + 1);
    A.col.reserve(used + slots);
    A.val.reserve(used + slots);
    A.ptr.push_back(0);
    for (int s = 0; s < slots; s++) {
        const int base = sliceStart[s / 32] + (s & 31), width = sliceWidth[s / 32];
        A.col.push_back(s);
        A.val.push_back(d[s]);
        for (int k = 0; k < width; k++) {
            const int c = col[base + 32 * (size_t)k];
            const float a = val[base + 32 * (size_t)k];
            if (c >= slots || a == 0.0f) continue;
            A.col.push_back(c);
            A.val.push_back(-(double)a);
        }
        A.ptr.push_back((int32_t)A.col.size());
    }
    tg_host::AmgHierarchy H;
    const std::string err = tg_host::amg_build(std::move(A), tg_host::AmgOptions(), &H);
    if (!err.empty()) return fail(h, TG_ERR_HOST, "tg_solve: " + err);
    if ((int)H.levels.size() > tgd::kAmgMaxLevels) return fail(h, TG_ERR_HOST, "tg_solve: too many multigrid levels");
    cudaError_t e = cudaSuccess;
    auto upI = [&](const std::vector<int32_t>& src) -> int32_t* {
        h->amgI.emplace_back();
        DBuf<int32_t>& b = h->amgI.back();
        if (e == cudaSuccess) e = b.alloc(std::max<size_t>(src.size(), 1));
        if (e == cudaSuccess && !src.empty())
            e = cudaMemcpy(b.p, src.data(), sizeof(int32_t) * src.size(), cudaMemcpyHostToDevice);
        return b.p;
    };
    auto upF = [&](const std::vector<double>& src) -> float* {
        std::vector<float> f(src.begin(), src.end());
        h->amgF.emplace_back();
        DBuf<float>& b = h->amgF.back();
        if (e == cudaSuccess) e = b.alloc(std::max<size_t>(f.size(), 1));
        if (e == cudaSuccess && !f.empty()) e = cudaMemcpy(b.p, f.data(), sizeof(float) * f.size(), cudaMemcpyHostToDevice);
        return b.p;
    };
    auto vec = [&](size_t n) -> float* {
        h->amgF.emplace_back();
        DBuf<float>& b = h->amgF.back();
        if (e == cudaSuccess) e = b.alloc(std::max<size_t>(n, 1));
        if (e == cudaSuccess) e = cudaMemset(b.p, 0, sizeof(float) * std::max<size_t>(n, 1));
        return b.p;
    };
    // the DBuf vectors must not reallocate while pointers into them are live
    h->amgI.reserve(8 * H.levels.size() + 4);
    h->amgF.reserve(8 * H.levels.size() + 4);
    // Lanes per CSR row, by a rule on the hierarchy alone: a row's sum is
    // formed in another order with other lanes, so lanes picked by their times
    // gave one specimen several sets of last digits, which a flight's last
    // point turns into 1e-3 of a voltage.  The power of two nearest a quarter
    // of the mean row length takes a row in about one round of loads (four per
    // lane); where the launch is bound by its rounds and not by its bytes, a
    // row is taken in one round: the restriction of the V rows up to 11,000
    // rows, and, under V systems whose passes leave little of them in L2, the
    // level-1 operator and deeper ones up to 7,000 rows.  These are the lanes
    // that timed trials of the V-cycle picked most often on 76 specimens of
    // 23k to 835k cells, ten times or more each (per matrix on 67% to 89% of
    // the grids); on the 7.3M-cell one they are what the trials picked.
    auto lanes = [](const tg_host::AmgCsr& M, bool oneRound) {
        const double per = M.rows > 0 ? (double)M.val.size() / M.rows / 4.0 : 1.0;
        int L = 2;
        while (L < 32 && per > L * (oneRound ? 1.0 : 1.4142135623730951)) L *= 2;
        return L;
    };
    constexpr int kRoundRowsR = 11000, kRoundRowsA = 7000, kRoundSlots = 25000;
    tgd::AmgDev g{};
    g.levels = (int)H.levels.size();
    for (int l = 0; l < g.levels; l++) {
        const tg_host::AmgLevel& L = H.levels[l];
        tgd::AmgDevLevel& D = g.lev[l];
        D.n = L.A.rows;
        if (l > 0) {
            D.a_ptr = upI(L.A.ptr);
            D.a_col = upI(L.A.col);
            D.a_val = upF(L.A.val);
            D.a_lanes = lanes(L.A, slots > kRoundSlots && (l == 1 || L.A.rows <= kRoundRowsA));
            std::vector<double> diag(L.A.rows, 1.0);
            for (int i = 0; i < L.A.rows; i++)
                for (int q = L.A.ptr[i]; q < L.A.ptr[i + 1]; q++)
                    if (L.A.col[q] == i && L.A.val[q] > 0.0) diag[i] = L.A.val[q];
            D.diag = upF(diag);
            D.b = vec(D.n);
            D.y = vec(D.n);
            D.x = vec(D.n);
            D.t = vec(D.n);
        }
        if (l + 1 < g.levels) {
            D.p_ptr = upI(L.P.ptr);
            D.p_col = upI(L.P.col);
            D.p_val = upF(L.P.val);
            D.r_ptr = upI(L.R.ptr);
            D.r_col = upI(L.R.col);
            D.r_val = upF(L.R.val);
            D.r_lanes = lanes(L.R, l == 0 && L.R.rows <= kRoundRowsR);
        }
    }
    g.y0 = vec((size_t)h->vCapacity + 1);
    g.t0 = vec((size_t)h->vCapacity + 1);
    g.coarse_inv = upF(H.coarse_inv);
    if (e != cudaSuccess) {
        h->amg_release();
        return cuda_check(h, e, "multigrid upload");
    }
    // the level-0 pass's load depth, which changes no sum, from timed trials
    for (int l = 0; l < tgd::kAmgMaxLevels; l++) h->amgTunedA[l] = h->amgTunedR[l] = 0.0f;
    g.fine_unroll = 8;
    if (amg_tune(g, h->vs(), slots, h->stream, h->amgTunedA, h->amgTunedR, &h->amgTunedFine) != 0) {
        h->amg_release();
        return cuda_check(h, cudaGetLastError(), "multigrid schedule tuning");
    }
    h->amg = g;
    h->amgReady = true;
    h->amgSlots = slots;
    *seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return TG_OK;
}

// the hierarchy build allocates on the host: no exception crosses the C ABI
static int amg_setup(tg_handle* h, double* seconds) {
    try {
        return amg_setup_impl(h, seconds);
    } catch (const std::exception& e) {
        h->amg_release();
        return fail(h, TG_ERR_HOST, std::string("tg_solve: multigrid setup: ") + e.what());
    }
}

// Single-reduction PCG on the V system until rho = r.r falls below rtol^2
// of its start value or maxIter is reached.  r (slot order) must hold
// the right-hand side; x receives the correction.  amg: the multigrid
// V-cycle as the preconditioner instead of the diagonal.
// fp64: the FP64 iterations (multigrid only), their right-hand side taken
// from the kept FP64 residuals by node.
static int run_vcg(tg_handle* h, double rtol, int maxIter, bool amg, int* itersOut, bool fp64 = false) {
    // the looped solve's body runs once before its cap is tested, and clears
    // the accumulators of the iteration after it
    const size_t need = 4 * (size_t)(std::max(maxIter, 1) + 2);
    if (h->vScal.n < need) CK(h->vScal.alloc(need));
    VSys v = h->vs();
    const int slots = h->vActive;
    const double rel2 = rtol * rtol;
    if (amg && !fp64 && h->launchMode == 2 && slots > 0) {
        if (!h->iterDev.p) CK(h->iterDev.alloc(1));
        if (!h->rel2Dev.p) CK(h->rel2Dev.alloc(2));
        if (!h->loopDone.p) CK(h->loopDone.alloc(1));
        VSys vg = v;
        vg.iter = h->iterDev.p;
        vg.rel2 = h->rel2Dev.p;
        const int rc = iteration_loop_graph(h, v, vg);
        if (rc != TG_OK) return rc;
        launch_vcg_replay_begin(h->iterDev.p, h->rel2Dev.p, rel2, maxIter, h->stream, h->vScal.p);
        // the whole solve in one launch: the loop stops itself
        CK(cudaGraphLaunch(h->loopExec, h->stream));
        g_launches.fetch_add(h->loopStartNodes, std::memory_order_relaxed);
        CK(cudaMemcpyAsync(&h->pin->loopIters[0], h->loopDone.p, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
        *itersOut = -1;  // pending: pin->loopIters[0] after the next sync
        return TG_OK;
    }
    CK(cudaMemsetAsync(h->vScal.p, 0, sizeof(double) * need, h->stream));
    if (fp64) {
        launch_vcg64_init(v, slots, h->resid.p, h->stream);
        launch_amg_vcycle(v, slots, h->amg, 0, -1.0, h->stream);
        launch_vcg64_spmv(v, slots, 0, -1.0, h->stream);
    } else {
        launch_vcg_init(v, slots, !amg, h->stream, amg ? h->amg.y0 : nullptr);
        if (amg) launch_amg_vcycle(v, slots, h->amg, 0, -1.0, h->stream, true);
        launch_vcg_spmv(v, slots, 0, -1.0, amg, h->stream);
    }
    // stop on the 2-norm of the residual (rho = r.r), the norm the outer
    // FP64 test uses: rho_it <= rtol^2 rho_0, tested by the kernels
    // themselves, so the iterations queue before rho_0 is read back
    // the multigrid FP32 iterations replay one captured iteration
    const bool replay = amg && !fp64 && h->launchMode >= 1 && slots > 0;
    if (replay) {
        if (!h->iterDev.p) CK(h->iterDev.alloc(1));
        if (!h->rel2Dev.p) CK(h->rel2Dev.alloc(2));
        VSys vg = v;
        vg.iter = h->iterDev.p;
        vg.rel2 = h->rel2Dev.p;
        const int rc = iteration_graph(h, vg);
        if (rc != TG_OK) return rc;
        launch_vcg_replay_begin(h->iterDev.p, h->rel2Dev.p, rel2, maxIter, h->stream);
    }
    int it = 0;
    // iterations queued before the first read: about as many as the last
    // solve took; then small batches
    int& last = amg ? h->lastItersAmg : h->lastItersJacobi;
    int batch = std::min(16, std::max(amg ? 2 : 8, last - (amg ? 1 : 4)));
    double* sb = h->pin->sb;  // scal[0..3], then the batch's iterations
    while (it < maxIter) {
        const int start = it;
        const int end = std::min(maxIter, it + batch);
        for (; it < end; it++) {
            if (fp64) {
                launch_vcg64_update(v, slots, it, rel2, h->stream);
                launch_amg_vcycle(v, slots, h->amg, it + 1, rel2, h->stream);
                launch_vcg64_spmv(v, slots, it + 1, rel2, h->stream);
                continue;
            }
            if (replay) {
                CK(cudaGraphLaunch(h->iterExec, h->stream));
                g_launches.fetch_add(h->iterNodes, std::memory_order_relaxed);
                continue;
            }
            launch_vcg_update(v, slots, it, rel2, !amg, h->stream, amg ? h->amg.y0 : nullptr);
            if (amg) launch_amg_vcycle(v, slots, h->amg, it + 1, rel2, h->stream, true);
            launch_vcg_spmv(v, slots, it + 1, rel2, amg, h->stream);
        }
        // rho after j iterations sits at scal[4j+3]; the kernels of later
        // iterations of the batch returned early once it met the target
        CK(cudaMemcpyAsync(sb, h->vScal.p, sizeof(double) * 4, cudaMemcpyDeviceToHost, h->stream));
        CK(cudaMemcpyAsync(sb + 4, h->vScal.p + 4 * (size_t)(start + 1), sizeof(double) * 4 * (end - start),
                           cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
        const double rho0 = sb[3];
        if (!(rho0 > 0.0)) {
            it = 0;
            break;
        }
        bool done = false;
        for (int j = start + 1; j <= end && !done; j++)
            if (sb[4 + 4 * (j - start - 1) + 3] <= rel2 * rho0) {
                it = j;
                done = true;
            }
        if (done) break;
        batch = amg ? 2 : 4;
    }
    last = it;
    *itersOut = it;
    return TG_OK;
}

int tg_solve(tg_handle* h, const tg_solve_opts* o, tg_solve_info* info) {
    DeviceScope dev_scope(h);
    if (!h || !o) return fail(h, TG_ERR_ARGUMENT, "tg_solve: null argument");
    if (o->max_inner < 0) return fail(h, TG_ERR_ARGUMENT, "tg_solve: max_inner below 0");
    if (o->inner_precision < 0 || o->inner_precision > 1)
        return fail(h, TG_ERR_ARGUMENT, "tg_solve: inner_precision 0 (FP32) or 1 (FP64)");
    if (o->inner_precision == 1 && (o->preconditioner != 1 || o->warm_start != 0))
        return fail(h, TG_ERR_ARGUMENT, "tg_solve: FP64 inner iterations take the multigrid preconditioner and a plain start");
    int rc = TG_OK;
    DevMesh m = h->dm();
    // ||b||^2 comes with the first residual of every solve (from a full pass
    // or from the kept values) and holds until the next removal
    bool needB = !h->bnormValid;
    VSys vsys = h->vs();
    CGVectors vN = h->cg();
    tg_solve_info inf{};
    double rel = 0.0;
    // a solve right after removals from a converged state records its
    // correction; with warm_start it starts from the previous one
    const bool fromEvent = h->converged && h->removalsSinceSolve > 0;
    const bool warm = fromEvent && h->histValid && (o->warm_start == 1 || o->warm_start == 2);
    const bool learnPredict = fromEvent && h->learner && (h->learnMode & 2) && o->warm_start == 2 && h->lastSite >= 0;
    // the first residual after removals from a converged state: the rows the
    // removals touched, from the kept residuals of the potentials as they
    // are; a recycled start then takes A hist off the V rows (FP32) and the
    // Neumann rows are recomputed.  The learned start then changes the
    // potentials of its graph's cells: their rows and their neighbours' are
    // recomputed in FP64 after the prediction, and the sums formed again.
    const bool incremental = h->residValid && fromEvent && !h->pendingOverflow && h->nPending > 0;
    const int nPending = h->nPending;
    h->residValid = h->pendingOverflow = false;
    h->nPending = 0;
    double* rv = h->resid.p;
    double* bv = h->resid.p + h->n;
    if (incremental) {
        CK(cudaMemcpyAsync(h->pendingDev.p, h->pin->pending, sizeof(int32_t) * nPending, cudaMemcpyHostToDevice,
                           h->stream));
        if (++h->resEpoch == INT32_MAX) {
            CK(cudaMemsetAsync(h->resStamp.p, 0, sizeof(int32_t) * (size_t)h->n, h->stream));
            h->resEpoch = 1;
        }
        launch_residual_rows(m, vsys, vN.r, h->pendingDev.p, nPending, h->resStamp.p, h->resEpoch, rv, bv, h->rsum.p,
                             h->stream);
        inf.residual_cells = nPending;
    }
    if (warm) launch_vcg_warm(m, vsys, h->vActive, 1.0f, h->stream);
    else if (fromEvent) CK(cudaMemsetAsync(vsys.hist, 0, sizeof(float) * ((size_t)h->vCapacity + 1), h->stream));
    // learned near field on top of the recycled far field (or the plain start
    // while there is no history); sample collection.  With a recycled start,
    // its FP32 first residual (r -= A hist) is taken before the prediction,
    // so that the predicted cells' rows can then be recomputed in FP64.
    const bool learnCollect = fromEvent && h->learner && (h->learnMode & 1) && h->lastSite >= 0;
    const bool warmFirst = learnPredict && incremental && warm;
    if (warmFirst) {
        CK(cudaMemsetAsync(h->rsum.p, 0, 2 * sizeof(double), h->stream));
        launch_vcg_warm_residual(vsys, h->vActive, h->rsum.p, h->stream);
    }
    if (learnPredict || learnCollect) {
        rc = learner_predict(h->learner, m, h->lastSite, h->stream, learnCollect, learnPredict, vsys.slot_of,
                             fromEvent ? vsys.hist : nullptr);
        if (rc != TG_OK) return fail(h, rc, std::string("tg_solve: ") + tg_learner_last_error(h->learner));
        if (learnPredict && incremental) {
            // the predicted cells' rows and their neighbours' from the new
            // potentials, with a fresh stamp (the removals' pass above may
            // have taken some of these rows before the prediction)
            const int32_t *cells = nullptr, *cellCount = nullptr;
            int cap = 0;
            learner_graph_cells(h->learner, &cells, &cellCount, &cap);
            if (++h->resEpoch == INT32_MAX) {
                CK(cudaMemsetAsync(h->resStamp.p, 0, sizeof(int32_t) * (size_t)h->n, h->stream));
                h->resEpoch = 1;
            }
            launch_residual_rows(m, vsys, vN.r, cells, cap, h->resStamp.p, h->resEpoch, rv, bv, h->rsum.p, h->stream,
                                 cellCount);
            if (warmFirst) {
                // the V rows' sum of squares from their FP32 residuals as
                // they now are, and the Neumann rows in full
                CK(cudaMemsetAsync(h->rsum.p, 0, 2 * sizeof(double), h->stream));
                launch_vcg_rnorm(vsys, h->vActive, h->rsum.p, h->stream);
                launch_residual(m, h->allN.p, h->countAllN, vN.r, h->rsum.p + 1, h->stream, nullptr, rv, nullptr);
            }
        }
    }
    h->converged = h->histValid = false;
    h->removalsSinceSolve = 0;
    const bool amg = o->preconditioner == 1;
    if (o->preconditioner < 0 || o->preconditioner > 1)
        return fail(h, TG_ERR_ARGUMENT, "tg_solve: preconditioner 0 (Jacobi) or 1 (multigrid)");
    const bool fp64 = o->inner_precision == 1;
    if (fp64 && h->vActive > 0 && !h->vVec64.p) {
        // first FP64 solve: the FP64 copies of the V system's couplings and
        // diagonals, kept in step by every later write of the FP32 ones
        const size_t stored = h->vVal.n, stride = (size_t)h->vCapacity + 1;
        cudaError_t e = h->vVal64.alloc(stored);
        if (e == cudaSuccess) e = h->vVec64.alloc(6 * stride);
        if (e == cudaSuccess) e = cudaMemsetAsync(h->vVal64.p, 0, sizeof(double) * stored, h->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(h->vVec64.p, 0, sizeof(double) * 6 * stride, h->stream);
        if (e != cudaSuccess) {
            h->vVal64.release();
            h->vVec64.release();
            return cuda_check(h, e, "tg_solve: FP64 inner system");
        }
        vsys = h->vs();
        launch_vcg64_derive(m, vsys, h->nnz, h->stream);
    }
    // (re)build the hierarchy when there is none or removals have grown the
    // system by 2% since
    if (amg && (!h->amgReady || h->vActive > h->amgSlots + h->amgSlots / 50)) {
        rc = amg_setup(h, &inf.setup_seconds);
        if (rc != TG_OK) return rc;
    }
    // looped and one-launch inner solves whose counts are still on their way
    bool loopPending = false, cgPending = false;
    for (int outer = 0;; outer++) {
        if (outer == 0 && incremental) {
            if (warm && !warmFirst) {
                CK(cudaMemsetAsync(h->rsum.p, 0, 2 * sizeof(double), h->stream));
                launch_vcg_warm_residual(vsys, h->vActive, h->rsum.p, h->stream);
                launch_residual(m, h->allN.p, h->countAllN, vN.r, h->rsum.p + 1, h->stream, nullptr, rv, nullptr);
            }
            needB = true;
        } else {
            // a full pass; the first one also takes the Dirichlet parts, so
            // that the kept values describe the rows as they are
            if (outer == 0) needB = true;
            CK(cudaMemsetAsync(h->rsum.p, 0, (needB ? 3 : 2) * sizeof(double), h->stream));
            launch_vcg_residual(m, vsys, h->allV.p, h->countAllV, h->rsum.p, needB ? h->rsum.p + 2 : nullptr,
                                h->stream, rv, bv);
            launch_residual(m, h->allN.p, h->countAllN, vN.r, h->rsum.p + 1, h->stream,
                            needB ? h->rsum.p + 2 : nullptr, rv, bv);
        }
        double* r2 = h->pin->r2;
        CK(cudaMemcpyAsync(r2, h->rsum.p, sizeof(double) * (needB ? 3 : 2), cudaMemcpyDeviceToHost, h->stream));
        rc = sync_status(h, "tg_solve residual");
        if (rc != TG_OK) return rc;
        if (loopPending) {
            // the looped inner solve's iterations came back with this read
            const int k = h->pin->loopIters[0];
            inf.inner += k;
            g_launches.fetch_add(h->loopNodes * k, std::memory_order_relaxed);
            h->lastItersAmg = k;
            loopPending = false;
        }
        if (cgPending) {
            const int k = h->pin->loopIters[1];
            inf.inner += k;
            inf.inner_neumann += k;
            cgPending = false;
        }
        // sums kept across removals can round to a little below zero
        r2[0] = std::max(r2[0], 0.0);
        r2[1] = std::max(r2[1], 0.0);
        if (needB) {
            h->bnorm2 = std::max(r2[2], 0.0);
            h->bnormValid = true;
            needB = false;
        }
        rel = h->bnorm2 > 0.0 ? std::sqrt((r2[0] + r2[1]) / h->bnorm2) : std::sqrt(r2[0] + r2[1]);
        if (outer == 0) inf.initial_rel_residual = rel;
        inf.outer = outer;
        inf.rel_residual = rel;
        // the first residual of a warm start taken from the kept values holds
        // A hist in FP32 only: it is not the FP64 test and never ends the
        // solve (the kept V-row values are also those before the start)
        if (rel <= o->rel_tol && !(outer == 0 && incremental && warm)) break;
        if (outer >= o->max_outer) {
            if (info) *info = inf;
            if (learnCollect) learner_collect_cancel(h->learner);
            return fail(h, TG_ERR_ITERATION_CAP, "tg_solve: outer iteration cap reached");
        }
        // inner reduction just sufficient for this step (not below the
        // configured one, which bounds the FP32 work of the first step)
        const double rtol = std::min(0.5, std::max(o->inner_rtol, 0.3 * o->rel_tol / rel));
        int itV = 0, itN = 0;
        if (h->vActive > 0 && r2[0] > 0.0) {
            rc = run_vcg(h, rtol, o->max_inner, amg, &itV, fp64);
            if (rc != TG_OK) return rc;
        }
        if (h->countAllN > 0) {
            // the Neumann rows' share of the global residual only has to fall
            // below 0.3 of the outer tolerance (the V rows' solve brings
            // theirs to about the same), whatever their own start
            const double floorN = 0.3 * o->rel_tol;
            const double floor2 = floorN * floorN * h->bnorm2;
            // one launch up to kCgSolveRows rows; beyond, a grid of them (a
            // cluster's eight SMs would be the bound)
            cgPending = h->launchMode >= 1 && h->countAllN <= kCgSolveRows;
            if (cgPending) {
                if (!h->cgDone.p) CK(h->cgDone.alloc(1));
                CK(launch_cg_solve(m, h->allN.p, h->countAllN, vN, vsys, fp64, rtol * rtol, floor2, o->max_inner,
                                   h->cgDone.p, h->stream));
                CK(cudaMemcpyAsync(&h->pin->loopIters[1], h->cgDone.p, sizeof(int32_t), cudaMemcpyDeviceToHost,
                                   h->stream));
            } else {
                launch_vcg_couple_neumann(m, vsys, h->allN.p, h->countAllN, vN.r, h->stream, fp64);
                rc = run_cg(h, h->allN.p, h->countAllN, rtol, o->max_inner, &itN, floor2);
                if (rc != TG_OK) return rc;
            }
        }
        if (itV < 0) {
            loopPending = true;
            itV = 0;
        }
        inf.inner += itV + itN;
        inf.inner_neumann += itN;
        if (fp64) launch_vcg64_apply(m, vsys, h->vActive, fromEvent, h->stream);
        else launch_vcg_apply(m, vsys, h->vActive, fromEvent, h->stream);
        if (!cgPending) launch_apply_correction(m, h->allN.p, h->countAllN, vN, h->stream);
    }
    h->selValid = false;
    h->converged = true;
    h->histValid = fromEvent;
    h->residValid = true;
    if (learnCollect) {
        rc = learner_collect_end(h->learner, m, h->stream);
        if (rc != TG_OK) return fail(h, rc, std::string("tg_solve: ") + tg_learner_last_error(h->learner));
    }
    if (info) *info = inf;
    return TG_OK;
}

int tg_amg_schedule(tg_handle* h, int32_t level, int32_t* rows, int32_t* a_lanes, int32_t* r_lanes, float* a_ms,
                    float* r_ms) {
    DeviceScope dev_scope(h);
    if (!h) return fail(h, TG_ERR_ARGUMENT, "tg_amg_schedule: null handle");
    if (!h->amgReady || level < 0 || level >= h->amg.levels)
        return fail(h, TG_ERR_ARGUMENT, "tg_amg_schedule: no such multigrid level (built at the first multigrid solve)");
    const tgd::AmgDevLevel& L = h->amg.lev[level];
    if (rows) *rows = level == 0 ? h->amgSlots : L.n;
    const bool csr = level >= 1 && level + 1 < h->amg.levels;
    const bool restr = level + 1 < h->amg.levels;
    // level 0: the loads per lane of its smoothing pass in place of lanes
    if (a_lanes) *a_lanes = csr ? L.a_lanes : (level == 0 ? h->amg.fine_unroll : 0);
    if (r_lanes) *r_lanes = restr ? L.r_lanes : 0;
    if (a_ms) *a_ms = csr ? h->amgTunedA[level] : (level == 0 ? h->amgTunedFine : 0.0f);
    if (r_ms) *r_ms = restr ? h->amgTunedR[level] : 0.0f;
    return TG_OK;
}

int tg_learner_attach(tg_handle* h, tg_learner* L, int32_t mode) {
    DeviceScope dev_scope(h);
    if (!h || mode < 0 || mode > 3 || (mode && !L)) return fail(h, TG_ERR_ARGUMENT, "tg_learner_attach: bad argument");
    if (mode == 0) {
        h->learner = nullptr;
        h->learnMode = 0;
        return TG_OK;
    }
    if (learner_device(L) != h->device)
        return fail(h, TG_ERR_ARGUMENT, "tg_learner_attach: the learner and the grid live on different devices");
    int maxRow = 0;
    for (int i = 0; i < h->n; i++) maxRow = std::max(maxRow, h->h_row_ptr[i + 1] - h->h_row_ptr[i]);
    const int rc = learner_attach_mesh(L, (size_t)h->n, maxRow);
    if (rc != TG_OK) return fail(h, rc, std::string("tg_learner_attach: ") + tg_learner_last_error(L));
    h->learner = L;
    h->learnMode = mode;
    return TG_OK;
}

int tg_field_o1(tg_handle* h, int32_t count, const int32_t* nodes, double* out) {
    DeviceScope dev_scope(h);
    if (!h || count < 0 || (count && (!nodes || !out))) return fail(h, TG_ERR_ARGUMENT, "tg_field_o1: bad argument");
    if (count == 0) return TG_OK;
    for (int32_t k = 0; k < count; k++)
        if (nodes[k] < 0 || nodes[k] >= h->n) return fail(h, TG_ERR_ARGUMENT, "tg_field_o1: node index out of range");
    int rc = stage(h, h->stageI, count);
    if (rc == TG_OK) rc = stage(h, h->stageD, 3 * (size_t)count);
    if (rc != TG_OK) return rc;
    CK(cudaMemcpyAsync(h->stageI.p, nodes, sizeof(int32_t) * count, cudaMemcpyHostToDevice, h->stream));
    launch_field_o1(h->dm(), h->stageI.p, count, h->stageD.p, h->stream);
    CK(cudaMemcpyAsync(out, h->stageD.p, sizeof(double) * 3 * count, cudaMemcpyDeviceToHost, h->stream));
    return sync_status(h, "tg_field_o1");
}

int tg_surface_init(tg_handle* h, int32_t vacuumId, int32_t* num) {
    DeviceScope dev_scope(h);
    if (!h || vacuumId < 0 || vacuumId > 127 || h->types[vacuumId].id < 0)
        return fail(h, TG_ERR_ARGUMENT, "tg_surface_init: unknown vacuum id");
    h->vacuumId = vacuumId;
    CK(cudaMemsetAsync(h->surfCount.p, 0, sizeof(int32_t), h->stream));
    launch_surface_init(h->dm(), h->sf(), vacuumId, h->stream);
    int rc = refresh_counts(h);
    if (rc == TG_OK) rc = sync_status(h, "tg_surface_init");
    if (num) *num = h->surfSlots;
    h->selValid = false;
    return rc;
}

int tg_surface_select(tg_handle* h, tg_select_info* info) { return tg_surface_select_mode(h, 0, 0.0f, info); }

// The selection's kernels and the copy of its keys and sums into pinned
// memory, queued on the handle's stream; select_decode reads them once the
// stream has been synchronised.
static int select_launch(tg_handle* h, int32_t mode, float temperature) {
    if (h->vacuumId < 0) return fail(h, TG_ERR_ARGUMENT, "tg_surface_select: surface not initialised");
    if (mode < 0 || mode > 3) return fail(h, TG_ERR_ARGUMENT, "tg_surface_select: probability mode 0..3");
    if (mode == 1 && !(temperature > 0.0f))
        return fail(h, TG_ERR_ARGUMENT, "tg_surface_select: Boltzmann probabilities need a temperature > 0");
    // ratios, scores and keys, then the candidate and the runner-ups, all
    // decoded on the device; one read at the end
    CK(cudaMemsetAsync(h->keys.p, 0, 7 * sizeof(unsigned long long), h->stream));
    CK(cudaMemsetAsync(h->acc.p, 0, 2 * sizeof(double), h->stream));
    launch_surface_select(h->dm(), h->sf(), h->surfSlots, mode, temperature, h->keys.p, h->acc.p, h->stream);
    launch_surface_best(h->sf(), h->surfSlots, h->acc.p, h->keys.p, h->stream);
    launch_surface_second(h->sf(), h->surfSlots, h->acc.p, h->keys.p, h->stream);
    CK(cudaMemcpyAsync(h->pin->keys, h->keys.p, 7 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(h->pin->sums, h->acc.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    return TG_OK;
}

static int select_decode(tg_handle* h, int32_t mode, tg_select_info* info);

int tg_surface_select_mode(tg_handle* h, int32_t mode, float temperature, tg_select_info* info) {
    DeviceScope dev_scope(h);
    if (!h || !info) return fail(h, TG_ERR_ARGUMENT, "tg_surface_select: null argument");
    int rc = select_launch(h, mode, temperature);
    if (rc != TG_OK) return rc;
    rc = sync_status(h, "tg_surface_select");
    if (rc != TG_OK) return rc;
    return select_decode(h, mode, info);
}

// The candidate, the runner-ups, the apex and the sums of the selection
// select_launch queued, from pinned memory (the stream has been
// synchronised since); sets the handle's selection.
static int select_decode(tg_handle* h, int32_t mode, tg_select_info* info) {
    unsigned long long k[7];
    std::memcpy(k, h->pin->keys, sizeof(k));
    const double sums[2] = {h->pin->sums[0], h->pin->sums[1]};
    tg_select_info s{};
    s.prob_mode = mode;
    s.ratio_sum = sums[0];
    s.score_sum = sums[1];
    if (k[0] == 0ull) {
        s.candidate = -1;
        s.apex = -1;
        s.num_surface = 0;
        *info = s;
        h->sel = s;
        h->selValid = true;
        return fail(h, TG_ERR_NO_SURFACE, "tg_surface_select: empty surface");
    }
    auto unkey = [](unsigned long long key, float* v) {
        const uint32_t hi = (uint32_t)(key >> 32);
        const uint32_t u = (hi & 0x80000000u) ? (hi & 0x7fffffffu) : ~hi;
        std::memcpy(v, &u, 4);
        return (int32_t)(~(uint32_t)key);
    };
    float bestRatio, zmax;
    const int bestRatioNode = unkey(k[0], &bestRatio);
    s.apex = unkey(k[1], &zmax);
    s.best_ratio = bestRatio;
    (void)bestRatioNode;
    h->surfMinNode = (int32_t)(~(uint32_t)k[2]);
    h->surfMaxNode = (int32_t)k[3] - 1;
    // the probabilities are score / sum in float, as the reference normalises
    float bestP = 0.0f;
    s.candidate = unkey(k[4], &bestP);
    if ((uint32_t)(k[4] >> 32) == 0u) bestP = std::numeric_limits<float>::quiet_NaN();
    float secondP = 0.0f, secondRatio = 0.0f;
    if (k[5]) unkey(k[5], &secondP);
    if (k[6]) unkey(k[6], &secondRatio);
    s.second_ratio = secondRatio;
    s.best_probability = bestP;
    s.second_probability = secondP;
    s.probability = bestP;
    s.num_surface = h->surfSlots;
    *info = s;
    h->sel = s;
    h->selValid = true;
    return TG_OK;
}

int tg_surface_pick(tg_handle* h, double u, int32_t* node, float* probability) {
    DeviceScope dev_scope(h);
    if (!h || !node) return fail(h, TG_ERR_ARGUMENT, "tg_surface_pick: null argument");
    if (!h->selValid || h->sel.candidate < 0) return fail(h, TG_ERR_ARGUMENT, "tg_surface_pick: no selection");
    // the smallest node T with sum_{surface i <= T} p_i >= u, by bisection
    // over node indices (the cumulative sum only grows at surface nodes)
    const float fsum = (float)h->sel.score_sum;
    auto prefix = [&](int upTo, double* out) -> int {
        CK(cudaMemsetAsync(h->acc.p, 0, sizeof(double), h->stream));
        launch_surface_prefix(h->sf(), h->surfSlots, fsum, upTo, h->acc.p, h->stream);
        CK(cudaMemcpyAsync(out, h->acc.p, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
        return sync_status(h, "tg_surface_pick");
    };
    int lo = h->surfMinNode, hi = h->surfMaxNode;
    double cum = 0.0;
    int rc = prefix(hi, &cum);
    if (rc != TG_OK) return rc;
    if (u > cum) {
        lo = hi;  // past the end: the last cell
    } else {
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if ((rc = prefix(mid, &cum)) != TG_OK) return rc;
            if (u > cum) lo = mid + 1;
            else hi = mid;
        }
    }
    *node = lo;
    if (probability) {
        int32_t slot = -1;
        CK(cudaMemcpyAsync(&slot, h->surfSlot.p + lo, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
        float sc = 0.0f;
        CK(cudaStreamSynchronize(h->stream));
        if (slot >= 0 && slot < h->surfSlots) {
            CK(cudaMemcpy(&sc, h->surfScore.p + slot, sizeof(float), cudaMemcpyDeviceToHost));
        }
        *probability = sc / fsum;
    }
    return TG_OK;
}

int tg_cell_values(tg_handle* h, int32_t count, const int32_t* nodes, float* phi, float* field, float* force) {
    DeviceScope dev_scope(h);
    if (!h || count < 0 || (!nodes && count != h->n))
        return fail(h, TG_ERR_ARGUMENT, "tg_cell_values: bad argument (nodes NULL needs count = N)");
    if (nodes)
        for (int32_t k = 0; k < count; k++)
            if (nodes[k] < 0 || nodes[k] >= h->n) return fail(h, TG_ERR_ARGUMENT, "tg_cell_values: node out of range");
    if (count == 0 || (!phi && !field && !force)) return TG_OK;
    int rc = stage(h, h->stageF, 7 * (size_t)count);
    if (rc == TG_OK && nodes) rc = stage(h, h->stageI, count);
    if (rc != TG_OK) return rc;
    float* dPhi = h->stageF.p;
    float* dField = dPhi + count;
    float* dForce = dField + 3 * (size_t)count;
    if (nodes) CK(cudaMemcpyAsync(h->stageI.p, nodes, sizeof(int32_t) * count, cudaMemcpyHostToDevice, h->stream));
    launch_cell_values(h->dm(), nodes ? h->stageI.p : nullptr, count, phi ? dPhi : nullptr, field ? dField : nullptr,
                       force ? dForce : nullptr, h->stream);
    if (phi) CK(cudaMemcpyAsync(phi, dPhi, sizeof(float) * count, cudaMemcpyDeviceToHost, h->stream));
    if (field) CK(cudaMemcpyAsync(field, dField, sizeof(float) * 3 * count, cudaMemcpyDeviceToHost, h->stream));
    if (force) CK(cudaMemcpyAsync(force, dForce, sizeof(float) * 3 * count, cudaMemcpyDeviceToHost, h->stream));
    return sync_status(h, "tg_cell_values");
}

int tg_surface_normals(tg_handle* h, int32_t count, const int32_t* nodes, float* normals) {
    DeviceScope dev_scope(h);
    if (!h || count < 0 || (count && (!nodes || !normals))) return fail(h, TG_ERR_ARGUMENT, "tg_surface_normals: bad argument");
    if (h->vacuumId < 0) return fail(h, TG_ERR_ARGUMENT, "tg_surface_normals: surface not initialised");
    for (int32_t k = 0; k < count; k++)
        if (nodes[k] < 0 || nodes[k] >= h->n) return fail(h, TG_ERR_ARGUMENT, "tg_surface_normals: node out of range");
    if (count == 0) return TG_OK;
    int rc = stage(h, h->stageF, 3 * (size_t)count);
    if (rc == TG_OK) rc = stage(h, h->stageI, count);
    if (rc == TG_OK) rc = stage(h, h->stageD, 9 * (size_t)count);
    if (rc != TG_OK) return rc;
    CK(cudaMemcpyAsync(h->stageI.p, nodes, sizeof(int32_t) * count, cudaMemcpyHostToDevice, h->stream));
    launch_surface_normals(h->dm(), h->stageI.p, count, h->vacuumId, h->stageD.p, h->stageF.p, h->stream);
    CK(cudaMemcpyAsync(normals, h->stageF.p, sizeof(float) * 3 * count, cudaMemcpyDeviceToHost, h->stream));
    return sync_status(h, "tg_surface_normals");
}

int tg_surface_cells(tg_handle* h, int32_t mode, float temperature, int32_t capacity, int32_t* count, int32_t* cells,
                     float* probability) {
    DeviceScope dev_scope(h);
    if (!h || !count || capacity < 0 || (capacity && (!cells || !probability)))
        return fail(h, TG_ERR_ARGUMENT, "tg_surface_cells: bad argument");
    *count = 0;
    tg_select_info info;
    int rc = tg_surface_select_mode(h, mode, temperature, &info);
    if (rc == TG_ERR_NO_SURFACE) return TG_OK;
    if (rc != TG_OK) return rc;
    std::vector<int32_t> list(h->surfSlots);
    std::vector<float> score(capacity > 0 ? h->surfSlots : 0);
    CK(cudaMemcpyAsync(list.data(), h->surfList.p, sizeof(int32_t) * h->surfSlots, cudaMemcpyDeviceToHost, h->stream));
    if (capacity > 0)
        CK(cudaMemcpyAsync(score.data(), h->surfScore.p, sizeof(float) * h->surfSlots, cudaMemcpyDeviceToHost, h->stream));
    rc = sync_status(h, "tg_surface_cells");
    if (rc != TG_OK) return rc;
    if (capacity == 0) {  // the count alone
        *count = (int32_t)(list.size() - std::count(list.begin(), list.end(), -1));
        return TG_OK;
    }
    std::vector<std::pair<int32_t, float>> set;
    set.reserve(h->surfSlots);
    for (int s = 0; s < h->surfSlots; s++)
        if (list[s] >= 0) set.emplace_back(list[s], score[s]);
    std::sort(set.begin(), set.end());
    // evap_compute_probabilities normalises each cell's value by the sum
    // over the set, in float
    const float fsum = (float)info.score_sum;
    for (size_t k = 0; k < set.size() && (int32_t)k < capacity; k++) {
        cells[k] = set[k].first;
        probability[k] = set[k].second / fsum;
    }
    *count = (int32_t)set.size();
    return TG_OK;
}

static std::string snapshot_name(const char* path, int32_t index) {
    char suffix[16];
    snprintf(suffix, sizeof(suffix), ".%08u", (unsigned)index);
    return std::string(path) + suffix;
}

int tg_log_grid(tg_handle* h, const char* path, int32_t index, int32_t binary, const uint32_t* numbers) {
    DeviceScope dev_scope(h);
    if (!h || !path) return fail(h, TG_ERR_ARGUMENT, "tg_log_grid: null argument");
    const int n = h->n;
    std::vector<float> phi(n), field(3 * (size_t)n), force(3 * (size_t)n);
    int rc = tg_cell_values(h, n, nullptr, phi.data(), field.data(), force.data());
    if (rc != TG_OK) return rc;
    std::vector<int8_t> t8(n);
    if ((rc = tg_get_types(h, t8.data())) != TG_OK) return rc;
    std::vector<int32_t> id(t8.begin(), t8.end());
    std::vector<uint32_t> num(n);
    for (int i = 0; i < n; i++) num[i] = numbers ? numbers[i] : (uint32_t)(i + 1);
    rc = tg_grid_log_write(snapshot_name(path, index).c_str(), binary, n, id.data(), num.data(), phi.data(),
                           field.data(), force.data());
    if (rc != TG_OK) return fail(h, rc, tg_last_error(nullptr));
    return TG_OK;
}

int tg_log_surface(tg_handle* h, const char* path, int32_t index, int32_t binary, int32_t withNeighbours,
                   int32_t mode, float temperature, const uint32_t* numbers) {
    DeviceScope dev_scope(h);
    if (!h || !path) return fail(h, TG_ERR_ARGUMENT, "tg_log_surface: null argument");
    const int n = h->n;
    int32_t nc = 0;
    int rc = tg_surface_cells(h, mode, temperature, 0, &nc, nullptr, nullptr);
    if (rc != TG_OK) return rc;
    std::vector<int32_t> cells(nc);
    std::vector<float> prob(nc);
    if (nc && (rc = tg_surface_cells(h, mode, temperature, nc, &nc, cells.data(), prob.data())) != TG_OK) return rc;
    std::vector<int8_t> t8(n);
    if ((rc = tg_get_types(h, t8.data())) != TG_OK) return rc;
    // LogSurface::prepare (logSurface.cpp:159-201): the cells, their
    // neighbour lists, and every cell and neighbour once, ascending
    std::vector<int32_t> type(nc), nptr(nc + 1, 0), nb;
    std::vector<uint32_t> num(nc);
    std::vector<char> mark(n, 0);
    for (int c = 0; c < nc; c++) {
        const int i = cells[c];
        type[c] = t8[i];
        num[c] = numbers ? numbers[i] : (uint32_t)(i + 1);
        mark[i] = 1;
        for (int q = h->h_row_ptr[i]; q < h->h_row_ptr[i + 1]; q++) {
            nb.push_back(h->h_col[q]);
            mark[h->h_col[q]] = 1;
        }
        nptr[c + 1] = (int32_t)nb.size();
    }
    std::vector<int32_t> nodes;
    for (int i = 0; i < n; i++)
        if (mark[i]) nodes.push_back(i);
    const int nn = (int)nodes.size();
    std::vector<float> phi(nn), field(3 * (size_t)nn), normal(3 * (size_t)nn, 0.0f), cellNormal(3 * (size_t)nc);
    if (nn && (rc = tg_cell_values(h, nn, nodes.data(), phi.data(), field.data(), nullptr)) != TG_OK) return rc;
    if (nc && (rc = tg_surface_normals(h, nc, cells.data(), cellNormal.data())) != TG_OK) return rc;
    for (int c = 0; c < nc; c++) {
        const size_t k = std::lower_bound(nodes.begin(), nodes.end(), cells[c]) - nodes.begin();
        for (int j = 0; j < 3; j++) normal[3 * k + j] = cellNormal[3 * (size_t)c + j];
    }
    rc = tg_surface_log_write(snapshot_name(path, index).c_str(), binary, nc, cells.data(), type.data(), num.data(),
                              prob.data(), withNeighbours ? nptr.data() : nullptr, nb.data(), nn, nodes.data(),
                              phi.data(), field.data(), normal.data());
    if (rc != TG_OK) return fail(h, rc, tg_last_error(nullptr));
    return TG_OK;
}

int tg_get_surface(tg_handle* h, int32_t capacity, int32_t* nodes, float* ratios, int32_t* count) {
    DeviceScope dev_scope(h);
    if (!h || !count) return fail(h, TG_ERR_ARGUMENT, "tg_get_surface: null argument");
    std::vector<int32_t> list(h->surfSlots);
    std::vector<float> rat(h->surfSlots);
    if (h->surfSlots) {
        CK(cudaMemcpyAsync(list.data(), h->surfList.p, sizeof(int32_t) * h->surfSlots, cudaMemcpyDeviceToHost, h->stream));
        CK(cudaMemcpyAsync(rat.data(), h->surfRatio.p, sizeof(float) * h->surfSlots, cudaMemcpyDeviceToHost, h->stream));
    }
    int rc = sync_status(h, "tg_get_surface");
    if (rc != TG_OK) return rc;
    int c = 0;
    for (int s = 0; s < h->surfSlots; s++) {
        if (list[s] < 0) continue;
        if (c < capacity) {
            if (nodes) nodes[c] = list[s];
            if (ratios) ratios[c] = rat[s];
        }
        c++;
    }
    *count = c;
    return TG_OK;
}

int tg_surface_normal(tg_handle* h, int32_t node, float normal[3]) {
    DeviceScope dev_scope(h);
    if (!h || node < 0 || node >= h->n || !normal) return fail(h, TG_ERR_ARGUMENT, "tg_surface_normal: bad argument");
    int rc = stage(h, h->stageF, 4);
    if (rc != TG_OK) return rc;
    // Surface_3d::Table::normal returns zero for nodes outside the surface set
    uint8_t f = 0;
    CK(cudaMemcpyAsync(&f, h->flags.p + node, 1, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    if (!(f & F_SURFACE)) {
        normal[0] = normal[1] = normal[2] = 0.0f;
        return TG_OK;
    }
    launch_surface_normal(h->dm(), h->sf(), node, h->vacuumId, h->stageF.p, h->stream);
    CK(cudaMemcpyAsync(normal, h->stageF.p, 3 * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    return sync_status(h, "tg_surface_normal");
}

// evap_takeAway on the device with one read back: the removal's result
// and the row and surface counts come back together; the cells that become
// free non-Neumann rows are appended to the V system, whose slot counter
// the host mirrors (an overflow raises S_CAPACITY at the next status read).
static int take_away_impl(tg_handle* h, int32_t node, int32_t capacity, int32_t* detached, int32_t* numDetached) {
    if (h->ncol > tg_handle::kMaxColours) return fail(h, TG_ERR_ARGUMENT, "tg_take_away: too many colours");
    tg_handle::Pinned* pin = h->pin;
    const int cap = (int)std::min<size_t>(h->result.n, 1024);
    launch_take_away(h->dm(), h->rl(), h->sf(), node, h->vacuumId, h->result.p, cap, h->stream);
    CK(cudaMemcpyAsync(pin->result, h->result.p, sizeof(int32_t) * cap, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(pin->counts, h->countVD.p, sizeof(int32_t) * h->ncol, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(pin->counts + h->ncol, h->countND.p, sizeof(int32_t) * h->ncol, cudaMemcpyDeviceToHost,
                       h->stream));
    CK(cudaMemcpyAsync(pin->misc, h->countAllD.p, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(pin->misc + 2, h->surfCount.p, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    int rc = sync_status(h, "tg_take_away");
    if (rc != TG_OK) return rc;
    std::memcpy(h->countV.data(), pin->counts, sizeof(int32_t) * h->ncol);
    std::memcpy(h->countN.data(), pin->counts + h->ncol, sizeof(int32_t) * h->ncol);
    h->countAllV = pin->misc[0];
    h->countAllN = pin->misc[1];
    h->surfSlots = std::min(pin->misc[2], h->n);
    const int nd = pin->result[0];
    // the flipped cells for the next solve's first residual; rows that move
    // between the V and Neumann classes, or out of the free rows, and lists
    // cut short by the result capacity take the full pass instead
    {
        const tg_type& vt0 = h->types[h->vacuumId];
        bool ok = nd + 1 < cap && h->nPending + 1 + nd <= (int)(sizeof(pin->pending) / sizeof(int32_t)) &&
                  !vt0.dirichlet;
        for (int k = -1; ok && k < nd; k++) {
            const int j = k < 0 ? node : pin->result[1 + k];
            const int t = h->h_type[j];
            if (t >= 0 && !h->types[t].dirichlet && h->types[t].neumann != vt0.neumann) ok = false;
        }
        if (ok) {
            pin->pending[h->nPending++] = node;
            for (int k = 0; k < nd; k++) pin->pending[h->nPending++] = pin->result[1 + k];
        } else {
            h->pendingOverflow = true;
        }
    }
    // the flipped cells and their neighbours join the vertex-field cells
    if (nd + 1 >= cap) {
        h->fieldAll = true;
    } else if (!h->fieldAll) {
        std::vector<int32_t> act;
        for (int k = -1; k < nd; k++) {
            const int f = k < 0 ? node : pin->result[1 + k];
            for (int q = h->h_row_ptr[f] - 1; q < h->h_row_ptr[f + 1]; q++) {
                const int j = q < h->h_row_ptr[f] ? f : h->h_col[q];
                if (!h->h_fieldActive[j]) {
                    h->h_fieldActive[j] = 1;
                    act.push_back(j);
                }
            }
        }
        if (!act.empty()) {
            const size_t na = act.size();
            if (na <= sizeof(pin->activated) / sizeof(int32_t)) {
                std::memcpy(pin->activated, act.data(), sizeof(int32_t) * na);
                CK(cudaMemcpyAsync(h->fieldCells.p + h->fieldCount, pin->activated, sizeof(int32_t) * na,
                                   cudaMemcpyHostToDevice, h->stream));
            } else {
                CK(cudaMemcpy(h->fieldCells.p + h->fieldCount, act.data(), sizeof(int32_t) * na,
                              cudaMemcpyHostToDevice));
            }
            h->fieldCount += (int)na;
        }
    }
    int nf = 0;
    if (!(h->h_type[node] >= 0 && h->types[h->h_type[node]].dirichlet == 0)) pin->flipped[nf++] = node;
    h->h_type[node] = (int8_t)h->vacuumId;
    for (int k = 0; k < nd && k + 1 < cap; k++) {
        const int j = pin->result[1 + k];
        if (h->types[h->h_type[j]].dirichlet) pin->flipped[nf++] = j;
        h->h_type[j] = (int8_t)h->vacuumId;
        if (detached && k < capacity) detached[k] = j;
    }
    if (numDetached) *numDetached = nd;
    // cells that became non-Neumann free rows join the V system
    const tg_type& vt = h->types[h->vacuumId];
    if (!vt.dirichlet && !vt.neumann && nf > 0) {
        if (h->vNext + nf > h->vCapacity) return fail(h, TG_ERR_ARGUMENT, "tg_take_away: V-system reserve exhausted");
        CK(cudaMemcpyAsync(h->stageI.p, pin->flipped, sizeof(int32_t) * nf, cudaMemcpyHostToDevice, h->stream));
        launch_vsys_add_rows(h->dm(), h->vs(), h->stageI.p, nf, h->stream);
        h->vNext += nf;
        h->vActive = (h->vNext + 31) / 32 * 32;
    }
    // cells that were free already (a removed non-Dirichlet species) keep
    // their rows, whose couplings the flip has changed
    if (nf < 1 + nd) {
        pin->flipped[512] = node;
        for (int k = 0; k < nd && k + 1 < cap; k++) pin->flipped[513 + k] = pin->result[1 + k];
        const int nr = 1 + std::min(nd, cap - 1);
        CK(cudaMemcpyAsync(h->stageI.p + 256, pin->flipped + 512, sizeof(int32_t) * nr, cudaMemcpyHostToDevice,
                           h->stream));
        launch_vsys_refresh(h->dm(), h->vs(), h->stageI.p + 256, nr, h->stream);
    }
    h->bnormValid = false;
    h->selValid = false;
    h->removalsSinceSolve++;
    h->lastSite = node;
    return TG_OK;
}

int tg_take_away(tg_handle* h, int32_t node, int32_t capacity, int32_t* detached, int32_t* numDetached) {
    DeviceScope dev_scope(h);
    if (!h || node < 0 || node >= h->n) return fail(h, TG_ERR_ARGUMENT, "tg_take_away: bad node");
    if (h->vacuumId < 0) return fail(h, TG_ERR_ARGUMENT, "tg_take_away: surface not initialised");
    const int rc = take_away_impl(h, node, capacity, detached, numDetached);
    if (rc != TG_OK) return rc;
    return sync_status(h, "tg_take_away (V rows)");
}

int tg_update_coordination(tg_handle* h) {
    DeviceScope dev_scope(h);
    if (!h) return fail(h, TG_ERR_ARGUMENT, "tg_update_coordination: null handle");
    h->residValid = false;
    launch_update_coordination(h->dm(), h->typeScratch.p, h->stream);
    return sync_status(h, "tg_update_coordination");
}

static TraceParams trace_params(const tg_handle* h, const tg_trace_opts* o) {
    TraceParams tp;
    tp.path = nullptr;
    tp.path_err = nullptr;
    tp.path_cap = 0;
    tp.dt0 = o->time_step;
    tp.dt_min = o->min_time_step;
    tp.tol = o->error_threshold;
    tp.max_steps = o->max_steps;
    tp.stepper_limit = o->stepper_limit;
    tp.walk_limit = o->walk_limit;
    tp.top_z = h->top_z;
    tp.integrator = o->integrator;
    tp.stepper = o->stepper;
    tp.precision = o->precision;
    tp.fp64_radius2 = o->fp64_radius * o->fp64_radius;
    return tp;
}

// Device path buffers for `slots` flights of `cap` points each.
static int stage_paths(tg_handle* h, size_t slots, int32_t cap) {
    int rc = stage(h, h->pathBuf, slots * (size_t)cap * 8);
    if (rc == TG_OK) rc = stage(h, h->pathErr, slots * 12);
    return rc;
}

// tg_trace, and tg_trace_path when cap > 0 (paths to host points/errors).
static int trace_impl(tg_handle* h, int32_t nIons, const float* start, const float* vel, const float* qm,
                      const int32_t* guess, const tg_trace_opts* o, tg_impact* out, int32_t cap,
                      tg_path_point* points, float* errors, const char* what) {
    if (!h || nIons < 0 || (nIons && (!start || !qm || !out)) || !o || cap < 0 ||
        (cap > 0 && nIons && (!points || !errors)))
        return fail(h, TG_ERR_ARGUMENT, std::string(what) + ": bad argument");
    if (!h->tet_v.p) return fail(h, TG_ERR_ARGUMENT, std::string(what) + ": mesh has no tetrahedra");
    if (o->precision < 0 || o->precision > 2 || !(o->fp64_radius >= 0.0))
        return fail(h, TG_ERR_ARGUMENT, std::string(what) + ": precision 0..2 and fp64_radius >= 0");
    if (nIons == 0) return TG_OK;
    if (guess)
        for (int32_t k = 0; k < nIons; k++)
            if (guess[k] < 0 || guess[k] >= h->ntets)
                return fail(h, TG_ERR_ARGUMENT, std::string(what) + ": tetrahedron guess out of range");
    int rc = stage(h, h->stageF, (size_t)nIons * 7);
    // more ions than the device holds at once: the flights that take the most
    // steps first, so that the others fill in behind them
    const bool ordered = nIons > trace_resident();
    if (rc == TG_OK) rc = stage(h, h->stageI, (size_t)nIons * (ordered ? 2 : 1));
    if (rc == TG_OK) rc = stage(h, h->stageImpact, nIons);
    if (rc == TG_OK && cap > 0) rc = stage_paths(h, nIons, cap);
    if (rc != TG_OK) return rc;
    float* dStart = h->stageF.p;
    float* dVel = h->stageF.p + 3 * (size_t)nIons;
    float* dQm = h->stageF.p + 6 * (size_t)nIons;
    CK(cudaMemcpyAsync(dStart, start, sizeof(float) * 3 * nIons, cudaMemcpyHostToDevice, h->stream));
    if (vel) CK(cudaMemcpyAsync(dVel, vel, sizeof(float) * 3 * nIons, cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(dQm, qm, sizeof(float) * nIons, cudaMemcpyHostToDevice, h->stream));
    if (guess) CK(cudaMemcpyAsync(h->stageI.p, guess, sizeof(int32_t) * nIons, cudaMemcpyHostToDevice, h->stream));
    else CK(cudaMemsetAsync(h->stageI.p, 0, sizeof(int32_t) * nIons, h->stream));
    int32_t* dOrder = nullptr;
    std::vector<int32_t> order;
    if (ordered) {
        // the step control bounds the error relative to each component, so an
        // ion beside a coordinate plane of the axis takes the shortest steps:
        // on a 4096-ion launch the ions whose smaller one of |x| and |y| is
        // below a tenth of the larger (an eighth of them) took 830 trials on
        // average and up to 2277, the others 390 and up to 1430
        order.resize(nIons);
        size_t head = 0, tail = nIons;
        for (int32_t k = 0; k < nIons; k++) {
            const float x = std::fabs(start[3 * (size_t)k]), y = std::fabs(start[3 * (size_t)k + 1]);
            if (std::min(x, y) < 0.1f * std::max(x, y)) order[head++] = k;
            else order[--tail] = k;
        }
        std::reverse(order.begin() + tail, order.end());
        dOrder = h->stageI.p + nIons;
        CK(cudaMemcpyAsync(dOrder, order.data(), sizeof(int32_t) * nIons, cudaMemcpyHostToDevice, h->stream));
    }
    TraceParams tp = trace_params(h, o);
    if (cap > 0) {
        tp.path = h->pathBuf.p;
        tp.path_err = h->pathErr.p;
        tp.path_cap = cap;
    }
    launch_vertex_fields(h->dm(), h->stream);  // once per call, from the current potentials
    launch_trace(h->dm(), nIons, dStart, vel ? dVel : nullptr, dQm, h->stageI.p, dOrder, tp, h->stageImpact.p, h->stream);
    CK(cudaMemcpyAsync(out, h->stageImpact.p, sizeof(tg_impact) * nIons, cudaMemcpyDeviceToHost, h->stream));
    if (cap > 0) {
        CK(cudaMemcpyAsync(points, h->pathBuf.p, sizeof(tg_path_point) * (size_t)nIons * cap, cudaMemcpyDeviceToHost,
                           h->stream));
        CK(cudaMemcpy2DAsync(errors, 6 * sizeof(float), h->pathErr.p, 12 * sizeof(float), 6 * sizeof(float), nIons,
                             cudaMemcpyDeviceToHost, h->stream));
    }
    return sync_status(h, what);
}

int tg_trace(tg_handle* h, int32_t nIons, const float* start, const float* vel, const float* qm,
             const int32_t* guess, const tg_trace_opts* o, tg_impact* out) {
    DeviceScope dev_scope(h);
    return trace_impl(h, nIons, start, vel, qm, guess, o, out, 0, nullptr, nullptr, "tg_trace");
}

int tg_trace_path(tg_handle* h, int32_t nIons, const float* start, const float* vel, const float* qm,
                  const int32_t* guess, const tg_trace_opts* o, int32_t cap, tg_impact* out, tg_path_point* points,
                  float* errors) {
    DeviceScope dev_scope(h);
    if (cap <= 0) return fail(h, TG_ERR_ARGUMENT, "tg_trace_path: cap must be positive");
    return trace_impl(h, nIons, start, vel, qm, guess, o, out, cap, points, errors, "tg_trace_path");
}

int tg_potential_at(tg_handle* h, int32_t n, const float* xyz, const int32_t* guess, float* out) {
    DeviceScope dev_scope(h);
    if (!h || n < 0 || (n && (!xyz || !out))) return fail(h, TG_ERR_ARGUMENT, "tg_potential_at: bad argument");
    if (n == 0) return TG_OK;
    if (!h->tet_v.p) return fail(h, TG_ERR_ARGUMENT, "tg_potential_at: mesh has no tetrahedra");
    if (guess)
        for (int32_t k = 0; k < n; k++)
            if (guess[k] < 0 || guess[k] >= h->ntets)
                return fail(h, TG_ERR_ARGUMENT, "tg_potential_at: tetrahedron guess out of range");
    int rc = stage(h, h->stageF, (size_t)n * 4);
    if (rc == TG_OK) rc = stage(h, h->stageI, n);
    if (rc != TG_OK) return rc;
    CK(cudaMemcpyAsync(h->stageF.p, xyz, sizeof(float) * 3 * n, cudaMemcpyHostToDevice, h->stream));
    if (guess) CK(cudaMemcpyAsync(h->stageI.p, guess, sizeof(int32_t) * n, cudaMemcpyHostToDevice, h->stream));
    else CK(cudaMemsetAsync(h->stageI.p, 0, sizeof(int32_t) * n, h->stream));
    launch_potential_at(h->dm(), n, h->stageF.p, h->stageI.p, 100000, h->stageF.p + 3 * (size_t)n, h->stream);
    CK(cudaMemcpyAsync(out, h->stageF.p + 3 * (size_t)n, sizeof(float) * n, cudaMemcpyDeviceToHost, h->stream));
    return sync_status(h, "tg_potential_at");
}

// Steps I-VI of one event.  With asyncImpact (a device slot) the flight of
// step V is queued on the trace stream and its impact left there; without,
// it runs through tg_trace and lands in rec->impact.
// The flight ring of tg_run_events, allocated at its first use.
static int ring_ready(tg_handle* h) {
    if (h->ringReady) return TG_OK;
    for (int r = 0; r < tg_handle::kRing; r++) {
        int leastPriority = 0, greatestPriority = 0;
        CK(cudaDeviceGetStreamPriorityRange(&leastPriority, &greatestPriority));
        CK(cudaStreamCreateWithPriority(&h->ringStream[r], cudaStreamNonBlocking, leastPriority));
        CK(cudaEventCreateWithFlags(&h->ringPhi[r], cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&h->ringDone[r], cudaEventDisableTiming));
        CK(cudaEventRecord(h->ringDone[r], h->ringStream[r]));
        CK(h->ringPhiBuf[r].alloc(h->n));
        CK(h->ringField[r].alloc(3 * (size_t)h->n));
        h->ringFull[r] = true;
    }
    h->ringReady = true;
    return TG_OK;
}

// Probability of a surface cell in the last selection (score / sum in
// float, as tg_surface_pick reports it); TG_ERR_ARGUMENT for a cell that is
// not on the surface.
static int surface_probability(tg_handle* h, int32_t node, float* probability) {
    if (node < 0 || node >= h->n) return fail(h, TG_ERR_ARGUMENT, "forced removal: node out of range");
    int32_t slot = -1;
    CK(cudaMemcpyAsync(&h->pin->node[1], h->surfSlot.p + node, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    slot = h->pin->node[1];
    if (slot < 0 || slot >= h->surfSlots)
        return fail(h, TG_ERR_ARGUMENT, "forced removal: node " + std::to_string(node) + " is not on the surface");
    float sc = 0.0f;
    CK(cudaMemcpy(&sc, h->surfScore.p + slot, sizeof(float), cudaMemcpyDeviceToHost));
    *probability = sc / (float)h->sel.score_sum;
    return TG_OK;
}

// callIndex: the event's position within the calling tg_run_event(s) call,
// which picks its forced removal (tg_event_opts.force_nodes)
static int run_event(tg_handle* h, const tg_event_opts* o, int32_t eventIndex, int32_t callIndex,
                     tg_event_record* rec, ImpactOut* asyncImpact) {
    if (h->vacuumId != o->vacuum_id) {
        int32_t ns;
        int rc = tg_surface_init(h, o->vacuum_id, &ns);
        if (rc != TG_OK) return rc;
    }
    if (o->prob_mode < 0 || o->prob_mode > 3 || o->choice_mode < 0 || o->choice_mode > 1)
        return fail(h, TG_ERR_ARGUMENT, "tg_run_event: probability mode 0..3, choice mode 0..1");
    if (o->trace.precision < 0 || o->trace.precision > 2 || !(o->trace.fp64_radius >= 0.0))
        return fail(h, TG_ERR_ARGUMENT, "tg_run_event: trace precision 0..2 and fp64_radius >= 0");
    int rc = TG_OK;
    if (!h->selValid || h->sel.prob_mode != o->prob_mode) {
        tg_select_info s;
        rc = tg_surface_select_mode(h, o->prob_mode, o->temperature, &s);
        if (rc != TG_OK) return rc;
    }
    std::memset(rec, 0, sizeof(*rec));
    const tg_select_info sel = h->sel;
    if (sel.candidate < 0) return fail(h, TG_ERR_NO_SURFACE, "tg_run_event: empty surface");
    // I) the candidate (evapMaximum, or evapMonteCarlo with the handle's
    // stream) and its state before removal
    int node = sel.candidate;
    float probability = sel.probability;
    if (o->choice_mode == 1) {
        if (!h->rngSeeded) {
            if (initstate_r(o->rng_seed, h->rngState, sizeof(h->rngState), &h->rng) != 0)
                return fail(h, TG_ERR_HOST, "tg_run_event: random stream");
            h->rngSeeded = true;
        }
        int32_t r = 0;
        random_r(&h->rng, &r);
        rc = tg_surface_pick(h, (double)r / (double)RAND_MAX, &node, &probability);
        if (rc != TG_OK) return rc;
    }
    if (o->force_nodes && callIndex < o->force_count) {
        node = o->force_nodes[callIndex];
        rc = surface_probability(h, node, &probability);
        if (rc != TG_OK) return rc;
    }
    rec->node = node;
    rec->type_id = h->h_type[node];
    rec->probability = probability;
    rec->best_probability = sel.best_probability;
    rec->second_probability = sel.second_probability;
    rec->best_ratio = sel.best_ratio;
    rec->second_ratio = sel.second_ratio;
    rec->scaling_reference = sel.best_ratio;
    // the state before removal (potential, field_o1, surface normal of the
    // candidate) is copied into pinned memory and read with the record at
    // the end of the event
    tg_handle::Pinned* pin = h->pin;
    pin->node[0] = node;
    CK(cudaMemcpyAsync(h->stageI.p + 512, &pin->node[0], sizeof(int32_t), cudaMemcpyHostToDevice, h->stream));
    launch_field_o1(h->dm(), h->stageI.p + 512, 1, h->stageD.p, h->stream);
    CK(cudaMemcpyAsync(&pin->before[0], h->phi64.p + node, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(&pin->before[1], h->stageD.p, 3 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    for (int k = 0; k < 3; k++) rec->apex[k] = sel.apex >= 0 ? h->h_xyz[3 * (size_t)sel.apex + k] : 0.0f;
    if (o->normal_enabled) {
        // the candidate is a surface cell by construction; the normal reads
        // the flags and types as they are before the removal, from copies,
        // on the auxiliary stream while the removal and the solve go on
        CK(cudaMemcpyAsync(h->snapFlags.p, h->flags.p, h->n, cudaMemcpyDeviceToDevice, h->stream));
        CK(cudaMemcpyAsync(h->snapType.p, h->type.p, h->n, cudaMemcpyDeviceToDevice, h->stream));
        CK(cudaEventRecord(h->evSnap, h->stream));
        CK(cudaStreamWaitEvent(h->auxStream, h->evSnap, 0));
        DevMesh ms = h->dm();
        ms.flags = h->snapFlags.p;
        ms.type = h->snapType.p;
        launch_surface_normal(ms, h->sf(), node, h->vacuumId, h->normalBuf.p, h->auxStream);
        CK(cudaMemcpyAsync(pin->normal, h->normalBuf.p, 3 * sizeof(float), cudaMemcpyDeviceToHost, h->auxStream));
        CK(cudaEventRecord(h->evNormal, h->auxStream));
    }
    const tg_type removed = h->types[h->h_type[node]];
    // II) removal
    int32_t nd = 0;
    rc = take_away_impl(h, node, 0, nullptr, &nd);
    if (rc != TG_OK) return rc;
    rec->detached = nd;
    if (h->coordinationActive) {
        h->residValid = false;
        launch_update_coordination(h->dm(), h->typeScratch.p, h->stream);
    }
    // III) relaxation
    if (o->relax_mode == 0) {
        int64_t it = 0;
        double dev = 0.0;
        int r1 = tg_local_relax(h, node, o->local_shell, o->local_threshold, o->local_cycle, o->local_queue, &it, &dev);
        if (r1 != TG_OK && r1 != TG_ERR_RELAX_FAULT && r1 != TG_ERR_ITERATION_CAP) return r1;
        rec->relax_iterations = (int32_t)it;
        if (o->global_steps > 0) {
            r1 = tg_relax_cycles(h, o->global_steps, &dev);
            if (r1 != TG_OK) return r1;
            rec->relax_iterations += o->global_steps;
        }
        if (o->refresh_interval > 0 && eventIndex % o->refresh_interval == 0) {
            r1 = tg_relax_threshold(h, o->refresh_threshold, o->refresh_cycle, o->refresh_queue, o->refresh_max_sweeps,
                                    &it, &dev);
            if (r1 != TG_OK && r1 != TG_ERR_RELAX_FAULT && r1 != TG_ERR_ITERATION_CAP) return r1;
            rec->relax_status = r1;
            rec->relax_iterations += (int32_t)it;
        }
        rc = tg_residual(h, &rec->rel_residual);
        if (rc != TG_OK) return rc;
    } else {
        tg_solve_info si;
        rc = tg_solve(h, &o->solve, &si);
        rec->relax_status = rc;
        if (rc != TG_OK && rc != TG_ERR_ITERATION_CAP) return rc;
        rec->relax_iterations = si.inner;
        rec->rel_residual = si.rel_residual;
    }
    // IV) fields, probabilities and the next candidate: queued here and
    // decoded after the event's one synchronisation at its end (only the
    // next event reads them)
    rc = select_launch(h, o->prob_mode, o->temperature);
    if (rc != TG_OK) return rc;
    h->selValid = false;
    // V) ion flight of the removed atom, VI) state after removal
    if (o->trace_enabled) {
        const float start[3] = {h->h_xyz[3 * (size_t)node], h->h_xyz[3 * (size_t)node + 1], h->h_xyz[3 * (size_t)node + 2]};
        // Trajectory_3d::eCharge / amu2kg (trajectory_3d.h:91-93) as floats
        const float charge = (float)removed.evap_charge * 1.60217733e-19f;
        const float mass = removed.mass * 1.660538782e-27f;
        const float qm = charge / mass;
        const int32_t guess = h->h_node_tet.empty() ? 0 : std::max(0, h->h_node_tet[node]);
        float vel[3] = {0.0f, 0.0f, 0.0f};
        if (o->initial_velocity) {
            // evap_initialVelocity (surface_3d.cpp:472-503): kinetic energies
            // split by two uniform draws, a random sign per component
            if (!h->rngSeeded) {
                if (initstate_r(o->rng_seed, h->rngState, sizeof(h->rngState), &h->rng) != 0)
                    return fail(h, TG_ERR_HOST, "tg_run_event: random stream");
                h->rngSeeded = true;
            }
            auto draw = [&]() {
                int32_t r = 0;
                random_r(&h->rng, &r);
                return r;
            };
            const double vmax = 2.0 * 1.3806504e-23 * (double)o->temperature / (double)removed.mass / 1.660538782e-27;
            float e2[3];
            e2[0] = (float)((double)draw() / RAND_MAX) * (float)vmax;
            e2[1] = (float)((double)draw() / RAND_MAX) * ((float)vmax - e2[0]);
            e2[2] = (float)vmax - e2[0] - e2[1];
            for (int c = 0; c < 3; c++) {
                vel[c] = std::sqrt(std::max(e2[c], 0.0f));
                if (draw() % 2) vel[c] = -vel[c];
            }
        }
        if (asyncImpact) {
            if (guess >= h->ntets || !h->tetpack.p) return fail(h, TG_ERR_ARGUMENT, "tg_run_events: no tetrahedra");
            rc = ring_ready(h);
            if (rc != TG_OK) return rc;
            const int r = h->ringNext;
            h->ringNext = (r + 1) % tg_handle::kRing;
            // the flight that used this slot (kRing events ago) is done with
            // its snapshots before this event's potentials replace them
            CK(cudaStreamWaitEvent(h->stream, h->ringDone[r], 0));
            CK(cudaMemcpyAsync(h->ringPhiBuf[r].p, h->phi64.p, sizeof(double) * h->n, cudaMemcpyDeviceToDevice,
                               h->stream));
            CK(cudaEventRecord(h->ringPhi[r], h->stream));
            CK(cudaStreamWaitEvent(h->ringStream[r], h->ringPhi[r], 0));
            // vertex fields from the snapshot on the slot's stream: they read
            // the couplings only through their zero pattern, which a flip to
            // the vacuum type never changes, so the next event's removal may
            // run meanwhile
            DevMesh mt = h->dm();
            mt.phi64 = h->ringPhiBuf[r].p;
            mt.phiTrace = h->ringPhiBuf[r].p;
            mt.vfield = h->ringField[r].p;
            mt.status = h->statusTrace.p;
            if (h->ringFull[r] || h->fieldAll) {
                launch_vertex_fields(mt, h->ringStream[r]);
                h->ringFull[r] = false;
            } else {
                launch_vertex_fields(mt, h->ringStream[r], h->fieldCells.p, h->fieldCount);
            }
            TraceParams tp = trace_params(h, &o->trace);
            if (o->path_cap > 0) {
                // this event's slot of the batch
                const size_t slot = (size_t)(asyncImpact - h->stageImpact.p);
                tp.path = h->pathBuf.p + slot * (size_t)o->path_cap * 8;
                tp.path_err = h->pathErr.p + 12 * slot;
                tp.path_cap = o->path_cap;
            }
            launch_trace_one(mt, start, vel, qm, guess, tp, asyncImpact, h->ringStream[r]);
            CK(cudaGetLastError());
            CK(cudaEventRecord(h->ringDone[r], h->ringStream[r]));
        } else {
            rc = trace_impl(h, 1, start, o->initial_velocity ? vel : nullptr, &qm, &guess, &o->trace, &rec->impact,
                            o->path_cap, o->path_points, o->path_errors, "tg_run_event");
            if (rc != TG_OK) return rc;
        }
    }
    // the state after removal, and one read of both
    launch_field_o1(h->dm(), h->stageI.p + 512, 1, h->stageD.p + 4, h->stream);
    CK(cudaMemcpyAsync(&pin->after[0], h->phi64.p + node, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(&pin->after[1], h->stageD.p + 4, 3 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    if (o->normal_enabled) CK(cudaStreamWaitEvent(h->stream, h->evNormal, 0));
    rc = sync_status(h, "tg_run_event");
    if (rc != TG_OK) return rc;
    {
        tg_select_info next;
        rc = select_decode(h, o->prob_mode, &next);
        if (rc != TG_OK && rc != TG_ERR_NO_SURFACE) return rc;
    }
    rec->phi_before = (float)pin->before[0];
    rec->phi_after = (float)pin->after[0];
    for (int k = 0; k < 3; k++) {
        rec->field_before[k] = (float)pin->before[1 + k];
        rec->field_after[k] = (float)pin->after[1 + k];
        if (o->normal_enabled) rec->normal[k] = pin->normal[k];
    }
    return TG_OK;
}

int tg_gemm_bf16(const uint16_t* A, const uint16_t* B, float* C, int32_t M, int32_t N, int32_t K) {
    if (!A || !B || !C || !gemm_shape_ok(M, N, K))
        return fail(nullptr, TG_ERR_ARGUMENT, "tg_gemm_bf16: M % 128, N in {64, 128}, K % 64 required");
    void *dA = nullptr, *dB = nullptr;
    float* dC = nullptr;
    int* dSt = nullptr;
    const size_t bytesA = sizeof(uint16_t) * (size_t)M * K, bytesB = sizeof(uint16_t) * (size_t)N * K;
    const size_t bytesC = sizeof(float) * (size_t)M * N;
    cudaError_t e = cudaMalloc(&dA, bytesA);
    if (e == cudaSuccess) e = cudaMalloc(&dB, bytesB);
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&dC), bytesC);
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&dSt), sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpy(dA, A, bytesA, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dB, B, bytesB, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(dSt, 0, sizeof(int));
    if (e == cudaSuccess) e = launch_gemm_bf16(dA, dB, dC, M, N, K, dSt, 0);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    int st = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&st, dSt, sizeof(int), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(C, dC, bytesC, cudaMemcpyDeviceToHost);
    cudaFree(dA);
    cudaFree(dB);
    cudaFree(dC);
    cudaFree(dSt);
    if (e != cudaSuccess) return fail(nullptr, TG_ERR_CUDA, std::string("tg_gemm_bf16: ") + cudaGetErrorString(e));
    if (st != 0) return status_code(nullptr, st, "tg_gemm_bf16");
    return TG_OK;
}

static bool path_opts_ok(const tg_event_opts* o) {
    return o->path_cap >= 0 && (o->path_cap == 0 || (o->path_points && o->path_errors));
}

int tg_run_event(tg_handle* h, const tg_event_opts* o, int32_t eventIndex, tg_event_record* rec) {
    DeviceScope dev_scope(h);
    if (!h || !o || !rec) return fail(h, TG_ERR_ARGUMENT, "tg_run_event: null argument");
    if (!path_opts_ok(o)) return fail(h, TG_ERR_ARGUMENT, "tg_run_event: path_cap < 0 or path buffers missing");
    if (o->force_count < 0) return fail(h, TG_ERR_ARGUMENT, "tg_run_event: force_count < 0");
    return run_event(h, o, eventIndex, 0, rec, nullptr);
}

int tg_run_events(tg_handle* h, const tg_event_opts* o, int32_t firstIndex, int32_t count, tg_event_record* recs,
                  int32_t* done) {
    DeviceScope dev_scope(h);
    if (!h || !o || count < 0 || (count && !recs)) return fail(h, TG_ERR_ARGUMENT, "tg_run_events: bad argument");
    if (!path_opts_ok(o)) return fail(h, TG_ERR_ARGUMENT, "tg_run_events: path_cap < 0 or path buffers missing");
    if (o->force_count < 0) return fail(h, TG_ERR_ARGUMENT, "tg_run_events: force_count < 0");
    if (done) *done = 0;
    int rc = stage(h, h->stageImpact, std::max(count, 1));
    if (rc == TG_OK && o->path_cap > 0 && o->trace_enabled) rc = stage_paths(h, std::max(count, 1), o->path_cap);
    if (rc != TG_OK) return rc;
    CK(cudaMemsetAsync(h->statusTrace.p, 0, sizeof(int), h->stream));
    int k = 0;
    for (; k < count; k++) {
        rc = run_event(h, o, firstIndex + k, k, &recs[k], h->stageImpact.p + k);
        if (rc != TG_OK) break;
    }
    // every flight queued so far completes before the impacts are read
    if (h->ringReady)
        for (int r = 0; r < tg_handle::kRing; r++) CK(cudaStreamSynchronize(h->ringStream[r]));
    CK(cudaStreamSynchronize(h->stream));
    if (o->trace_enabled && k > 0) {
        std::vector<ImpactOut> imp(k);
        CK(cudaMemcpy(imp.data(), h->stageImpact.p, sizeof(ImpactOut) * k, cudaMemcpyDeviceToHost));
        for (int j = 0; j < k; j++) std::memcpy(&recs[j].impact, &imp[j], sizeof(tg_impact));
        if (o->path_cap > 0) {
            CK(cudaMemcpy(o->path_points, h->pathBuf.p, sizeof(tg_path_point) * (size_t)k * o->path_cap,
                          cudaMemcpyDeviceToHost));
            CK(cudaMemcpy2D(o->path_errors, 6 * sizeof(float), h->pathErr.p, 12 * sizeof(float), 6 * sizeof(float), k,
                            cudaMemcpyDeviceToHost));
        }
        int st = 0;
        CK(cudaMemcpy(&st, h->statusTrace.p, sizeof(int), cudaMemcpyDeviceToHost));
        if (st != 0) {
            CK(cudaMemset(h->statusTrace.p, 0, sizeof(int)));
            if (rc == TG_OK) rc = status_code(h, st, "tg_run_events flights");
        }
    }
    if (done) *done = k;
    return rc;
}

int tg_run_tips(tg_handle* const* handles, int32_t count, const tg_event_opts* opts, int32_t firstIndex,
                tg_event_record* recs, float* latency_ms, int32_t* status, int32_t threads) {
    if (count < 0 || (count && (!handles || !opts || !recs || !latency_ms || !status)))
        return fail(nullptr, TG_ERR_ARGUMENT, "tg_run_tips: bad argument");
    for (int32_t k = 0; k < count; k++) {
        if (!handles[k]) return fail(nullptr, TG_ERR_ARGUMENT, "tg_run_tips: null handle");
        for (int32_t j = 0; j < k; j++)
            if (handles[j] == handles[k]) return fail(nullptr, TG_ERR_ARGUMENT, "tg_run_tips: a handle listed twice");
    }
    int T = threads > 0 ? threads : (int)std::max(1u, std::thread::hardware_concurrency());
    T = std::max(1, std::min(T, (int)count));
    // tip k goes to worker k % T: a handle is only ever driven by one thread
    auto work = [&](int t) {
        for (int32_t k = t; k < count; k += T) {
            const auto t0 = std::chrono::steady_clock::now();
            int32_t done = 0;
            status[k] = tg_run_events(handles[k], &opts[k], firstIndex, 1, &recs[k], &done);
            latency_ms[k] = (float)std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0)
                                .count();
        }
    };
    if (T == 1) {
        work(0);
    } else {
        std::vector<std::thread> pool;
        try {
            pool.reserve(T);
            for (int t = 0; t < T; t++) pool.emplace_back(work, t);
        } catch (const std::exception& e) {
            for (auto& th : pool) th.join();
            return fail(nullptr, TG_ERR_HOST, std::string("tg_run_tips: starting host threads: ") + e.what());
        }
        for (auto& th : pool) th.join();
    }
    for (int32_t k = 0; k < count; k++)
        if (status[k] != TG_OK) {
            g_error = "tg_run_tips: tip " + std::to_string(k) + ": " + handles[k]->err;
            return status[k];
        }
    return TG_OK;
}

}  // extern "C"

// ---- field_o1 without allocation ----
//
// tg_field_o1 stages its node list and results in per-handle device buffers
// that grow with cudaMalloc when a call asks for more nodes than any call
// before it.  Some callers cannot allocate at that point: a host whose
// device memory is fully committed to the mesh and to another allocator's
// pool (a caching allocator that already holds the rest of the 180 GB), or a
// real-time loop that must not take the driver's allocation lock between
// events.  tg_field_o1_noalloc serves them from a fixed scratch array that
// is part of this library's device image, so it makes no allocation call.
namespace {

constexpr int kNoAllocMaxDevices = 64;
// nodes (int32) first, then the fields (3 doubles per node); both offsets
// are multiples of 256 bytes
constexpr size_t kNoAllocNodesBytes = sizeof(int32_t) * (size_t)TG_FIELD_O1_NOALLOC_MAX;
constexpr size_t kNoAllocBytes = kNoAllocNodesBytes + 3 * sizeof(double) * (size_t)TG_FIELD_O1_NOALLOC_MAX;
static_assert(kNoAllocNodesBytes % 256 == 0, "field offset must stay 256-byte aligned");
static __device__ __align__(256) unsigned char g_field_scratch[kNoAllocBytes];

std::mutex g_noalloc_mutex;
void* g_noalloc_ptr[kNoAllocMaxDevices] = {};

// Device address of the scratch on the handle's device, looked up once per
// device with that device current (the caller's DeviceScope makes it so; the
// lookup may load this library's device image onto the device).
int noalloc_scratch(tg_handle* h, unsigned char** out) {
    const int dev = h->device;
    if (dev < 0 || dev >= kNoAllocMaxDevices)
        return fail(h, TG_ERR_ARGUMENT, "tg_field_o1_noalloc: device ordinal beyond the 64 the scratch table covers");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        CK(cudaGetSymbolAddress(&p, g_field_scratch));
        g_noalloc_ptr[dev] = p;
    }
    *out = static_cast<unsigned char*>(g_noalloc_ptr[dev]);
    return TG_OK;
}

}  // namespace

extern "C" {

int tg_field_o1_noalloc(tg_handle* h, int32_t count, const int32_t* nodes, double* out) {
    DeviceScope dev_scope(h);
    if (!h || count < 0 || (count && (!nodes || !out)))
        return fail(h, TG_ERR_ARGUMENT, "tg_field_o1_noalloc: bad argument");
    if (count > TG_FIELD_O1_NOALLOC_MAX)
        return fail(h, TG_ERR_ARGUMENT,
                    "tg_field_o1_noalloc: " + std::to_string(count) + " nodes exceed the fixed scratch of " +
                        std::to_string(TG_FIELD_O1_NOALLOC_MAX) + " nodes; split the list or call tg_field_o1");
    for (int32_t k = 0; k < count; k++)
        if (nodes[k] < 0 || nodes[k] >= h->n)
            return fail(h, TG_ERR_ARGUMENT, "tg_field_o1_noalloc: node index out of range");
    unsigned char* base = nullptr;
    int rc = noalloc_scratch(h, &base);
    if (rc != TG_OK || count == 0) return rc;
    int32_t* dNodes = reinterpret_cast<int32_t*>(base);
    double* dOut = reinterpret_cast<double*>(base + kNoAllocNodesBytes);
    // Nothing in the scratch has to start at zero: the node list is copied
    // in and the kernel writes every one of the count results.  The
    // handle's status word, which the kernel may set, is cleared by
    // sync_status whenever it is found set.
    CK(cudaMemcpyAsync(dNodes, nodes, sizeof(int32_t) * count, cudaMemcpyHostToDevice, h->stream));
    launch_field_o1(h->dm(), dNodes, count, dOut, h->stream);
    CK(cudaMemcpyAsync(out, dOut, sizeof(double) * 3 * count, cudaMemcpyDeviceToHost, h->stream));
    return sync_status(h, "tg_field_o1_noalloc");
}

}  // extern "C"
