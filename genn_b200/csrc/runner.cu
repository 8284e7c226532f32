// C ABI of the B200 backend (include/genn_b200.h) and the runner behind it.
//
// A runner is the counterpart of one loaded librunner.so of the reference: it
// owns the stream, the device-resident step counters, the merged-group tables
// and the captured step graph.  The time-step path allocates nothing and never
// synchronises; the host only enqueues (one cudaGraphLaunch per block of steps).
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <algorithm>
#include <cctype>
#include <cstdarg>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "genn_b200.h"
#include "common.cuh"
#include "neuron_update.cuh"
#include "presynaptic_update.cuh"
#include "postsynaptic_update.cuh"
#include "init.cuh"
#include "fused_step.cuh"
#include "urgent.cuh"
#include "stream_step.cuh"
#include "tiled.cuh"
#include "dense_batch.cuh"
#include "sparse_batch.cuh"
#include "procedural.cuh"
#include "resident.h"
#include "memory.h"
#include "record.cuh"

#include <cub/device/device_scan.cuh>

using namespace b200;

namespace
{
thread_local std::string g_lastError;

int fail(int code, const char *fmt, ...)
{
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_lastError = buf;
    return code;
}

#define CUDA_TRY(expr)                                                                           \
    do {                                                                                         \
        cudaError_t _e = (expr);                                                                 \
        if(_e != cudaSuccess) {                                                                  \
            return fail(B200_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e),   \
                        __FILE__, __LINE__);                                                     \
        }                                                                                        \
    } while(0)

constexpr size_t STAGE_BYTES = 256 * 1024 - 64;  // page-locked buffer of a runner through which small arrays reach pageable memory
constexpr size_t LARGE_PULL = 4u << 20;      // arrays from here on are copied out by several threads
constexpr uint64_t FIRST_BLOCK = 64;         // steps of the first launch of the target-resident kernel in a call, the next has twice as many:
constexpr uint64_t QUIET_BLOCK = 2048;       // a network that was busy at first is soon tried again; once a call has passed quietly
constexpr uint64_t LONG_CALL = 10000;        // steps of a first call in the middle of which the host looks whether the other kernel has taken over
constexpr uint64_t LONG_HOLD = 512;          // steps of that kernel's turn from which its own tables are made (with rings: 2 - 20 ms)
constexpr uint64_t WINDOW_STEPS = 4;         // steps of a launch from which they are done in windows where they can be
constexpr double MOST_LOSS = 1.0e6;          // ns that a call of the target-resident kernel may lose with no launch behind it, for each of the
constexpr unsigned int MOST_QUIET = 50;      // quiet calls before it, up to this many (a launch for nothing: 4 us, a tenth of a short call)
constexpr size_t ARRAY_TAIL_PAD = 256;     // vector loads may read up to 15 bytes past the last element

template<typename T>
struct DeviceTable
{
    T *d = nullptr;
    unsigned int *blockStart = nullptr;
    unsigned int num = 0;
    unsigned int blocks = 0;

    void release(cudaStream_t s)
    {
        poolFree(d, s);
        poolFree(blockStart, s);
        d = nullptr; blockStart = nullptr; num = 0; blocks = 0;
    }

    cudaError_t upload(const std::vector<T> &items, const std::vector<unsigned int> &starts, cudaStream_t s)
    {
        release(s);
        num = (unsigned int)items.size();
        if(num == 0) return cudaSuccess;
        blocks = starts.back();
        cudaError_t e = poolAlloc(&d, sizeof(T) * num, s);
        if(e != cudaSuccess) return e;
        e = poolAlloc(&blockStart, sizeof(unsigned int) * starts.size(), s);
        if(e != cudaSuccess) return e;
        e = cudaMemcpyAsync(d, items.data(), sizeof(T) * num, cudaMemcpyHostToDevice, s);
        if(e != cudaSuccess) return e;
        e = cudaMemcpyAsync(blockStart, starts.data(), sizeof(unsigned int) * starts.size(), cudaMemcpyHostToDevice, s);
        if(e != cudaSuccess) return e;
        return cudaStreamSynchronize(s);
    }
};

struct Timer
{
    double seconds = 0.0;
};
}   // anonymous namespace

// (Everything the host writes into device memory goes through the runner's stream, which does not wait for the legacy one:
// a plain cudaMemcpy may return while its transfer is still on the way, and a kernel launched behind it on another stream
// would read what was there before.)

// Device buffer that is freed on every early return of a build function unless it was handed over.
struct ScopedDevice
{
    cudaStream_t stream;
    void *p = nullptr;
    explicit ScopedDevice(cudaStream_t s) : stream(s) {}
    ~ScopedDevice() { poolFree(p, stream); }
    template<typename T> T *as() const { return static_cast<T*>(p); }
    void *release() { void *q = p; p = nullptr; return q; }
};

constexpr unsigned int PROFILE_MAX_CTAS = 1024;     // per-CTA cycle counters of option "fused_profile"

struct b200_runner
{
    int device = 0;
    float dt = 0.1f;
    unsigned long long seed = 0;
    unsigned int batch = 1;
    cudaStream_t stream = nullptr;
    StepState *state = nullptr;
    std::unordered_map<void*, size_t> arrays;
    unsigned char *stage = nullptr;         // STAGE_BYTES, page-locked: pulls of small arrays land here
    unsigned int *hostWord = nullptr;       // page-locked: the device's error word
    std::mutex staging;                     // held by the thread whose transfer uses either
    // recording list (record.cuh): chunk counts, header and pairs on the device, header and pairs on the host
    unsigned int *recCounts = nullptr;
    RecordHeader *recList = nullptr, *recHost = nullptr;
    size_t recChunks = 0, recCapacity = 0;
    size_t recLast = 0;                     // pairs of the last pull

    std::vector<b200_neuron_group> neuronGroups;
    std::vector<b200_synapse_group> synapseGroups;
    std::map<std::string, std::vector<b200_custom_update_group>> customUpdates;
    bool dirty = true;

    DeviceTable<b200_neuron_group> neuronTable;
    DeviceTable<b200_synapse_group> sparseTable, postSpanTable, learnTable, proceduralTable, drawnTable, denseTable, scatterTable;
    DeviceTable<b200_synapse_group> scatterRows;    // the groups of scatterTable, for presynapticSparseKernel
    bool drawnNormal = false, drawnWide = false;    // proceduralDrawnKernel: every weight Normal; element numbers beyond 32 bits
    unsigned int ahead = 0, advance = 1;    // place of the step being enqueued in its block of steps (see chainPhase)
    ScatterTarget *scatterTargets = nullptr;
    ScatterPart *scatterParts = nullptr;    // sparseBatchKernel: what every CTA does
    unsigned int scatterGrid = 0, scatterCells = 0, scatterDepth = 0, scatterPiece = 0;
    size_t scatterSmem = 0;
    // sparseBatchKernel's start and flush take longer than presynapticSparseKernel needs for a few spikes: it is used ("armed")
    // while the largest spike count of the steps before (peakHost below) reaches this many spikes a copy
    float scatterMinSpikes = SCATTER_MIN_SPIKES;
    bool scatterArmed = false;
    unsigned int scatterQuiet = 0;
    unsigned long long scatterSources = ~0ull;      // neuron groups whose spikes it delivers
    uint4 *denseParts = nullptr;            // denseBatchKernel: what every CTA does

    // persistent fused-step path (batch 1, SPARSE non-learning groups only)
    bool fusedEligible = false;
    bool useFused = true;
    unsigned int fusedBlocksPerSM = 0;      // 0: as many as fit (occupancy query)
    unsigned int fusedGrid = 0;
    unsigned int *fusedSlotStart = nullptr;
    FusedSource *fusedSources = nullptr;
    uint2 *fusedItems = nullptr;
    unsigned int fusedNumSources = 0;
    unsigned int fusedNumItems = 0;
    size_t fusedSmemBytes = 0;
    bool fusedStage = false;
    const void *fusedKernel = nullptr;
    int fusedPerSM = 0;
    unsigned long long *fusedBarrier = nullptr;
    unsigned long long fusedLaunches = 0;
    bool fusedProfile = false;
    unsigned long long *fusedCtaCycles = nullptr;
    // one-step lag of the persistent kernel (fused_step.cuh): allowed while every
    // synapse has a dendritic delay of at least one step
    bool useLag = true;
    bool lagAgreed = false;         // sharded model: the host checked that every process is eligible
    bool lagStale = true;           // delay arrays may have changed since the last scan
    bool lagEligible = false;
    std::vector<b200_synapse_group> fusedGroups;    // host copy of the SPARSE groups the kernel serves
    // split delivery (fused_step.cuh): private tables of the synapses that arrive in the same step
    bool useSplit = true;
    int streamWarpsWanted = -1;                     // -1: as many as the neuron slots leave free, 0: none
    unsigned int streamWarps = 0;                   // of the current tables (0: fusedStepKernel)
    unsigned int slotsPerCta = 0;
    std::vector<unsigned int> urgentStride;         // per SPARSE group: its longest urgent row (0: none)
    unsigned int *urgentOffsets = nullptr;          // row offsets of all groups, one after the other
    uint2 *urgentEntries = nullptr;
    FusedUrgent *fusedUrgent = nullptr;             // device copy for the kernel, or NULL
    enum Schedule { PLAIN = 0, SPLIT = 1, LAG = 2, EMIT = 3 };
    // "deliver at emission" mode (near.cuh): near synapses of all groups, one row per source neuron
    bool useEmit = true;
    bool nearExported = false;              // nearTable is an allocation of its own, which other processes map
    uint2 *nearTable = nullptr;             // rows of every source neuron (synapses onto THIS process's neurons)
    NearRing *nearRings = nullptr;          // device copies, [world][numRings] and [world][neuron groups]
    NearSpace *nearSpaces = nullptr;
    unsigned int numRings = 0;
    // sharded model: built by b200_near_export / b200_near_import / b200_near_finish
    std::vector<NearRing> nearRingsHost;            // this process's rings
    std::vector<unsigned long long> nearCellHost;   // per neuron group: first entry of its rows in nearTable
    std::vector<unsigned int> nearShiftHost;        // per neuron group: row length shift (0xFFFFFFFF: no rows)
    std::vector<uint2*> nearImported;               // per neuron group: the rows of this process's neurons, one block per process
    std::vector<NearSpace> nearSpacesAll;           // [neuron groups]
    std::vector<bool> nearPeerDone;                 // per process: its blocks have been copied in
    bool emitAgreed = false;                        // every process exported, imported and qualified
    bool nearDataStale = false;                     // synapse arrays changed after the exchange
    Schedule schedule = PLAIN;

    void freeNearTable()
    {
        if(nearTable) {
            if(nearExported) cudaFree(nearTable);
            else poolFree(nearTable, stream);
        }
        nearTable = nullptr;
    }

    void dropNear()
    {
        freeNearTable();
        poolFree(nearRings, stream);
        poolFree(nearSpaces, stream);
        for(uint2 *p : nearImported) if(p) cudaFree(p);
        nearImported.clear();
        nearRings = nullptr; nearSpaces = nullptr; numRings = 0;
        emitAgreed = false;
    }

    void dropUrgent()
    {
        urgentStride.clear();
        poolFree(urgentOffsets, stream);
        poolFree(urgentEntries, stream);
        poolFree(fusedUrgent, stream);
        urgentOffsets = nullptr; urgentEntries = nullptr; fusedUrgent = nullptr;
        if(!emitAgreed) dropNear();
    }

    // spike exchange of a sharded model
    unsigned char *arena = nullptr;
    size_t arenaBytes = 0;
    // data-parallel runs: communicator for the all-reduce inside batch-reduce custom updates, and the
    // buffer the reduced values of a group are packed into for it
    void *ncclComm = nullptr;
    unsigned int ncclWorld = 1;
    float *reducePacked = nullptr;
    size_t reducePackedElements = 0;
    // queues for near synapses between processes (near.cuh), behind the caller's part of the arena
    size_t queueOffset = 0;
    unsigned int queueWords = NEAR_QUEUE_WORDS;
    bool useNearQueues = true;
    bool queuesAgreed = false;                  // every process runs the same grid, which the queues are numbered by
    unsigned int peerGrid[B200_MAX_RANKS] = {};
    unsigned char *peerArena[B200_MAX_RANKS] = {};
    bool peerLocal[B200_MAX_RANKS] = {};    // mapped by pointer (same process): nothing to close
    unsigned char **peerTable = nullptr;     // device copy of peerArena
    unsigned int rank = 0, world = 1;
    size_t flagsOffset = 0;
    bool sharded() const { return world > 1; }

    // target-tiled delivery of heavy steps on the one-launch-per-kernel path (tiled.cuh): private
    // re-packed copy of the non-learning SPARSE groups
    bool useTiled = true;
    float tiledTicketEvents = 2048.0f, tiledTicketCost = 256.0f;     // (swept on Potjans x1 with a quarter of the neurons spiking)
    float tiledMinEvents = 1.0e6f;          // estimated events of a step from which the tiled kernel takes it
    bool tiledReady = false, tiledStale = true;
    // The tiled kernels cost two launches per step even when they find nothing to do, so they are only
    // launched ("armed") while the network's recent activity could reach the threshold: the neuron kernel
    // keeps the largest spike count of a step in StepState::peak_spikes, the host fetches it (asynchronously,
    // into page-locked memory) behind every block of steps and looks at it before the next block
    bool tiledArmed = false;
    unsigned int *peakHost = nullptr;
    cudaEvent_t peakEvent = nullptr;
    bool peakPending = false, peakSeen = false;
    unsigned int peakSteps = 0;             // steps since the count was last fetched
    unsigned int quietBlocks = 0;
    double eventsPerSpike = 0.0;
    std::string tiledWhyNot;
    TiledTile *tiledTiles = nullptr;
    TiledSource *tiledSources = nullptr;
    unsigned int *tiledRunStart = nullptr, *tiledCtaStart = nullptr, *tiledPairBatches = nullptr;
    void *tiledKeys = nullptr;
    float *tiledWeights = nullptr;
    TiledPair *tiledPairs = nullptr;
    double *tiledPairPrefix = nullptr;
    unsigned char *tiledServed = nullptr;
    unsigned int tiledNumPairs = 0, tiledNumSources = 0, tiledPostBits = 10, tiledGrid = 0;
    size_t tiledSmemBytes = 0;
    unsigned long long tiledSynapses = 0;

    void dropTiled()
    {
        void *bufs[] = {tiledTiles, tiledSources, tiledRunStart, tiledCtaStart, tiledPairBatches, tiledKeys, tiledWeights,
                        tiledPairs, tiledPairPrefix, tiledServed};
        for(void *b : bufs) poolFree(b, stream);
        tiledTiles = nullptr; tiledSources = nullptr; tiledRunStart = nullptr; tiledCtaStart = nullptr;
        tiledPairBatches = nullptr; tiledKeys = nullptr; tiledWeights = nullptr; tiledPairs = nullptr;
        tiledPairPrefix = nullptr; tiledServed = nullptr;
        tiledReady = false;
    }

    // target-resident kernel (resident.h): private copy of the SPARSE groups cut by CTA, message buffers
    bool useResident = true;
    bool residentAsked = false;             // the caller asked for it by name (and says so when it writes an exposed array)
    std::vector<void*> exposed;             // arrays that the program writes by itself (b200_array_expose)
    bool tiledChosen = false;               // the caller set what arms the tiled kernels: they serve whatever they can
    bool scheduleChosen = false;            // the caller picked a schedule of the other persistent kernels
    bool residentStale = true, residentReady = false;
    bool residentOld = false;               // only weights have changed since the copy was made: it is filled again where it lies
    // A program that changes the synapses again and again would pay for a copy every time: it is made (or filled) again when the steps on
    // the model's other path, which reads the arrays, have cost as much as that
    unsigned long long residentRent = 0;    // steps left to do there
    double residentCells = 0.0;             // entries of the copy, millions
    unsigned long long residentBuilds = 0, residentLaunches = 0;
    struct ResidentPair { unsigned int delay_class, src, first, count; };
    std::vector<ResidentPair> residentPairs;            // what the copy is filled from
    const b200_synapse_group *residentGroups = nullptr; // (device)
    const unsigned int *residentTargets = nullptr, *residentDepths = nullptr;
    std::string residentWhyNot;
    unsigned int residentCtas = 0, residentWarps = 0;       // 0: chosen by size
    unsigned int residentGrid = 0, residentBlock = 0;
    size_t residentSmem = 0;
    unsigned long long residentCleared = ~0ull;             // steps done when the message buffers were last cleared (~0: they are not)
    size_t residentMailBytes = 0, windowMailBytes = 0;
    const void *residentKernel = nullptr;
    ResidentLaunch resident{};
    bool useWindow = true, windowReady = false;             // windows of steps (resident_window.cuh)
    ResidentWindow window{};
    const void *windowKernel = nullptr;
    size_t windowSmem = 0;
    unsigned int windowBlock = 0, windowWeight = 0;
    bool windowMayOverflow = false;                         // a step may have more spikes than its list holds: a launch has to follow
    std::vector<void*> residentBuffers;
    // busy networks (resident.h): the kernel with a grid barrier takes over
    volatile unsigned long long *residentHold = nullptr;    // page-locked: until which step it goes on
    bool residentHandsOver = false;         // the model's other path is that kernel (else: one launch per kernel, call by call)
    float residentPatience = 200.0f;        // us
    bool residentPatienceChosen = false;
    double residentWorst = 0.0;             // ns that a step could lose, were every neuron to fire
    double residentSources = 0.0;           // neurons with synapses
    bool residentSteeper = false;           // groups with rings, whose spikes cost more here
    unsigned long long residentHoldSeen = 0;
    unsigned int residentQuiet = 0;         // calls since the host last saw that it had to

    void dropResident()
    {
        for(void *p : residentBuffers) poolFree(p, stream);
        residentBuffers.clear();
        residentReady = windowReady = false;
        residentCleared = ~0ull;
    }

    // options
    unsigned int spikeLanes = 16;
    bool countEvents = false;
    bool useGraph = true;
    unsigned int graphSteps = 100;
    bool timing = false;

    // captured graph of `graphLen` steps for a given recording length
    cudaGraphExec_t graphExec = nullptr;
    unsigned int graphLen = 0;
    unsigned long long graphNumRec = 0;

    std::map<std::string, Timer> timers;
    cudaEvent_t evA = nullptr, evB = nullptr, evC = nullptr, evD = nullptr;
    unsigned long long launches = 0;
    unsigned long long hostTimestep = 0, hostStepsDone = 0;

    void dropGraph()
    {
        if(graphExec) cudaGraphExecDestroy(graphExec);
        graphExec = nullptr;
        graphLen = 0;
    }
};

namespace
{
template<typename F>
int withIndType(unsigned int bytes, F f)
{
    switch(bytes) {
    case 1: return f(uint8_t());
    case 2: return f(uint16_t());
    case 4: return f(uint32_t());
    default: return fail(B200_ERR_INVALID, "index width %u is not 1, 2 or 4", bytes);
    }
}

// Kernel instances by (max fused postsynaptic models, max current sources) of
// any neuron group: the smallest covering instance is used.
struct NeuronShape { int npsm, ncs; };

NeuronShape neuronShape(const b200_runner *r)
{
    unsigned int p = 0, c = 0;
    for(const auto &g : r->neuronGroups) {
        p = std::max(p, g.num_psm);
        c = std::max(c, g.num_cs);
    }
    NeuronShape s;
    s.npsm = (p <= 1) ? 1 : (p <= 2) ? 2 : B200_MAX_PSM;
    s.ncs = (c == 0) ? 0 : (c == 1) ? 1 : B200_MAX_CS;
    return s;
}

template<typename F>
int withNeuronShape(const b200_runner *r, F f)
{
    const NeuronShape s = neuronShape(r);
#define B200_SHAPE(P, C) if(s.npsm == P && s.ncs == C) return f(std::integral_constant<int, P>(), std::integral_constant<int, C>())
    B200_SHAPE(1, 0); B200_SHAPE(1, 1); B200_SHAPE(1, B200_MAX_CS);
    B200_SHAPE(2, 0); B200_SHAPE(2, 1); B200_SHAPE(2, B200_MAX_CS);
    B200_SHAPE(B200_MAX_PSM, 0); B200_SHAPE(B200_MAX_PSM, 1); B200_SHAPE(B200_MAX_PSM, B200_MAX_CS);
#undef B200_SHAPE
    return fail(B200_ERR_INVALID, "no kernel instance for this neuron shape");
}


// Tables of the persistent fused-step kernel for the current schedule: spike
// sources, the two item lists of each, thread slots, shared-memory budget, grid.
int buildFusedTables(b200_runner *r)
{
    poolFree(r->fusedSlotStart, r->stream);
    r->fusedSlotStart = nullptr;
    poolFree(r->fusedSources, r->stream);
    r->fusedSources = nullptr;
    poolFree(r->fusedItems, r->stream);
    r->fusedItems = nullptr;
    if(!r->fusedEligible) return B200_OK;
    const std::vector<b200_synapse_group> &sparse = r->fusedGroups;
    std::vector<unsigned int> slotStart{0};
    for(const auto &g : r->neuronGroups) slotStart.push_back(slotStart.back() + ((g.num_update + 31u) & ~31u));
    std::vector<FusedSource> sources;
    std::vector<std::vector<uint2>> perSource;
    std::vector<std::vector<uint2>> perSourceUrgent;
    for(size_t gi = 0; gi < sparse.size(); gi++) {
        const auto &g = sparse[gi];
        // which list the group's full-row chunks go to, and whether it has a table of urgent synapses
        const bool ring = g.max_den_delay >= 2 && g.d;
        const bool later = (r->schedule == b200_runner::LAG) || (r->schedule == b200_runner::EMIT) ||
                           (r->schedule == b200_runner::SPLIT && ring);
        const unsigned int urgentStride = (r->schedule == b200_runner::SPLIT && gi < r->urgentStride.size())
            ? r->urgentStride[gi] : 0u;
        // a sharded source population contributes one source per process section
        const unsigned int sections = std::max(1u, g.src_sections);
        const unsigned int chunks = (g.row_stride + 3 + FUSED_CHUNK - 1) / FUSED_CHUNK;
        for(unsigned int sec = 0; sec < sections; sec++) {
            const unsigned int *cntPtr = g.src_spk_cnt + sec * g.src_cnt_section_stride;
            size_t si = 0;
            for(; si < sources.size(); si++) {
                if(sources[si].spk_cnt == cntPtr && sources[si].delay == g.axonal_delay) break;
            }
            if(si == sources.size()) {
                FusedSource src{};
                src.spk_cnt = cntPtr;
                src.spk = g.src_spk + sec * g.src_spk_section_stride;
                src.num_src = g.src_spk_slot_stride ? g.src_spk_slot_stride : g.num_src;   // list capacity
                src.slots = g.src_delay_slots;
                src.delay = g.axonal_delay;
                src.spk_tag = g.src_spk_tag
                    ? reinterpret_cast<const unsigned long long*>(g.src_spk_tag + sec * g.src_cnt_section_stride) : nullptr;
                src.spk_wire = g.src_spk_wire
                    ? reinterpret_cast<const unsigned long long*>(g.src_spk_wire + sec * g.src_spk_section_stride) : nullptr;
                sources.push_back(src);
                perSource.emplace_back();
                perSourceUrgent.emplace_back();
            }
            auto &rows = later ? perSource[si] : perSourceUrgent[si];
            for(unsigned int c = 0; c < chunks; c++) rows.push_back(make_uint2((unsigned int)gi, c));
            for(unsigned int c = 0; c < (urgentStride + 31u) / 32u; c++) {
                perSourceUrgent[si].push_back(make_uint2((unsigned int)gi, c | FUSED_URGENT_TABLE));
            }
        }
    }
    std::vector<uint2> items;
    for(size_t si = 0; si < sources.size(); si++) {
        sources[si].item_begin = (unsigned int)items.size();
        sources[si].item_count = (unsigned int)perSource[si].size();
        items.insert(items.end(), perSource[si].begin(), perSource[si].end());
        sources[si].urgent_begin = (unsigned int)items.size();
        sources[si].urgent_count = (unsigned int)perSourceUrgent[si].size();
        items.insert(items.end(), perSourceUrgent[si].begin(), perSourceUrgent[si].end());
    }
    if(sources.size() > FUSED_MAX_SOURCES) {
        return fail(B200_ERR_INVALID, "%zu spike sources exceed the %u the persistent kernel handles",
                    sources.size(), (unsigned int)FUSED_MAX_SOURCES);
    }
    r->fusedNumSources = (unsigned int)sources.size();
    r->fusedNumItems = (unsigned int)items.size();
    r->fusedSmemBytes = align16(sizeof(b200_neuron_group) * r->neuronGroups.size()) +
                        align16(sizeof(b200_synapse_group) * sparse.size()) +
                        align16(sizeof(FusedSource) * sources.size()) + align16(sizeof(uint2) * items.size()) +
                        align16(sizeof(unsigned int) * slotStart.size()) +
                        (r->fusedUrgent ? align16(sizeof(FusedUrgent) * sparse.size()) : 0) +
                        (r->schedule == b200_runner::EMIT
                            ? align16(sizeof(NearRing) * r->numRings * r->world) +
                              align16(sizeof(NearSpace) * r->neuronGroups.size()) : 0);
    r->fusedStage = r->fusedSmemBytes <= 200 * 1024;
    {
        // SPLIT schedule: the warp-specialised kernel, if the neuron slots (dealt out evenly over one
        // CTA per SM) leave at least four warps per CTA free for streaming
        r->streamWarps = 0;
        r->slotsPerCta = 0;
        int sms = 0;
        CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
        // (a sharded model on the split schedule measured faster on one set of warps: its chain waits
        // for the other GPUs anyway, and the stream warps' fences compete with it)
        const bool wanted = r->streamWarpsWanted > 0 ||
                            (r->streamWarpsWanted < 0 && !(r->sharded() && r->schedule == b200_runner::SPLIT));
        if((r->schedule == b200_runner::SPLIT || r->schedule == b200_runner::EMIT) && r->fusedStage && wanted && sms > 0) {
            const unsigned int perCta = ((slotStart.back() + sms - 1) / sms + 31u) & ~31u;
            const unsigned int warps = FUSED_BLOCK / 32;
            const unsigned int chainMin = std::max(8u, perCta / 32u);
            // (a sharded model keeps the block's last warp for publishing its spike counts)
            const unsigned int publisher = r->sharded() ? 1u : 0u;
            if(chainMin + 4u + publisher <= warps) {
                unsigned int stream = warps - chainMin - publisher;
                if(r->streamWarpsWanted > 0) stream = std::min(stream, (unsigned int)r->streamWarpsWanted);
                r->streamWarps = stream;
                r->slotsPerCta = perCta;
            }
        }
        if(r->schedule == b200_runner::EMIT && !r->streamWarps) {
            // no room for the warp-specialised kernel after all: plain schedule
            r->schedule = b200_runner::PLAIN;
            return buildFusedTables(r);
        }
        int e = withNeuronShape(r, [&](auto P, auto C) -> int {
            const void *kernel = r->streamWarps ? streamKernelFor(decltype(P)::value, decltype(C)::value, r->sharded())
                                                : fusedKernelFor(decltype(P)::value, decltype(C)::value);
            r->fusedKernel = kernel;
            if(r->fusedStage) {
                CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)r->fusedSmemBytes));
            }
            int perSM = 0;
            CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kernel, FUSED_BLOCK,
                                                                   r->fusedStage ? r->fusedSmemBytes : 0));
            r->fusedPerSM = perSM;
            return B200_OK;
        });
        if(e) return e;
    }
    CUDA_TRY(poolAlloc(&r->fusedSlotStart, sizeof(unsigned int) * slotStart.size(), r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->fusedSlotStart, slotStart.data(), sizeof(unsigned int) * slotStart.size(), cudaMemcpyHostToDevice, r->stream));
    if(!sources.empty()) {
        CUDA_TRY(poolAlloc(&r->fusedSources, sizeof(FusedSource) * sources.size(), r->stream));
        CUDA_TRY(cudaMemcpyAsync(r->fusedSources, sources.data(), sizeof(FusedSource) * sources.size(), cudaMemcpyHostToDevice, r->stream));
        CUDA_TRY(poolAlloc(&r->fusedItems, sizeof(uint2) * items.size(), r->stream));
        CUDA_TRY(cudaMemcpyAsync(r->fusedItems, items.data(), sizeof(uint2) * items.size(), cudaMemcpyHostToDevice, r->stream));
    }
    if(!r->fusedBarrier) CUDA_TRY(poolAlloc(&r->fusedBarrier, sizeof(unsigned long long), r->stream));
    int perSM = r->fusedPerSM, sms = 0, coop = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
    CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, r->device));
    if(perSM < 1 || !coop) {
        r->fusedEligible = false;
    }
    else {
        if(r->fusedBlocksPerSM) perSM = std::min<int>(perSM, (int)r->fusedBlocksPerSM);
        if(r->streamWarps) perSM = 1;       // its neuron slots were dealt out for one CTA per SM
        r->fusedGrid = (unsigned int)(perSM * sms);
    }
    return B200_OK;
}

// What the CTAs of denseBatchKernel do: (columns, sources) parts of every group, about as many as the chip holds at once so
// that no last wave is nearly empty.  A part has at least 64 sources (below that its sums cost more than its rows) and at
// most DENSE_WINDOW.
int buildDense(b200_runner *r, const std::vector<b200_synapse_group> &dense)
{
    poolFree(r->denseParts, r->stream);
    r->denseParts = nullptr;
    r->denseTable.release(r->stream);
    if(dense.empty()) return B200_OK;
    int sms = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
    const unsigned int words = (r->batch + DENSE_COPIES - 1u) / DENSE_COPIES;
    unsigned long long strips = 0;
    for(const auto &g : dense) strips += (g.num_trg + DENSE_COLS - 1u) / DENSE_COLS;
    const unsigned int wanted = std::max(1u, (unsigned int)((unsigned long long)sms * DENSE_PER_SM / std::max(1ull, strips * words)));
    std::vector<uint4> parts;
    for(unsigned int gi = 0; gi < dense.size(); gi++) {
        const auto &g = dense[gi];
        const unsigned int chunks = std::max(std::min(wanted, std::max(1u, g.num_src / 64u)), (g.num_src + DENSE_WINDOW - 1u) / DENSE_WINDOW);
        const unsigned int per = chunks ? (g.num_src + chunks - 1u) / chunks : 0u;
        for(unsigned int first = 0; first < g.num_src; first += per) {
            const unsigned int n = std::min(per, g.num_src - first);
            for(unsigned int col = 0; col < g.num_trg; col += DENSE_COLS) parts.push_back(make_uint4(gi, col, first, n));
        }
    }
    if(parts.empty()) return B200_OK;
    CUDA_TRY(cudaFuncSetAttribute(denseBatchKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DENSE_SMEM));
    CUDA_TRY(poolAlloc(&r->denseParts, sizeof(uint4) * parts.size(), r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->denseParts, parts.data(), sizeof(uint4) * parts.size(), cudaMemcpyHostToDevice, r->stream));
    CUDA_TRY(r->denseTable.upload(dense, {0u, (unsigned int)parts.size()}, r->stream));
    return B200_OK;
}

// Whether sparseBatchKernel delivers a SPARSE group: a batched network (one copy has the target-resident kernel, and the
// tiled kernels where that does not apply), no learning, a target buffer that fits a CTA's shared memory.
bool scatterServes(const b200_runner *r, const b200_synapse_group &g)
{
    if(r->batch < 2 || r->sharded() || r->tiledChosen || g.wu_model == B200_WU_STDP) return false;
    const unsigned long long cells = (unsigned long long)std::max(1u, g.max_den_delay) * g.num_trg;
    // (two pieces of the widest kind for every warp have to fit besides: the groups of a model share one ring size, so a model
    // without delays stops at 29 900 targets where its own six bytes a synapse would do for 34 500)
    if(cells * sizeof(float) > SCATTER_SMEM - 2u * SCATTER_WARPS * SCATTER_PIECE * 9u - 128u) return false;
    if(((reinterpret_cast<size_t>(g.ind) | reinterpret_cast<size_t>(g.g) | reinterpret_cast<size_t>(g.d) |
         reinterpret_cast<size_t>(g.max_den_delay ? g.den_delay : g.out_post)) & 15u) != 0u) return false;
    unsigned int groups = 0;
    for(const auto &o : r->synapseGroups) {
        if((o.max_den_delay ? o.den_delay : o.out_post) == (g.max_den_delay ? g.den_delay : g.out_post)) groups++;
    }
    return groups <= SCATTER_MOST_SOURCES;
}

// Where the neuron kernel's spike-count peaks land (allocated with the tables that need them; never on the time-step path).
int ensurePeak(b200_runner *r)
{
    if(r->peakHost) return B200_OK;
    CUDA_TRY(hostAcquire(reinterpret_cast<void**>(&r->peakHost), sizeof(unsigned int)));
    CUDA_TRY(cudaEventCreateWithFlags(&r->peakEvent, cudaEventDisableTiming));
    *r->peakHost = 0u;
    return B200_OK;
}

// The CTAs of sparseBatchKernel: one per SM as far as there are not more (buffer, copy) pairs; a buffer gets as many as its
// part of all synapses.
int buildScatter(b200_runner *r, std::vector<b200_synapse_group> &scatter)
{
    poolFree(r->scatterTargets, r->stream);
    poolFree(r->scatterParts, r->stream);
    r->scatterTargets = nullptr;
    r->scatterParts = nullptr;
    r->scatterTable.release(r->stream);
    r->scatterRows.release(r->stream);
    if(scatter.empty()) return B200_OK;
    auto buffer = [](const b200_synapse_group &g) { return g.max_den_delay ? g.den_delay : g.out_post; };
    std::stable_sort(scatter.begin(), scatter.end(), [&](const b200_synapse_group &a, const b200_synapse_group &b) { return buffer(a) < buffer(b); });
    std::vector<ScatterTarget> targets;
    std::vector<double> weight;
    double all = 0.0;
    unsigned int cells = 0, pieceBytes = 0;
    for(unsigned int i = 0; i < scatter.size(); i++) {
        const auto &g = scatter[i];
        if(targets.empty() || targets.back().cells != buffer(g)) {
            targets.push_back(ScatterTarget{buffer(g), std::max(1u, g.max_den_delay) * g.num_trg, i, 0u});
            weight.push_back(0.0);
        }
        targets.back().num_groups++;
        const double synapses = (double)g.num_src * g.row_stride + 1.0;
        weight.back() += synapses;
        all += synapses;
        cells = std::max(cells, targets.back().num_cells);
        pieceBytes = std::max(pieceBytes, SCATTER_PIECE * (g.ind_bytes + 4u + (g.max_den_delay ? 1u : 0u)));
    }
    int sms = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
    std::vector<ScatterPart> parts;
    for(unsigned int t = 0; t < targets.size(); t++) {
        const unsigned int shares = std::max(1u, (unsigned int)((double)sms * weight[t] / all / r->batch));
        for(unsigned int b = 0; b < r->batch; b++) {
            for(unsigned int s = 0; s < shares; s++) parts.push_back(ScatterPart{t, b, s, shares});
        }
    }
    r->scatterGrid = (unsigned int)parts.size();
    r->scatterCells = cells;
    r->scatterPiece = pieceBytes;
    const size_t sums = (size_t)((cells + 31u) & ~31u) * sizeof(float);
    r->scatterDepth = std::min<unsigned int>(SCATTER_MOST_DEPTH, (unsigned int)((SCATTER_SMEM - sums) / (SCATTER_WARPS * pieceBytes)));
    r->scatterSmem = sums + (size_t)r->scatterDepth * SCATTER_WARPS * pieceBytes;
    CUDA_TRY(cudaFuncSetAttribute(sparseBatchKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)r->scatterSmem));
    CUDA_TRY(poolAlloc(&r->scatterTargets, sizeof(ScatterTarget) * targets.size(), r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->scatterTargets, targets.data(), sizeof(ScatterTarget) * targets.size(), cudaMemcpyHostToDevice, r->stream));
    CUDA_TRY(poolAlloc(&r->scatterParts, sizeof(ScatterPart) * parts.size(), r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->scatterParts, parts.data(), sizeof(ScatterPart) * parts.size(), cudaMemcpyHostToDevice, r->stream));
    CUDA_TRY(r->scatterTable.upload(scatter, {0u, r->scatterGrid}, r->stream));
    std::vector<unsigned int> starts{0u};
    for(const auto &g : scatter) starts.push_back(starts.back() + (g.row_stride + 3u + PRE_TILE - 1u) / PRE_TILE);
    CUDA_TRY(r->scatterRows.upload(scatter, starts, r->stream));
    if(const int e = ensurePeak(r)) return e;
    r->scatterSources = 0;
    for(size_t ni = 0; ni < std::min<size_t>(r->neuronGroups.size(), 64); ni++) {
        for(const auto &g : scatter) if(g.src_spk_cnt == r->neuronGroups[ni].spk_cnt) r->scatterSources |= 1ull << ni;
    }
    if(!r->peakSeen) {
        // before anything has been counted: twenty spikes a second of every source neuron
        std::vector<const void*> sources;
        double neurons = 0.0;
        for(const auto &g : scatter) {
            if(std::find(sources.begin(), sources.end(), g.src_spk_cnt) != sources.end()) continue;
            sources.push_back(g.src_spk_cnt);
            neurons += g.num_src;
        }
        r->scatterArmed = neurons * 20.0e-3 * r->dt >= r->scatterMinSpikes;
    }
    return B200_OK;
}

int prepare(b200_runner *r)
{
    if(!r->dirty) return B200_OK;
    r->dropGraph();
    // neuron groups: padded to whole blocks
    {
        std::vector<unsigned int> starts{0};
        for(const auto &g : r->neuronGroups) {
            starts.push_back(starts.back() + (g.num_update + NEURON_BLOCK - 1) / NEURON_BLOCK);
        }
        CUDA_TRY(r->neuronTable.upload(r->neuronGroups, starts, r->stream));
    }
    std::vector<b200_synapse_group> sparse, postSpan, learn, procedural, drawn, dense, scatter;
    std::vector<unsigned int> sparseStarts{0}, postSpanStarts{0}, learnStarts{0}, proceduralStarts{0};
    for(const auto &g : r->synapseGroups) {
        if(g.connectivity == B200_CONN_SPARSE && scatterServes(r, g)) {
            scatter.push_back(g);
        }
        else if(g.connectivity == B200_CONN_SPARSE) {
            sparse.push_back(g);
            // +3: tiles are aligned to the array, not to the row
            sparseStarts.push_back(sparseStarts.back() + (g.row_stride + 3 + PRE_TILE - 1) / PRE_TILE);
        }
        else if(r->batch > 1 && g.connectivity == B200_CONN_DENSE && g.wu_model != B200_WU_STDP && g.num_src >= DENSE_LEAST_SOURCES) {
            dense.push_back(g);
        }
        else if(g.connectivity == B200_CONN_BITMASK || g.connectivity == B200_CONN_DENSE) {
            postSpan.push_back(g);
            postSpanStarts.push_back(postSpanStarts.back() + (g.row_stride + PRE_BLOCK - 1) / PRE_BLOCK);
        }
        else if(g.connectivity == B200_CONN_PROCEDURAL) {
            const unsigned int T = connectSubRows(g.proc_connect, g.proc_connect_params);
            if(T > 32u || (T & (T - 1u))) return fail(B200_ERR_INVALID, "procedural group: %u sub-rows per row (a power of two of at most 32 is supported)", T);
            const bool prob = (g.proc_connect == B200_CONNECT_FIXED_PROBABILITY || g.proc_connect == B200_CONNECT_FIXED_PROBABILITY_NO_AUTAPSE);
            // drawn weights need a place in the row and most of the work: the two-phase kernel
            if(prob && g.wu_model != B200_WU_STATIC_PULSE_CONSTANT_WEIGHT) {
                drawn.push_back(g);
            }
            else {
                procedural.push_back(g);
                proceduralStarts.push_back(proceduralStarts.back() + 1);
            }
        }
        else {
            return fail(B200_ERR_INVALID, "connectivity %u is not supported by this build", g.connectivity);
        }
        if(g.wu_model == B200_WU_STDP) {
            learn.push_back(g);
            const unsigned int width = (g.connectivity == B200_CONN_SPARSE) ? g.col_stride : g.num_src;
            learnStarts.push_back(learnStarts.back() + (width + POST_BLOCK - 1) / POST_BLOCK);
        }
    }
    CUDA_TRY(r->sparseTable.upload(sparse, sparseStarts, r->stream));
    CUDA_TRY(r->postSpanTable.upload(postSpan, postSpanStarts, r->stream));
    {
        int e = buildDense(r, dense);
        if(e == B200_OK) e = buildScatter(r, scatter);
        if(e) return e;
    }
    CUDA_TRY(r->learnTable.upload(learn, learnStarts, r->stream));
    CUDA_TRY(r->proceduralTable.upload(procedural, proceduralStarts, r->stream));
    CUDA_TRY(r->drawnTable.upload(drawn, {0u, (unsigned int)drawn.size()}, r->stream));
    r->drawnNormal = true;
    r->drawnWide = false;
    for(const auto &g : drawn) {
        r->drawnNormal = r->drawnNormal && g.proc_weight_init == B200_INIT_NORMAL;
        r->drawnWide = r->drawnWide || (unsigned long long)g.num_src * g.row_stride > 0xFFFFFFFFull;
    }

    // ---- tables of the persistent fused-step kernel --------------------------------
    r->fusedEligible = (r->batch == 1 && postSpan.empty() && dense.empty() && scatter.empty() && learn.empty() && procedural.empty() && drawn.empty() &&
                        !r->neuronGroups.empty());
    r->fusedGroups = sparse;
    r->lagStale = true;
    r->tiledStale = r->residentStale = true;
    r->residentRent = 0;
    r->schedule = b200_runner::PLAIN;
    r->dropUrgent();
    {
        const int e = buildFusedTables(r);
        if(e) return e;
    }

    // ---- ring period: least common multiple of every ring size ----------------------
    {
        unsigned long long period = 1;
        auto fold = [&period](unsigned int n) {
            if(n < 2) return;
            unsigned long long a = period, b = n;
            while(b) { const unsigned long long t = a % b; a = b; b = t; }
            period = period / a * n;
        };
        for(const auto &g : r->neuronGroups) {
            fold(g.num_delay_slots);
            for(unsigned int p = 0; p < g.num_psm; p++) fold(g.psm[p].max_den_delay);
        }
        for(const auto &g : r->synapseGroups) {
            fold(g.src_delay_slots);
            fold(g.trg_delay_slots);
            fold(g.max_den_delay);
        }
        if(period > (1ull << 30)) return fail(B200_ERR_INVALID, "ring sizes have no common period below 2^30");
        const unsigned int ring[2] = {(unsigned int)(r->hostStepsDone % period), (unsigned int)period};
        CUDA_TRY(cudaMemcpyAsync(&r->state->phase, ring, sizeof(ring), cudaMemcpyHostToDevice, r->stream));
    }
    r->dirty = false;
    return B200_OK;
}


// Near-synapse table of the "deliver at emission" schedule; leaves r->schedule alone if the model
// does not qualify (a group without a delay ring of three slots or more, an axonal delay, a ring
// that is not a postsynaptic model of a neuron group, too few free warps for streaming).
int buildNearTables(b200_runner *r, bool forExport = false)
{
    const auto &groups = r->fusedGroups;
    const size_t n = groups.size(), numNeuronGroups = r->neuronGroups.size();
    if(n == 0) return B200_OK;
    unsigned int slots = 0;
    for(const auto &g : r->neuronGroups) slots += (g.num_update + 31u) & ~31u;
    int sms = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
    const unsigned int perCta = ((slots + sms - 1) / sms + 31u) & ~31u;
    if(std::max(8u, perCta / 32u) + 4u > FUSED_BLOCK / 32) return B200_OK;      // no room for stream warps
    std::vector<NearRing> rings;
    std::vector<unsigned int> ringOf(n), sourceOf(n);
    for(size_t gi = 0; gi < n; gi++) {
        const auto &g = groups[gi];
        // the stream reads a spike list up to two steps after it was written: delay 0 and four slots
        if(g.max_den_delay < 3 || !g.d || g.axonal_delay != 0 || g.src_delay_slots < 4 || g.num_src >= (1u << 24)) return B200_OK;
        bool found = false;
        for(size_t ni = 0; ni < numNeuronGroups && !found; ni++) {
            const auto &ng = r->neuronGroups[ni];
            for(unsigned int p = 0; p < ng.num_psm && !found; p++) {
                if(ng.psm[p].den_delay == g.den_delay && ng.psm[p].max_den_delay == g.max_den_delay &&
                   ng.num_neurons == g.num_trg) {
                    size_t ri = 0;
                    for(; ri < rings.size(); ri++) if(rings[ri].den_delay == g.den_delay) break;
                    if(ri == rings.size()) rings.push_back(NearRing{g.den_delay, g.max_den_delay, g.num_trg});
                    ringOf[gi] = (unsigned int)ri;
                    found = true;
                }
            }
        }
        if(!found || rings.size() > NEAR_MAX_RINGS) return B200_OK;
        if(forExport) {
            // the other processes reduce into this ring over NVLink: it has to lie in the exchange arena
            const unsigned char *ring = reinterpret_cast<const unsigned char*>(g.den_delay);
            if(ring < r->arena || ring >= r->arena + r->arenaBytes) return B200_OK;
        }
        found = false;
        for(size_t ni = 0; ni < numNeuronGroups && !found; ni++) {
            const auto &ng = r->neuronGroups[ni];
            // the spiking thread looks its row up by neuron id.  One process: it updates the whole
            // population.  Sharded: the rows are built for all source neurons here and handed to
            // the processes that own them (b200_near_import); this process's own list section
            // is `rank` sections into the population's lists.
            const unsigned int *own = g.src_spk_cnt + (forExport ? (size_t)r->rank * g.src_cnt_section_stride : 0);
            if(ng.spk_cnt == own && ng.num_neurons == g.num_src &&
               (forExport || (ng.first_neuron == 0 && ng.num_update == ng.num_neurons))) {
                sourceOf[gi] = (unsigned int)ni;
                found = true;
            }
        }
        if(!found) return B200_OK;
    }
    // rows of every source population, counted first: the longest fixes the population's row length
    std::vector<unsigned long long> rowBase(numNeuronGroups + 1, 0);
    for(size_t ni = 0; ni < numNeuronGroups; ni++) rowBase[ni + 1] = rowBase[ni] + r->neuronGroups[ni].num_neurons;
    const unsigned long long totalRows = rowBase[numNeuronGroups];
    if(totalRows == 0 || totalRows >= (1ull << 31)) return B200_OK;
    // (both freed on every way out of this function; a table left behind by a failed build is dropped with the
    // runner's other near tables)
    ScopedDevice cursorHold(r->stream), badHold(r->stream);
    CUDA_TRY(poolAlloc(&cursorHold.p, sizeof(unsigned int) * totalRows, r->stream));
    unsigned int *const cursor = cursorHold.as<unsigned int>();
    CUDA_TRY(cudaMemsetAsync(cursor, 0, sizeof(unsigned int) * totalRows, r->stream));
    for(size_t gi = 0; gi < n; gi++) {
        const auto &g = groups[gi];
        if(!g.num_src) continue;
        nearCountKernel<<<std::min(1184u, (g.num_src + 7u) / 8u), 256, 0, r->stream>>>(g, cursor + rowBase[sourceOf[gi]]);
        CUDA_TRY(cudaPeekAtLastError());
        r->launches++;
    }
    std::vector<unsigned int> counts(totalRows);
    CUDA_TRY(cudaMemcpyAsync(counts.data(), cursor, sizeof(unsigned int) * totalRows, cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    std::vector<unsigned long long> firstCell(numNeuronGroups, 0ull);
    std::vector<unsigned int> shifts(numNeuronGroups, 0xFFFFFFFFu);
    unsigned long long cells = 0;
    for(size_t ni = 0; ni < numNeuronGroups; ni++) {
        bool isSource = false;
        for(size_t gi = 0; gi < n; gi++) isSource = isSource || sourceOf[gi] == ni;
        if(!isSource) continue;
        unsigned int longest = 0;
        for(unsigned long long row = rowBase[ni]; row < rowBase[ni + 1]; row++) longest = std::max(longest, counts[row]);
        unsigned int shift = 5;
        while((1u << shift) < longest) shift++;
        // a population most of whose synapses are near gains nothing from this schedule
        if(shift > 10) return B200_OK;
        firstCell[ni] = cells;
        shifts[ni] = shift;
        cells += (unsigned long long)r->neuronGroups[ni].num_neurons << shift;
    }
    if(cells >= (1ull << 33)) return B200_OK;      // 64 GB of table: not worth it
    CUDA_TRY(cudaMemsetAsync(cursor, 0, sizeof(unsigned int) * totalRows, r->stream));
    CUDA_TRY(poolAlloc(&badHold.p, sizeof(unsigned int), r->stream));
    unsigned int *const bad = badHold.as<unsigned int>();
    CUDA_TRY(cudaMemsetAsync(bad, 0, sizeof(unsigned int), r->stream));
    r->nearExported = forExport;
    CUDA_TRY(forExport ? cudaMalloc(&r->nearTable, sizeof(uint2) * (cells + 1)) : poolAlloc(&r->nearTable, sizeof(uint2) * (cells + 1), r->stream));
    CUDA_TRY(cudaMemsetAsync(r->nearTable, 0, sizeof(uint2) * (cells + 1), r->stream));
    for(size_t gi = 0; gi < n; gi++) {
        const auto &g = groups[gi];
        if(!g.num_src) continue;
        const unsigned int blocks = std::min(1184u, (g.num_src + 7u) / 8u);
        const unsigned int src = sourceOf[gi];
        const int e = withIndType(g.ind_bytes, [&](auto tag) -> int {
            using IndT = decltype(tag);
            nearFillKernel<IndT><<<blocks, 256, 0, r->stream>>>(g, ringOf[gi], cursor + rowBase[src],
                                                                r->nearTable + firstCell[src], shifts[src], bad);
            return B200_OK;
        });
        if(e) return e;
        CUDA_TRY(cudaPeekAtLastError());
        r->launches++;
    }
    unsigned int isBad = 0;
    CUDA_TRY(cudaMemcpyAsync(&isBad, bad, sizeof(unsigned int), cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    if(isBad) {
        r->freeNearTable();
        return B200_OK;
    }
    r->numRings = (unsigned int)rings.size();
    r->nearRingsHost = rings;
    r->nearCellHost = firstCell;
    r->nearShiftHost = shifts;
    if(forExport) return B200_OK;       // the owners of the source neurons take their rows from here
    std::vector<NearSpace> spaces(numNeuronGroups);
    for(size_t ni = 0; ni < numNeuronGroups; ni++) spaces[ni] = NearSpace{r->nearTable + firstCell[ni], shifts[ni], 0u, shifts[ni], 0u};
    CUDA_TRY(poolAlloc(&r->nearRings, sizeof(NearRing) * rings.size(), r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->nearRings, rings.data(), sizeof(NearRing) * rings.size(), cudaMemcpyHostToDevice, r->stream));
    CUDA_TRY(poolAlloc(&r->nearSpaces, sizeof(NearSpace) * spaces.size(), r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->nearSpaces, spaces.data(), sizeof(NearSpace) * spaces.size(), cudaMemcpyHostToDevice, r->stream));
    r->schedule = b200_runner::EMIT;
    return B200_OK;
}

// Choose the schedule of the persistent kernel from the dendritic delays that
// are actually in the arrays, and build what it needs:
//   LAG    every SPARSE group has a delay ring and no synapse arrives in the same
//          step: spikes are delivered one step late, one grid barrier per step;
//   SPLIT  the synapses that do arrive in the same step are copied into tables of
//          their own and delivered before the neuron update, all others after it;
//   PLAIN  everything before the neuron update.
int refreshSchedule(b200_runner *r)
{
    r->lagStale = false;
    r->lagEligible = false;
    r->schedule = b200_runner::PLAIN;
    r->dropUrgent();
    if(!r->fusedEligible) return B200_OK;
    const auto &groups = r->fusedGroups;
    const size_t n = groups.size();
    // rows of every group with a delay ring, one after the other, each group with one extra
    // cell so that offsets[row + 1] exists for its last row
    std::vector<size_t> rowBase(n, 0);
    size_t totalRows = 0;
    bool anyRing = false;
    for(size_t gi = 0; gi < n; gi++) {
        const auto &g = groups[gi];
        if(g.max_den_delay < 2 || !g.d || g.num_src == 0) continue;
        anyRing = true;
        rowBase[gi] = totalRows;
        totalRows += (size_t)g.num_src + 1;
    }
    if((r->useLag || r->useSplit) && anyRing && totalRows < (1ull << 31)) {
        CUDA_TRY(poolAlloc(&r->urgentOffsets, sizeof(unsigned int) * (totalRows + 1), r->stream));
        CUDA_TRY(cudaMemsetAsync(r->urgentOffsets, 0, sizeof(unsigned int) * (totalRows + 1), r->stream));
        for(size_t gi = 0; gi < n; gi++) {
            const auto &g = groups[gi];
            if(g.max_den_delay < 2 || !g.d || g.num_src == 0) continue;
            urgentCountKernel<<<std::min(1184u, (g.num_src + 7u) / 8u), 256, 0, r->stream>>>(g, r->urgentOffsets + rowBase[gi]);
            CUDA_TRY(cudaPeekAtLastError());
            r->launches++;
        }
        // counts -> offsets on the host (a few MB once per change of the delay arrays)
        std::vector<unsigned int> cells(totalRows + 1);
        CUDA_TRY(cudaMemcpyAsync(cells.data(), r->urgentOffsets, sizeof(unsigned int) * (totalRows + 1),
                                 cudaMemcpyDeviceToHost, r->stream));
        CUDA_TRY(cudaStreamSynchronize(r->stream));
        r->urgentStride.assign(n, 0u);
        unsigned long long total = 0;
        for(size_t gi = 0; gi < n; gi++) {
            const auto &g = groups[gi];
            if(g.max_den_delay < 2 || !g.d || g.num_src == 0) continue;
            unsigned int longest = 0;
            for(size_t row = 0; row <= g.num_src; row++) {
                unsigned int &cell = cells[rowBase[gi] + row];
                const unsigned int len = (row < g.num_src) ? cell : 0u;
                longest = std::max(longest, len);
                cell = (unsigned int)total;
                total += len;
            }
            r->urgentStride[gi] = longest;
        }
        // a list read one step late, with a peer possibly writing two steps ahead, needs delay + 4 slots
        bool lagOk = (total == 0);
        for(size_t gi = 0; gi < n; gi++) {
            const auto &g = groups[gi];
            if(g.max_den_delay < 2 || !g.d || g.axonal_delay + 4 > g.src_delay_slots) lagOk = false;
        }
        r->lagEligible = lagOk;
        if(r->useLag && lagOk && (!r->sharded() || r->lagAgreed)) {
            r->schedule = b200_runner::LAG;
        }
        else if(r->useEmit && r->sharded() && r->emitAgreed) {
            if(r->nearDataStale) {
                return fail(B200_ERR_STATE, "synapse arrays of a sharded model changed after its processes exchanged "
                                            "their near-synapse tables: run b200_near_export / import / finish again");
            }
            r->schedule = b200_runner::EMIT;        // tables exchanged between the processes beforehand
        }
        else if(r->useEmit && !r->sharded() && r->streamWarpsWanted != 0 && r->fusedStage) {
            const int e = buildNearTables(r);
            if(e) return e;
        }
        if(r->schedule != b200_runner::PLAIN) {
            // decided
        }
        else if(r->useSplit && total < (1ull << 31)) {
            r->schedule = b200_runner::SPLIT;
            if(total) {
                CUDA_TRY(cudaMemcpyAsync(r->urgentOffsets, cells.data(), sizeof(unsigned int) * (totalRows + 1),
                                         cudaMemcpyHostToDevice, r->stream));
                CUDA_TRY(poolAlloc(&r->urgentEntries, sizeof(uint2) * total, r->stream));
                std::vector<FusedUrgent> table(n);
                for(size_t gi = 0; gi < n; gi++) {
                    const auto &g = groups[gi];
                    table[gi] = FusedUrgent{r->urgentOffsets + rowBase[gi], r->urgentEntries, r->urgentStride[gi], 0u};
                    if(!r->urgentStride[gi]) continue;
                    const unsigned int blocks = std::min(1184u, (g.num_src + 7u) / 8u);
                    const int e = withIndType(g.ind_bytes, [&](auto tag) -> int {
                        using IndT = decltype(tag);
                        urgentFillKernel<IndT><<<blocks, 256, 0, r->stream>>>(g, r->urgentOffsets + rowBase[gi], r->urgentEntries);
                        return B200_OK;
                    });
                    if(e) return e;
                    CUDA_TRY(cudaPeekAtLastError());
                    r->launches++;
                }
                CUDA_TRY(poolAlloc(&r->fusedUrgent, sizeof(FusedUrgent) * n, r->stream));
                CUDA_TRY(cudaMemcpyAsync(r->fusedUrgent, table.data(), sizeof(FusedUrgent) * n, cudaMemcpyHostToDevice, r->stream));
                CUDA_TRY(cudaStreamSynchronize(r->stream));
            }
        }
        if(!r->urgentEntries) {
            poolFree(r->urgentOffsets, r->stream);
            r->urgentOffsets = nullptr;
            r->urgentStride.assign(n, 0u);
        }
    }
    return buildFusedTables(r);
}

// true if [p, p + bytes) overlaps an array the delay scan depends on
bool touchesDelays(const b200_runner *r, const void *p, size_t bytes)
{
    const unsigned char *a = static_cast<const unsigned char*>(p), *b = a + bytes;
    auto overlaps = [&](const void *start, size_t size) {
        const unsigned char *s0 = static_cast<const unsigned char*>(start);
        return s0 && a < s0 + size && b > s0;
    };
    for(const auto &g : r->fusedGroups) {
        if(!g.max_den_delay || !g.d) continue;
        const size_t synapses = (size_t)g.num_src * g.row_stride;
        // the urgent tables copy indices and weights, the schedule depends on delays and row lengths
        if(overlaps(g.d, synapses) || overlaps(g.row_length, sizeof(unsigned int) * g.num_src) ||
           overlaps(g.ind, synapses * g.ind_bytes) || overlaps(g.g, synapses * sizeof(float))) return true;
    }
    return false;
}

// Which arrays of SPARSE groups that private copies are made from [p, p + bytes) overlaps: 1 weights, 2 any other.
unsigned int touchesSparse(const b200_runner *r, const void *p, size_t bytes)
{
    const unsigned char *a = static_cast<const unsigned char*>(p), *b = a + bytes;
    auto overlaps = [&](const void *start, size_t size) {
        const unsigned char *s0 = static_cast<const unsigned char*>(start);
        return s0 && a < s0 + size && b > s0;
    };
    unsigned int which = 0;
    for(const auto &g : r->synapseGroups) {
        if(g.connectivity != B200_CONN_SPARSE || g.wu_model == B200_WU_STDP) continue;
        const size_t synapses = (size_t)g.num_src * g.row_stride;
        if(overlaps(g.g, synapses * sizeof(float))) which |= 1u;
        if(overlaps(g.d, synapses) || overlaps(g.row_length, sizeof(unsigned int) * g.num_src) || overlaps(g.ind, synapses * g.ind_bytes)) which |= 2u;
    }
    return which;
}

// [p, p + bytes) gets other values: the private copies made from it have to be made again before they are next used.
void arrayWritten(b200_runner *r, const void *p, size_t bytes)
{
    if(touchesDelays(r, p, bytes)) { r->lagStale = true; r->nearDataStale = true; }
    const unsigned int which = touchesSparse(r, p, bytes);
    if(!which) return;
    r->tiledStale = true;
    if(!r->residentReady || r->residentStale) {
        r->residentStale = true;
        return;
    }
    if(which & 2u) r->residentStale = true;
    else r->residentOld = true;
    // Filling takes 12 us and 6.2 for every million entries, making anew 100 and 60 (allocations, two waits); a step here takes some
    // 3.3 us less.  With rings the other path would have to make its own table of delay-0 and -1 synapses first, which takes longer.
    bool rings = false;
    for(unsigned int a = 0; a < r->resident.num_delays; a++) rings = rings || r->resident.kind[a] == RESIDENT_SPLIT;
    const double cost = r->residentStale ? 100.0 + 60.0 * r->residentCells : 12.0 + 6.2 * r->residentCells;
    r->residentRent = rings ? 0ull : (unsigned long long)(cost / 3.3);
}

// `goal`: not 0: the launch does what a launch of the target-resident kernel in front of it leaves of the steps up to there.
// `quick`: no time to look at the arrays.
int launchFused(b200_runner *r, unsigned long long numSteps, unsigned long long numRec, unsigned long long goal = 0, bool quick = false)
{
    if((goal || quick) && r->lagStale) {
        // the schedule that needs no private copies of them (at a hundred spikes a step and more it is as fast as the others)
        if(r->schedule != b200_runner::PLAIN) {
            r->schedule = b200_runner::PLAIN;
            r->dropUrgent();
            if(const int e = buildFusedTables(r)) return e;
        }
    }
    else if(r->lagStale) {
        const bool was = r->lagEligible;
        const int e = refreshSchedule(r);
        if(e) return e;
        if(r->sharded() && r->lagAgreed && r->useLag && was && !r->lagEligible) {
            return fail(B200_ERR_STATE, "a synapse with dendritic delay 0 appeared after the processes of this sharded "
                                        "model agreed to deliver spikes one step late");
        }
    }
    FusedLaunch L;
    L.lag = (r->schedule == b200_runner::LAG) ? 1u : 0u;
    L.skip_urgent = (r->schedule == b200_runner::SPLIT) ? 1u : 0u;
    L.urgent = r->fusedUrgent;
    L.stream_warps = r->streamWarps;
    L.slots_per_cta = r->slotsPerCta;
    L.emit = (r->schedule == b200_runner::EMIT) ? 1u : 0u;
    L.num_rings = r->numRings;
    L.near_rings = r->nearRings;
    L.near_spaces = r->nearSpaces;
    L.queue_words = (r->sharded() && L.emit && r->useNearQueues && r->queuesAgreed) ? r->queueWords : 0u;
    L.queue_count = NEAR_QUEUE_COUNT;
    L.publisher = (r->sharded() && r->streamWarps) ? 1u : 0u;
    L.queue_offset = r->queueOffset;
    L.neuron.groups = r->neuronTable.d;
    L.neuron.block_start = r->neuronTable.blockStart;
    L.neuron.num_groups = r->neuronTable.num;
    L.neuron.batch = 1;
    L.neuron.dt = r->dt;
    L.neuron.seed = r->seed;
    L.neuron.num_recording_timesteps = numRec;
    L.neuron.state = r->state;
    L.neuron.count_events = r->countEvents ? 1u : 0u;
    L.neuron.ahead = L.neuron.advance = 0u;
    L.slot_start = r->fusedSlotStart;
    L.sgroups = r->sparseTable.d;
    L.sources = r->fusedSources;
    L.items = r->fusedItems;
    L.num_sources = r->fusedNumSources;
    L.num_sgroups = r->sparseTable.num;
    L.num_items = r->fusedNumItems;
    L.stage_in_smem = r->fusedStage ? 1u : 0u;
    L.count_events = r->countEvents ? 1u : 0u;
    L.profile = r->fusedProfile ? 1u : 0u;
    L.cta_cycles = (r->fusedProfile && r->fusedGrid <= PROFILE_MAX_CTAS) ? r->fusedCtaCycles : nullptr;
    L.num_steps = numSteps;
    L.goal = goal;
    L.barrier = r->fusedBarrier;
    L.rank = r->rank;
    L.world = r->world;
    L.arena = r->arena;
    L.peer_table = r->peerTable;
    if(r->sharded()) {
        for(unsigned int p = 0; p < r->world; p++) {
            if(p != r->rank && !r->peerArena[p]) return fail(B200_ERR_STATE, "exchange arena of rank %u has not been opened", p);
        }
        for(const auto &g : r->neuronGroups) {
            const unsigned char *c = reinterpret_cast<const unsigned char*>(g.spk_cnt), *s = reinterpret_cast<const unsigned char*>(g.spk);
            const unsigned char *t = reinterpret_cast<const unsigned char*>(g.spk_tag);
            const unsigned char *w = reinterpret_cast<const unsigned char*>(g.spk_wire);
            if(c < r->arena || c >= r->arena + r->arenaBytes || s < r->arena || s >= r->arena + r->arenaBytes ||
               t < r->arena || t >= r->arena + r->arenaBytes || w < r->arena || w >= r->arena + r->arenaBytes) {
                return fail(B200_ERR_INVALID, "spike arrays of a sharded model must live in the exchange arena");
            }
        }
    }
    if(!goal) CUDA_TRY(cudaMemsetAsync(r->fusedBarrier, 0, sizeof(unsigned long long), r->stream));      // (else the launch in front of it did)
    void *args[] = {&L};
    CUDA_TRY(cudaLaunchCooperativeKernel(r->fusedKernel, dim3(r->fusedGrid), dim3(FUSED_BLOCK), args,
                                         r->fusedStage ? r->fusedSmemBytes : 0, r->stream));
    if(!goal) r->launches++;        // (two launches that share their steps count as one)
    r->fusedLaunches++;
    return B200_OK;
}

SynapseLaunch synapseLaunch(const b200_runner *r, const DeviceTable<b200_synapse_group> &t)
{
    SynapseLaunch L;
    L.groups = t.d;
    L.block_start = t.blockStart;
    L.num_groups = t.num;
    L.batch = r->batch;
    L.dt = r->dt;
    L.seed = r->seed;
    L.state = r->state;
    L.count_events = r->countEvents ? 1u : 0u;
    L.ahead = r->ahead;
    L.tiled_served = nullptr;
    return L;
}

struct ScopedTimer
{
    b200_runner *r;
    std::string name;
    bool on;
    ScopedTimer(b200_runner *r_, const std::string &n, bool capturing) : r(r_), name(n), on(r_->timing && !capturing)
    {
        if(on) cudaEventRecord(r->evA, r->stream);
    }
    ~ScopedTimer()
    {
        if(on) {
            cudaEventRecord(r->evB, r->stream);
            cudaEventSynchronize(r->evB);
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, r->evA, r->evB);
            r->timers[name].seconds += ms * 1e-3;
        }
    }
};

using TiledKernel = void (*)(const TiledLaunch);
TiledKernel tiledKernelFor(bool key16, bool weights)
{
    if(key16) return weights ? tiledDeliverKernel<uint16_t, true> : tiledDeliverKernel<uint16_t, false>;
    return weights ? tiledDeliverKernel<uint32_t, true> : tiledDeliverKernel<uint32_t, false>;
}

// (Re)build the private tile-major copy of the non-learning SPARSE groups (tiled.cuh).  Not on the
// time-step path: runs when the per-kernel path is first used and after the arrays it copies changed.
int buildTiled(b200_runner *r)
{
    r->dropTiled();
    r->tiledStale = false;
    r->tiledWhyNot.clear();
    if(!r->useTiled) { r->tiledWhyNot = "switched off"; return B200_OK; }
    if(r->sharded()) { r->tiledWhyNot = "sharded models run on the persistent kernel"; return B200_OK; }
    // the SPARSE groups in the order of sparseTable; the non-learning ones are served
    std::vector<b200_synapse_group> sparse;
    for(const auto &g : r->synapseGroups) if(g.connectivity == B200_CONN_SPARSE && !scatterServes(r, g)) sparse.push_back(g);
    std::vector<unsigned char> served(sparse.size(), 0);
    struct Target { float *ptr; unsigned int n, depth, stride, tiles, firstTile, firstTable, rows, firstSource; std::vector<size_t> groups; };
    std::vector<Target> targets;
    unsigned int maxDepth = 1;
    unsigned long long slots = 0;
    bool anyWeights = false;
    for(size_t i = 0; i < sparse.size(); i++) {
        const auto &g = sparse[i];
        if(g.wu_model == B200_WU_STDP || g.src_sections > 1) continue;
        float *ptr = g.max_den_delay ? g.den_delay : g.out_post;
        const unsigned int depth = std::max(1u, g.max_den_delay);
        auto it = std::find_if(targets.begin(), targets.end(), [&](const Target &t) { return t.ptr == ptr; });
        if(it == targets.end()) {
            targets.push_back(Target{ptr, g.num_trg, depth, 0, 0, 0, 0, 0, 0, {}});
            it = targets.end() - 1;
        }
        if(it->n != g.num_trg || it->depth != depth) { r->tiledWhyNot = "groups disagree on the shape of a shared target"; return B200_OK; }
        it->groups.push_back(i);
        served[i] = 1;
        maxDepth = std::max(maxDepth, depth);
        slots += (unsigned long long)g.num_src * g.row_stride;
        anyWeights = anyWeights || (g.g != nullptr && g.wu_model != B200_WU_STATIC_PULSE_CONSTANT_WEIGHT);
    }
    if(targets.empty()) { r->tiledWhyNot = "no non-learning SPARSE group"; return B200_OK; }
    for(const auto &t : targets) {
        if(t.groups.size() > TILED_MAX_SOURCES) { r->tiledWhyNot = "too many synapse groups onto one target"; return B200_OK; }
    }
    if(slots >= (1ull << 32)) { r->tiledWhyNot = "more than 2^32 synapse slots"; return B200_OK; }
    if(maxDepth > TILED_ACC_FLOATS || maxDepth > 4096u) { r->tiledWhyNot = "delay ring too deep for a shared-memory tile"; return B200_OK; }
    const bool key16 = (maxDepth <= 64u);
    const unsigned int postBits = key16 ? 10u : 20u;
    unsigned int numTiles = 0, entries = 0, numSources = 0;
    for(auto &t : targets) {
        t.stride = std::min(std::min(1u << postBits, TILED_ACC_FLOATS / t.depth), std::max(t.n, 1u));
        t.tiles = (t.n + t.stride - 1) / t.stride;
        t.rows = 1;
        for(size_t gi : t.groups) t.rows += sparse[gi].num_src;
        t.firstTile = numTiles;
        t.firstTable = entries;
        t.firstSource = numSources;
        const unsigned long long e = (unsigned long long)entries + (unsigned long long)t.tiles * t.rows;
        if(e >= (1ull << 32)) { r->tiledWhyNot = "run-start tables exceed 2^32 entries"; return B200_OK; }
        entries = (unsigned int)e;
        numTiles += t.tiles;
        numSources += (unsigned int)t.groups.size();
    }
    if(numTiles > 65535u) { r->tiledWhyNot = "more than 65535 tiles"; return B200_OK; }

    // ---- count, scan, place ---------------------------------------------------------------------
    ScopedDevice count(r->stream), runStart(r->stream), scanTemp(r->stream), keys(r->stream), weights(r->stream);
    CUDA_TRY(poolAlloc(&count.p, sizeof(unsigned int) * ((size_t)entries + 1), r->stream));
    CUDA_TRY(poolAlloc(&runStart.p, sizeof(unsigned int) * ((size_t)entries + 1), r->stream));
    CUDA_TRY(cudaMemsetAsync(count.p, 0, sizeof(unsigned int) * ((size_t)entries + 1), r->stream));
    std::vector<TiledBuildGroup> build;
    std::vector<TiledSource> sources;
    for(auto &t : targets) {
        unsigned int rowBase = 0;
        for(size_t gi : t.groups) {
            const auto &g = sparse[gi];
            TiledBuildGroup B{};
            B.row_length = g.row_length; B.ind = g.ind; B.d = g.max_den_delay ? g.d : nullptr;
            B.g = (g.wu_model == B200_WU_STATIC_PULSE_CONSTANT_WEIGHT) ? nullptr : g.g;
            B.num_src = g.num_src; B.row_stride = g.row_stride; B.ind_bytes = g.ind_bytes; B.num_trg = g.num_trg;
            B.depth = t.depth; B.first_tile = t.firstTile; B.stride = t.stride; B.row_base = rowBase;
            B.rows_per_tile = t.rows; B.first_table = t.firstTable; B.const_weight = g.wu_params[0];
            build.push_back(B);
            TiledSource S{};
            S.spk_cnt = g.src_spk_cnt; S.spk = g.src_spk; S.num_src = g.num_src; S.src_delay_slots = g.src_delay_slots;
            S.axonal_delay = g.axonal_delay; S.row_base = rowBase; S.const_weight = g.wu_params[0]; S.mean_row = 0.0f;
            sources.push_back(S);
            rowBase += g.num_src;
        }
    }
    auto launchBuild = [&](int pass) -> int {
        for(const auto &B : build) {
            const unsigned long long total = (unsigned long long)B.num_src * B.row_stride;
            if(!total) continue;
            const unsigned int blocks = (unsigned int)std::min<unsigned long long>((total + 255) / 256, 148ull * 16ull);
            if(key16) tiledBuildKernel<uint16_t><<<blocks, 256, 0, r->stream>>>(B, pass, count.as<unsigned int>(), runStart.as<unsigned int>(),
                                                                            keys.as<uint16_t>(), weights.as<float>(), postBits, r->state);
            else tiledBuildKernel<uint32_t><<<blocks, 256, 0, r->stream>>>(B, pass, count.as<unsigned int>(), runStart.as<unsigned int>(),
                                                                       keys.as<uint32_t>(), weights.as<float>(), postBits, r->state);
            r->launches++;
        }
        CUDA_TRY(cudaPeekAtLastError());
        return B200_OK;
    };
    if(const int e = launchBuild(0)) return e;
    size_t tempBytes = 0;
    CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tempBytes, count.as<unsigned int>(), runStart.as<unsigned int>(), (int)(entries + 1), r->stream));
    CUDA_TRY(poolAlloc(&scanTemp.p, std::max<size_t>(tempBytes, 16), r->stream));
    CUDA_TRY(cub::DeviceScan::ExclusiveSum(scanTemp.p, tempBytes, count.as<unsigned int>(), runStart.as<unsigned int>(), (int)(entries + 1), r->stream));
    unsigned int total = 0;
    CUDA_TRY(cudaMemcpyAsync(&total, runStart.as<unsigned int>() + entries, sizeof(total), cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    CUDA_TRY(poolAlloc(&keys.p, std::max<size_t>((size_t)total * (key16 ? 2 : 4), 16), r->stream));
    if(anyWeights) CUDA_TRY(poolAlloc(&weights.p, std::max<size_t>((size_t)total * sizeof(float), 16), r->stream));
    CUDA_TRY(cudaMemsetAsync(count.p, 0, sizeof(unsigned int) * ((size_t)entries + 1), r->stream));
    if(const int e = launchBuild(1)) return e;

    // ---- tiles, sources and (tile, source) pairs -----------------------------------------------------
    std::vector<unsigned int> hostRuns((size_t)entries + 1);
    CUDA_TRY(cudaMemcpyAsync(hostRuns.data(), runStart.p, sizeof(unsigned int) * hostRuns.size(), cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    std::vector<TiledTile> tiles(numTiles);
    std::vector<TiledPair> pairs;
    {
        size_t firstSource = 0;
        for(auto &t : targets) {
            std::vector<unsigned long long> groupSynapses(t.groups.size(), 0);
            for(unsigned int i = 0; i < t.tiles; i++) {
                TiledTile &T = tiles[t.firstTile + i];
                T.target = t.ptr; T.num_trg = t.n; T.depth = t.depth; T.first_trg = i * t.stride;
                T.num_tile = std::min(t.stride, t.n - i * t.stride); T.stride = t.stride;
                T.first_source = t.firstSource; T.num_sources = (unsigned int)t.groups.size();
                T.table = t.firstTable + i * t.rows;
                for(size_t si = 0; si < t.groups.size(); si++) {
                    const auto &g = sparse[t.groups[si]];
                    const size_t base = (size_t)T.table + sources[firstSource + si].row_base;
                    const unsigned long long syn = hostRuns[base + g.num_src] - hostRuns[base];
                    groupSynapses[si] += syn;
                    if(syn) {
                        pairs.push_back(TiledPair{(unsigned short)(t.firstTile + i), (unsigned short)si,
                                                  (float)((double)syn / std::max(1u, g.num_src))});
                    }
                }
            }
            // per source: synapses per source neuron, for the event estimate of a step
            for(size_t si = 0; si < t.groups.size(); si++) {
                const auto &g = sparse[t.groups[si]];
                sources[firstSource + si].mean_row = g.num_src ? (float)((double)groupSynapses[si] / g.num_src) : 0.0f;
            }
            firstSource += t.groups.size();
        }
    }
    if(pairs.empty()) { r->tiledWhyNot = "no synapses"; return B200_OK; }
    if((unsigned long long)pairs.size() * r->batch >= (1ull << 31)) { r->tiledWhyNot = "too many (tile, source, batch) pairs"; return B200_OK; }
    int sms = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
    const unsigned int grid = (unsigned int)sms;
    size_t smem = 0;
    for(const auto &T : tiles) smem = std::max(smem, sizeof(float) * T.depth * T.stride);
    auto toDevice = [&](const void *host, size_t bytes, void **out) -> int {
        CUDA_TRY(poolAlloc(out, std::max<size_t>(bytes, 16), r->stream));
        CUDA_TRY(cudaMemcpyAsync(*out, host, bytes, cudaMemcpyHostToDevice, r->stream));
        return B200_OK;
    };
    int e = toDevice(tiles.data(), sizeof(TiledTile) * tiles.size(), (void**)&r->tiledTiles);
    if(!e) e = toDevice(sources.data(), sizeof(TiledSource) * sources.size(), (void**)&r->tiledSources);
    if(!e) e = toDevice(pairs.data(), sizeof(TiledPair) * pairs.size(), (void**)&r->tiledPairs);
    if(!e) e = toDevice(served.data(), served.size(), (void**)&r->tiledServed);
    if(e) { r->dropTiled(); return e; }
    // scratch of the per-step work partition
    {
        const size_t perStep = pairs.size() * r->batch;
        cudaError_t ce = poolAlloc(&r->tiledPairBatches, sizeof(unsigned int) * perStep, r->stream);
        if(ce == cudaSuccess) ce = poolAlloc(&r->tiledPairPrefix, sizeof(double) * perStep, r->stream);
        if(ce == cudaSuccess) ce = poolAlloc(&r->tiledCtaStart, sizeof(unsigned int) * 2 * (grid + 1), r->stream);
        if(ce != cudaSuccess) { r->dropTiled(); CUDA_TRY(ce); }
    }
    CUDA_TRY(cudaFuncSetAttribute(tiledKernelFor(key16, anyWeights), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    r->tiledRunStart = static_cast<unsigned int*>(runStart.release());
    r->tiledKeys = keys.release();
    r->tiledWeights = static_cast<float*>(weights.release());
    r->tiledNumPairs = (unsigned int)pairs.size();
    r->tiledNumSources = numSources;
    r->tiledPostBits = postBits;
    r->tiledGrid = grid;
    r->tiledSmemBytes = smem;
    r->tiledSynapses = total;
    if(const int err = ensurePeak(r)) return err;
    r->tiledReady = true;
    {
        unsigned long long neurons = 0;
        for(const auto &ng : r->neuronGroups) neurons += ng.num_neurons;
        r->eventsPerSpike = neurons ? (double)r->tiledSynapses / (double)neurons : 0.0;
    }
    return B200_OK;
}

TiledLaunch tiledLaunch(const b200_runner *r)
{
    TiledLaunch L;
    L.ahead = r->ahead;
    L.tiles = r->tiledTiles; L.sources = r->tiledSources; L.run_start = r->tiledRunStart; L.keys = r->tiledKeys;
    L.weights = r->tiledWeights; L.pairs = r->tiledPairs; L.pair_batches = r->tiledPairBatches;
    L.pair_prefix = r->tiledPairPrefix; L.cta_start = r->tiledCtaStart; L.num_pairs = r->tiledNumPairs;
    L.num_sources = r->tiledNumSources; L.grid = r->tiledGrid;
    L.batch = r->batch; L.post_bits = r->tiledPostBits; L.min_events = r->tiledMinEvents; L.state = r->state;
    L.count_events = r->countEvents ? 1u : 0u;
    L.ticket_events = r->tiledTicketEvents; L.ticket_cost = r->tiledTicketCost;
    L.profile = (r->fusedProfile && r->tiledGrid <= PROFILE_MAX_CTAS) ? r->fusedCtaCycles : nullptr;
    return L;
}

// Counts (pass 0) or places (pass 1) the synapses of the target-resident kernel's copy.  Placed again over what it holds, other
// weights of the same synapses fill the same places (in another order within a run).
int residentPass(b200_runner *r, int which, unsigned int *longest, unsigned long long *totals)
{
    const ResidentLaunch &L = r->resident;
    const size_t numGroups = r->neuronGroups.size(), runsPerCta = (size_t)L.num_delays * numGroups;
    int sms = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
    for(const auto &pr : r->residentPairs) {
        ResidentBuild B;
        B.groups = r->residentGroups + pr.first;
        B.target = r->residentTargets + pr.first;
        B.num_groups = pr.count;
        B.num_src = r->neuronGroups[pr.src].num_neurons;
        B.unit_start = L.unit_start; B.columns = L.columns; B.depth = r->residentDepths; B.grid = r->residentGrid;
        B.runs_stride = (unsigned int)runsPerCta;
        if(!B.num_src) continue;
        const size_t at = (size_t)pr.delay_class * numGroups + pr.src;
        B.late = (L.kind[pr.delay_class] == RESIDENT_LATE);
        B.split = (L.kind[pr.delay_class] == RESIDENT_SPLIT);
        // longest run of every (CTA, pair), then longest head of every pair
        B.near_longest = longest ? longest + runsPerCta * r->residentGrid + at : nullptr;
        B.synapses = totals ? totals + at : nullptr;
        CUDA_TRY(residentBuild(B, which, longest ? longest + at : nullptr, L.runs ? L.runs + at : nullptr, const_cast<uint2*>(L.entries), r->state,
                               std::min(B.num_src, (unsigned int)sms * 8u), r->stream));
        r->launches++;
    }
    return B200_OK;
}

// (Re)build the tables of the target-resident kernel; leaves residentReady false, with the reason, where the model does
// not qualify.  Runs when a block of steps is first asked for and after the arrays it copies changed.
int buildResident(b200_runner *r)
{
    r->dropResident();
    r->residentStale = r->residentOld = false;
    r->residentRent = 0;
    r->residentBuilds++;
    r->residentWhyNot.clear();
    auto no = [&](const char *why) { r->residentWhyNot = why; return B200_OK; };
    if(r->batch != 1 || r->sharded()) return no("batch or sharded model");
    const size_t numGroups = r->neuronGroups.size();
    if(!numGroups || numGroups > RESIDENT_MAX_GROUPS || r->synapseGroups.empty()) return no("no groups, or too many");
    int sms = 0, coop = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
    CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, r->device));
    if(!coop) return no("no cooperative launch");
    ResidentLaunch &L = r->resident;
    L = ResidentLaunch{};
    r->residentHandsOver = r->fusedEligible;

    // ---- ring depths, axonal delays, who feeds whom --------------------------------------------------------
    std::vector<unsigned int> unitStart{0}, depths, delays;
    unsigned int maxSlots = 0;
    for(const auto &g : r->neuronGroups) {
        if(g.first_neuron != 0 || g.num_update != g.num_neurons || g.num_neurons >= (1u << 24)) return no("partly updated population");
        if(g.spike_times) return no("spike times");
        unitStart.push_back(unitStart.back() + (g.num_neurons + 31u) / 32u);
        maxSlots = std::max(maxSlots, g.num_delay_slots);
        for(unsigned int p = 0; p < g.num_psm; p++) {
            const unsigned int d = std::max(1u, g.psm[p].max_den_delay);
            if(std::find(depths.begin(), depths.end(), d) == depths.end()) depths.push_back(d);
        }
    }
    if(depths.empty()) depths.push_back(1u);
    const unsigned int units = unitStart.back();
    if(depths.size() > RESIDENT_CLASSES || units == 0) return no("too many ring depths");
    struct Link { size_t syn; unsigned int src, trg, psm, delayClass; };
    std::vector<Link> links;
    for(size_t i = 0; i < r->synapseGroups.size(); i++) {
        const auto &g = r->synapseGroups[i];
        if(g.connectivity == B200_CONN_PROCEDURAL || g.wu_model == B200_WU_STDP) return no("procedural or learning group");
        Link l{i, ~0u, ~0u, 0u, 0u};
        for(unsigned int ni = 0; ni < numGroups; ni++) {
            const auto &ng = r->neuronGroups[ni];
            if(ng.spk_cnt == g.src_spk_cnt && ng.num_neurons == g.num_src) l.src = ni;
            for(unsigned int p = 0; p < ng.num_psm; p++) {
                const bool same = g.max_den_delay ? (ng.psm[p].den_delay == g.den_delay && ng.psm[p].max_den_delay == g.max_den_delay)
                                                  : (!ng.psm[p].max_den_delay && ng.psm[p].out_post == g.out_post);
                if(same && ng.num_neurons == g.num_trg) { l.trg = ni; l.psm = p; }
            }
        }
        if(l.src == ~0u || l.trg == ~0u) return no("a group's source or target is not a population of the model");
        auto it = std::find(delays.begin(), delays.end(), g.axonal_delay);
        if(it == delays.end()) { delays.push_back(g.axonal_delay); it = delays.end() - 1; }
        l.delayClass = (unsigned int)(it - delays.begin());
        links.push_back(l);
    }
    if(delays.size() > RESIDENT_CLASSES) return no("too many axonal delays");
    const unsigned int numDelays = (unsigned int)delays.size();
    // what of each class has to be delivered before the neuron update (resident.h)
    bool anyLate = false;
    for(unsigned int a = 0; a < numDelays; a++) {
        bool rings = true, noRing = true;
        for(const auto &l : links) {
            const auto &g = r->synapseGroups[l.syn];
            if(l.delayClass != a) continue;
            if(g.connectivity != B200_CONN_SPARSE || g.max_den_delay < 2) rings = false;
            if(g.max_den_delay) noRing = false;
        }
        L.kind[a] = rings ? RESIDENT_SPLIT : (noRing && delays[a] >= 1u) ? RESIDENT_LATE : RESIDENT_IMMEDIATE;
        anyLate = anyLate || L.kind[a] == RESIDENT_LATE;
    }
    // buffers per input: the ring, one, or two that a LATE class fills and empties in turn
    for(auto &d : depths) if(d == 1u && anyLate) d = 2u;
    std::sort(depths.begin(), depths.end());
    depths.erase(std::unique(depths.begin(), depths.end()), depths.end());
    auto depthOf = [&](const b200_psm &psm) {
        const unsigned int d = psm.max_den_delay ? psm.max_den_delay : anyLate ? 2u : 1u;
        return (unsigned int)(std::find(depths.begin(), depths.end(), d) - depths.begin());
    };

    // ---- windows of steps (resident_window.cuh) ----------------------------------------------------------------
    ResidentWindow &win = r->window;
    win = ResidentWindow{};
    bool windowed = r->useWindow && numDelays == 1 && depths.size() == 1;
    unsigned long long sourceGroups = 0, freeGroups = 0, sourceNeurons = 0;
    for(const auto &l : links) sourceGroups |= 1ull << l.src;
    for(size_t ni = 0; ni < numGroups; ni++) {
        const auto &g = r->neuronGroups[ni];
        for(unsigned int p = 0; p < g.num_psm; p++) windowed = windowed && !g.psm[p].max_den_delay;
        if(!((sourceGroups >> ni) & 1ull)) continue;
        sourceNeurons += g.num_neurons;
        if((g.model == B200_NEURON_POISSON || g.model == B200_NEURON_SPIKE_SOURCE_ARRAY) && !g.num_psm && !g.num_cs) freeGroups |= 1ull << ni;
    }
    if(windowed) {
        const unsigned int after = delays[0] + 1u;
        if(freeGroups == sourceGroups) {
            // (a list that holds every source: a launch cannot stop short of where the sources have got to)
            win.feed = 1u;
            win.free_groups = freeGroups;
            win.steps = (unsigned int)std::min<unsigned long long>(RESIDENT_WINDOW_MOST, RESIDENT_WINDOW_LIST / std::max(1ull, sourceNeurons));
            win.cap = (unsigned int)std::min<unsigned long long>(sourceNeurons, RESIDENT_WINDOW_LIST);
            win.buffers = 4u;
        }
        else {
            for(win.lag = 1; after % win.lag || after / win.lag > RESIDENT_WINDOW_MOST; win.lag++) {}
            win.steps = after / win.lag;
            win.cap = (unsigned int)std::min<unsigned long long>(sourceNeurons, RESIDENT_LIST);
            win.buffers = windowBuffers(2u * win.lag + 2u);
            windowed = win.cap >= sourceNeurons || r->residentHandsOver;      // (before it is rounded up)
        }
        win.cap = (win.cap + 3u) & ~3u;         // (entries are read four at a time)
        windowed = windowed && win.steps >= RESIDENT_WINDOW_LEAST;
    }

    // ---- how many CTAs, how many warps ----------------------------------------------------------------------
    const NeuronShape shape = neuronShape(r);
    cudaFuncAttributes attr{};
    const bool oneClass = depths.size() == 1 && numDelays == 1;
    CUDA_TRY(cudaFuncGetAttributes(&attr, residentKernelFor(shape.npsm, shape.ncs, oneClass, RESIDENT_BLOCK)));     // (both instances share as much)
    unsigned int numSpans = 0;
    for(const auto &l : links) numSpans += (r->synapseGroups[l.syn].connectivity != B200_CONN_SPARSE);
    const unsigned int longestDelay = *std::max_element(delays.begin(), delays.end()), shortest = *std::min_element(delays.begin(), delays.end());
    const unsigned int history = std::min(longestDelay + 1u, maxSlots);
    // event counts of Poisson sources: the cumulative probabilities b200_poisson_inverse would add up
    std::vector<float> poisson;
    if(shape.ncs == 1) {
        for(const auto &g : r->neuronGroups) {
            float p = g.num_cs ? g.cs[0].params[2] : 1.0f, sum = p;
            for(unsigned int i = 0; i < 64u; i++) {
                poisson.push_back(sum);
                p = B200_FDIV(B200_FMUL(p, g.cs[0].params[3]), (float)(i + 1u));
                sum = B200_FADD(sum, p);
            }
        }
    }
    size_t tables = 0;
    auto place = [&](size_t bytes) { const unsigned int at = (unsigned int)tables; tables += align16(bytes); return at; };
    L.at.groups = place(sizeof(b200_neuron_group) * numGroups);
    L.at.unit_start = place(sizeof(unsigned int) * (numGroups + 1));
    L.at.unit_first = place(sizeof(unsigned int) * units);
    L.at.columns = place(sizeof(unsigned int) * RESIDENT_UNITS * B200_MAX_PSM);
    L.at.runs = place(sizeof(ResidentRun) * numDelays * numGroups);
    L.at.rows = place(sizeof(unsigned long long) * numDelays * numGroups);
    L.at.spans = place(sizeof(ResidentSpan) * numSpans);
    L.at.poisson = place(sizeof(float) * poisson.size());
    bool draws = false;
    for(const auto &g : r->neuronGroups) draws = draws || g.model == B200_NEURON_POISSON;
    L.at.undrawn = place(draws ? sizeof(unsigned int) * RESIDENT_BLOCK : 0);
    L.at.history = place(sizeof(unsigned int) * history * RESIDENT_UNITS);
    L.at.acc = place(0);
    int optin = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, r->device));
    const size_t room = (size_t)optin - attr.sharedSizeBytes;
    size_t windowRoom = 0;
    if(windowed) {
        CUDA_TRY(cudaFuncGetAttributes(&attr, residentWindowKernelFor(shape.npsm, shape.ncs)));
        windowRoom = (size_t)optin - attr.sharedSizeBytes;
        win.ring = std::max(history, win.steps);
    }
    auto groupOf = [&](unsigned int u) { return (unsigned int)(std::upper_bound(unitStart.begin(), unitStart.end(), u) - unitStart.begin()) - 1u; };
    std::vector<unsigned int> columns, ctaColumns;
    unsigned int grid = 0;
    size_t accFloats = 0;
    auto layOut = [&](unsigned int G) {
        columns.assign((size_t)G * RESIDENT_UNITS * B200_MAX_PSM, 0u);
        ctaColumns.assign((size_t)G * RESIDENT_CLASSES, 0u);
        accFloats = 0;
        for(unsigned int c = 0; c < G; c++) {
            size_t floats = 0;
            for(unsigned int u = c, w = 0; u < units; u += G, w++) {
                const auto &g = r->neuronGroups[groupOf(u)];
                for(unsigned int p = 0; p < g.num_psm; p++) {
                    const unsigned int cls = depthOf(g.psm[p]);
                    unsigned int &cols = ctaColumns[(size_t)c * RESIDENT_CLASSES + cls];
                    columns[((size_t)c * RESIDENT_UNITS + w) * B200_MAX_PSM + p] = (cls << 16) | cols;
                    cols += 32u;
                }
            }
            for(size_t k = 0; k < depths.size(); k++) floats += (size_t)depths[k] * ctaColumns[(size_t)c * RESIDENT_CLASSES + k];
            accFloats = std::max(accFloats, floats);
        }
    };
    const unsigned int most = std::min<unsigned int>((unsigned int)sms, RESIDENT_MAX_CTAS);
    auto copiesFor = [](unsigned int G) { return std::min(32u, (G + RESIDENT_READERS - 1u) / RESIDENT_READERS); };
    // the list and the ballots lie where the other kernel's input buffers begin, the buffers of a window behind them
    auto windowBytes = [&] {
        win.list_at = L.at.history;
        win.words_at = win.list_at + (unsigned int)align16(sizeof(unsigned int) * win.steps * win.cap);
        win.acc_at = win.words_at + (unsigned int)align16(sizeof(unsigned int) * win.ring * RESIDENT_UNITS);
        return win.acc_at + accFloats / depths[0] * win.steps * sizeof(float);
    };
    if(windowed) {
        // (a window's messages cost little, and its deliveries and updates are shared by all SMs.  us a step on 48 / 100 / 148 CTAs: 1000 ->
        // 10 000 neurons 0.30 / 0.26 / 0.26, BITMASK 2003 x 5009 0.60 / 0.50 / 0.49, DENSE 4096 x 4096 1.11 / 1.04 / 0.85, 100 000 neurons
        // with conductances 1.35 / 1.36 / 1.32.)  Calls of one to three steps go through them one by one on the same grid, for which
        // the synapses are laid out: us a call of 1 / 2 / 3 steps, here and on the grid of the rule below: 1000 -> 10 000 10.2 / 12.8 /
        // 16.0 and 10.0 / 12.4 / 14.4, BITMASK 11.7 / 16.5 / 20.6 and 11.3 / 16.5 / 19.7, 5000 neurons with conductances 10.9 / 14.6 / 17.1 and
        // 10.7 / 13.9 / 17.0, 100 000 14.3 / 20.8 / 26.2 and 14.5 / 20.7 / 26.2; with a fetch behind each call 30.0 - 50.4 and 30.0 - 50.0.
        const unsigned int G = std::min(std::max(r->residentCtas ? r->residentCtas : most, (units + RESIDENT_UNITS - 1u) / RESIDENT_UNITS), std::min(most, units));
        // Messages: room for every neuron in every step of `buffers` windows, about as much as a spike queue of that delay (100 000 neurons, 199
        // steps: 84 MB beside 81).  No more than a quarter of the free memory (what the pool may keep needs no asking).
        const unsigned int perCta = (units + G - 1u) / G;
        win.body = perCta * 32u * win.steps;
        const size_t headBytes = sizeof(ulonglong2) * win.buffers * copiesFor(G) * RESIDENT_HEADS;
        r->windowMailBytes = headBytes + sizeof(unsigned short) * win.buffers * G * win.body;
        size_t freeBytes = POOL_KEEP * 4, totalBytes = 0;
        if(r->windowMailBytes > freeBytes / 4) CUDA_TRY(cudaMemGetInfo(&freeBytes, &totalBytes));
        if(perCta <= RESIDENT_UNITS && r->windowMailBytes <= freeBytes / 4) {
            layOut(G);
            r->windowSmem = windowBytes();
            if(tables + accFloats * sizeof(float) <= room && r->windowSmem <= windowRoom) grid = G;
        }
        windowed = grid != 0u;
    }
    if(!windowed) {
        // Units of 32 neurons for a CTA.  More CTAs share the work of a step but lengthen the exchange.  us a step, this rule / the
        // best of seven grids from 16 to 148 CTAs (at which): SPARSE 1000 + 1000 3.0 / 2.9 (64), 3000 3.5 / 3.5, 5000 4.2 / 4.2,
        // 10 000 4.4 / 3.8 (32), 20 000 6.3 / 5.3 (64), 50 000 6.8 / 6.7; with rings 1000 2.6 / 2.5, 3000 3.4 / 3.1 (16), 8000 5.9
        // / 4.4 (32), 20 000 7.9 / 7.8; DENSE 1000 x 1000 2.9 / 2.7 (64), 2000 x 2000 3.5 / 3.2 (148), 1000 x 4000 3.3 / 3.2, 8000 x
        // 8000 8.1 / 8.1; BITMASK 2000 x 2000 3.7 / 3.2 (148), 1000 x 4000 3.5 / 3.1 (32), 8000 x 8000 5.0 / 4.8.  So the lines are
        // coarse: within a fifth of the best in all of 25 but one.
        bool rings = false;
        for(unsigned int a = 0; a < numDelays; a++) rings = rings || L.kind[a] == RESIDENT_SPLIT;
        const unsigned int perCta = numSpans ? 2u : rings ? 4u : 10u;
        unsigned int G = r->residentCtas ? r->residentCtas : std::max(32u, (units + perCta - 1u) / perCta);
        G = std::min(std::min(std::max(G, (units + RESIDENT_UNITS - 1u) / RESIDENT_UNITS), most), units);
        for(;; G = std::min(most, G + (G + 7u) / 8u)) {
            if((units + G - 1u) / G <= RESIDENT_UNITS) {
                layOut(G);
                if(tables + accFloats * sizeof(float) <= room) { grid = G; break; }
            }
            if(G == most) break;
        }
        if(!grid) return no("more neurons, or deeper rings, than the SMs hold");
    }
    const unsigned int neuronWarps = (units + grid - 1u) / grid;
    // (warps without neurons ask for the messages and build this CTA's own)
    unsigned int warps = r->residentWarps ? r->residentWarps : std::max(numSpans ? 16u : 8u, neuronWarps + (grid + 31u) / 32u);
    if(neuronWarps <= RESIDENT_FEW / 32u && !r->residentWarps) warps = std::min(warps, RESIDENT_FEW / 32u);
    warps = std::min(std::max(warps, std::max(neuronWarps, (grid + 31u) / 32u)), RESIDENT_UNITS);
    r->windowBlock = 32u * (r->residentWarps ? warps : RESIDENT_UNITS);
    r->residentKernel = residentKernelFor(shape.npsm, shape.ncs, oneClass, warps * 32u);

    auto device = [&](size_t bytes, void **out) -> int {
        CUDA_TRY(poolAlloc(out, std::max<size_t>(bytes, 16), r->stream));
        r->residentBuffers.push_back(*out);
        return B200_OK;
    };
    auto upload = [&](const void *host, size_t bytes, void **out) -> int {
        if(const int err = device(bytes, out)) return err;
        CUDA_TRY(cudaMemcpyAsync(*out, host, bytes, cudaMemcpyHostToDevice, r->stream));
        return B200_OK;
    };
    std::vector<unsigned int> unitFirst(units);
    for(unsigned int u = 0; u < units; u++) unitFirst[u] = (groupOf(u) << 24) | ((u - unitStart[groupOf(u)]) * 32u);
    unsigned int *dUnitStart = nullptr, *dUnitFirst = nullptr, *dColumns = nullptr, *dCtaColumns = nullptr, *dDepths = nullptr;
    if(const int err = upload(unitStart.data(), sizeof(unsigned int) * unitStart.size(), (void**)&dUnitStart)) return err;
    if(const int err = upload(unitFirst.data(), sizeof(unsigned int) * unitFirst.size(), (void**)&dUnitFirst)) return err;
    if(const int err = upload(columns.data(), sizeof(unsigned int) * columns.size(), (void**)&dColumns)) return err;
    if(const int err = upload(ctaColumns.data(), sizeof(unsigned int) * ctaColumns.size(), (void**)&dCtaColumns)) return err;
    if(const int err = upload(depths.data(), sizeof(unsigned int) * depths.size(), (void**)&dDepths)) return err;

    // ---- runs of the SPARSE groups ----------------------------------------------------------------------------
    const size_t runsPerCta = (size_t)numDelays * numGroups;
    std::vector<ResidentRun> runs(runsPerCta * grid, ResidentRun{0, 0, 0});
    std::vector<b200_synapse_group> sorted;
    std::vector<unsigned int> targets;
    std::vector<b200_runner::ResidentPair> &pairs = r->residentPairs;
    pairs.clear();
    for(unsigned int a = 0; a < numDelays; a++) {
        for(unsigned int ni = 0; ni < numGroups; ni++) {
            b200_runner::ResidentPair pr{a, ni, (unsigned int)sorted.size(), 0u};
            for(const auto &l : links) {
                const auto &g = r->synapseGroups[l.syn];
                if(l.delayClass != a || l.src != ni) continue;
                L.sources[a] |= 1ull << ni;
                if(g.connectivity != B200_CONN_SPARSE) continue;
                sorted.push_back(g);
                targets.push_back((l.trg << 8) | l.psm);
                pr.count++;
            }
            if(pr.count) pairs.push_back(pr);
        }
    }
    for(unsigned int a = 0; a < numDelays; a++) L.source_groups |= L.sources[a];
    std::vector<unsigned long long> rowStarts(runsPerCta, 0ull);
    r->residentCells = 0.0;
    L.num_delays = numDelays;
    ResidentRun *dRuns = nullptr;
    uint2 *dEntries = nullptr;
    if(!pairs.empty()) {
        unsigned long long cells = 0;
        ScopedDevice totals(r->stream), longest(r->stream);
        if(const int err = upload(sorted.data(), sizeof(b200_synapse_group) * sorted.size(), (void**)&r->residentGroups)) return err;
        if(const int err = upload(targets.data(), sizeof(unsigned int) * targets.size(), (void**)&r->residentTargets)) return err;
        r->residentDepths = dDepths;
        L.unit_start = dUnitStart;
        L.columns = dColumns;
        r->residentGrid = grid;
        const size_t numLongest = runs.size() + runsPerCta;
        CUDA_TRY(poolAlloc(&longest.p, sizeof(unsigned int) * numLongest, r->stream));
        CUDA_TRY(poolAlloc(&totals.p, sizeof(unsigned long long) * runsPerCta, r->stream));
        std::vector<unsigned long long> synapses(runsPerCta, 0ull);
        std::vector<unsigned int> longestHost(numLongest);
        auto count = [&]() -> int {
            CUDA_TRY(cudaMemsetAsync(longest.p, 0, sizeof(unsigned int) * numLongest, r->stream));
            CUDA_TRY(cudaMemsetAsync(totals.p, 0, sizeof(unsigned long long) * runsPerCta, r->stream));
            if(const int err = residentPass(r, 0, longest.as<unsigned int>(), totals.as<unsigned long long>())) return err;
            CUDA_TRY(cudaMemcpyAsync(synapses.data(), totals.p, sizeof(unsigned long long) * runsPerCta, cudaMemcpyDeviceToHost, r->stream));
            CUDA_TRY(cudaMemcpyAsync(longestHost.data(), longest.p, sizeof(unsigned int) * numLongest, cudaMemcpyDeviceToHost, r->stream));
            CUDA_TRY(cudaStreamSynchronize(r->stream));
            return B200_OK;
        };
        if(const int err = count()) return err;
        // the heads stand in front of the update: worth it while they are a few loads
        bool again = false;
        for(size_t pair = 0; pair < runsPerCta; pair++) {
            if(longestHost[runs.size() + pair] > RESIDENT_NEAR_MOST && L.kind[pair / numGroups] == RESIDENT_SPLIT) {
                L.kind[pair / numGroups] = RESIDENT_IMMEDIATE;
                again = true;
            }
        }
        if(again) if(const int err = count()) return err;
        for(size_t pair = 0; pair < runsPerCta; pair++) {
            const unsigned int near = longestHost[runs.size() + pair], a = (unsigned int)(pair / numGroups);
            unsigned int row = 0;
            for(unsigned int c = 0; c < grid; c++) {
                ResidentRun &run = runs[c * runsPerCta + pair];
                run.place = ((unsigned long long)near << 48) | (cells + row);
                run.length = ((near + longestHost[c * runsPerCta + pair] + 3u) & ~3u) - near;
                row += near + run.length;
                L.chunks[a] = std::max(L.chunks[a], (run.length + RESIDENT_CHUNK - 1u) / RESIDENT_CHUNK);
                win.run_groups = std::max(win.run_groups, (run.length + 31u) / 32u);
            }
            rowStarts[pair] = cells;
            cells += (unsigned long long)row * r->neuronGroups[pair % numGroups].num_neurons;
            L.near_most[a] = std::max(L.near_most[a], near);
            for(unsigned int c = 0; c < grid; c++) runs[c * runsPerCta + pair].row = row;
        }
        for(unsigned int a = 0; a < numDelays; a++) L.near_share[a] = L.near_most[a] ? (unsigned int)(((1ull << 32) + L.near_most[a] - 1u) / L.near_most[a]) : 0u;
        // what a spike costs here above what it costs the kernel with a grid barrier
        r->residentWorst = r->residentSources = 0.0;
        r->residentSteeper = false;
        for(unsigned int a = 0; a < numDelays; a++) {
            double sources = 0.0, all = 0.0;
            for(size_t ni = 0; ni < numGroups; ni++) {
                if(!((L.sources[a] >> ni) & 1ull)) continue;
                sources += r->neuronGroups[ni].num_neurons;
                all += (double)synapses[a * numGroups + ni];
            }
            const double here = (RESIDENT_RUN_COST * L.chunks[a] + RESIDENT_NEAR_COST * L.near_most[a] / 32.0) / warps;
            // (a model that the grid-barrier kernels do not take has only presynapticSparseKernel, no faster than this one per
            // spike, and the tiled kernels, whose launches and flush take some 35 us)
            const double there = !r->residentHandsOver ? 0.0 : (L.kind[a] == RESIDENT_SPLIT ? 0.02 : 0.0085) * all / std::max(1.0, sources);
            L.weight[a] = (unsigned int)std::min(std::max(0.0, here - there) + 0.5, (double)RESIDENT_MOST_WEIGHT);
            if(windowed) {
                const double inWindows = RESIDENT_WINDOW_COST * win.run_groups * 32.0 / r->windowBlock;
                r->windowWeight = (unsigned int)std::min(std::max(0.0, inWindows - there) + 0.5, (double)RESIDENT_MOST_WEIGHT);
            }
            r->residentSources += sources;
            r->residentSteeper = r->residentSteeper || (L.kind[a] == RESIDENT_SPLIT && L.weight[a]);
            r->residentWorst += sources * L.weight[a] + std::max(0.0, sources / RESIDENT_LIST - 1.0) * RESIDENT_PIECE_COST;
            // (with rings the exchange, which grows with the grid, and the heads stand in front of the update: at ten spikes a step
            // 63 CTAs gain 3.0 us on the other kernel, 148 gain 1.5)
            const unsigned int spare = !r->residentHandsOver ? 35000u : (L.kind[a] == RESIDENT_LATE) ? 4000u :
                (L.kind[a] == RESIDENT_SPLIT) ? 4500u - std::min(2500u, 15u * grid) : 3300u;
            L.spare = L.spare ? std::min(L.spare, spare) : spare;
        }
        for(unsigned int a = 0; a < numDelays; a++) L.quiet[a] = L.weight[a] ? L.spare / (2u * L.weight[a]) : RESIDENT_LIST;
        // padded runs of a network with few synapses per (source neuron, CTA) pair can take several times the room of its
        // arrays: the copy may use a quarter of what is free
        size_t freeBytes = POOL_KEEP * 4, totalBytes = 0;       // (what the pool may keep needs no asking)
        if(cells * sizeof(uint2) > freeBytes / 4) CUDA_TRY(cudaMemGetInfo(&freeBytes, &totalBytes));
        if(cells * sizeof(uint2) > freeBytes / 4) { r->dropResident(); return no("the padded copy of the synapses would take more than a quarter of the free memory"); }
        // (a table that stays in L2 once it has been read needs no fetching ahead: measured on tables of up to half of it)
        int l2 = 0;
        CUDA_TRY(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, r->device));
        L.prefetch = cells * sizeof(uint2) > (size_t)l2 / 2 ? 1u : 0u;
        if(const int err = device(sizeof(uint2) * cells, (void**)&dEntries)) return err;
        CUDA_TRY(cudaMemsetAsync(dEntries, 0xFF, sizeof(uint2) * cells, r->stream));
        if(const int err = upload(runs.data(), sizeof(ResidentRun) * runs.size(), (void**)&dRuns)) return err;
        L.runs = dRuns;
        L.entries = dEntries;
        r->residentCells = 1e-6 * (double)cells;
        if(const int err = residentPass(r, 1, nullptr, nullptr)) return err;
        CUDA_TRY(cudaStreamSynchronize(r->stream));         // (the temporaries go out of scope)
    }
    else if(const int err = upload(runs.data(), sizeof(ResidentRun) * runs.size(), (void**)&dRuns)) return err;

    // ---- DENSE and BITMASK groups ---------------------------------------------------------------------------------
    std::vector<ResidentSpan> spans;
    for(const auto &l : links) {
        const auto &g = r->synapseGroups[l.syn];
        if(g.connectivity == B200_CONN_SPARSE) continue;
        const bool constant = (g.wu_model == B200_WU_STATIC_PULSE_CONSTANT_WEIGHT);
        spans.push_back(ResidentSpan{constant ? nullptr : g.g, g.connectivity == B200_CONN_BITMASK ? g.gp : nullptr, g.wu_params[0], g.row_stride,
                                     g.num_trg, l.delayClass, l.src, l.trg, l.psm, g.num_src});
    }
    if(const int err = upload(spans.data(), sizeof(ResidentSpan) * spans.size(), (void**)&L.spans)) return err;
    if(const int err = upload(rowStarts.data(), sizeof(unsigned long long) * rowStarts.size(), (void**)&L.rows)) return err;
    if(!poisson.empty()) {
        if(const int err = upload(poisson.data(), sizeof(float) * poisson.size(), (void**)&L.poisson)) return err;
    }

    // ---- messages ---------------------------------------------------------------------------------------------------
    L.buffers = longestDelay + shortest + 3u;
    L.history = history;
    const unsigned int mostIds = neuronWarps * 32u;
    L.more_words = (mostIds - RESIDENT_CELL_IDS + RESIDENT_MORE_IDS - 1u) / RESIDENT_MORE_IDS;
    L.copies = copiesFor(grid);
    const size_t headWords = (size_t)L.buffers * L.copies * grid * 2u, moreWords = (size_t)L.buffers * grid * L.more_words;
    void *mail = nullptr;
    r->residentMailBytes = sizeof(unsigned long long) * (headWords + moreWords + 1u);
    if(const int err = device(r->residentMailBytes, &mail)) return err;
    L.inbox = static_cast<ulonglong2*>(mail);
    L.more = static_cast<unsigned long long*>(mail) + headWords;
    L.leave = L.more + moreWords;
    // (memory of the pool: the word that another model, or this one before, left there could be the one that is waited for)
    CUDA_TRY(cudaMemsetAsync(L.leave, 0, sizeof(unsigned long long), r->stream));

    L.unit_start = dUnitStart; L.unit_first = dUnitFirst; L.columns = dColumns; L.cta_columns = dCtaColumns; L.runs = dRuns; L.entries = dEntries;
    L.num_spans = numSpans; L.num_units = units;
    L.num_depths = (unsigned int)depths.size();
    L.num_delays = numDelays;
    for(size_t i = 0; i < depths.size(); i++) L.depth[i] = depths[i];
    for(size_t i = 0; i < delays.size(); i++) L.delay[i] = delays[i];
    L.acc_floats = (unsigned int)accFloats;
    r->residentGrid = grid;
    r->residentBlock = warps * 32u;
    r->residentSmem = tables + accFloats * sizeof(float);
    CUDA_TRY(cudaFuncSetAttribute(r->residentKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
    if(!r->residentHold) {
        void *word = nullptr;
        CUDA_TRY(hostAcquire(&word, sizeof(unsigned long long)));
        r->residentHold = static_cast<volatile unsigned long long*>(word);
        *r->residentHold = 0ull;
    }
    L.hold = const_cast<unsigned long long*>(r->residentHold);
    if(windowed) {
        if(const int err = device(sizeof(ulonglong2) * win.buffers * L.copies * RESIDENT_HEADS, (void**)&win.heads)) return err;
        if(const int err = device(sizeof(unsigned short) * win.buffers * grid * win.body, (void**)&win.bodies)) return err;
        CUDA_TRY(cudaMemsetAsync(win.heads, 0, sizeof(ulonglong2) * win.buffers * L.copies * RESIDENT_HEADS, r->stream));
        r->windowKernel = residentWindowKernelFor(shape.npsm, shape.ncs);
        CUDA_TRY(cudaFuncSetAttribute(r->windowKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)windowRoom));
        r->windowMayOverflow = win.cap < sourceNeurons;
        r->windowReady = true;
    }
    r->residentReady = true;
    return B200_OK;
}

// Whether a launch of so many steps goes through them in windows.
bool useWindows(const b200_runner *r, unsigned long long numSteps)
{
    return r->windowReady && numSteps >= WINDOW_STEPS;
}

// `done`: steps done when the launch begins; `leave`: a launch of the kernel with a grid barrier follows for what it leaves.
int launchResident(b200_runner *r, unsigned long long numSteps, unsigned long long numRec, unsigned long long done, bool leave)
{
    ResidentLaunch &L = r->resident;
    L.neuron.groups = r->neuronTable.d;
    L.neuron.block_start = r->neuronTable.blockStart;
    L.neuron.num_groups = r->neuronTable.num;
    L.neuron.batch = 1;
    L.neuron.dt = r->dt;
    L.neuron.seed = r->seed;
    L.neuron.num_recording_timesteps = numRec;
    L.neuron.state = r->state;
    L.neuron.count_events = r->countEvents ? 1u : 0u;
    L.neuron.ahead = L.neuron.advance = 0u;
    L.count_events = r->countEvents ? 1u : 0u;
    L.num_steps = (unsigned int)numSteps;
    L.may_leave = leave ? 1u : 0u;
    L.patience = (unsigned int)std::min(1000.0 * r->residentPatience, (double)RESIDENT_MOST_DEBT - 1.0);
    L.barrier = r->fusedBarrier;
    L.launch = ++r->residentLaunches;
    if(useWindows(r, numSteps)) {
        bool clear = false;
        r->window.epoch = windowNextEpoch(r->window.epoch, &clear);
        if(clear) CUDA_TRY(cudaMemsetAsync(r->window.heads, 0, sizeof(ulonglong2) * r->window.buffers * L.copies * RESIDENT_HEADS, r->stream));
        ResidentWindowLaunch A{L, r->window};
        if(r->residentHandsOver) {
            A.L.spare = RESIDENT_WINDOW_SPARE;
            A.L.weight[0] = r->windowWeight;
        }
        void *args[] = {&A};
        CUDA_TRY(cudaLaunchCooperativeKernel(r->windowKernel, dim3(r->residentGrid), dim3(r->windowBlock), args, r->windowSmem, r->stream));
        r->launches++;
        r->fusedLaunches++;
        return B200_OK;
    }
    // a message word is known by the last 20 bits of its step: before they repeat, no old word may be left.  (Steps on other
    // paths count too: they leave the words of earlier steps where they are.)
    if(r->residentCleared == ~0ull || done + numSteps - r->residentCleared >= RESIDENT_TAG_STEPS - 1ull) {
        CUDA_TRY(cudaMemsetAsync(L.inbox, 0, r->residentMailBytes, r->stream));
        r->residentCleared = done;
    }
    void *args[] = {&L};
    CUDA_TRY(cudaLaunchCooperativeKernel(r->residentKernel, dim3(r->residentGrid), dim3(r->residentBlock), args, r->residentSmem, r->stream));
    r->launches++;
    r->fusedLaunches++;
    return B200_OK;
}

// Whether b200_step_time takes the target-resident kernel (its tables are built if they were not).
int chooseResident(b200_runner *r, bool *yes)
{
    *yes = false;
    // (a private copy would not see what the program writes into an array by itself)
    for(void *p : r->exposed) if(!r->residentAsked && touchesSparse(r, p, 1)) return B200_OK;
    if(!r->useFused || !r->useResident || r->scheduleChosen || r->timing || r->sharded() || r->batch != 1) return B200_OK;
    if(r->residentStale && !(r->residentReady && r->residentRent)) {
        if(const int e = buildResident(r)) { r->dropResident(); return e; }
    }
    *yes = r->residentReady;
    return B200_OK;
}

// The copy as the arrays are now (nothing, if it is).
int refreshResident(b200_runner *r)
{
    r->residentRent = 0;
    if(r->residentStale) {
        const int e = buildResident(r);
        if(e) r->dropResident();
        return e;
    }
    if(r->residentOld) {
        r->residentOld = false;
        return residentPass(r, 1, nullptr, nullptr);
    }
    return B200_OK;
}

// Before steps are enqueued (or captured) on the one-launch-per-kernel path.
int ensureTiled(b200_runner *r)
{
    if(r->sparseTable.num && (r->tiledStale || (r->useTiled && !r->tiledReady && r->tiledWhyNot.empty()))) {
        r->dropGraph();
        return buildTiled(r);
    }
    return B200_OK;
}

// (`force`: an update the caller asked for on its own, with spike lists of its choosing)
bool tiledActive(const b200_runner *r, bool force = false)
{
    return r->tiledReady && (force || r->tiledArmed || r->tiledMinEvents == 0);
}

// Whether sparseBatchKernel delivers the groups it can.
bool scatterActive(const b200_runner *r)
{
    return r->scatterArmed || r->scatterMinSpikes <= 0.0f;
}

// A kernel of the one-launch-per-kernel path: its blocks may be placed while the kernel before it runs (chainWait).
template<typename P, typename A>
cudaError_t chain(const b200_runner *r, void (*kernel)(P), dim3 grid, unsigned int block, size_t smem, const A &params)
{
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(block);
    config.dynamicSmemBytes = smem;
    config.stream = r->stream;
    config.attrs = &early;
    config.numAttrs = r->timing ? 0u : 1u;      // (timed kernels do not overlap)
    return cudaLaunchKernelEx(&config, kernel, params);
}

// Spikes of a copy that blocks take side by side: with a learning rule an event is a chain of dependent loads, so every
// block the chip holds at once (16 of 128 threads an SM) should have a spike; without one the rows are long and 16 will do.
unsigned int spikeLanesFor(const b200_runner *r, unsigned int blocks)
{
    if(r->learnTable.num == 0) return r->spikeLanes;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device);
    return std::max(r->spikeLanes, std::min(256u, (unsigned int)sms * 16u / std::max(1u, blocks * r->batch)));
}

int enqueueSynapses(b200_runner *r, bool capturing, bool force = false)
{
    if(r->sparseTable.num) {
        ScopedTimer tm(r, "presynaptic_update", capturing);
        SynapseLaunch S = synapseLaunch(r, r->sparseTable);
        if(tiledActive(r, force)) {
            // the step's estimated events decide which of the two kernels delivers the served groups
            const TiledLaunch T = tiledLaunch(r);
            CUDA_TRY(chain(r, tiledDecideKernel, 1, TILED_BLOCK, 0, T));
            CUDA_TRY(chain(r, tiledKernelFor(r->tiledPostBits == 10u, r->tiledWeights != nullptr), r->tiledGrid, TILED_BLOCK, r->tiledSmemBytes, T));
            r->launches += 2;
            S.tiled_served = r->tiledServed;
        }
        const dim3 grid(r->sparseTable.blocks, spikeLanesFor(r, r->sparseTable.blocks), r->batch);
        CUDA_TRY(chain(r, presynapticSparseKernel, grid, PRE_BLOCK, 0, S));
        r->launches++;
    }
    if(r->postSpanTable.num) {
        ScopedTimer tm(r, "presynaptic_update", capturing);
        const dim3 grid(r->postSpanTable.blocks, 1, r->batch);
        CUDA_TRY(chain(r, presynapticPostSpanKernel, grid, PRE_BLOCK, 0, synapseLaunch(r, r->postSpanTable)));
        r->launches++;
    }
    if(r->denseTable.num) {
        ScopedTimer tm(r, "presynaptic_update", capturing);
        const dim3 grid(r->denseTable.blocks, 1, (r->batch + DENSE_COPIES - 1u) / DENSE_COPIES);
        CUDA_TRY(chain(r, denseBatchKernel, grid, DENSE_BLOCK, DENSE_SMEM, DenseLaunch{synapseLaunch(r, r->denseTable), r->denseParts}));
        r->launches++;
    }
    if(r->scatterTable.num && !force && !scatterActive(r)) {
        ScopedTimer tm(r, "presynaptic_update", capturing);
        const dim3 grid(r->scatterRows.blocks, spikeLanesFor(r, r->scatterRows.blocks), r->batch);
        CUDA_TRY(chain(r, presynapticSparseKernel, grid, PRE_BLOCK, 0, synapseLaunch(r, r->scatterRows)));
        r->launches++;
    }
    else if(r->scatterTable.num) {
        ScopedTimer tm(r, "presynaptic_update", capturing);
        CUDA_TRY(chain(r, sparseBatchKernel, r->scatterGrid, SCATTER_BLOCK, r->scatterSmem,
                       ScatterLaunch{synapseLaunch(r, r->scatterTable), r->scatterTargets, r->scatterParts, r->scatterCells, r->scatterDepth, r->scatterPiece}));
        r->launches++;
    }
    if(r->proceduralTable.num) {
        ScopedTimer tm(r, "presynaptic_update", capturing);
        // (spike, sub-row) items spread over the whole device; the spike count is only known there
        int sms = 0;
        CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
        const dim3 grid((unsigned int)sms * 8u, r->proceduralTable.num, r->batch);
        CUDA_TRY(chain(r, presynapticProceduralKernel, grid, PROC_BLOCK, 0, synapseLaunch(r, r->proceduralTable)));
        r->launches++;
    }
    if(r->drawnTable.num) {
        ScopedTimer tm(r, "presynaptic_update", capturing);
        // (the number of spikes is only known on the device: as many blocks as the chip holds take them in turn)
        int sms = 0;
        CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
        const dim3 grid((unsigned int)sms * PROC_PER_SM, r->drawnTable.num, r->batch);
        const ProceduralLaunch P{synapseLaunch(r, r->drawnTable), proceduralKeys(r->seed)};
        auto kernel = r->drawnNormal ? (r->drawnWide ? proceduralDrawnKernel<true, true> : proceduralDrawnKernel<true, false>)
                                     : proceduralDrawnKernel<false, true>;
        CUDA_TRY(chain(r, kernel, grid, DRAWN_BLOCK, 0, P));
        r->launches++;
    }
    if(r->learnTable.num) {
        ScopedTimer tm(r, "postsynaptic_update", capturing);
        const dim3 grid(r->learnTable.blocks, spikeLanesFor(r, r->learnTable.blocks), r->batch);
        CUDA_TRY(chain(r, postsynapticUpdateKernel, grid, POST_BLOCK, 0, synapseLaunch(r, r->learnTable)));
        r->launches++;
    }
    CUDA_TRY(cudaPeekAtLastError());
    return B200_OK;
}

int enqueueNeurons(b200_runner *r, unsigned long long numRec, bool capturing)
{
    if(r->neuronTable.num == 0) return fail(B200_ERR_STATE, "no neuron groups registered");
    ScopedTimer tm(r, "neuron_update", capturing);
    NeuronLaunch L;
    L.groups = r->neuronTable.d;
    L.block_start = r->neuronTable.blockStart;
    L.num_groups = r->neuronTable.num;
    L.batch = r->batch;
    L.dt = r->dt;
    L.seed = r->seed;
    L.num_recording_timesteps = numRec;
    L.state = r->state;
    L.count_events = r->countEvents ? 1u : 0u;
    L.ahead = r->ahead;
    L.advance = r->advance;
    L.peak_groups = (r->scatterTable.num && !r->tiledReady) ? r->scatterSources : ~0ull;
    // (as many blocks as are on the chip at once: thousands of blocks for a few loads each spend their time starting, and
    // counting themselves one after another in the ticket)
    int sms = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
    const unsigned long long items = (unsigned long long)r->neuronTable.blocks * r->batch;
    const bool four = items >= (unsigned long long)sms * NEURON_WARPS_WANTED;
    const dim3 grid((unsigned int)std::min<unsigned long long>(four ? (items + 3u) / 4u : items, (unsigned long long)sms * NEURON_BLOCKS_PER_SM));
    int e = withNeuronShape(r, [&](auto P, auto C) -> int {
        constexpr int NPSM = decltype(P)::value, NCS = decltype(C)::value;
        auto launch = [&](dim3 blocks, auto *staged, auto *direct) -> int {
            if(neuronStaged(L.num_groups, items, (unsigned int)sms, r->postSpanTable.num || r->denseTable.num)) {
                CUDA_TRY(chain(r, staged, blocks, NEURON_BLOCK, neuronTableBytes(L.num_groups), L));
            }
            else CUDA_TRY(chain(r, direct, blocks, NEURON_BLOCK, 0, L));
            return B200_OK;
        };
        // (with many inputs or sources four words would not fit the registers)
        if constexpr(NPSM + NCS <= 4) {
            if(four) return launch(grid, neuronUpdateKernel<NPSM, NCS, 4, true>, neuronUpdateKernel<NPSM, NCS, 4, false>);
        }
        return launch(dim3((unsigned int)std::min<unsigned long long>(items, (unsigned long long)sms * NEURON_BLOCKS_PER_SM)),
                      neuronUpdateKernel<NPSM, NCS, 1, true>, neuronUpdateKernel<NPSM, NCS, 1, false>);
    });
    if(e) return e;
    r->launches++;
    CUDA_TRY(cudaPeekAtLastError());
    return B200_OK;
}

// Behind a block of steps of the per-kernel path: the block's largest spike count on its way to the host.
int fetchPeak(b200_runner *r)
{
    if(!r->peakHost || r->peakPending) return B200_OK;      // (an earlier block's copy still under way: keep it)
    CUDA_TRY(cudaMemcpyAsync(r->peakHost, &r->state->peak_spikes, sizeof(unsigned int), cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaMemsetAsync(&r->state->peak_spikes, 0, sizeof(unsigned int), r->stream));
    CUDA_TRY(cudaEventRecord(r->peakEvent, r->stream));
    r->peakPending = true;
    r->peakSteps = 0;
    return B200_OK;
}

// Before a block of steps: choose kernels by the last spike count that has arrived.
int pollPeak(b200_runner *r)
{
    if(!r->peakPending || cudaEventQuery(r->peakEvent) != cudaSuccess) return B200_OK;
    r->peakPending = false;
    r->peakSeen = true;
    const double peak = (double)*r->peakHost;
    if(r->tiledReady) {
        const double estimate = peak * r->eventsPerSpike;
        const bool was = r->tiledArmed;
        if(estimate * 4.0 >= (double)r->tiledMinEvents) {
            r->tiledArmed = true;
            r->quietBlocks = 0;
        }
        else if(r->tiledArmed && estimate * 16.0 < (double)r->tiledMinEvents && ++r->quietBlocks >= 3) {
            r->tiledArmed = false;
        }
        if(was != r->tiledArmed) r->dropGraph();        // the captured steps launch other kernels now
    }
    if(r->scatterTable.num) {
        const double least = (double)r->scatterMinSpikes * r->batch;
        const bool was = r->scatterArmed;
        if(peak >= least) {
            r->scatterArmed = true;
            r->scatterQuiet = 0;
        }
        else if(r->scatterArmed && peak * 2.0 < least && ++r->scatterQuiet >= 3) r->scatterArmed = false;
        if(was != r->scatterArmed) r->dropGraph();
    }
    return B200_OK;
}

int enqueueStep(b200_runner *r, unsigned long long numRec, bool capturing)
{
    int e = enqueueSynapses(r, capturing);
    if(e) return e;
    return enqueueNeurons(r, numRec, capturing);
}

unsigned int kernelsPerStep(const b200_runner *r)
{
    return 1u + (r->sparseTable.num ? (tiledActive(r) ? 3u : 1u) : 0u) + (r->postSpanTable.num ? 1u : 0u) + (r->denseTable.num ? 1u : 0u) + (r->scatterTable.num ? 1u : 0u) + (r->learnTable.num ? 1u : 0u) +
           (r->proceduralTable.num ? 1u : 0u) + (r->drawnTable.num ? 1u : 0u);
}

int buildGraph(b200_runner *r, unsigned int len, unsigned long long numRec)
{
    r->dropGraph();
    cudaGraph_t graph = nullptr;
    const unsigned long long before = r->launches;
    CUDA_TRY(cudaStreamBeginCapture(r->stream, cudaStreamCaptureModeThreadLocal));
    int e = B200_OK;
    for(unsigned int i = 0; i < len && e == B200_OK; i++) {
        r->ahead = i;
        r->advance = (i + 1u == len) ? len : 0u;
        e = enqueueStep(r, numRec, true);
    }
    r->ahead = 0;
    r->advance = 1;
    cudaError_t ce = cudaStreamEndCapture(r->stream, &graph);
    r->launches = before;       // capture enqueues nothing
    if(e) {
        if(graph) cudaGraphDestroy(graph);
        return e;
    }
    CUDA_TRY(ce);
    ce = cudaGraphInstantiate(&r->graphExec, graph, 0);
    cudaGraphDestroy(graph);
    CUDA_TRY(ce);
    r->graphLen = len;
    r->graphNumRec = numRec;
    return B200_OK;
}
}   // anonymous namespace

extern "C" {

const char *b200_last_error(void)
{
    return g_lastError.c_str();
}

int b200_device_count(int *count)
{
    CUDA_TRY(cudaGetDeviceCount(count));
    return B200_OK;
}

int b200_runner_create(int device, double dt, uint64_t seed, uint32_t batch_size, b200_runner **out)
{
    if(!out || batch_size == 0) return fail(B200_ERR_INVALID, "bad arguments to b200_runner_create");
    CUDA_TRY(cudaSetDevice(device));
    b200_runner *r = new b200_runner();
    r->device = device;
    r->dt = (float)dt;
    r->seed = seed;
    r->batch = batch_size;
    CUDA_TRY(cudaStreamCreateWithFlags(&r->stream, cudaStreamNonBlocking));
    CUDA_TRY(poolAlloc(&r->state, sizeof(StepState), r->stream));
    CUDA_TRY(cudaMemsetAsync(r->state, 0, sizeof(StepState), r->stream));
    {
        const unsigned long long limits[3] = {BARRIER_SPIN_LIMIT, EXCHANGE_SPIN_LIMIT, (unsigned long long)STREAM_WAIT_CYCLES};
        CUDA_TRY(cudaMemcpyAsync(&r->state->barrier_spin_limit, limits, sizeof(limits), cudaMemcpyHostToDevice, r->stream));
        const unsigned int polls = COPY_WAITS;
        CUDA_TRY(cudaMemcpyAsync(&r->state->copy_wait_limit, &polls, sizeof(polls), cudaMemcpyHostToDevice, r->stream));
    }
    CUDA_TRY(cudaEventCreate(&r->evA));
    CUDA_TRY(cudaEventCreate(&r->evB));
    CUDA_TRY(cudaEventCreate(&r->evC));
    CUDA_TRY(cudaEventCreate(&r->evD));
    CUDA_TRY(hostAcquire(reinterpret_cast<void**>(&r->stage), STAGE_BYTES + 64));
    r->hostWord = reinterpret_cast<unsigned int*>(r->stage + STAGE_BYTES);
    *out = r;
    return B200_OK;
}

/* ---- NCCL, resolved when first needed: the library that is already in the process (a host application
 *      that bootstraps with torch.distributed has loaded one) or the system's.  The reference's CUDA backend
 *      exports ncclGenerateUniqueID / ncclGetUniqueID / ncclInitCommunicator from the generated library
 *      and emits one ncclAllReduce per reduction target (backends/cuda/backend.cc:219-226, 1360-1389,
 *      backendCUDAHIP.h:240-292); here the targets of a group travel as ONE buffer. ------------------- */
namespace
{
struct NcclId { char internal[128]; };                  // ncclUniqueId
struct NcclApi
{
    void *lib = nullptr;
    int (*getUniqueId)(NcclId*) = nullptr;
    int (*commInitRank)(void**, int, NcclId, int) = nullptr;
    int (*allReduce)(const void*, void*, size_t, int, int, void*, cudaStream_t) = nullptr;
    int (*commDestroy)(void*) = nullptr;
    const char *(*getErrorString)(int) = nullptr;
};
constexpr int NCCL_FLOAT32 = 7, NCCL_SUM = 0, NCCL_MAX = 2;     // ncclDataType_t / ncclRedOp_t values of nccl.h

NcclApi *ncclApi()
{
    static NcclApi api;
    if(api.lib) return &api;
    void *lib = dlopen("libnccl.so.2", RTLD_NOW | RTLD_NOLOAD);
    if(!lib) lib = dlopen("libnccl.so.2", RTLD_NOW | RTLD_LOCAL);
    if(!lib) lib = dlopen("libnccl.so", RTLD_NOW | RTLD_LOCAL);
    if(!lib) return nullptr;
    api.getUniqueId = reinterpret_cast<decltype(api.getUniqueId)>(dlsym(lib, "ncclGetUniqueId"));
    api.commInitRank = reinterpret_cast<decltype(api.commInitRank)>(dlsym(lib, "ncclCommInitRank"));
    api.allReduce = reinterpret_cast<decltype(api.allReduce)>(dlsym(lib, "ncclAllReduce"));
    api.commDestroy = reinterpret_cast<decltype(api.commDestroy)>(dlsym(lib, "ncclCommDestroy"));
    api.getErrorString = reinterpret_cast<decltype(api.getErrorString)>(dlsym(lib, "ncclGetErrorString"));
    if(!api.getUniqueId || !api.commInitRank || !api.allReduce || !api.commDestroy || !api.getErrorString) return nullptr;
    api.lib = lib;
    return &api;
}
}   // namespace

#define NCCL_TRY(api, call) do { const int e_ = (call); if(e_ != 0) return fail(B200_ERR_CUDA, "NCCL: %s (%s)", (api)->getErrorString(e_), #call); } while(0)

int b200_runner_destroy(b200_runner *r)
{
    if(!r) return B200_OK;
    cudaSetDevice(r->device);
    cudaStreamSynchronize(r->stream);
    r->dropGraph();
    r->neuronTable.release(r->stream);
    r->sparseTable.release(r->stream);
    r->postSpanTable.release(r->stream);
    r->denseTable.release(r->stream);
    poolFree(r->denseParts, r->stream);
    r->scatterTable.release(r->stream);
    r->scatterRows.release(r->stream);
    poolFree(r->scatterTargets, r->stream);
    poolFree(r->scatterParts, r->stream);
    r->proceduralTable.release(r->stream);
    r->drawnTable.release(r->stream);
    r->learnTable.release(r->stream);
    poolFree(r->fusedSlotStart, r->stream);
    poolFree(r->fusedSources, r->stream);
    poolFree(r->fusedItems, r->stream);
    poolFree(r->fusedBarrier, r->stream);
    r->dropUrgent();
    r->dropNear();
    poolFree(r->fusedCtaCycles, r->stream);
    r->dropTiled();
    r->dropResident();
    for(unsigned int p = 0; p < B200_MAX_RANKS; p++) {
        if(r->peerArena[p] && !r->peerLocal[p]) cudaIpcCloseMemHandle(r->peerArena[p]);
    }
    hostRelease(r->stage);
    poolFree(r->recCounts, r->stream);
    poolFree(r->recList, r->stream);
    hostRelease(r->recHost);
    hostRelease(r->peakHost);
    hostRelease(const_cast<unsigned long long*>(r->residentHold));
    if(r->peakEvent) cudaEventDestroy(r->peakEvent);
    if(r->ncclComm && ncclApi()) ncclApi()->commDestroy(r->ncclComm);
    poolFree(r->reducePacked, r->stream);
    if(r->arena) cudaFree(r->arena);
    poolFree(r->peerTable, r->stream);
    for(auto &a : r->arrays) poolFree(a.first, r->stream);
    poolFree(r->state, r->stream);
    cudaEventDestroy(r->evA);
    cudaEventDestroy(r->evB);
    cudaEventDestroy(r->evC);
    cudaEventDestroy(r->evD);
    cudaStreamDestroy(r->stream);
    delete r;
    return B200_OK;
}

int b200_array_alloc(b200_runner *r, size_t bytes, void **device_ptr)
{
    if(!r || !device_ptr) return fail(B200_ERR_INVALID, "bad arguments to b200_array_alloc");
    CUDA_TRY(cudaSetDevice(r->device));
    void *p = nullptr;
    CUDA_TRY(poolAlloc(&p, bytes + ARRAY_TAIL_PAD, r->stream));
    CUDA_TRY(cudaMemsetAsync(p, 0, bytes + ARRAY_TAIL_PAD, r->stream));
    r->arrays[p] = bytes;
    *device_ptr = p;
    return B200_OK;
}

int b200_host_alloc(b200_runner *r, size_t bytes, void **host_ptr)
{
    if(!r || !host_ptr) return fail(B200_ERR_INVALID, "bad arguments to b200_host_alloc");
    CUDA_TRY(cudaSetDevice(r->device));
    CUDA_TRY(hostAcquire(host_ptr, bytes ? bytes : 1));
    return B200_OK;
}

int b200_host_register(void *host_ptr, size_t bytes)
{
    const cudaError_t e = cudaHostRegister(host_ptr, bytes, cudaHostRegisterPortable);
    if(e == cudaSuccess) return B200_OK;
    cudaGetLastError();         // (a page that is locked already, say: not an error of anything that follows)
    return fail(B200_ERR_CUDA, "%s (page-locking %llu bytes)", cudaGetErrorString(e), (unsigned long long)bytes);
}

int b200_host_unregister(void *host_ptr)
{
    CUDA_TRY(cudaHostUnregister(host_ptr));
    return B200_OK;
}

int b200_host_free(b200_runner *r, void *host_ptr)
{
    (void)r;
    hostRelease(host_ptr);
    return B200_OK;
}

// The arena a process allocates: the caller's bytes, then the near-synapse queues of both step parities
// from every process (the same layout in every process: peers address each other's arenas by offset).
static size_t exchangeQueueOffset(size_t bytes) { return (bytes + 255) & ~(size_t)255; }
static size_t exchangeTotalBytes(size_t bytes)
{
    return exchangeQueueOffset(bytes) + (size_t)2 * B200_MAX_RANKS * NEAR_QUEUE_COUNT * NEAR_QUEUE_WORDS * sizeof(unsigned long long)
        + ARRAY_TAIL_PAD;
}

int b200_exchange_alloc(b200_runner *r, size_t bytes, void **device_ptr)
{
    if(!r || !device_ptr || bytes == 0) return fail(B200_ERR_INVALID, "bad arguments to b200_exchange_alloc");
    if(r->arena) return fail(B200_ERR_STATE, "the exchange arena has already been allocated");
    CUDA_TRY(cudaSetDevice(r->device));
    void *p = nullptr;
    const size_t total = exchangeTotalBytes(bytes);
    CUDA_TRY(cudaMalloc(&p, total));
    CUDA_TRY(cudaMemsetAsync(p, 0, total, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));         // (peers write into it as soon as they know its handle)
    r->arena = static_cast<unsigned char*>(p);
    r->arenaBytes = bytes;
    r->queueOffset = exchangeQueueOffset(bytes);
    *device_ptr = p;
    return B200_OK;
}

int b200_exchange_bytes(b200_runner *r, size_t *bytes)
{
    if(!r || !r->arena || !bytes) return fail(B200_ERR_STATE, "no exchange arena");
    *bytes = exchangeTotalBytes(r->arenaBytes);
    return B200_OK;
}

int b200_exchange_get_handle(b200_runner *r, void *handle_64_bytes)
{
    if(!r || !r->arena || !handle_64_bytes) return fail(B200_ERR_STATE, "no exchange arena");
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "IPC handle size");
    cudaIpcMemHandle_t h;
    CUDA_TRY(cudaIpcGetMemHandle(&h, r->arena));
    memcpy(handle_64_bytes, &h, sizeof(h));
    return B200_OK;
}

int b200_exchange_open_peer(b200_runner *r, uint32_t peer_rank, const void *handle_64_bytes)
{
    if(!r || peer_rank >= B200_MAX_RANKS || !handle_64_bytes) return fail(B200_ERR_INVALID, "bad peer rank");
    if(r->peerArena[peer_rank]) return fail(B200_ERR_STATE, "peer %u already opened", peer_rank);
    CUDA_TRY(cudaSetDevice(r->device));
    cudaIpcMemHandle_t h;
    memcpy(&h, handle_64_bytes, sizeof(h));
    void *p = nullptr;
    CUDA_TRY(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess));
    r->peerArena[peer_rank] = static_cast<unsigned char*>(p);
    if(!r->peerTable) CUDA_TRY(poolAlloc(&r->peerTable, sizeof(unsigned char*) * B200_MAX_RANKS, r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->peerTable, r->peerArena, sizeof(unsigned char*) * B200_MAX_RANKS, cudaMemcpyHostToDevice, r->stream));
    return B200_OK;
}

int b200_exchange_set_peer(b200_runner *r, uint32_t peer_rank, void *device_ptr)
{
    if(!r || peer_rank >= B200_MAX_RANKS || !device_ptr) return fail(B200_ERR_INVALID, "bad peer rank or pointer");
    if(r->peerArena[peer_rank]) return fail(B200_ERR_STATE, "peer %u already opened", peer_rank);
    CUDA_TRY(cudaSetDevice(r->device));
    r->peerArena[peer_rank] = static_cast<unsigned char*>(device_ptr);
    if(!r->peerTable) CUDA_TRY(poolAlloc(&r->peerTable, sizeof(unsigned char*) * B200_MAX_RANKS, r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->peerTable, r->peerArena, sizeof(unsigned char*) * B200_MAX_RANKS, cudaMemcpyHostToDevice, r->stream));
    r->peerLocal[peer_rank] = true;
    return B200_OK;
}

/* ---- sharded "deliver at emission": every process builds the near-synapse rows of ALL source neurons
 *      onto its own neurons, then hands each process the rows of that process's neurons ------------- */
int b200_near_export(b200_runner *r, void *handle_64_bytes, uint64_t *meta, uint32_t meta_words)
{
    if(!r || !handle_64_bytes || !meta) return fail(B200_ERR_INVALID, "null argument");
    CUDA_TRY(cudaSetDevice(r->device));
    int e = prepare(r);
    if(e) return e;
    r->emitAgreed = false;
    r->dropNear();
    memset(handle_64_bytes, 0, 64);
    const size_t groups = r->neuronGroups.size();
    if(meta_words < 3 + 2 * groups) return fail(B200_ERR_INVALID, "meta array too short: %zu words needed", 3 + 2 * groups);
    meta[0] = 0; meta[1] = groups; meta[2] = 0;
    if(!r->sharded() || !r->fusedEligible || !r->useEmit || r->streamWarpsWanted == 0 || !r->fusedStage) return B200_OK;
    e = buildNearTables(r, true);
    if(e) return e;
    if(!r->nearTable) return B200_OK;       // does not qualify
    cudaIpcMemHandle_t h;
    CUDA_TRY(cudaIpcGetMemHandle(&h, r->nearTable));
    memcpy(handle_64_bytes, &h, sizeof(h));
    meta[0] = 1; meta[2] = (uint64_t)r->numRings | ((uint64_t)r->fusedGrid << 32);
    for(size_t ni = 0; ni < groups; ni++) {
        meta[3 + 2 * ni] = r->nearCellHost[ni];
        meta[4 + 2 * ni] = r->nearShiftHost[ni];
    }
    r->nearImported.assign(groups, nullptr);
    r->nearSpacesAll.assign(groups, NearSpace{nullptr, 0xFFFFFFFFu, 0u, 0u, 0u});
    r->nearPeerDone.assign(r->world, false);
    r->nearDataStale = false;
    return B200_OK;
}

int b200_near_import(b200_runner *r, uint32_t peer_rank, const void *handle_64_bytes, const uint64_t *meta,
                     const uint32_t *common_shift)
{
    if(!r || !handle_64_bytes || !meta || !common_shift || peer_rank >= r->world) return fail(B200_ERR_INVALID, "bad arguments to b200_near_import");
    const size_t groups = r->neuronGroups.size();
    if(r->nearImported.size() != groups || r->nearPeerDone.size() != r->world) return fail(B200_ERR_STATE, "b200_near_export has to come first");
    if(!meta[0] || meta[1] != groups || (uint32_t)meta[2] != r->numRings) return fail(B200_ERR_STATE, "process %u does not qualify or runs another model", peer_rank);
    r->peerGrid[peer_rank] = (unsigned int)(meta[2] >> 32);
    CUDA_TRY(cudaSetDevice(r->device));
    const uint2 *table = r->nearTable;
    void *mapped = nullptr;
    if(peer_rank != r->rank) {
        cudaIpcMemHandle_t h;
        memcpy(&h, handle_64_bytes, sizeof(h));
        CUDA_TRY(cudaIpcOpenMemHandle(&mapped, h, cudaIpcMemLazyEnablePeerAccess));
        table = static_cast<const uint2*>(mapped);
    }
    unsigned int worldShift = 0;
    while((1u << worldShift) < r->world) worldShift++;
    // Rows of this process's neurons: [neuron][process][1 << common shift] entries, zero padded.  The
    // block of process `peer_rank` is copied out of that process's table, whose rows may be shorter.
    for(size_t ni = 0; ni < groups; ni++) {
        const uint32_t shift = (uint32_t)meta[4 + 2 * ni], common = common_shift[ni];
        if(shift == 0xFFFFFFFFu || common == 0xFFFFFFFFu) continue;
        if(shift > common || common + worldShift > 12) return fail(B200_ERR_INVALID, "bad common row length for neuron group %zu", ni);
        const auto &ng = r->neuronGroups[ni];
        const size_t rowCells = (size_t)1 << (common + worldShift);
        if(!r->nearImported[ni]) {
            CUDA_TRY(cudaMalloc(&r->nearImported[ni], sizeof(uint2) * (rowCells * ng.num_update + 1)));
            CUDA_TRY(cudaMemsetAsync(r->nearImported[ni], 0, sizeof(uint2) * (rowCells * ng.num_update + 1), r->stream));
            r->nearSpacesAll[ni] = NearSpace{r->nearImported[ni], common + worldShift, ng.first_neuron, common, 0u};
        }
        if(ng.num_update) {
            CUDA_TRY(cudaMemcpy2DAsync(r->nearImported[ni] + ((size_t)peer_rank << common), sizeof(uint2) * rowCells,
                                  table + meta[3 + 2 * ni] + ((size_t)ng.first_neuron << shift), sizeof(uint2) << shift,
                                  sizeof(uint2) << shift, ng.num_update, cudaMemcpyDeviceToDevice, r->stream));
        }
    }
    CUDA_TRY(cudaDeviceSynchronize());
    if(mapped) CUDA_TRY(cudaIpcCloseMemHandle(mapped));
    r->nearPeerDone[peer_rank] = true;
    return B200_OK;
}

/* After EVERY process has imported from every process (the caller synchronises them): free the full table
 * and switch the schedule on (`agreed` != 0) or drop everything. */
int b200_near_finish(b200_runner *r, int agreed)
{
    if(!r) return fail(B200_ERR_INVALID, "null runner");
    CUDA_TRY(cudaSetDevice(r->device));
    if(!agreed || r->nearPeerDone.size() != r->world) {
        r->dropNear();
        r->lagStale = true;
        return B200_OK;
    }
    for(uint32_t p = 0; p < r->world; p++) {
        if(!r->nearPeerDone[p]) return fail(B200_ERR_STATE, "the rows held by process %u have not been imported", p);
        if(p != r->rank && !r->peerArena[p]) return fail(B200_ERR_STATE, "exchange arena of rank %u has not been opened", p);
    }
    r->freeNearTable();
    // the rings of every process as this process sees them: same offset in the peer's arena
    std::vector<NearRing> rings((size_t)r->world * r->numRings);
    for(uint32_t p = 0; p < r->world; p++) {
        for(uint32_t i = 0; i < r->numRings; i++) {
            NearRing ring = r->nearRingsHost[i];
            if(p != r->rank) {
                ring.den_delay = reinterpret_cast<float*>(r->peerArena[p] + (reinterpret_cast<unsigned char*>(ring.den_delay) - r->arena));
            }
            rings[(size_t)p * r->numRings + i] = ring;
        }
    }
    poolFree(r->nearRings, r->stream);
    poolFree(r->nearSpaces, r->stream);
    CUDA_TRY(poolAlloc(&r->nearRings, sizeof(NearRing) * rings.size(), r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->nearRings, rings.data(), sizeof(NearRing) * rings.size(), cudaMemcpyHostToDevice, r->stream));
    CUDA_TRY(poolAlloc(&r->nearSpaces, sizeof(NearSpace) * r->nearSpacesAll.size(), r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->nearSpaces, r->nearSpacesAll.data(), sizeof(NearSpace) * r->nearSpacesAll.size(), cudaMemcpyHostToDevice, r->stream));
    r->emitAgreed = true;
    r->queuesAgreed = r->fusedGrid <= NEAR_QUEUE_COUNT;
    for(uint32_t p = 0; p < r->world; p++) {
        if(r->peerGrid[p] != r->fusedGrid) r->queuesAgreed = false;
    }
    r->lagStale = true;
    return B200_OK;
}

int b200_exchange_configure(b200_runner *r, uint32_t rank, uint32_t world)
{
    if(!r || world == 0 || world > B200_MAX_RANKS || rank >= world) return fail(B200_ERR_INVALID, "bad rank/world");
    if(world > 1 && !r->arena) return fail(B200_ERR_STATE, "no exchange arena");
    r->rank = rank;
    r->world = world;
    r->dirty = true;
    return B200_OK;
}

int b200_array_free(b200_runner *r, void *device_ptr)
{
    auto it = r->arrays.find(device_ptr);
    if(it == r->arrays.end()) return fail(B200_ERR_INVALID, "pointer was not allocated by this runner");
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    CUDA_TRY(poolFree(device_ptr, r->stream));
    r->arrays.erase(it);
    r->exposed.erase(std::remove(r->exposed.begin(), r->exposed.end(), device_ptr), r->exposed.end());
    return B200_OK;
}

int b200_array_push(b200_runner *r, void *device_ptr, const void *host, size_t bytes)
{
    CUDA_TRY(cudaMemcpyAsync(device_ptr, host, bytes, cudaMemcpyHostToDevice, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    arrayWritten(r, device_ptr, bytes);
    return B200_OK;
}

int b200_array_pull(b200_runner *r, void *host, const void *device_ptr, size_t bytes)
{
    if(bytes <= STAGE_BYTES) {
        // to page-locked memory and on from there: the driver's own way into pageable memory takes 15 us however
        // few the bytes, this one 8 (40 KB)
        std::lock_guard<std::mutex> lock(r->staging);
        CUDA_TRY(cudaMemcpyAsync(r->stage, device_ptr, bytes, cudaMemcpyDeviceToHost, r->stream));
        CUDA_TRY(cudaStreamSynchronize(r->stream));
        memcpy(host, r->stage, bytes);
        return B200_OK;
    }
    if(bytes >= LARGE_PULL) {
        CUDA_TRY(pullLarge(host, device_ptr, bytes, 1u, false, r->device, r->stream));
        return B200_OK;
    }
    CUDA_TRY(cudaMemcpyAsync(host, device_ptr, bytes, cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    return B200_OK;
}

int b200_array_pull_u32(b200_runner *r, uint32_t *host, const void *device_ptr, uint32_t elem_bytes, uint64_t count)
{
    if(!r || (count && (!host || !device_ptr))) return fail(B200_ERR_INVALID, "null argument to b200_array_pull_u32");
    if(elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4) return fail(B200_ERR_INVALID, "element size %u is not 1, 2 or 4", elem_bytes);
    if(count) CUDA_TRY(pullLarge(host, device_ptr, count, elem_bytes, true, r->device, r->stream));
    return B200_OK;
}

int b200_array_memset(b200_runner *r, void *device_ptr, int value, size_t bytes)
{
    CUDA_TRY(cudaMemsetAsync(device_ptr, value, bytes, r->stream));
    arrayWritten(r, device_ptr, bytes);
    return B200_OK;
}

int b200_array_expose(b200_runner *r, void *device_ptr)
{
    // (also one inside the exchange arena of a sharded model: nothing is copied from there)
    if(!r || !device_ptr) return fail(B200_ERR_INVALID, "null argument to b200_array_expose");
    if(std::find(r->exposed.begin(), r->exposed.end(), device_ptr) == r->exposed.end()) r->exposed.push_back(device_ptr);
    return B200_OK;
}

int b200_push_neuron_update_group(b200_runner *r, uint32_t idx, const b200_neuron_group *g)
{
    if(!r || !g) return fail(B200_ERR_INVALID, "null argument");
    if(g->num_psm > B200_MAX_PSM || g->num_cs > B200_MAX_CS) return fail(B200_ERR_INVALID, "too many children");
    if(g->num_delay_slots < 2) return fail(B200_ERR_INVALID, "num_delay_slots must be at least 2");
    if(g->first_neuron + g->num_update > g->num_neurons) return fail(B200_ERR_INVALID, "update slice out of range");
    if(g->first_neuron & 31u) return fail(B200_ERR_INVALID, "first_neuron must be a multiple of 32");
    if(!g->spk_cnt || !g->spk) return fail(B200_ERR_INVALID, "spike arrays missing");
    if(idx >= r->neuronGroups.size()) r->neuronGroups.resize(idx + 1);
    r->neuronGroups[idx] = *g;
    r->dirty = true;
    return B200_OK;
}

int b200_validate_synapse_group(const b200_synapse_group *g)
{
    if(!g) return fail(B200_ERR_INVALID, "null argument");
    if(g->connectivity == B200_CONN_SPARSE) {
        if(!g->row_length || !g->ind) return fail(B200_ERR_INVALID, "SPARSE group without row_length/ind");
        if(g->ind_bytes != 1 && g->ind_bytes != 2 && g->ind_bytes != 4) return fail(B200_ERR_INVALID, "bad ind_bytes");
    }
    if(g->connectivity == B200_CONN_BITMASK) {
        if(!g->gp || (g->row_stride & 31u)) return fail(B200_ERR_INVALID, "BITMASK needs gp and a row stride padded to 32");
        if(g->wu_model != B200_WU_STATIC_PULSE_CONSTANT_WEIGHT) return fail(B200_ERR_INVALID, "BITMASK carries no per-synapse variables");
    }
    if(g->connectivity == B200_CONN_PROCEDURAL) {
        if(g->proc_connect != B200_CONNECT_FIXED_PROBABILITY && g->proc_connect != B200_CONNECT_FIXED_PROBABILITY_NO_AUTAPSE &&
           g->proc_connect != B200_CONNECT_FIXED_NUMBER_POST_WITH_REPLACEMENT) {
            return fail(B200_ERR_INVALID, "PROCEDURAL connectivity needs a snippet that builds rows without stored lengths");
        }
        if(g->wu_model != B200_WU_STATIC_PULSE && g->wu_model != B200_WU_STATIC_PULSE_CONSTANT_WEIGHT) {
            return fail(B200_ERR_INVALID, "PROCEDURAL connectivity supports StaticPulse and StaticPulseConstantWeight");
        }
        if(!g->row_stride) return fail(B200_ERR_INVALID, "PROCEDURAL group without a row stride (longest row)");
    }
    if(g->wu_model != B200_WU_STATIC_PULSE_CONSTANT_WEIGHT && g->connectivity != B200_CONN_PROCEDURAL && !g->g) {
        return fail(B200_ERR_INVALID, "weight array missing");
    }
    if(g->wu_model == B200_WU_STATIC_PULSE_DENDRITIC_DELAY && (!g->d || !g->den_delay || !g->max_den_delay)) {
        return fail(B200_ERR_INVALID, "dendritic delay group without d/den_delay");
    }
    // the kernels switch on max_den_delay: a ring depth means "read d, add into den_delay"
    if(g->max_den_delay && (!g->den_delay || (!g->d && g->connectivity != B200_CONN_PROCEDURAL))) {
        return fail(B200_ERR_INVALID, "max_den_delay set but d or den_delay missing");
    }
    if(g->max_den_delay && g->wu_model != B200_WU_STATIC_PULSE_DENDRITIC_DELAY && g->connectivity != B200_CONN_PROCEDURAL) {
        return fail(B200_ERR_INVALID, "max_den_delay set on a weight update model that does not call addToPostDelay");
    }
    if((g->max_den_delay || g->wu_model == B200_WU_STATIC_PULSE_DENDRITIC_DELAY) &&
       (g->connectivity == B200_CONN_BITMASK || g->connectivity == B200_CONN_DENSE)) {
        return fail(B200_ERR_INVALID, "dendritic delay is supported on SPARSE connectivity only");
    }
    if(!g->max_den_delay && !g->out_post) return fail(B200_ERR_INVALID, "out_post missing");
    if(g->connectivity == B200_CONN_SPARSE) {
        // rows are read as aligned groups of four synapses counted from the array base
        if(g->g && ((uintptr_t)g->g & 15u)) return fail(B200_ERR_INVALID, "g must be 16-byte aligned");
        if((uintptr_t)g->ind & (4u * g->ind_bytes - 1u)) return fail(B200_ERR_INVALID, "ind must be aligned to four indices");
        if(g->d && ((uintptr_t)g->d & 3u)) return fail(B200_ERR_INVALID, "d must be 4-byte aligned");
    }
    if(g->wu_model == B200_WU_STDP) {
        if(!g->src_spike_times || !g->trg_spike_times || !g->trg_spk || !g->trg_spk_cnt) {
            return fail(B200_ERR_INVALID, "learning group without spike times");
        }
        if(g->connectivity == B200_CONN_SPARSE && (!g->col_length || !g->remap)) {
            return fail(B200_ERR_INVALID, "learning SPARSE group without remap");
        }
        if(g->back_prop_delay + 2 > g->trg_delay_slots) {
            return fail(B200_ERR_INVALID, "back-propagation delay exceeds the target spike queue");
        }
    }
    if(g->axonal_delay + 2 > g->src_delay_slots) return fail(B200_ERR_INVALID, "axonal delay exceeds the source spike queue");
    return B200_OK;
}

int b200_push_synapse_group(b200_runner *r, uint32_t idx, const b200_synapse_group *g)
{
    if(!r || !g) return fail(B200_ERR_INVALID, "null argument");
    if(const int e = b200_validate_synapse_group(g)) return e;
    if(idx >= r->synapseGroups.size()) r->synapseGroups.resize(idx + 1);
    r->synapseGroups[idx] = *g;
    r->dirty = true;
    return B200_OK;
}

int b200_push_custom_update(b200_runner *r, const char *name, uint32_t idx, const b200_custom_update_group *u)
{
    if(!r || !name || !u) return fail(B200_ERR_INVALID, "null argument");
    auto &v = r->customUpdates[name];
    if(idx >= v.size()) v.resize(idx + 1);
    v[idx] = *u;
    return B200_OK;
}

int b200_set_option(b200_runner *r, const char *name, double value)
{
    const std::string n(name);
    // (an option that picks a schedule of the other persistent kernels asks for those kernels)
    if(n == "use_lag" || n == "use_emit" || n == "use_split" || n == "stream_warps") r->scheduleChosen = true;
    if(n == "spike_lanes") r->spikeLanes = std::max(1u, (unsigned int)value);
    else if(n == "count_events") r->countEvents = (value != 0.0);
    else if(n == "use_graph") r->useGraph = (value != 0.0);
    else if(n == "use_fused") r->useFused = (value != 0.0);
    else if(n == "use_resident") {
        r->useResident = r->residentAsked = (value != 0.0);
        r->scheduleChosen = false;
        if(!r->useResident && !r->residentBuffers.empty()) {
            // its copy of the synapses goes back
            CUDA_TRY(cudaSetDevice(r->device));
            r->dropResident();
            r->residentStale = true;
            r->residentRent = 0;
        }
    }
    else if(n == "use_windows") { r->useWindow = (value != 0.0); r->residentStale = true; r->residentRent = 0; }
    else if(n == "resident_ctas") { r->residentCtas = (unsigned int)std::max(0.0, value); r->residentStale = true; r->residentRent = 0; }
    else if(n == "resident_warps") { r->residentWarps = (unsigned int)std::max(0.0, value); r->residentStale = true; r->residentRent = 0; }
    else if(n == "resident_patience") {
        // (0: leaves in front of the first spike that costs more here)
        r->residentPatience = (float)std::max(0.0, value);
        r->residentPatienceChosen = true;
    }
    else if(n == "use_lag") { r->useLag = (value != 0.0); r->lagStale = true; }
    else if(n == "use_split") { r->useSplit = (value != 0.0); r->lagStale = true; }
    else if(n == "use_near_queues") r->useNearQueues = (value != 0.0);
    else if(n == "near_queue_words") {
        if(value < 2.0 || value > (double)NEAR_QUEUE_WORDS) return fail(B200_ERR_INVALID, "near_queue_words must lie in [2, %u]", NEAR_QUEUE_WORDS);
        r->queueWords = (unsigned int)value;
    }
    else if(n == "use_emit") { r->useEmit = (value != 0.0); r->lagStale = true; }
    else if(n == "stream_warps") { r->streamWarpsWanted = (int)value; r->lagStale = true; }
    else if(n == "lag_agreed") { r->lagAgreed = (value != 0.0); r->lagStale = true; }
    else if(n == "rescan_delays") {
        r->lagStale = true;
        for(const auto &g : r->synapseGroups) if(g.row_length) arrayWritten(r, g.row_length, sizeof(unsigned int) * g.num_src);
    }
    else if(n == "fused_profile") {
        // (the per-CTA cycle counters are allocated here, not on the time-step path)
        r->fusedProfile = (value != 0.0);
        if(r->fusedProfile && !r->fusedCtaCycles) {
            CUDA_TRY(cudaSetDevice(r->device));
            CUDA_TRY(poolAlloc(&r->fusedCtaCycles, sizeof(unsigned long long) * 5 * PROFILE_MAX_CTAS, r->stream));
            CUDA_TRY(cudaMemsetAsync(r->fusedCtaCycles, 0, sizeof(unsigned long long) * 5 * PROFILE_MAX_CTAS, r->stream));
        }
    }
    else if(n == "fused_blocks_per_sm") { r->fusedBlocksPerSM = (unsigned int)value; r->dirty = true; }
    else if(n == "graph_steps") r->graphSteps = std::max(1u, (unsigned int)value);
    else if(n == "barrier_spin_limit" || n == "exchange_spin_limit" || n == "stream_wait_cycles") {
        // limits of the waits inside the persistent kernels (polls, polls, SM cycles); a wait that runs out
        // makes the launch return early and b200_synchronize report it
        if(value < 1.0) return fail(B200_ERR_INVALID, "%s must be at least 1", name);
        const unsigned long long v = (unsigned long long)value;
        unsigned long long *dst = (n == "barrier_spin_limit") ? &r->state->barrier_spin_limit
                                : (n == "exchange_spin_limit") ? &r->state->exchange_spin_limit
                                : reinterpret_cast<unsigned long long*>(&r->state->stream_wait_cycles);
        CUDA_TRY(cudaStreamSynchronize(r->stream));
        CUDA_TRY(cudaMemcpyAsync(dst, &v, sizeof(v), cudaMemcpyHostToDevice, r->stream));
    }
    else if(n == "copy_wait_limit") {
        // polls for a copy into shared memory; 0: none is waited for, so that every step of the kernels that use them fails
        const unsigned int polls = (unsigned int)std::min(std::max(0.0, value), 4.0e9);
        CUDA_TRY(cudaStreamSynchronize(r->stream));
        CUDA_TRY(cudaMemcpyAsync(&r->state->copy_wait_limit, &polls, sizeof(polls), cudaMemcpyHostToDevice, r->stream));
    }
    else if(n == "scatter_min_spikes") { r->scatterMinSpikes = (float)value; r->peakSeen = false; r->dirty = true; }
    else if(n == "use_tiled") { r->useTiled = (value != 0.0); r->tiledStale = true; }
    else if(n == "tiled_min_events") { r->tiledMinEvents = (float)value; r->tiledChosen = r->dirty = true; }
    else if(n == "tiled_ticket_events") { r->tiledTicketEvents = std::max(1.0f, (float)value); r->dropGraph(); }
    else if(n == "tiled_ticket_cost") { r->tiledTicketCost = std::max(0.0f, (float)value); r->dropGraph(); }
    else return fail(B200_ERR_INVALID, "unknown option %s", name);
    r->dropGraph();
    return B200_OK;
}

int b200_initialize(b200_runner *r)
{
    CUDA_TRY(cudaSetDevice(r->device));
    return prepare(r);
}

int b200_initialize_sparse(b200_runner *r)
{
    CUDA_TRY(cudaSetDevice(r->device));
    return prepare(r);
}

int b200_init_var(b200_runner *r, void *device_ptr, uint32_t elem_bytes, uint64_t count,
                  uint32_t snippet, const float *params, uint32_t rng_stream)
{
    r->lagStale = true;
    r->tiledStale = r->residentStale = true;
    InitParams prm{};
    for(int i = 0; i < 4; i++) prm.p[i] = params ? params[i] : 0.0f;
    const unsigned int blocks = (unsigned int)std::min<uint64_t>((count + INIT_BLOCK - 1) / INIT_BLOCK, 148u * 32u);
    if(count == 0) return B200_OK;
    if(elem_bytes == 4) {
        initVarKernel<float><<<blocks, INIT_BLOCK, 0, r->stream>>>((float*)device_ptr, count, snippet, prm, r->seed, rng_stream);
    }
    else if(elem_bytes == 1) {
        initVarKernel<uint8_t><<<blocks, INIT_BLOCK, 0, r->stream>>>((uint8_t*)device_ptr, count, snippet, prm, r->seed, rng_stream);
    }
    else return fail(B200_ERR_INVALID, "element size %u not supported", elem_bytes);
    r->launches++;
    CUDA_TRY(cudaPeekAtLastError());
    return B200_OK;
}

int b200_init_sparse_connectivity(b200_runner *r, uint32_t snippet, const float *params,
                                  uint32_t num_src, uint32_t num_trg, uint32_t row_stride,
                                  uint32_t ind_bytes, uint32_t trg_begin, uint32_t trg_end,
                                  uint32_t *row_length, void *ind, uint32_t rng_stream)
{
    r->lagStale = true;
    r->tiledStale = r->residentStale = true;
    if(trg_end > num_trg || trg_begin >= trg_end) return fail(B200_ERR_INVALID, "bad target range");
    InitParams prm{};
    for(int i = 0; i < 4; i++) prm.p[i] = params ? params[i] : 0.0f;
    return withIndType(ind_bytes, [&](auto tag) -> int {
        using IndT = decltype(tag);
        if(snippet == B200_CONNECT_FIXED_NUMBER_PRE_WITH_REPLACEMENT) {
            CUDA_TRY(cudaMemsetAsync(row_length, 0, sizeof(uint32_t) * num_src, r->stream));
            const unsigned int n = trg_end - trg_begin;
            initFixedNumberPreKernel<IndT><<<(n + INIT_BLOCK - 1) / INIT_BLOCK, INIT_BLOCK, 0, r->stream>>>(
                (unsigned int)prm.p[0], num_src, row_stride, trg_begin, trg_end, row_length, ind, r->seed, rng_stream, r->state);
        }
        else {
            initSparseConnectivityKernel<IndT><<<(num_src + INIT_BLOCK - 1) / INIT_BLOCK, INIT_BLOCK, 0, r->stream>>>(
                snippet, prm, num_src, row_stride, trg_begin, trg_end, row_length, ind, r->seed, rng_stream, r->state);
        }
        r->launches++;
        CUDA_TRY(cudaPeekAtLastError());
        return B200_OK;
    });
}

int b200_init_sparse_vars(b200_runner *r, const uint32_t *row_length, uint32_t num_src,
                          uint32_t row_stride, void *device_ptr, uint32_t elem_bytes,
                          uint32_t snippet, const float *params, uint32_t rng_stream)
{
    r->lagStale = true;
    r->tiledStale = r->residentStale = true;
    InitParams prm{};
    for(int i = 0; i < 4; i++) prm.p[i] = params ? params[i] : 0.0f;
    const uint64_t total = (uint64_t)num_src * row_stride;
    if(total == 0) return B200_OK;
    const unsigned int blocks = (unsigned int)std::min<uint64_t>((total + INIT_BLOCK - 1) / INIT_BLOCK, 148u * 32u);
    if(elem_bytes == 4) {
        initSparseVarKernel<float><<<blocks, INIT_BLOCK, 0, r->stream>>>((float*)device_ptr, row_length, num_src, row_stride, snippet, prm, r->seed, rng_stream);
    }
    else if(elem_bytes == 1) {
        initSparseVarKernel<uint8_t><<<blocks, INIT_BLOCK, 0, r->stream>>>((uint8_t*)device_ptr, row_length, num_src, row_stride, snippet, prm, r->seed, rng_stream);
    }
    else return fail(B200_ERR_INVALID, "element size %u not supported", elem_bytes);
    r->launches++;
    CUDA_TRY(cudaPeekAtLastError());
    return B200_OK;
}

int b200_build_remap(b200_runner *r, const uint32_t *row_length, const void *ind, uint32_t ind_bytes,
                     uint32_t num_src, uint32_t num_trg, uint32_t row_stride, uint32_t col_stride,
                     uint32_t *col_length, uint32_t *remap)
{
    const uint64_t total = (uint64_t)num_src * row_stride;
    CUDA_TRY(cudaMemsetAsync(col_length, 0, sizeof(uint32_t) * num_trg, r->stream));
    if(total == 0) return B200_OK;
    const unsigned int blocks = (unsigned int)std::min<uint64_t>((total + INIT_BLOCK - 1) / INIT_BLOCK, 148u * 32u);
    return withIndType(ind_bytes, [&](auto tag) -> int {
        using IndT = decltype(tag);
        buildRemapKernel<IndT><<<blocks, INIT_BLOCK, 0, r->stream>>>(row_length, ind, num_src, num_trg, row_stride,
                                                                     col_stride, col_length, remap, r->state);
        r->launches++;
        CUDA_TRY(cudaPeekAtLastError());
        return B200_OK;
    });
}

int b200_update_synapses(b200_runner *r)
{
    int e = prepare(r);
    if(e) return e;
    e = ensureTiled(r);
    if(e) return e;
    return enqueueSynapses(r, false, true);
}

int b200_update_neurons(b200_runner *r, uint64_t num_recording_timesteps)
{
    int e = prepare(r);
    if(e) return e;
    e = enqueueNeurons(r, num_recording_timesteps, false);
    if(e == B200_OK) {
        r->hostTimestep++;
        r->hostStepsDone++;
    }
    return e;
}

int b200_step_time(b200_runner *r, uint64_t num_steps, uint64_t num_recording_timesteps)
{
    int e = prepare(r);
    if(e) return e;
    uint64_t left = num_steps;
    if(r->sharded() && !(r->useFused && r->fusedEligible && !r->timing)) {
        return fail(B200_ERR_STATE, "a sharded model runs on the persistent kernel only (batch 1, SPARSE "
                                    "non-learning groups, per-kernel timing off)");
    }
    bool resident = false;
    if(num_steps && (e = chooseResident(r, &resident)) != B200_OK) return e;
    // (a busy network without the kernel with a grid barrier: one launch per kernel, call by call)
    if(resident && !r->residentHandsOver) {
        if(r->hostStepsDone < *r->residentHold) resident = false;
        else if(num_steps <= r->residentRent) {
            r->residentRent -= num_steps;
            resident = false;
        }
        else {
            if((e = refreshResident(r)) != B200_OK) return e;
            resident = r->residentReady;
        }
    }
    if(resident) {
        if(*r->residentHold != r->residentHoldSeen) {
            r->residentHoldSeen = *r->residentHold;
            r->residentQuiet = r->hostStepsDone > r->residentHoldSeen + 2u * FIRST_BLOCK ? 1u : 0u;       // (it has gone on since)
        }
        // (a model's first call, of many steps and with rings: worth waiting once, behind its first blocks, for whether the other kernel has
        // taken over, since that one is faster with tables of its own)
        bool look = r->residentHandsOver && r->residentSteeper && r->lagStale && !r->residentQuiet && num_steps >= LONG_CALL;
        // (one step of it could use up the patience, or be more than the list holds, and how it begins is not known yet)
        const bool sudden = r->residentHandsOver && !r->residentQuiet && r->residentSources > RESIDENT_LIST;
        uint64_t block = !r->residentHandsOver ? RESIDENT_TAG_STEPS / 2 : sudden ? FIRST_BLOCK : QUIET_BLOCK;
        while(left) {
            const uint64_t done = r->hostStepsDone + (num_steps - left);
            if(look && num_steps - left >= LONG_HOLD) {
                look = false;
                CUDA_TRY(cudaStreamSynchronize(r->stream));
                if(done < *r->residentHold && (e = refreshSchedule(r)) != B200_OK) return e;
            }
            if(r->residentHandsOver && done < *r->residentHold) {
                const uint64_t n = std::min<uint64_t>(left, *r->residentHold - done);
                e = launchFused(r, n, num_recording_timesteps, 0, *r->residentHold - done < LONG_HOLD);
                if(e) return e;
                left -= n;
                r->residentRent -= std::min<unsigned long long>(r->residentRent, n);
                continue;
            }
            if(r->residentRent || !r->residentReady) {
                const uint64_t n = r->residentReady ? std::min<uint64_t>(left, r->residentRent) : left;
                e = launchFused(r, n, num_recording_timesteps);
                if(e) return e;
                left -= n;
                r->residentRent -= std::min<unsigned long long>(r->residentRent, n);
                continue;
            }
            if(r->residentStale || r->residentOld) {
                if((e = refreshResident(r)) != B200_OK) return e;
                continue;
            }
            const uint64_t n = std::min<uint64_t>(left, std::min<uint64_t>(block, RESIDENT_TAG_STEPS / 2));
            const bool leave = r->residentHandsOver && (r->residentPatienceChosen || (r->windowMayOverflow && useWindows(r, n)) || (double)n * r->residentWorst > MOST_LOSS * (1u + std::min(r->residentQuiet, MOST_QUIET)));
            e = launchResident(r, n, num_recording_timesteps, done, leave);
            if(e == B200_OK && leave) e = launchFused(r, n, num_recording_timesteps, done + n);
            if(e) return e;
            left -= n;
            block *= 2;
        }
        r->residentQuiet++;
    }
    else if(r->useFused && r->fusedEligible && !r->timing) {
        while(left) {
            const uint64_t n = std::min<uint64_t>(left, 1ull << 20);
            e = launchFused(r, n, num_recording_timesteps);
            if(e) return e;
            left -= n;
        }
    }
    else if((e = ensureTiled(r)) != B200_OK || (e = pollPeak(r)) != B200_OK) {
        return e;
    }
    else if(r->useGraph && !r->timing && num_steps >= 2) {
        const unsigned int len = (unsigned int)std::min<uint64_t>(num_steps, r->graphSteps);
        if(!r->graphExec || r->graphLen > num_steps || r->graphNumRec != num_recording_timesteps ||
           (r->graphLen != len && r->graphLen != r->graphSteps)) {
            e = buildGraph(r, len, num_recording_timesteps);
            if(e) return e;
        }
        while(left >= r->graphLen) {
            CUDA_TRY(cudaGraphLaunch(r->graphExec, r->stream));
            r->launches += (unsigned long long)r->graphLen * kernelsPerStep(r);
            left -= r->graphLen;
            if(r->scatterTable.num && !r->peakSeen && left >= 4ull * r->graphLen) {
                // a model's first steps, and many more behind them: worth waiting, once, for what they have to say
                if((e = fetchPeak(r)) != B200_OK) return e;
                CUDA_TRY(cudaEventSynchronize(r->peakEvent));
                const unsigned int len = r->graphLen;
                if((e = pollPeak(r)) != B200_OK) return e;
                if(!r->graphExec && (e = buildGraph(r, len, num_recording_timesteps)) != B200_OK) return e;
            }
        }
    }
    for(; left; left--) {
        e = enqueueStep(r, num_recording_timesteps, false);
        if(e) return e;
    }
    if((r->tiledReady || r->scatterTable.num) && !resident && !(r->useFused && r->fusedEligible && !r->timing)) {
        // (three more entries in the stream: not behind every call of a few steps)
        r->peakSteps += (unsigned int)std::min<uint64_t>(num_steps, 1u << 20);
        if(r->tiledReady || r->peakSteps >= 64u || !r->peakSeen) {
            e = fetchPeak(r);
            if(e) return e;
        }
    }
    r->hostTimestep += num_steps;
    r->hostStepsDone += num_steps;
    return B200_OK;
}


int b200_nccl_unique_id(void *id_128_bytes)
{
    if(!id_128_bytes) return fail(B200_ERR_INVALID, "null id buffer");
    NcclApi *api = ncclApi();
    if(!api) return fail(B200_ERR_STATE, "libnccl.so.2 could not be loaded: %s", dlerror());
    NcclId id;
    NCCL_TRY(api, api->getUniqueId(&id));
    memcpy(id_128_bytes, &id, sizeof(id));
    return B200_OK;
}

int b200_nccl_init(b200_runner *r, const void *id_128_bytes, uint32_t rank, uint32_t world)
{
    if(!r || !id_128_bytes || world == 0 || rank >= world) return fail(B200_ERR_INVALID, "bad arguments to b200_nccl_init");
    if(r->ncclComm) return fail(B200_ERR_STATE, "the communicator has already been created");
    NcclApi *api = ncclApi();
    if(!api) return fail(B200_ERR_STATE, "libnccl.so.2 could not be loaded: %s", dlerror());
    CUDA_TRY(cudaSetDevice(r->device));
    NcclId id;
    memcpy(&id, id_128_bytes, sizeof(id));
    NCCL_TRY(api, api->commInitRank(&r->ncclComm, (int)world, id, (int)rank));
    r->ncclWorld = world;
    return B200_OK;
}

// A custom update group.  `phases`: bit 0 reduce over the batch, bit 1 write back.  With a communicator
// (data-parallel run: every process holds a share of the batch) the reduced values of ALL updates of the
// group are packed into one buffer, sums first, combined with one all-reduce per operation on the
// runner's stream, and written back from there: no host synchronisation anywhere.
static int runCustomUpdate(b200_runner *r, const char *name, unsigned int phases)
{
    auto it = r->customUpdates.find(name);
    if(it == r->customUpdates.end()) return fail(B200_ERR_INVALID, "no custom update group '%s'", name);
    ScopedTimer tm(r, std::string("custom_update_") + name, false);
    const bool combine = r->ncclComm && r->ncclWorld > 1 && phases == 3u;
    auto blocksFor = [](uint64_t n) { return (unsigned int)std::min<uint64_t>((n + REDUCE_BLOCK - 1) / REDUCE_BLOCK, 148u * 16u); };
    // (a write-back changes the variable itself: weights, say, that private copies hold)
    for(const auto &u : it->second) {
        arrayWritten(r, u.target, sizeof(float) * u.num_elements);
        if(u.broadcast && (phases & 2u)) arrayWritten(r, u.source, sizeof(float) * u.num_elements * r->batch);
    }
    if(!combine) {
        for(const auto &u : it->second) {
            if(u.num_elements == 0) continue;
            batchReduceKernel<<<blocksFor(u.num_elements), REDUCE_BLOCK, 0, r->stream>>>(u, r->batch, phases, nullptr);
            r->launches++;
        }
        CUDA_TRY(cudaPeekAtLastError());
        return B200_OK;
    }
    // layout of the packed buffer: every update's segment starts on a 16-byte boundary
    std::vector<size_t> offset(it->second.size(), 0);
    size_t total = 0, sums = 0;
    for(int pass = 0; pass < 2; pass++) {
        for(size_t i = 0; i < it->second.size(); i++) {
            const auto &u = it->second[i];
            if((u.op == B200_REDUCE_SUM) != (pass == 0)) continue;
            offset[i] = total;
            total += (u.num_elements + 3) & ~(uint64_t)3;
        }
        if(pass == 0) sums = total;
    }
    if(total > r->reducePackedElements) {
        CUDA_TRY(cudaStreamSynchronize(r->stream));
        if(r->reducePacked) CUDA_TRY(poolFree(r->reducePacked, r->stream));
        r->reducePacked = nullptr;
        CUDA_TRY(poolAlloc(&r->reducePacked, sizeof(float) * total, r->stream));
        CUDA_TRY(cudaMemsetAsync(r->reducePacked, 0, sizeof(float) * total, r->stream));
        r->reducePackedElements = total;
    }
    for(size_t i = 0; i < it->second.size(); i++) {
        const auto &u = it->second[i];
        if(u.num_elements == 0) continue;
        batchReduceKernel<<<blocksFor(u.num_elements), REDUCE_BLOCK, 0, r->stream>>>(u, r->batch, 1u, r->reducePacked + offset[i]);
        r->launches++;
    }
    CUDA_TRY(cudaPeekAtLastError());
    NcclApi *api = ncclApi();
    if(sums) NCCL_TRY(api, api->allReduce(r->reducePacked, r->reducePacked, sums, NCCL_FLOAT32, NCCL_SUM, r->ncclComm, r->stream));
    if(total > sums) NCCL_TRY(api, api->allReduce(r->reducePacked + sums, r->reducePacked + sums, total - sums, NCCL_FLOAT32, NCCL_MAX, r->ncclComm, r->stream));
    for(size_t i = 0; i < it->second.size(); i++) {
        const auto &u = it->second[i];
        if(u.num_elements == 0) continue;
        batchReduceKernel<<<blocksFor(u.num_elements), REDUCE_BLOCK, 0, r->stream>>>(u, r->batch, 2u, r->reducePacked + offset[i]);
        r->launches++;
    }
    CUDA_TRY(cudaPeekAtLastError());
    return B200_OK;
}

int b200_custom_update(b200_runner *r, const char *name)
{
    return runCustomUpdate(r, name, 3u);
}

int b200_custom_update_reduce(b200_runner *r, const char *name)
{
    return runCustomUpdate(r, name, 1u);
}

int b200_custom_update_broadcast(b200_runner *r, const char *name)
{
    return runCustomUpdate(r, name, 2u);
}

// The device's error word as a status.  A time-out leaves every CTA out of the kernel: the word is cleared for the next one.
static int reportDeviceError(b200_runner *r, unsigned int err)
{
    if(!err) return B200_OK;
    cudaMemsetAsync(&r->state->error, 0, sizeof(unsigned int), r->stream);
    r->residentCleared = ~0ull;         // (a launch that gave up may have left messages of steps that count again)
    return fail(B200_ERR_DEVICE_CHECK, "device-side check failed (flags 0x%x:%s%s%s%s%s%s)", err,
                (err & ERR_SPIKE_OVERFLOW) ? " spike list overflow" : "",
                (err & ERR_IND_RANGE) ? " index or row length out of range" : "",
                (err & ERR_DELAY_RANGE) ? " a synapse arriving in the same step appeared after the schedule was chosen (option rescan_delays)" : "",
                (err & ERR_BARRIER_TIMEOUT) ? " grid barrier timed out" : "",
                (err & ERR_EXCHANGE_TIMEOUT) ? " spikes of another process did not arrive in time" : "",
                (err & ERR_COPY_TIMEOUT) ? " a copy into shared memory was not waited for any longer" : "");
}

int b200_synchronize(b200_runner *r)
{
    std::lock_guard<std::mutex> lock(r->staging);
    CUDA_TRY(cudaMemcpyAsync(r->hostWord, &r->state->error, sizeof(unsigned int), cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    return reportDeviceError(r, *r->hostWord);
}

int b200_get_timestep(b200_runner *r, uint64_t *timestep)
{
    *timestep = r->hostTimestep;
    return B200_OK;
}

int b200_set_timestep(b200_runner *r, uint64_t timestep)
{
    const unsigned long long t = timestep;
    CUDA_TRY(cudaMemcpyAsync(&r->state->timestep, &t, sizeof(t), cudaMemcpyHostToDevice, r->stream));
    r->hostTimestep = timestep;
    return B200_OK;
}

int b200_get_steps_done(b200_runner *r, uint64_t *steps)
{
    *steps = r->hostStepsDone;
    return B200_OK;
}

int b200_get_counter(b200_runner *r, const char *name, uint64_t *value)
{
    const std::string n(name);
    if(n == "stream_warps") {
        int e = prepare(r);
        if(e) return e;
        if(r->fusedEligible && r->lagStale) {
            e = refreshSchedule(r);
            if(e) return e;
        }
        *value = r->streamWarps;
        return B200_OK;
    }
    if(n == "resident") {
        // whether b200_step_time takes the target-resident kernel
        int e = prepare(r);
        bool yes = false;
        if(!e) e = chooseResident(r, &yes);
        if(e) return e;
        *value = yes ? 1u : 0u;
        return B200_OK;
    }
    if(n == "resident_bytes") {
        *value = r->residentReady ? (uint64_t)(r->residentCells * 1e6 * sizeof(uint2) + 0.5) : 0u;
        return B200_OK;
    }
    if(n == "resident_message_bytes") {
        *value = r->residentReady ? r->residentMailBytes + (r->windowReady ? r->windowMailBytes : 0u) : 0u;
        return B200_OK;
    }
    if(n == "resident_builds") {
        // how often the copy has been made (not: filled again with other weights)
        *value = r->residentBuilds;
        return B200_OK;
    }
    if(n == "window_steps") {
        // steps of a window (resident_window.cuh), 0 where that kernel does not apply
        int e = prepare(r);
        bool yes = false;
        if(!e) e = chooseResident(r, &yes);
        if(e) return e;
        *value = yes && r->windowReady ? r->window.steps : 0u;
        return B200_OK;
    }
    if(n == "resident_hold") {
        // the step until which the kernel with a grid barrier takes a busy network's steps
        CUDA_TRY(cudaStreamSynchronize(r->stream));
        *value = r->residentHold ? *r->residentHold : 0u;
        return B200_OK;
    }
    if(n == "schedule") {
        // of the next persistent launch: 0 everything before the neuron update, 1 only the synapses that
        // arrive in the same step before it (split delivery), 2 spikes one step late (one barrier per step)
        int e = prepare(r);
        if(e) return e;
        if(r->fusedEligible && r->lagStale) {
            e = refreshSchedule(r);
            if(e) return e;
        }
        *value = (uint64_t)r->schedule;
        return B200_OK;
    }
    if(n == "tiled_armed") {
        // whether the next block of steps on the one-launch-per-kernel path launches the tiled kernels
        *value = tiledActive(r) ? 1u : 0u;
        return B200_OK;
    }
    if(n == "scatter_armed") {
        // whether the next block of steps of a batched network sums its SPARSE groups in shared memory
        int e = prepare(r);
        if(!e) e = pollPeak(r);
        if(e) return e;
        *value = (r->scatterTable.num && scatterActive(r)) ? 1u : 0u;
        return B200_OK;
    }
    if(n == "tiled_ready" || n == "tiled_synapses" || n == "heavy") {
        // the target-tiled copy of the SPARSE groups (built when the one-launch-per-kernel path is first
        // used) / the verdict of the last step's event estimate
        if(n == "heavy") {
            unsigned int h = 0;
            CUDA_TRY(cudaStreamSynchronize(r->stream));
            CUDA_TRY(cudaMemcpy(&h, &r->state->heavy, sizeof(h), cudaMemcpyDeviceToHost));
            *value = h;
            return B200_OK;
        }
        int e = prepare(r);
        if(!e) e = ensureTiled(r);
        if(e) return e;
        *value = (n == "tiled_ready") ? (r->tiledReady ? 1u : 0u) : r->tiledSynapses;
        return B200_OK;
    }
    if(n == "lag_eligible" || n == "lag") {
        // whether this process may deliver spikes one step late (scans the delay arrays if
        // they changed) / whether its next persistent launch will
        int e = prepare(r);
        if(e) return e;
        if(r->fusedEligible && r->lagStale) {
            e = refreshSchedule(r);
            if(e) return e;
        }
        const bool can = r->useLag && r->fusedEligible && r->lagEligible;
        *value = (n == "lag") ? (r->useFused && r->fusedEligible && r->schedule == b200_runner::LAG) : can;
        return B200_OK;
    }
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    StepState s;
    CUDA_TRY(cudaMemcpy(&s, r->state, sizeof(s), cudaMemcpyDeviceToHost));
    if(n == "synaptic_events") *value = s.synaptic_events;
    else if(n == "spikes") *value = s.spikes;
    else if(n == "cycles_presynaptic") *value = s.phase_cycles[0];
    else if(n == "cycles_barrier_a") *value = s.phase_cycles[1];
    else if(n == "cycles_neuron") *value = s.phase_cycles[2];
    else if(n == "cycles_barrier_b") *value = s.phase_cycles[3];
    else if(n.size() >= 6 && n.size() <= 7 && n.compare(0, 5, "probe") == 0 && atoi(n.c_str() + 5) >= 0 && atoi(n.c_str() + 5) < 12 &&
            isdigit((unsigned char)n[5])) *value = s.probe[atoi(n.c_str() + 5)];
    else if(n == "timestep") *value = s.timestep;
    else if(n == "steps_done") *value = s.steps_done;
    else return fail(B200_ERR_INVALID, "unknown counter %s", name);
    return B200_OK;
}

/* Per-CTA phase cycles of the persistent kernel (option "fused_profile"): out[cta*4 + phase]. */
int b200_get_cta_cycles(b200_runner *r, uint64_t *out, uint32_t max_ctas, uint32_t *num_ctas)
{
    *num_ctas = 0;
    if(!r->fusedCtaCycles) return B200_OK;
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    const uint32_t n = std::min<uint32_t>(max_ctas, r->fusedGrid);
    CUDA_TRY(cudaMemcpy(out, r->fusedCtaCycles, sizeof(uint64_t) * 4 * n, cudaMemcpyDeviceToHost));
    if(max_ctas >= 2 * r->fusedGrid) {
        // trailing block: cycles from step start to the spike-header barrier
        CUDA_TRY(cudaMemcpy(out + 4ull * n, r->fusedCtaCycles + 4ull * r->fusedGrid, sizeof(uint64_t) * n, cudaMemcpyDeviceToHost));
    }
    *num_ctas = n;
    return B200_OK;
}

/* Which time-step path b200_step_time will take: 2 target-stationary persistent kernel,
 * 1 persistent kernel with global reductions, 0 one launch per kernel.  `why` (may be NULL)
 * receives the reason the faster paths were not chosen. */
int b200_get_step_path(b200_runner *r, int *path, char *why, size_t why_bytes)
{
    const int e = prepare(r);
    if(e) return e;
    *path = (r->useFused && r->fusedEligible) ? 1 : 0;
    if(why && why_bytes) snprintf(why, why_bytes, "%s", r->fusedEligible ? "" : "batch > 1, or groups that are not SPARSE and non-learning");
    return B200_OK;
}

int b200_enable_timing(b200_runner *r, int enabled)
{
    r->timing = (enabled != 0);
    return B200_OK;
}

int b200_get_timer(b200_runner *r, const char *name, double *seconds)
{
    auto it = r->timers.find(name);
    *seconds = (it == r->timers.end()) ? 0.0 : it->second.seconds;
    return B200_OK;
}

int b200_reset_timers(b200_runner *r)
{
    r->timers.clear();
    return B200_OK;
}

int b200_get_kernel_launches(b200_runner *r, uint64_t *launches)
{
    *launches = r->launches;
    return B200_OK;
}

// Time `num_steps` steps with CUDA events recorded on the runner's own stream
// (events of another stream would not see this work).  Synchronises.
int b200_step_time_timed(b200_runner *r, uint64_t num_steps, uint64_t num_recording_timesteps, float *milliseconds)
{
    int e = prepare(r);
    if(e) return e;
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    CUDA_TRY(cudaEventRecord(r->evC, r->stream));
    e = b200_step_time(r, num_steps, num_recording_timesteps);
    if(e) return e;
    CUDA_TRY(cudaEventRecord(r->evD, r->stream));
    CUDA_TRY(cudaEventSynchronize(r->evD));
    CUDA_TRY(cudaEventElapsedTime(milliseconds, r->evC, r->evD));
    return B200_OK;
}

int b200_pull_recording(b200_runner *r, uint32_t num_arrays, const uint32_t *const *words, const uint64_t *num_words,
                        uint32_t capacity, const void **pairs, uint64_t *num_pairs)
{
    if(!r || (num_arrays && (!words || !num_words)) || !pairs || !num_pairs) return fail(B200_ERR_INVALID, "null argument to b200_pull_recording");
    CUDA_TRY(cudaSetDevice(r->device));
    *pairs = nullptr;
    *num_pairs = 0;
    uint64_t total = 0, chunks = 0;
    for(uint32_t i = 0; i < num_arrays; i++) {
        total += num_words[i];
        chunks += (num_words[i] + RECORD_CHUNK - 1) / RECORD_CHUNK;
    }
    if(total > 0xFFFFFFFFull) return fail(B200_ERR_INVALID, "word indices beyond 32 bits");
    if(chunks == 0) return b200_synchronize(r);
    if(chunks > r->recChunks || capacity > r->recCapacity) {
        CUDA_TRY(cudaStreamSynchronize(r->stream));
        poolFree(r->recCounts, r->stream);
        poolFree(r->recList, r->stream);
        hostRelease(r->recHost);
        r->recCounts = nullptr; r->recList = nullptr; r->recHost = nullptr;
        r->recChunks = r->recCapacity = 0;
        const size_t bytes = sizeof(RecordHeader) + sizeof(uint2) * (size_t)capacity;
        CUDA_TRY(poolAlloc(&r->recCounts, sizeof(unsigned int) * chunks, r->stream));
        CUDA_TRY(poolAlloc(&r->recList, bytes, r->stream));
        CUDA_TRY(hostAcquire(reinterpret_cast<void**>(&r->recHost), bytes));
        r->recChunks = chunks;
        r->recCapacity = capacity;
    }
    static_assert(sizeof(RecordHeader) == sizeof(uint2), "the pairs follow the header");
    uint2 *list = reinterpret_cast<uint2*>(r->recList + 1);
    auto perArrays = [&](auto launch) {
        RecordArrays A;
        A.first_chunk = 0;
        uint32_t base = 0;
        for(uint32_t first = 0; first < num_arrays; first += RECORD_ARRAYS) {
            A.num = 0;
            A.chunk_start[0] = 0;
            for(uint32_t i = first; i < std::min(num_arrays, first + RECORD_ARRAYS); i++) {
                A.words[A.num] = words[i];
                A.num_words[A.num] = (unsigned int)num_words[i];
                A.base[A.num] = base;
                base += (uint32_t)num_words[i];
                A.num++;
                A.chunk_start[A.num] = A.chunk_start[A.num - 1] + (unsigned int)((num_words[i] + RECORD_CHUNK - 1) / RECORD_CHUNK);
            }
            if(A.chunk_start[A.num]) launch(A);
            A.first_chunk += A.chunk_start[A.num];
        }
    };
    perArrays([&](const RecordArrays &A) {
        recordCountKernel<<<A.chunk_start[A.num], RECORD_BLOCK, 0, r->stream>>>(A, r->recCounts);
        r->launches++;
    });
    perArrays([&](const RecordArrays &A) {
        recordListKernel<<<A.chunk_start[A.num], RECORD_BLOCK, 0, r->stream>>>(A, r->recCounts, (unsigned int)chunks, r->recList, list, capacity, r->state);
        r->launches++;
    });
    CUDA_TRY(cudaPeekAtLastError());
    // header and, in the same copy, about as many pairs as the last pull brought; what is left in a second one
    const size_t first = std::min<size_t>(capacity, r->recLast + r->recLast / 4 + 512);
    CUDA_TRY(cudaMemcpyAsync(r->recHost, r->recList, sizeof(RecordHeader) + sizeof(uint2) * first, cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    const size_t count = r->recHost->count;
    *num_pairs = count;
    if(count <= capacity) {
        r->recLast = count;
        uint2 *host = reinterpret_cast<uint2*>(r->recHost + 1);
        if(count > first) {
            CUDA_TRY(cudaMemcpyAsync(host + first, list + first, sizeof(uint2) * (count - first), cudaMemcpyDeviceToHost, r->stream));
            CUDA_TRY(cudaStreamSynchronize(r->stream));
        }
        *pairs = host;
    }
    return reportDeviceError(r, r->recHost->error);
}

int b200_decode_recording(const uint32_t *words, const void *pairs, uint64_t num_pairs, uint32_t base, uint32_t rows, uint32_t batch,
                          uint32_t words_per_row, uint32_t first_row, uint32_t num_neurons, uint32_t first_id, double start, double dt,
                          uint64_t *counts, double *const *times, uint32_t *const *ids)
{
    if((!words && !pairs && num_pairs) || !counts || !rows || !batch || !words_per_row || first_row >= rows ||
       num_neurons > 32ull * words_per_row || num_neurons + 32ull <= 32ull * words_per_row || (ids && !times)) {
        return fail(B200_ERR_INVALID, "bad arguments to b200_decode_recording");
    }
    decodeRecording(words, static_cast<const uint32_t*>(pairs), num_pairs, base, rows, batch, words_per_row, first_row, num_neurons, first_id,
                    start, dt, counts, times, ids);
    return B200_OK;
}

int b200_pull_spikes(b200_runner *r, const uint32_t *count_ptr, const uint32_t *list_ptr, uint32_t capacity, uint32_t *ids, uint32_t *num)
{
    if(!r || !count_ptr || !list_ptr || !ids || !num) return fail(B200_ERR_INVALID, "null argument to b200_pull_spikes");
    // count, error word and the first ids in one synchronisation
    const uint32_t first = std::min<uint32_t>(capacity, STAGE_BYTES / sizeof(uint32_t));
    std::lock_guard<std::mutex> lock(r->staging);
    CUDA_TRY(cudaMemcpyAsync(r->hostWord + 1, count_ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaMemcpyAsync(r->hostWord, &r->state->error, sizeof(uint32_t), cudaMemcpyDeviceToHost, r->stream));
    if(first) CUDA_TRY(cudaMemcpyAsync(r->stage, list_ptr, sizeof(uint32_t) * first, cudaMemcpyDeviceToHost, r->stream));
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    const uint32_t n = std::min(r->hostWord[1], capacity);
    memcpy(ids, r->stage, sizeof(uint32_t) * std::min(n, first));
    if(n > first) {
        CUDA_TRY(cudaMemcpyAsync(ids + first, list_ptr + first, sizeof(uint32_t) * (n - first), cudaMemcpyDeviceToHost, r->stream));
        CUDA_TRY(cudaStreamSynchronize(r->stream));
    }
    *num = n;
    return reportDeviceError(r, r->hostWord[0]);
}

int b200_timed_begin(b200_runner *r)
{
    if(!r) return fail(B200_ERR_INVALID, "null runner");
    int e = prepare(r);
    if(e) return e;
    CUDA_TRY(cudaStreamSynchronize(r->stream));
    CUDA_TRY(cudaEventRecord(r->evC, r->stream));
    return B200_OK;
}

int b200_timed_end(b200_runner *r, float *milliseconds)
{
    if(!r || !milliseconds) return fail(B200_ERR_INVALID, "null argument");
    CUDA_TRY(cudaEventRecord(r->evD, r->stream));
    CUDA_TRY(cudaEventSynchronize(r->evD));
    CUDA_TRY(cudaEventElapsedTime(milliseconds, r->evC, r->evD));
    return B200_OK;
}

}   // extern "C"
