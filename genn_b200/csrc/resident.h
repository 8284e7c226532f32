// Target-resident persistent time-step kernel.
//
// A step of a batch-1 network is a dependent chain, not traffic: neuron update -> who spiked -> their synapses ->
// neuron update.  The kernels that share the input buffers between CTAs (fused_step.cuh, stream_step.cuh) pay for that
// chain at L2 distance several times over: spike-list atomics, a grid barrier with its release and acquire, the
// lists, the rows, reductions into L2, the buffers read back.  Here everything but the spikes stays inside the CTA:
//
//   * neurons are dealt out in units of 32 (one recording word) over the CTAs, unit u to CTA u % G: state in registers,
//     input buffers and dendritic-delay rings in shared memory;
//   * every CTA delivers ALL spikes, each onto its own neurons only.  A private copy of the SPARSE groups (built from
//     the caller's arrays, rebuilt when they change) holds, per source neuron and CTA, the synapses of all groups onto
//     that CTA's neurons as one run of 8-byte entries (ring slot and column, weight).  Runs of one source population
//     onto one CTA have the same padded length, so a spike's id leads to its entries in one memory round trip; the
//     runs of one source neuron lie side by side (one address translation per spike, not one per spike and CTA).
//     DENSE rows and BITMASK words are read where they are: a unit of 32 targets is 128 bytes or one word of a row;
//   * the only thing that crosses CTAs is one message per CTA and step: two 64-bit words (step number, spike count, the
//     first seven ids); further ids wait at the sender.  Every word carries its step number, so readers poll the
//     cells themselves: the all-gather IS the barrier, with no fence, no counter and no list.  A message is stored
//     once for every RESIDENT_READERS CTAs: with one copy for all, polling it grew from 1.8 k cycles at 32 CTAs to
//     8 k at 148, and with a copy for each the sender's stores took 10 cycles apiece, 1.6 k at 148.  (A step of 77 169 neurons
//     on 148 CTAs with 20 / 12 / 8 / 5 readers a copy: 4.17 / 4.15 / 4.07 / 4.04 us.)  A cell is
//     written again `buffers` steps later; its sender has by then received messages that every reader sent after it had
//     read this one.
//
// What has to be in place before the neuron update of a step is kept small.  Groups of one axonal delay form a class:
//
//   IMMEDIATE  the runs (and DENSE / BITMASK rows) of the step's spikes are added before the update;
//   SPLIT      every group has a delay ring: only synapses of dendritic delay 0 are needed at once.  They stand at the head of
//              every run, all heads of a step's spikes are one line of entries for the threads of the CTA, and the rest is
//              fetched behind them, while the neurons are updated, and added after that.  (They were rows of their own, one
//              per source neuron, which every CTA read whole.  us a step before / now, rings of 16, 1000 synapses: 4000 + 4000
//              neurons 3.74 / 3.00 at 10 spikes a step, 17.6 / 8.5 at 100; 40 000 + 40 000 neurons 3.56 / 2.89, 10.9 / 5.5);
//   LATE       no group has a ring and the axonal delay is a step or more: the spikes of the NEXT step are known
//              already, so their runs are fetched and added behind the update too, into the second of two buffers.
//              CTAs then run up to the delay apart, and no step waits for another SM or for memory.
//
// Busy networks.  Every CTA handles every spike, so a spike costs each of them the same, however many they are: about
// RESIDENT_RUN_COST ns of a warp for every chunk of its run and RESIDENT_NEAR_COST for every 32 entries of its head, where
// the kernels with a grid barrier share its synapses out (8.5 ps each; 20 with rings) behind a step that costs 2 to 4 us more
// to begin with.  A step of 10 000 + 10 000 neurons, 1000 synapses each: 3.3 us at 10 spikes a step (6.6 with the barrier),
// 7.5 at 100 (7.7), 16.5 at 300 (11.3), 163 at 3000 (62); 20 000 + 20 000, 200 synapses: 3.3 (6.5), 6.3 (6.8), 12.2 (6.9), 107
// (15); 4000 + 4000 with rings of 16, 1000 synapses: 3.0 (6.0), 8.5 (8.3), 22 (11.9), 69 at 1000 (23).  So a launch keeps
// account of what it loses: every spike delivered adds its class's `weight`, every step takes off `spare`, and when the sum
// passes `patience` the launch ends with the next step's list.  A launch of the other kernel that the host has put behind it does the rest
// up to the same step, and goes on for `resident_rest` steps, twice as many every time this happens, before this kernel is tried again.  All
// CTAs count the same spikes, so they leave at the same step without a word.  More spikes in one step than the list holds are left to
// the other kernel at once (models with one delay, up to 20 units a CTA): the messages' further ids are fetched by one lane per
// sender, 0.3 ms for every 2048 of them.
//
// Networks whose spikes need several steps, or come from populations without inputs, go through windows of steps instead
// (resident_window.cuh); there a spike costs the less and the account is kept window by window.
//
// Memory between launches is what every other path leaves: the first steps of a launch take the spikes of the steps
// before it from the spike lists, the last ones write them.
#pragma once

#include <cuda_runtime.h>

#include "neuron_update.cuh"
#include "window_tags.h"

namespace b200
{
constexpr unsigned int RESIDENT_BLOCK = 768;            // most threads of a CTA: 80 registers each
constexpr unsigned int RESIDENT_FEW = 640;              // threads up to which another instance has 96
constexpr unsigned int RESIDENT_UNITS = RESIDENT_BLOCK / 32;    // most units of 32 neurons of a CTA
constexpr unsigned int RESIDENT_MAX_CTAS = 256;
constexpr unsigned int RESIDENT_MAX_GROUPS = 64;        // neuron groups (a bit mask says which are sources)
constexpr unsigned int RESIDENT_CLASSES = 4;            // distinct ring depths / distinct axonal delays
constexpr unsigned int RESIDENT_LIST = 2048;            // spikes delivered between two barriers of a CTA
constexpr unsigned int RESIDENT_READERS = 5;            // CTAs that poll one copy of the messages (a lane stores each: at most 32 copies)
constexpr unsigned int RESIDENT_LOADS = 4;              // loads of a run that a lane has in flight
constexpr unsigned int RESIDENT_CHUNK = 32 * RESIDENT_LOADS;    // entries of a run that one warp takes
constexpr unsigned int RESIDENT_NEAR_LOADS = 4;         // entries of the runs' heads that a lane has in flight
constexpr unsigned int RESIDENT_DENSE_SPIKES = 8;       // rows of a DENSE group whose loads a lane has in flight
constexpr unsigned int RESIDENT_NEAR_MOST = 64;         // most delay-0 synapses of a run for a SPLIT class
constexpr float RESIDENT_RUN_COST = 560.0f, RESIDENT_NEAR_COST = 280.0f;        // ns of a warp for a chunk of a run / of heads
constexpr unsigned int RESIDENT_PIECE_COST = 300000;    // ns of a step with more spikes than the list holds, for every list of them
constexpr unsigned int RESIDENT_MOST_WEIGHT = 1000, RESIDENT_MOST_DEBT = 1u << 30;      // ns
constexpr unsigned int RESIDENT_REST = 48;              // steps on the other kernel, the first time
constexpr unsigned int RESIDENT_MOST_REST = 1u << 20;
constexpr unsigned int RESIDENT_PAD = 0xFFFFFFFFu;      // key of a padding entry
constexpr unsigned long long RESIDENT_TAG_STEPS = 1ull << 20;       // step numbers of messages are 20 bits
constexpr unsigned int RESIDENT_HEAD_IDS = 3, RESIDENT_MORE_IDS = 4;    // ids in a first word / in a further word
constexpr unsigned int RESIDENT_CELL_IDS = RESIDENT_HEAD_IDS + RESIDENT_MORE_IDS;  // ids in the two words of an inbox cell

enum ResidentClass { RESIDENT_IMMEDIATE = 0, RESIDENT_SPLIT = 1, RESIDENT_LATE = 2 };

// entry key of a run: ring class << 30 | delay << 16 | column
struct ResidentRun              // runs of one (axonal delay, source population) pair onto one CTA
{
    unsigned long long place;   // entries of the head (delay-0 synapses of a SPLIT class) << 48 | first entry of the run of source neuron 0
    unsigned int length;        // entries behind the head (0: none); with the head a multiple of four
    unsigned int row;           // entries between two source neurons: the runs of all CTAs
    __host__ __device__ unsigned int near() const { return (unsigned int)(place >> 48); }
    __host__ __device__ unsigned long long base() const { return place & 0xFFFFFFFFFFFFull; }
};

struct ResidentSpan             // a DENSE or BITMASK group
{
    const float *g;             // DENSE weights or NULL (constant)
    const unsigned int *gp;     // BITMASK words or NULL
    float weight;               // constant weight
    unsigned int row_stride;    // BITMASK: bits of a row
    unsigned int num_trg;
    unsigned int delay_class;
    unsigned int src_group, trg_group, psm;
    unsigned int num_src;
};

// Where the tables of a CTA lie in its dynamic shared memory (bytes): constants of the launch, so no thread keeps pointers.
struct ResidentLayout
{
    unsigned int groups, unit_start, unit_first, columns, runs, rows, spans, poisson, undrawn, history, acc;
};

struct ResidentLaunch
{
    NeuronLaunch neuron;
    ResidentLayout at;
    const unsigned int *unit_start;     // [num_groups + 1] units of 32 neurons before each group
    const unsigned int *unit_first;     // [num_units] neuron group << 24 | first neuron of the unit
    const unsigned int *columns;        // [grid][RESIDENT_UNITS][B200_MAX_PSM] ring class << 16 | first column
    const unsigned int *cta_columns;    // [grid][RESIDENT_CLASSES] columns of each ring class
    const ResidentRun *runs;            // [grid][delay classes][num_groups]
    const unsigned long long *rows;     // [delay classes][num_groups] where the runs of source neuron 0 begin
    const uint2 *entries;
    const float *poisson;               // [num_groups][64] distribution of the event count of a group's one Poisson source, or NULL
    const ResidentSpan *spans;
    unsigned int num_spans;
    unsigned int num_units;
    unsigned int num_depths, depth[RESIDENT_CLASSES];       // buffers per input: ring depths; without a ring 1, or 2 with a LATE class
    unsigned int num_delays, delay[RESIDENT_CLASSES];       // axonal delays
    unsigned int kind[RESIDENT_CLASSES];                    // ResidentClass of each delay
    unsigned long long source_groups;                       // groups with outgoing synapses of any delay
    unsigned long long sources[RESIDENT_CLASSES];           // neuron groups with outgoing synapses of that delay
    unsigned int chunks[RESIDENT_CLASSES];                  // warp items of the longest run of that delay (0: no runs)
    unsigned int near_most[RESIDENT_CLASSES];               // entries of the longest head of that delay (0: no heads)
    unsigned int near_share[RESIDENT_CLASSES];              // 2^32 / near_most, rounded up
    unsigned int acc_floats;            // shared memory of the input buffers
    unsigned int history;               // steps whose spike lists the launch has to leave behind
    unsigned int buffers;               // message buffers
    unsigned int more_words;            // words behind the cell a message may need
    ulonglong2 *inbox;                  // [buffers][copies][sender]
    unsigned int copies;
    unsigned int prefetch;              // 1: the runs do not stay in L2: a spiking neuron's are fetched ahead of its message
    unsigned long long *more;           // [buffers][sender][more_words]
    unsigned long long *leave;          // number of the launch at whose end the spike lists may be written
    unsigned long long launch;          // number of this launch: no other of the runner has it, and none is 0
    unsigned int num_steps;
    unsigned int count_events;
    unsigned int weight[RESIDENT_CLASSES];  // ns that a spike of that delay costs above what it costs the other kernel
    unsigned int quiet[RESIDENT_CLASSES];   // spikes of a step that cost half of `spare`: up to there nothing is accounted
    unsigned int spare;                     // ns that a step without spikes costs less than there
    unsigned int patience;                  // ns
    unsigned int may_leave;                 // 1: a launch of the other kernel follows that does what this one leaves
    unsigned long long *hold;               // page-locked: the host's copy of StepState::resident_hold
    unsigned long long *barrier;            // of the launch that follows: zeroed by this one
};

// the runs of one pair are counted (pass 0) and placed (pass 1) by one launch each
struct ResidentBuild
{
    const b200_synapse_group *groups;   // the SPARSE groups of one (axonal delay, source population) pair
    const unsigned int *target;         // per group: neuron group << 8 | postsynaptic model of its target
    unsigned int num_groups, num_src;
    const unsigned int *unit_start, *columns;
    const unsigned int *depth;          // buffers per input, by ring class
    unsigned int late;                  // 1: LATE class: every synapse arrives one step after its delivery
    unsigned int split;                 // 1: SPLIT class: delay-0 synapses stand at the head of a run
    unsigned int *near_longest;         // longest head of a run
    unsigned long long *synapses;       // all of the pair
    unsigned int grid;
    unsigned int runs_stride;           // distance between the pair's runs of two CTAs
};

// ---- windows of steps (resident_window.cuh) ----------------------------------------------------------
// Where no spike of a window of steps reaches anybody in that window, CTAs exchange once a window.
constexpr unsigned int RESIDENT_WINDOW_MOST = 16;       // most steps of a window
constexpr unsigned int RESIDENT_WINDOW_LEAST = 4;       // fewest
constexpr unsigned int RESIDENT_WINDOW_INLINE = 3;      // entries that travel with the head
constexpr unsigned int RESIDENT_HEADS = RESIDENT_MAX_CTAS + RESIDENT_UNITS;     // (those of a reading warp lie side by side, the last of each short)
constexpr unsigned int RESIDENT_WINDOW_LIST = 40960;    // spikes of a window that the list has room for (160 KB)

constexpr unsigned int RESIDENT_WINDOW_SPARE = 5500;    // ns that a step without spikes costs less than on the kernel with a grid barrier
// ns of a warp for 32 entries of a run.  us a step at 10 / 100 / 300 / 1000 / 3000 spikes, in windows and with a grid barrier: 10 000 -> 10 000
// neurons, 1000 synapses 1.0 / 3.1 / 7.0 / 20 / 56 and 6.8 / 7.9 / 11.4 / 24 / 61, 8000 -> 80 000, 500 synapses 1.0 / 2.8 / 5.8 / 17 / 47
// and 6.6 / 7.0 / 7.2 / 10.3 / 19.
constexpr float RESIDENT_WINDOW_COST = 430.0f;

struct ResidentWindow
{
    unsigned int steps;                 // of a window
    unsigned int feed;                  // 1: the spikes come from populations without inputs, which are a window ahead of the others
    unsigned int lag;                   // else: windows between a spike's and the one it arrives in
    unsigned int cap;                   // spikes of one step that the list has room for
    unsigned int ring;                  // steps whose ballots are kept
    unsigned int buffers;               // of messages
    unsigned int body;                  // most spikes of a message
    unsigned int run_groups;            // groups of 32 entries of the longest run (0: no runs)
    unsigned int list_at, words_at, acc_at;     // in dynamic shared memory, behind the tables of ResidentLayout
    unsigned int epoch;                 // of the launch (window_tags.h)
    unsigned long long free_groups;     // populations without inputs (FEED)
    ulonglong2 *heads;                  // [buffers][copies][RESIDENT_HEADS] tag << 20 | spikes, short tag << 48 | the first three entries
    unsigned short *bodies;             // [buffers][grid][body] step of the window << 10 | unit of the CTA << 5 | neuron
};

struct ResidentWindowLaunch
{
    ResidentLaunch L;
    ResidentWindow W;
};

// kernels: resident.cu, resident_window.cu
const void *residentWindowKernelFor(int npsm, int ncs);
const void *residentKernelFor(int npsm, int ncs, bool one_class, unsigned int threads);
cudaError_t residentBuild(const ResidentBuild &B, int pass, unsigned int *longest, const ResidentRun *runs, uint2 *entries, StepState *state,
                          unsigned int blocks, cudaStream_t stream);
}   // namespace b200
