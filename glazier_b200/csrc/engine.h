// Internal interface between the host engine (engine.cu) and the kernel
// files. Nothing here crosses the C ABI.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "device.cuh"

namespace glz {

constexpr int kMaxSpecies = 8;
constexpr int kMaxTypes = 64;

// Lattice geometry. A plane has d == 1, dim == 2, four colours; a volume has
// dim == 3 and eight.
struct Geometry {
    int w, h, d, dim, ncol, sites;
    int n_off;          // energy neighbourhood (lattice.rs:69-88)
    int off[26][3];
    int ring_n;         // positions of the connectivity veto's ring, 0 when off
    int nm;             // exact moment sums per cell: 5 in a plane, 9 in a volume
    // w, h and their halves (a colour's targets per row and rows per plane)
    // as multiply-shift dividers; set_dividers fills them from w and h
    Divider div_w, div_h, div_hw, div_hh;
};

inline void set_dividers(Geometry &g) {
    g.div_w = make_divider((uint32_t)g.w);
    g.div_h = make_divider((uint32_t)g.h);
    g.div_hw = make_divider((uint32_t)(g.w / 2 > 0 ? g.w / 2 : 1));
    g.div_hh = make_divider((uint32_t)(g.h / 2 > 0 ? g.h / 2 : 1));
}

// A type's target volume or surface as the kernels' tables hold it: zero where
// the term's weight is zero, so that the term is a finite number times zero
// whatever target the model states for it (infinite, NaN, or past f32).
inline float weighted_target(double target, float weight) { return weight != 0.0f ? (float)target : 0.0f; }

// Per-type tables in device memory, row-major [type][...], index 0 the medium.
struct TypeTables {
    const float *contact;       // n_types * n_types
    const float *target_volume, *lambda_volume, *target_surface, *lambda_surface;
    const double *target_length, *lambda_length, *division_volume, *death_rate;
    const uint8_t *connected;
    const float *chemotaxis, *secretion, *uptake;  // n_types * n_species
    const float *external;                         // n_types * 3: the drift vector
    const float *max_activity, *lambda_activity;   // the motility (Act) term
    const double *lambda_nematic;
};

// The tables a sweep prices with sit in one allocation (an engine's, or a
// replica's of the ensemble up to lambda_surface), in this order, so a block
// copies them into shared memory as one run of words: byte offsets for
// n types and ns species. The first `lean` bytes are all that contact, volume
// and surface terms read.
struct TypeLayout {
    int contact, target_volume, lambda_volume, target_surface, lambda_surface, lean;
    int target_length, lambda_length, lambda_nematic;
    int max_activity, lambda_activity, external, chemotaxis, connected, bytes;
    __host__ __device__ constexpr TypeLayout(int n, int ns)
        : contact(0), target_volume(4 * n * n), lambda_volume(target_volume + 4 * n),
          target_surface(lambda_volume + 4 * n), lambda_surface(target_surface + 4 * n), lean(lambda_surface + 4 * n),
          target_length((lean + 7) / 8 * 8), lambda_length(target_length + 8 * n),
          lambda_nematic(lambda_length + 8 * n), max_activity(lambda_nematic + 8 * n),
          lambda_activity(max_activity + 4 * n), external(lambda_activity + 4 * n), chemotaxis(external + 12 * n),
          connected(chemotaxis + 4 * n * ns), bytes((connected + n + 3) / 4 * 4) {}
};
constexpr int kSmemTypes = 16;  // tables of up to this many types are held in shared memory

// The per-cell tallies a colour pass reads, in the rotation that gives every
// pass a snapshot without an extra launch:
//   the value at the start of pass p is B[p % 2] + D[(p + 2) % 3];
//   pass p adds its changes into D[p % 3], and on the way writes
//   B[(p + 1) % 2] = B[p % 2] + D[(p + 2) % 3] and clears D[(p + 1) % 3],
//   none of which any thread of pass p reads.
// `vol_surf` words hold (volume, surface); `mom` holds nm int64 sums per cell.
struct Tallies {
    int2 *vs_base[2];
    long long *vs_delta[3];
    long long *mom_base[2];
    long long *mom_delta[3];
    int *vol_by_colour;  // ncol per cell: only the current colour's entry changes in a pass
    int *anchor;         // 4 per cell (x, y, z, unused): the integer origin of the moment sums
};

// The device clock of an engine whose steps replay from one captured CUDA
// graph: the kernels of a step read the step's number, its first pass's
// number and each species' current field buffer here, so the same graph
// serves every step; the graph's last node advances it.
struct EngineClock {
    long long step;       // Monte Carlo steps completed
    long long pass;       // colour passes completed
    unsigned field_cur;   // bit s: the buffer (0 or 1) holding species s
    unsigned field_flip;  // bit s: species s takes an odd number of sub-steps, so its buffer flips each step
};

struct SweepLaunch {
    Geometry g;
    TypeTables t;
    int n_types, n_species;
    float beta;  // (float)(1 / T), rounded once on the host
    int colour;
    int32_t step;
    uint64_t key_pick, key_accept;  // stream_key(seed, step, colour, 0 / 1)
    uint32_t *labels;
    const uint8_t *cell_type;
    // this pass's view of the tallies
    const int2 *vs_base;
    const long long *vs_prev;
    unsigned long long *vs_cur;
    int2 *vs_next_base;
    long long *vs_clear;
    const long long *mom_base;
    const long long *mom_prev;
    unsigned long long *mom_cur;
    long long *mom_next_base;
    long long *mom_clear;
    int *vol_by_colour;
    const int *anchor;
    int n_labels;
    // Population models keep their live label count in device memory (it
    // changes on the device when cells divide); n_labels is then the
    // capacity and kernels read the count here. Null otherwise.
    const int *n_live;
    int uniform_type;  // the type of every label when they share one, else -1
    int uniform_contact_exact;  // J m is exact in f32 for every |m| <= n_off (see sweep.cu)
    float uniform_contact;      // J[type][type] when uniform
    float u_target_volume, u_lambda_volume, u_target_surface, u_lambda_surface;
    int has_length, tracks, has_chemotaxis, has_external, has_motility, has_nematic;
    // the nematic field, (Q_xx, Q_xy) per site; its per-cell sums ride in the
    // moment words after the geometric ones (g.nm counts both)
    const float *nematic;
    // Motility reads labels and activity two sites from the target, where
    // same-colour targets change during the pass, so a pass with it leaves
    // both as they were and lists its accepted copies for launch_apply_copies.
    const float *activity;
    uint4 *pending;  // target, new label, its type's maximum activity (f32 bits)
    int *pending_count;  // this pass's, and the other pass parity's (cleared for the next pass)
    int *pending_clear;
    int use_tma;
    int lean;                // price contact, volume and surface only: no length, chemotaxis, connectivity or moment tracking
    int direct;              // take the direct kernel
    int compact;             // the direct kernel queues unlike copies before pricing them: 1 per warp, 2 per block
    int direct_span;         // targets a block (a streaming warp) of the queueing direct kernel takes
    int rotate_share;        // labels whose tallies a direct block rotates (without n_live)
    int max_ctas;            // > 0 caps the persistent grid (each CTA then walks more tiles)
    const void *tensor_map;  // CUtensorMap in device-visible memory, or null
    int *error_flag;
    // A clocked launch (the direct kernel only) takes its step, draws, tally
    // slots and field buffers from `clock` at run time: from this pass's
    // colour, the seed, every tally array and the field buffers.
    const EngineClock *clock;
    uint64_t seed;
    Tallies tal;
    float *field_buf;    // two buffers per species, species-major
    unsigned field_cur;  // bit s: the buffer holding species s (a clocked launch reads the clock's)
};

cudaError_t launch_sweep(const SweepLaunch &a, cudaStream_t stream);

// Every requested MCS of a lean model with nothing between its passes in one
// launch (the cluster sweep, the band sweep).
struct ResidentLaunch {
    SweepLaunch a;           // static fields; the pass fields are set per pass
    uint64_t seed;
    int32_t step0;           // the first MCS's step number
    int mcs;                 // MCS to run
    long long pass0;         // the first pass's number (the tally rotation's phase)
    int2 *vs_base[2];
    long long *vs_delta[3];
    unsigned *barrier;       // [0] arrivals, [1] barriers completed; zero at launch
};

// Targets a pass from which the direct kernel queues a block's unlike copies
// (of a lean plane: more than 148 SMs' four blocks of 256 take at once; of a
// volume; of a plane with terms past contact, volume and surface) and from
// which each warp streams over a run of its own (of a lean plane: more than
// one wave of gathering blocks holds; of the others).
constexpr int kDirectGatherFrom = 148 * 4 * 256 + 1;
constexpr int kDirectGatherVolumeFrom = 5 << 14;
constexpr int kDirectGatherEveryFrom = (1 << 16) + 1;
constexpr int kDirectCompactPlaneFrom = 148 * 4 * 512 + 1;
constexpr int kDirectCompactFrom = 1 << 20;

// Every requested MCS of a small lean plane in one thread-block cluster holding
// it in shared memory; cudaErrorNotSupported (nothing launched) when it does not fit one.
cudaError_t launch_cluster_sweep(const ResidentLaunch &r, cudaStream_t stream);

// Every MCS of a call (or one MCS, when fields run between steps) of a large
// lean plane in one cooperative launch: one CTA per SM streams its band of
// rows through shared memory, a grid barrier between passes (band.cu).
// cudaErrorNotSupported (nothing launched) when the plane does not suit it.
cudaError_t launch_band_sweep(const ResidentLaunch &r, cudaStream_t stream);
// Whether a plane of this width and height suits the band sweep on the
// current device (rows whole 16-byte units, a ring of enough rows).
bool band_sweep_fits(int w, int h);

// Apply a motility pass's listed copies: the label, and the activity of a
// type with a maximum (lib.rs:696-698); then clear the next pass's count.
cudaError_t launch_apply_copies(const SweepLaunch &a, float *activity, cudaStream_t stream);

// The activity's memory runs down by one each Monte Carlo step
// (lib.rs:426-432, motility.rs).
cudaError_t launch_activity_decay(float *activity, int sites, cudaStream_t stream);

// The batched ensemble: independent replicas of one neighbourhood, all their
// runs of targets (or tiles) in one launch per colour. Replica state lives in flat
// arrays; each replica's SweepLaunch holds its static fields (geometry,
// tables, absolute label/type/colour-count pointers) and the kernel patches
// the per-pass ones from the clock.
struct EnsembleClock {
    long long step;  // Monte Carlo steps completed
    long long pass;  // colour passes completed
};

struct EnsembleReplica {
    SweepLaunch a;
    long long cell_off;  // first entry of this replica in the flat per-cell arrays
    uint64_t seed;
};

struct EnsembleLaunch {
    int n;             // replicas
    int total_tiles;
    int colour;
    int max_ctas;
    const EnsembleReplica *replicas;
    const void *maps;        // one CUtensorMap per replica (64-byte aligned), or null
    const int *tile_prefix;  // n + 1 entries, in schedule order
    const int *order;        // schedule position -> replica
    const EnsembleClock *clock;
    int2 *vs_base[2];
    long long *vs_delta[3];
    long long total_cells;
    int ncol;
    int uniform_contact_exact;
    int *error_flag;
    // 0: the windowed persistent kernel (128 x 32 tiles); 1, 2, 3: one block
    // per tile of 32 x 8, 16 x 16 or 64 x 4 targets of a plane, priced where
    // they lie (tile_prefix and total_tiles then count those tiles);
    // kEnsembleRuns: a block per run of kEnsembleRun consecutive targets of a
    // replica (total_tiles counts the runs)
    int tile_shape;
    const int2 *runs;  // per run: its replica, its first target
    // The colour schedule of the direct shapes: 0 a launch per colour pass;
    // 1 every pass of the step in one cooperative launch, blocks striding
    // over the tiles, a grid barrier (bounded, error flag 4) between passes.
    int one_launch;
    unsigned *barrier;  // [0] arrivals, [1] barriers completed; zero at launch
};

constexpr int kEnsembleRuns = 4;    // the tile shape of runs
constexpr int kEnsembleRun = 1024;  // targets a run

// Targets per tile along x and y of ensemble tile shape `shape` (1, 2, 3).
inline void ensemble_tile(int shape, int &bx, int &by) {
    bx = shape == 1 ? 32 : (shape == 2 ? 16 : 64);
    by = 256 / bx;
}

cudaError_t launch_ensemble_sweep(const EnsembleLaunch &e, int dim, int n_off, bool uniform, cudaStream_t stream);
cudaError_t launch_clock_advance(EnsembleClock *clock, int ncol, cudaStream_t stream);
int ensemble_grid_cap(int dim, int n_off, bool uniform);

struct FieldLaunch {
    Geometry g;
    int n_types, n_species;
    int round;
    float d[kMaxSpecies], decay[kMaxSpecies];
    int active[kMaxSpecies], last[kMaxSpecies];
    const uint32_t *labels;
    const uint8_t *cell_type;
    const float *secretion, *uptake;
    // the infection rule (an extension): the uptake of species infect_species
    // by cells of type infect_from adds into dose[label], in units of 2^-24
    int infect_species = -1;  // -1: no rule
    int infect_from;
    unsigned long long *dose;
    // Two buffers per species, species-major: a round reads the one that
    // field_cur (or, clocked, the clock) and the round give, and writes the
    // other. field_cur is as at the step's start in every round.
    float *field_buf = nullptr;
    unsigned field_cur = 0;
    const EngineClock *clock = nullptr;
};

cudaError_t launch_field_round(const FieldLaunch &a, cudaStream_t stream);

// Fixed-point scale of the infection dose: an uptake amount u adds
// rint(u * 2^24), so the sum is exact and its order does not matter.
constexpr float kDoseScale = 16777216.0f;

// Recount every tally from the lattice into base slot `slot`, clearing every
// delta word: volume, per-colour volume, surface, anchor (first site in scan
// order) and the exact moment sums.
struct RecountLaunch {
    Geometry g;
    uint32_t *labels;
    int n_labels;
    int2 *vs_base;
    long long *mom_base;
    long long *vs_delta[3];
    long long *mom_delta[3];
    int *vol_by_colour;
    int *anchor;
    int *first;  // scratch per label: its first site in scan order
    int tracks;
    const float *nematic;  // with the nematic term: its sums follow the moments
    // Set to 2 when a label is not below n_labels; the recount of a lattice
    // from outside (without `flags`) then makes the site medium, so that no
    // sweep indexes an array with it.
    int *error_flag;
    // Population models: the live count in device memory (n_labels is then
    // the capacity).
    const int *n_live;
    // The recount at a population step's end: the two steps' event flags (it
    // runs only when this step's, by the step's or the clock's parity, are
    // nonzero; the step's own kernels have then cleared the tallies and found
    // the first sites).
    const int *flags;
    const EngineClock *clock;
    long long step;
};

cudaError_t launch_recount(const RecountLaunch &a, cudaStream_t stream);

// Fold the pending deltas into the base: B[s] += D[pd]; D[pd] = 0.
// With `n_live` (device memory) the count is read there and n_labels is the
// capacity.
cudaError_t launch_settle(int2 *vs_base, long long *vs_delta, long long *mom_base, long long *mom_delta, int nm,
                          int n_labels, int tracks, const int *n_live, cudaStream_t stream);
// Advance an engine's clock by one step of `ncol` passes.
cudaError_t launch_engine_clock_advance(EngineClock *clock, int ncol, cudaStream_t stream);

// The medium's volume and unlike-bond surface, counted from the lattice
// (the sweep keeps no tally for label 0).
cudaError_t launch_medium_count(const Geometry &g, const uint32_t *labels, unsigned long long *out,
                                cudaStream_t stream);

struct PopulationLaunch {
    Geometry g;
    TypeTables t;
    uint32_t *labels;
    uint8_t *cell_type;
    int n_types;
    int n_labels;            // without n_live
    int cap;
    int has_pop, tracks;     // has_pop 0: the infection rule alone
    int *n_live;             // the live label count; the decision adds the daughters to it
    Tallies tal;
    int base_slot;           // of the settled tallies (a step has an even number of passes: its start's)
    int *vol_by_colour;
    const int *anchor;
    uint64_t key_death;      // stream_key(seed, step, kPopulationStream, 0)
    long long step, pass;    // the step's number; the pass count at its end
    const EngineClock *clock;  // clocked: step and pass from here, with `seed`
    uint64_t seed;
    // the infection rule (infect_from -1: none)
    int infect_from, infect_to;
    long long infect_threshold;
    const unsigned long long *dose;
    // scratch, cap entries each
    unsigned char *mode;
    double *plan;            // 6 per cell: centroid, axis
    int *moved;
    uint32_t *daughter;
    int *first;
    int *flags;              // two steps' event flags, by the step's parity
    int *ticket;             // blocks done counting
    // Where the host sees the count (mapped memory): (step << 32) | the count
    // before that step's divisions, written when seen_step >= 0.
    unsigned long long *seen;
    long long seen_step;
};

__device__ __forceinline__ int population_parity(const PopulationLaunch &a) {
    return (int)((a.clock ? a.clock->step : a.step) & 1);
}

// Have the pages of a host buffer that a copy is about to fill mapped in one
// call: a fresh buffer's pages otherwise fault one by one inside the driver's
// copy, which takes five times as long as the copy itself (51 MB in 64
// lattices: 22 ms, 15 with this, 4.3 into pages already mapped). Changes no
// content, and does nothing to a buffer that has its pages.
void prefault(void *p, size_t bytes);

// Record the message glz_last_error() returns on this thread, and clear CUDA's
// own record of the thread's last error.
void set_last_error(const std::string &msg);

}  // namespace glz

struct glz_gpu;

namespace glz {

// An engine's steps replayed inside another graph (the batched ensemble):
// whether its steps replay from a captured graph at all; the clock set from
// its counters before a run of replays; its clocked step as a graph, with the
// version of its per-label arrays the graph holds; before each replay, room
// for that step's divisions (syncing `replays` first when it must read its
// count; a growth changes the version and the graph must be captured anew);
// after each replay, its counters; after the run, its count and error flag.
bool engine_replays(const glz_gpu *h);
int engine_begin_replays(glz_gpu *h);
int engine_step_graph(glz_gpu *h, cudaGraph_t *out, uint64_t *version);
int engine_before_replay(glz_gpu *h, cudaStream_t replays, uint64_t *version);
void engine_after_replay(glz_gpu *h);
int engine_end_replays(glz_gpu *h);

// A step's per-label end: the infection rule, division and death; a
// population model's recount (launch_recount with `flags`) follows it.
cudaError_t launch_step_labels(const PopulationLaunch &a, cudaStream_t stream);

}  // namespace glz
