// kernels.h: host-side launchers of the decision engine's CUDA stages.
//
// Every stage takes a list of frame jobs (FrameJob, device memory) so one launch scores several
// frames -- the leaf B frames of a mini-GOP, or frames of several streams of different sizes --
// and each CTA finds its job and unit from a prefix table of the jobs' unit counts.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace celv2cu {

constexpr int kMaxJobs = 32;

// The superblocks [sb0, sb0 + sbs) of a job.
struct SbRange {
  int job, sb0, sbs;
};

// Units of one stage as prefix sums: part p -- a job, or in the superblock stages (intra, inter,
// finalize) a range of its superblocks -- owns units [prefix[p], prefix[p + 1]).
// queue: the stage's work queue in device memory (zero before the launch) -- a persistent grid's
// CTAs take units from it in order until it runs dry; null: one CTA per unit (blockIdx.x).
struct WorkList {
  int nparts;
  int prefix[kMaxJobs + 1];
  SbRange part[kMaxJobs];
  unsigned* queue;
};

// The next unit of this CTA into `unit` (every thread gets it); false when the stage is done.
// Starts with a barrier, so the previous unit's shared state is free for the next one (slot: two ints
// of shared memory, used in turn). No CTA ever waits for another: a drained queue simply ends the loop.
__device__ __forceinline__ bool take_unit(const WorkList& w, int& unit, int& iter, int* slot) {
  const int total = w.prefix[w.nparts];
  if (!w.queue) {
    if (iter++) return false;
    unit = blockIdx.x;
    return unit < total;
  }
  int* s = slot + (iter++ & 1);
  if (threadIdx.x == 0) *s = (int)atomicAdd(w.queue, 1u);
  __syncthreads();
  unit = *s;
  return unit < total;
}

// CTAs of a persistent grid for a kernel: the SM count times the CTAs an SM holds, at most units.
int persistent_grid(const void* kernel, int threads, size_t smem, int units);

// Unit u's part (a linear scan: at most kMaxJobs parts).
__device__ __forceinline__ int part_of(const WorkList& w, int u) {
  int j = 0;
  while (j + 1 < w.nparts && u >= w.prefix[j + 1]) j++;
  return j;
}

// A plane to make from its uploaded samples (packed rows of the padded width): its pyramid with
// margins. shift: bit depth - 8 of 16-bit samples, -1: 8-bit samples.
struct PlaneIn {
  const void* raw;
  int shift;
  DevPyramid pyr;
};
struct PlaneSet {
  int n;
  PlaneIn p[kMaxRefs + 1];
};
// Level 0 with its margin and the pyramid of every plane of the set, from their samples.
void launch_pyramid(const PlaneSet& s, cudaStream_t st);
// The quarter-pel phase planes of every plane of the set (pyr.lv[0] alone is read).
void launch_phases(const PlaneSet& s, cudaStream_t st);

// Motion search of one pyramid level for every (job, reference, 8x8 cell), whole-pel (level 0's
// field in quarter pels). Units: me_units(nrefs, fcols[level], frows[level], cells) per job (groups
// of `cells` cells of one reference; cells 7, 15 or 30).
int me_units(int nrefs, int cols, int rows, int cells);
// The cells per CTA to run a level of `cells` cells (all jobs and references) with, `configured` or fewer.
int me_level_cells(long long cells, int configured);
void launch_me_level(const FrameJob* jobs, const WorkList& w, int level, int cells, cudaStream_t st);
// Level 0's quarter-pel refinement, in place. Units: refine_units(nrefs, fcols[0], frows[0]) per job.
int refine_units(int nrefs, int cols, int rows);
void launch_me_refine(const FrameJob* jobs, const WorkList& w, cudaStream_t st);

// Intra SATDs of every candidate block and mode. Units: the parts' superblocks (split further by the
// launcher where they are few).
void launch_intra(const FrameJob* jobs, const WorkList& w, cudaStream_t st);

// Each reference's best candidate MV per candidate block, the distinct MVs of a superblock taken
// in chunks of at most `chunk` (<= 64). Units: nrefs times the parts' superblocks. Units that keep
// their 64-level blocks are scored whole (k_inter); with `regions` (some job has keep words) a
// second kernel scores the others region by region, draining `region_queue` (zero beforehand).
void launch_inter(const FrameJob* jobs, const WorkList& w, int chunk, bool regions, unsigned* region_queue,
                  cudaStream_t st);

// The window the inter stage loads of a phase plane for a motion vector (its box): bytes, rows.
void inter_window(unsigned& bytes, unsigned& rows);

// Per-block choice, compound, partition choice and the decision records. Units: the parts' superblocks.
void launch_finalize(const FrameJob* jobs, const WorkList& w, cudaStream_t st);

// The learned pruner's decision rule (pruner.cu): per output group the probability a kept option needs
// (references, intra, block levels, intra modes), and the band around them inside which a superblock
// falls back to the full search.
struct PrunerThresholds {
  float ref, intra, level, mode, band;
};
// The jobs of a batch with features or a network: entry i owns superblocks [prefix[i], prefix[i + 1]).
struct NetList {
  int n;
  int prefix[kMaxJobs + 1];
  struct Entry {
    int job, nrefs;
    float* feats;         // superblocks x CELV2_PRUNER_FEATURES
    const float* params;  // the network's parameters
    const void* wb;       // and their bf16 copies (infer_weights: infer_weight_elems() elements)
    uint32_t* keep;       // the keep words it writes
    PrunerThresholds th;
  } e[kMaxJobs];
};
// Every entry's features; the network and the keep words of every superblock of the list.
void launch_features(const FrameJob* jobs, const NetList& l, cudaStream_t st);
void launch_infer(const NetList& l, cudaStream_t st);
size_t infer_weight_elems();
void infer_weights(const float* params, void* wb, cudaStream_t st);

}  // namespace celv2cu
