/*
 * kernels.h - device data layouts and host-callable launchers of the
 * transport and reduction kernels.
 */
#ifndef PTG_KERNELS_H
#define PTG_KERNELS_H

#include <cuda_runtime.h>
#include <stdint.h>

namespace ptg {

/* ---------------- plain FP64 kernel ------------------------------------- */

/* Built geometry in device memory, FP64 structure of arrays (the
   ptg_geometry fields the transport reads). */
struct Geo64 {
  const double* vertex;      /* closed polygons, 3 per vertex        */
  const double* normal;      /* 3 per surface                        */
  const double* tangent;     /* 9 per surface, column-major          */
  const double* center;      /* 3 per surface                        */
  const double* radius;
  const double* spec;
  const double* tparam;
  const int* shape;
  const int* nvertex;
  const int* vbegin;
  const int* kind_trans;
  const int* gout;
  const int* internal;
  const int* incident;
  const int* grain_begin;
  const int* grain_incident;
  const double* grain_gen;   /* 3 per grain                          */
  double box[3];
  double scope[2];
  int face_kind[6];
  int kind_grain, ngrain, igrain_fill, nmaterial;
  double max_omega;
};

/* Per task: lambda [nm] (1e10 ballistic, <= 0 skipped), cos/sin of the
   incident angle, mode omega. */
struct Task64 {
  double lambda, cth, sth, omega;
};

/* Most facet planes of a grain: the tail phase's balls take one a lane. */
constexpr int kMaxPlanes = 32;

/* GeoF32.has_ext of the FP32 kernels that read a chunk table. */
constexpr int kChunkTableExt = 1;

/* Work queue of a run: chunk c is particles [j, j + size), j = (c % per_task)
   size, of task order[c / per_task], clipped to np_local. */
struct ChunkQueue {
  const int* order;          /* tasks, longest expected trajectories first      */
                             /* (NULL: as they are numbered)                    */
  int32_t per_task, size, np_local;
};

struct Run64 {
  const Task64* task;
  int64_t ntask;
  int64_t np;                 /* particles per task (all ranks)          */
  int64_t np_local;           /* particles of this rank per task         */
  int32_t rank, nranks;
  uint32_t k0, k1, c1;        /* Philox key and stream word              */
  int64_t max_flights;
  int32_t ref_quirks;
  unsigned long long* counts; /* [ntask]                                 */
  unsigned long long* lost;   /* [ntask]                                 */
  unsigned long long* stats;  /* flights, lost, capped, samples          */
  /* replay of one task (replay_task >= 0) */
  int64_t replay_task;
  int* end_side;
  unsigned* flights;
  double* final_pos;
  /* persistent kernels: the work queue, scheduling and tail list of RunF32
     (kTail64Units float4 per phonon; queue[4] phonons on the list) */
  ChunkQueue chunks;
  int32_t nchunk;
  int* queue;
  int32_t regen_threshold, fast_steps, coop_lanes, grace_steps;
  float fast_lambda_max;
  float round_lambda_max;    /* phonons with a longer MFP end in the drain     */
  float4* tail;
  int32_t tail_cap;
  int32_t* tail_order;
  int32_t* tail_hist;
};

cudaError_t launch_plain_fp64(const Geo64& g, const Run64& r, cudaStream_t st, int* grid,
                              int* block);

/* ---------------- persistent FP32 kernel -------------------------------- */

/* Surface record types in the FP32 blob. */
/* REC_CAP: capped cylinder, its (unit axis, half length) in the edge array */
enum { REC_POLY = 1, REC_SPHERE = 2, REC_CYL = 3, REC_CAP = 4 };
enum { REC_INTERIOR = 1 << 8 };

/* Offsets (in 16-byte units) of the sections of the FP32 geometry blob. */
struct BlobLayout {
  int hot;          /* float4[2*nsurf]: A = shape data, B = int4 (type, e0, ne, geom) */
  int cold;         /* float4[3*nsurf]: (t1,spec) (t2,tparam) (n, kind|gout<<8)      */
  int edge;         /* float4[nedge]  : in-plane inward edge normal m, m.v           */
  int cand_begin;   /* int[ngrain_total+1]                                           */
  int cand;         /* int[ncand]                                                    */
  int start;        /* voronoi: float4 (generatrix, grain); bricks: int2 (surf, grain) */
  int bvh_root;     /* int[ngrain_total]: root node of the grain's BVH, -1 linear scan */
  int plane_begin;  /* int[ngrain_total+1]: a BVH grain's distinct planes (facet_planes) */
  int plane;        /* float4: outward unit normal, offset                            */
  int nplane;       /* planes in the blob (0: no grain has them)                      */
  int bvh_node;     /* float4[2*nnode]: (lo, a) (hi, b), see bvh.cpp                  */
  int nbvh;         /* BVH nodes in the blob (0: every grain scans linearly)          */
  int ncap;         /* capped-cylinder records in the blob                            */
  int total;        /* blob size in 16-byte units                                    */
  int nstart;
};

struct GeoF32 {
  const float4* blob;  /* device blob (global memory)                    */
  BlobLayout lay;
  float box[3];
  float scope[2];
  float eps;           /* absolute geometric tolerance [nm]              */
  int periodic_mask;   /* bit f set: box face f is periodic              */
  int kind_grain, igrain_fill, nmaterial;
  int stage_smem;      /* 1: copy the blob to shared memory (bulk copy)  */
  int node_stage;      /* else: float4 units of the BVH node region (its  */
                       /*    top levels, breadth first) copied instead    */
  int has_ext;         /* 1: a BVH or capped cylinders (kernels built for  */
                       /*    them; the others leave both out), 2: a grain  */
                       /*    with facet planes as well                    */
};

/* One geometry of a batched launch (device table, read through the cache). */
struct GeoEntry {
  const float4* blob;
  BlobLayout lay;
  float box[3];
  float scope[2];
  float eps;
  float fast_lambda_max;
  int periodic_mask, kind_grain, igrain_fill, nmaterial;
  long long np;                /* particles per task of this geometry        */
  unsigned k0, k1, c1;         /* Philox key and stream word                 */
  int task_base;               /* first global task of this geometry         */
  int nsurf;                   /* its surfaces (adjoint replay)               */
  int adj_base;                /* its adjoint accumulators' first element    */
};

/* Per task (FP32): lambda (inf = ballistic, <= 0 skipped), cos, sin, omega/max_omega */
struct RunF32 {
  const float4* task;
  ChunkQueue chunks;          /* the chunks, longest expected trajectories first   */
  const int4* chunk;          /* their table (task, first local particle, count, 0),
                                 read instead by batches and by the kernels for a
                                 BVH or capped cylinders without facet planes
                                 (kChunkTableExt) */
  int32_t nchunk;
  int64_t np;
  int32_t rank, nranks;
  uint32_t k0, k1, c1;
  uint32_t max_flights;
  int32_t ref_quirks;
  int32_t regen_threshold;
  int32_t fast_steps;         /* a quarter of the most ball flights per iteration,
                                 but for the last group's (0: off)                 */
  float fast_lambda_max;      /* tasks with a smaller MFP use the fast path           */
  int32_t coop_lanes;         /* once the queue is dry, a warp with at most this many
                                 live phonons moves them to the tail list, where
                                 each gets a warp of its own that advances it 32
                                 flights a round (0: off)                         */
  int32_t grace_steps;        /* passes a warp's long-MFP phonons (no fast path) get
                                 after the queue is dry before they go to the list
                                 too (grace_passes)                               */
  float4* tail;               /* tail list: kTailUnits float4 per phonon           */
  int32_t tail_cap;           /* its capacity in phonons                           */
  int32_t* tail_order;        /* the tail phase takes list slots in this order
                                 (launch_tail_order), else front then back         */
  int32_t* tail_hist;         /* order buckets' histogram and cursors
                                 (kTailOrderExtra ints, zeroed before the drain)   */
  int32_t stage_test;         /* test only: set up the shared-memory staging
                                 barrier without issuing the copy, so its
                                 bounded wait runs out (PTG_ERR_TIMEOUT)          */
  unsigned long long* counts;
  unsigned long long* lost;
  /* flights, lost, capped, samples, max trajectory flights,
     t_start and t_drain (the largest complement, 0: none), t_end (max) in
     globaltimer ns,
     flights taken with the intersection test, safe balls built */
  unsigned long long* stats;
  int* queue;                 /* [0] next chunk, [1] error flags, [2] / [4] phonons
                                 put at the front / back of the tail list, [3]
                                 next tail-list phonon, [5] tail-list requests
                                 (8 ints) */
  /* adjoint support */
  unsigned long long* tlist;  /* mode 1: sample ids of transmitted phonons         */
  unsigned long long tlist_cap;
  const unsigned long long* alist;  /* mode 2: sample ids to replay               */
  long long alist_n;
  const float* wsample;       /* mode 2: d kappa / d T_task / np, per task         */
  double* adj;                /* mode 2: [kAdjBatches][nsurf + 1] accumulators     */
  int nsurf;
  /* mode 3: per replayed sample, positions (3 floats) at trace_off[t] ..
     trace_off[t+1] (trace NULL: counting pass), position count and exit */
  float* trace;
  const long long* trace_off;
  long long* trace_npos;
  int* trace_end;
  /* batched launch: geometry table and the geometry of every global task */
  const GeoEntry* geos;
  const int* task_geo;
};

/* u64 statistics slots of a transport launch: 0 flights, 1 lost, 2 capped,
   3 samples, 4 longest trajectory, 5-7 globaltimer start / queue dry / end,
   8 full-test flights, 9 safe balls, 10 listed samples, 11 replay
   mismatches, 12 cooperative rounds, 13 cooperative flights, 14 BVH boxes,
   15 surfaces tested, 16 flights of phonons handed to the tail phase before
   the hand-over, 17 flights of phonons that ended in the tail phase. */
constexpr int kStatSlots = 24;

/* Scheduling defaults of the persistent kernel (ptg_options 0 = these):
   idle lanes before a warp refills, fast-path flights per lane and
   iteration (structures whose grains are scanned linearly take short
   fast-path bursts, their full flights being cheap: thin film 16.5 ->
   15.8 ms, Voronoi 312 -> 305 ms at 4 against 8; those with a BVH or capped
   cylinders amortise dearer full flights over longer ones: C3 766 / 740 /
   733 ms and C4 3877 -> 3817 ms at 4 / 8 / 12, and with three drain blocks
   per SM C4 3661 -> 3592 ms at 12 -> 20; the batched launch keeps 8). */
constexpr int kDefaultRegen = 2;
constexpr int kDefaultFastSteps = 8;
constexpr int kDefaultFastStepsPlain = 4;
constexpr int kDefaultFastStepsExt = 20;
inline int default_fast_steps(const GeoF32& g) {
  return g.has_ext ? kDefaultFastStepsExt : kDefaultFastStepsPlain;
}

/* Passes (one full flight per lane each) that the drain phase gives its
   long-MFP phonons once the queue is dry, before it hands them to the tail
   phase like the diffusive ones.  Most of them leave the box within a few
   dozen flights, most flights ending at a surface, and a round of the tail
   phase then advances one phonon by a single flight: a warp that takes them
   one after the other needs about 2000 cycles a flight, a drain pass about
   3500 for 32 of them.  So they stay where the tail phase would get many per
   warp (120 000 phonons, MFP 150 nm in a 200 nm cube: 432 -> 209 us; 3.6e6
   ballistic ones among spheres: 1107 -> 710 us) and go at once where it gets
   few (3200 phonons in a porous film, MFP 100 nm: 229 us against 248 with 16
   passes, 260 with 32).  The two are equal at 4 to 8 phonons per warp, and
   16 and 32 passes at about 40.  Behind a BVH a pass waits for 32 tree walks,
   so the line lies higher (64 spheres and 16 capped cylinders, 2e5 phonons,
   MFP 150 nm: 6.0 -> 3.1 ms, a mesh with 17 a warp, 2000 nm: 2.6 -> 2.1; but 14
   a warp, ballistic: lattice of 5^3 cubes 2.27 ms against 2.00 without the
   passes, a prism 0.55 against 0.46).  Below 40 the longest MFP also has to be
   a quarter of the smallest box side: shorter ones outlive the passes (MFP 10
   nm among a sphere and a cylinder, 14 a warp: 1.49 against 1.37 ms).  The
   adjoint's two passes hand over at once: their tail is a few long
   trajectories, which the passes only delay (9.9 ms against 10.5 with 16). */
inline int grace_passes(int64_t samples, int64_t tail_warps, bool bvh, double longest_mfp, double box_min) {
  if (samples >= 40 * tail_warps) return 32;
  return samples >= (bvh ? 16 : 6) * tail_warps && longest_mfp >= 0.25 * box_min ? 16 : 0;
}

/* Replays are split in this many interleaved batches (sample % kAdjBatches)
   whose spread gives the standard error of the adjoint estimates. */
constexpr int kAdjBatches = 8;
/* kernel modes: forward, forward + list of transmitted samples, adjoint replay */
/* forward tallies; + list of transmitted samples; adjoint replay of a list;
   trace replay of a list (one-lane full flights, positions recorded) */
enum { MODE_FORWARD = 0, MODE_LIST = 1, MODE_ADJOINT = 2, MODE_TRACE = 3 };

cudaError_t launch_persistent_fp32(const GeoF32& g, const RunF32& r, int grid, int block,
                                   size_t smem, cudaStream_t st, int mode = MODE_FORWARD);
/* Fills the chunk table of the queue's nchunk chunks. */
cudaError_t launch_expand_chunks(const ChunkQueue& q, int nchunk, int4* chunks, cudaStream_t st);
/* Orders the tail list for the tail phase, longest expected remaining walk
   first, into order (tail_cap ints) from the buckets' histogram that the drain
   phase fills as it hands phonons over (hist: kTailOrderExtra ints with the
   buckets' cursors, zeroed by the caller before the drain).  One kernel between
   the drain and the tail launch on the same stream. */
constexpr int kTailOrderExtra = 256;
cudaError_t launch_tail_order(const float4* tail, int units, int tail_cap, const int* queue,
                              int32_t* order, int32_t* hist, cudaStream_t st);
/* The FP64 pair: the same queue and list, FP64 flights; the blob of g32 gives
   the bounds for balls and BVH walks. */
cudaError_t drain64_occupancy(int block, int* blocks_per_sm, int ext);
cudaError_t tail64_occupancy(int block, int* blocks_per_sm, int ext);
cudaError_t launch_drain64(const Geo64& g, const GeoF32& g32, const Run64& r, int grid, int block,
                           cudaStream_t st);
cudaError_t launch_tail64(const Geo64& g, const GeoF32& g32, const Run64& r, int grid, int block,
                          cudaStream_t st);
/* The FP32 tail phase (forward, list and adjoint modes): the phonons the drain
   phase left in r.tail, one per warp. */
cudaError_t launch_tail_fp32(const GeoF32& g, const RunF32& r, int grid, int block, size_t smem,
                             cudaStream_t st, int mode = MODE_FORWARD);
cudaError_t tail_occupancy(int block, size_t smem, int* blocks_per_sm, int mode = MODE_FORWARD,
                           int ext = 0, bool whole = true);
/* Batched launch over several geometries (geometry in global memory):
   forward, list (ids of transmitted samples as (global task << 32) |
   particle) or adjoint replay of such a list. */
cudaError_t launch_persistent_batch(const RunF32& r, int grid, int block, cudaStream_t st,
                                    int ext, int mode, bool tail);
cudaError_t persistent_batch_occupancy(int block, int* blocks_per_sm, int ext, int mode, bool tail);
/* float4 per phonon in the tail list: the state of a phonon handed from the
   drain phase to the tail phase (position, direction, free path, MFP, the
   ball centre and radii, grain, last surface, task, omega, sample id,
   flight, adjoint terms, second ball). */
constexpr int kTailUnits = 7;
/* ... and in the FP64 one: (ball centre, ball radii squared) in FP32, then
   position, direction, free path and MFP in FP64, (grain and surface last
   met, order bucket, grain), (task, sample id, flight).  Both layouts hold
   the order bucket at word 26. */
constexpr int kTail64Units = 8;
/* Shared memory for staged BVH nodes when the whole blob is not staged:
   64 KB, the top ten or so levels of the trees, small enough that two
   blocks of the tail kernel (kStaticSmem of its own at most) still fit on an
   SM. */
constexpr int kNodeStageUnits = 4096;
constexpr size_t kStaticSmem = 27 * 1024;
/* Dynamic shared memory of a transport launch: the whole blob, or the
   staged BVH nodes, or none. */
inline size_t dynamic_smem_bytes(const GeoF32& g, size_t blob_bytes) {
  if (g.stage_smem) return blob_bytes;
  return (size_t)g.node_stage * 16u;
}
/* Violations recorded by the bounds-checked build (PT_CHECK); other builds
   return cudaErrorNotSupported. */
cudaError_t check_report(long long* count, int* code, int* index, bool reset);
cudaError_t check_report_planes(long long* count, int* code, int* index, bool reset);
cudaError_t check_report_batch(long long* count, int* code, int* index, bool reset);
cudaError_t check_report_fp64(long long* count, int* code, int* index, bool reset);
/* The part of the FP32 kernels built for facet planes, behind
   launch_persistent_fp32, launch_tail_fp32 and their occupancies. */
cudaError_t planes_occupancy(int block, size_t smem, int* blocks_per_sm, int mode, bool whole, bool tail);
cudaError_t launch_planes(const GeoF32& g, const RunF32& r, int grid, int block, size_t smem, cudaStream_t st,
                          int mode, bool tail);
/* Residency of the persistent kernel for a block size and shared memory. */
cudaError_t persistent_occupancy(int block, size_t smem, int* blocks_per_sm,
                                 int mode = MODE_FORWARD, int ext = 0, bool whole = true);

/* ---------------- FP64 kappa reduction ---------------------------------- */

struct ReduceIn {
  const unsigned long long* counts;  /* [ntask]                          */
  int64_t nmode;
  int32_t nangle, ns, kind_mfp, nbins;
  double np;                         /* particles per task                */
  double dS;                         /* Simpson step * 1.5 * Lx           */
  double tnorm;                      /* 0.75 * Lx                         */
  const double* coef;                /* [nangle] Simpson c_a sin cos      */
  const double* K;                   /* [nmode]                           */
  const double* W;                   /* [nmode]                           */
  const double* mfp_m;               /* [nmode] bulk MFP [m]              */
  const int* bin;                    /* [nmode]                           */
  const double* grid;                /* [ns] (GRID)                       */
  /* scratch and outputs */
  double* tc;                        /* [nmode] kappa per mode            */
  double* kv;                        /* [nmode] kappa variance per mode   */
  double* bw;                        /* [nmode] W * <T>                   */
  double* bv;                        /* [nmode] W^2 var<T>                */
  double* emfp_nm;                   /* [nmode]                           */
  double* transmit;                  /* [nmode*ns*nangle] or null         */
  double* result;                    /* [2 + 3*nbins]: kappa, var, (sumW, sumWT, sumW2V) per bin */
};

cudaError_t launch_kappa_reduce(const ReduceIn& in, cudaStream_t st);

/* Batched reduction: the same spectrum for ngeo geometries whose counts are
   stored one after another (ntask_per_geo each); per geometry np and box x.
   result: [ngeo][2 + 3*nbins]. */
struct ReduceBatchIn {
  ReduceIn base;               /* counts, coef, K, W, mfp_m, bin, grid, nbins... */
  int ngeo;
  long long ntask_per_geo;
  const double* np_geo;        /* [ngeo] */
  const double* dS_geo;        /* [ngeo] */
  const double* tnorm_geo;     /* [ngeo] */
};
cudaError_t launch_kappa_reduce_batch(const ReduceBatchIn& in, cudaStream_t st);

}  // namespace ptg

#endif
