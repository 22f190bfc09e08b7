// b2d_dev.h — records shared by the host planner and the CUDA kernels.
//
// Device layout: every world (one Solver) is a self-contained block of device
// memory holding all of its arrays; a DWorld record (in a device table) holds
// the world's parameters and pointers into its block.  Work lists name
// (world, item) pairs, so a batch or a serving pool is just a table of worlds.
// Solver particles stay in insertion order, exactly like the reference's
// Vec<Particle> (src/solver.rs:24).
#pragma once
#include <cstdint>

// CUDA's vector types (plain C structs, usable by the host compiler too)
#include <vector_functions.h>
#include <vector_types.h>

#include <cstring>

namespace b2d {

// Collision extension flags (not in the reference; see solve_dynamic_collisions).
enum : uint32_t { COLLIDE_PP = 1u, COLLIDE_PC = 2u, COLLIDE_PPOLY = 4u };
// World flag set by the planner: every solver particle of this world belongs
// to a body that the shared-memory link executor runs, so that executor
// enters each particle into the collision grid (a slot insert, or the
// sorted grid's count) as it stores the body back: no separate insert or
// count kernel for this world.
constexpr uint32_t GRID_IN_LINKS = 8u;

// Schedule op ids on the host: a body-local link index, or a body-local
// particle index with this bit set (bounds + integrate).
constexpr uint32_t OP_INTEG = 0x80000000u;
// Second word of a link op whose first word is the link index (bodies of more
// than 65,535 particles, whose endpoints do not fit one word).
constexpr uint32_t OP_WIDE = 0xFFFFFFFFu;

// A body is a set of solver particles run by one executor unit: a union of
// whole link-connected components, so no link crosses two bodies.
struct DBody {
  uint32_t i0, np;       // particle list bidx[i0 .. i0+np) (world indices, ascending)
  uint32_t l0, nl;       // links lab[l0 .. l0+nl) (serial bodies: lrec) in execution order
  uint32_t sched;        // schedule id (group executors); serial bodies: links of the first
                         // half, which runs beside the second half of the pass before it
                         // a lag (flags >> BODY_LAG_SHIFT) behind (0: the links run in one chain)
  uint32_t local;        // 1: link endpoints are body-local; 0: world indices
  uint32_t first;        // bidx[i0 + i] == first + i for every i, else NO_FIRST
  uint32_t flags;        // BODY_*
};
// Every link's stiffness is exactly 1: the executors keep no stiffness.
// Every rest length is below 2^100 in magnitude: the fused-arithmetic link
// solve (kernels.cuh, link_solve_fused) may run.
// A serial executor's body.
// One whose consecutive links (within each half) share one particle: it is
// carried from link to link in registers.
enum : uint32_t { BODY_UNIT = 1u, BODY_RANGE = 2u, BODY_SERIAL = 4u, BODY_CARRY = 8u };
constexpr uint32_t BODY_LAG_SHIFT = 8;
// Mark on a link endpoint of a serial body in two chains: no later link of
// the pass moves this particle (it is integrated right after).
constexpr uint32_t LINK_FINAL = 0x80000000u;
// A carried body's record {x, y, ..}: y is the endpoint that the link before
// hands on, x the other one.  On x: the link is (y, x), not (x, y).  On y: y is
// handed on once more, else x is.
constexpr uint32_t LINK_SWAPPED = 0x40000000u, LINK_KEEP = 0x40000000u;
constexpr uint32_t LINK_INDEX = 0x3FFFFFFFu;
constexpr uint32_t NO_FIRST = 0xFFFFFFFFu;

// a serial record's endpoints in the link's order (carried: its body is one of
// BODY_CARRY; others may index past LINK_INDEX)
__host__ __device__ inline uint2 record_ends(const uint4& r, bool carried) {
  const uint32_t mask = carried ? LINK_INDEX : ~LINK_FINAL;
  const uint32_t x = r.x & mask, y = r.y & mask;
  return carried && (r.x & LINK_SWAPPED) ? uint2{y, x} : uint2{x, y};
}

struct DPoly {
  uint32_t v0, nv;       // vertices
  uint32_t l0, nl;       // polygon links (polygon-local indices)
  uint32_t is_static, pad;
};

// A level schedule is stored as a stream of self-describing chunks of at most
// SCHED_CHUNK_WORDS 32-bit words, each 16-byte aligned so that one bulk copy
// (TMA, cp.async.bulk) moves it into shared memory:
//   word 0            rounds in the chunk
//   words 1..         the end of each round, counted in the chunk's ops, and
//                     the last one twice more, so that an executor can load
//                     two rounds ahead without a test.  Link-pass schedules:
//                     the end; whole-update schedules: (end of the round's
//                     link ops) | (end of the round) << 16
//   (pad to an even word)
//   then two words per op, a round's link ops first:
//     link op    {a | b << 16, link index}   (body-local endpoints; bodies
//                                             of up to 65535 particles)
//                {link index, OP_WIDE}       (larger bodies)
//     integrate  {p | p << 16, 0}            (up to 65535 particles)
//                {p, 0}                      (larger bodies)
// A round is a whole level, or a piece of one (of at most DSched::tl link ops
// in schedules for the shared-memory executor); a group barrier follows it.
constexpr uint32_t SCHED_CHUNK_WORDS = 4096;
// words before the ops of a chunk of n rounds
constexpr uint32_t sched_head_words(uint32_t n) { return (n + 4u) & ~1u; }
// shared bytes after each executor group's schedule area: two mbarriers and
// two flag words
constexpr uint32_t GROUP_TAIL_BYTES = 32;
// Threads of a group executor's CTA, one group or several: at most 512 link
// and 256 integrate threads in a whole update; a link pass, whose launches may
// have more bodies than SMs, stays within the 64 registers that let two CTAs
// of 512 threads share an SM (200 cloths of 32x32, a pass: 44 us; with 70
// registers 61 us).
constexpr uint32_t group_threads_max(bool full) { return full ? 768u : 512u; }
struct DSched {
  uint32_t chunk0, nchunks;  // chunk_off / chunk_len entries
  uint32_t nlvl, nops;
  uint32_t off, words;       // the chunks are contiguous: stream[off, off + words)
  uint32_t tl, ti;           // threads that run link ops and integrate ops (shared-memory and
                             // flow executors; 0 in schedules for the other executors)
};

// Flow schedules (large bodies, k_exec_flow): the C CTAs of a cluster each run
// their own ops of every level, in chunks like the above (DSched::off: C
// records of FLOW_REC_WORDS words, below), except that
//   a round's word is   link ops end | round end << 11 | level % 32 << 22
//                       (the two after the last carry the next round's level)
//   an op is            {a | b << 16, k | to(a) << 16 | to(b) << 23}
//                       with k the CTA's own link index; to(x), where the
//                       particle goes after this op: bit 0 set when its next
//                       user is another CTA, bits 1-3 that CTA, bits 4-6 one
//                       less than the levels until it has to be there
// and one more op {lo | lo << 16, 0} ends each chunk (in no round), so that a
// chunk without ops has one to read.
constexpr uint32_t FLOW_REC_WORDS = 16;
enum : uint32_t {            // words of a CTA's record
  FR_CHUNK0, FR_NCHUNKS,     // its chunks: chunk_off / chunk_len entries
  FR_LO, FR_WINDOW,          // body-local ids [lo, lo + window) have a slot here
  FR_OWN0, FR_OWN1,          // particles it integrates
  FR_LINKS, FR_NLINKS,       // stream offset: body link of each of its link indices
  FR_LOAD, FR_NLOAD,         // particles that start here
  FR_STORE, FR_NSTORE,       // particles that end here
  FR_EXPECT, FR_NLEVELS,     // per level: particles that have to arrive before it
};
// shared bytes beside a flow CTA's state: the cluster's addresses, arrival, progress and fill
// barriers, the flags, the chunk count of each fill buffer
constexpr uint32_t FLOW_TAIL_BYTES = 512;
constexpr uint32_t STREAM_BUFFERS = 2 * SCHED_CHUNK_WORDS * 4;  // two fill buffers of a chunk
constexpr uint32_t FLOW_MAX_C = 8;     // CTAs in a cluster
constexpr uint32_t FLOW_AHEAD = 8;     // most levels between a send and its deadline
constexpr uint32_t FLOW_BARS = 32;     // arrival barriers, by level % FLOW_BARS
constexpr uint32_t FLOW_SKEW = 16;     // levels between the CTAs' progress checks: a sender is at
                                       // most this far ahead of a receiver, so a deadline is less
                                       // than FLOW_BARS levels past the receiver's level
static_assert(FLOW_SKEW + FLOW_AHEAD < FLOW_BARS, "arrival barriers must not wrap");

// 1 / c when c is a positive normal power of two (then x / c == x * (1/c)
// exactly for every x: both round the same real number), else 0.
inline float pow2_reciprocal(float c) {
  uint32_t u;
  std::memcpy(&u, &c, 4);
  const uint32_t e = (u >> 23) & 0xFFu;
  if ((u >> 31) || (u & 0x7FFFFFu) || e == 0u || e == 255u) return 0.0f;
  const int ne = 254 - (int)e;  // 2^(127 - (e - 127)) has exponent field 254 - e
  if (ne < 1 || ne > 254) return 0.0f;
  const uint32_t r = (uint32_t)ne << 23;
  float f;
  std::memcpy(&f, &r, 4);
  return f;
}

struct DWorld {
  // parameters
  float gx, gy;          // 0 + gravity: the acceleration at integrate time
  float bx, by, bw, bh;  // Bounds pos / size (src/solver.rs:13-17)
  float h;               // dt * (1 / sub_steps) (src/solver.rs:107-108)
  float radius, cell;    // extension: particle radius, grid cell
  uint32_t S, I;         // sub_steps, link iterations
  uint32_t flags;        // COLLIDE_* bits
  uint32_t slot;         // stable id (hash salt for the shared grid)
  uint32_t np, nb, nc, ncl, ng;
  uint32_t gb0, gmask;   // extension grid: this world's buckets [gb0, gb0 + gmask]
  uint32_t gp0;          // extension grid: this world's particle scratch offset
  float icell;           // 1 / cell when cell is a power of two (exact), else 0
  // solver particles
  float2* pos[2];        // ping-pong positions; pos[0] holds the state between steps
  float2* prev;
  // bodies and links
  DBody* bodies;
  uint32_t* bidx;
  uint2* lab;
  float* lrest;
  float* lstiff;
  uint4* lrec;           // serial bodies' links: {a, b, rest bits, stiffness bits}, endpoints
                         // body-local with their LINK_ marks
  // circles (src/circle.rs:4-8) and circle links
  float2* cpos; float2* cprev; float2* cacc;
  float* crad; uint32_t* cstatic;
  uint2* clab; float* clrest;
  // polygons (src/polygon.rs:7-14)
  DPoly* polys;
  float2* vpos; float2* vprev; float2* vacc;
  float2* pcenter;
  float4* paabb;
  uint2* plab; float* plrest;
  uint32_t* stage_off;   // polygon-pair test offsets, see stage_pair
  uint32_t* stage_pr;    // polygon pair of each stage: self | other << 16
};

// Shared (engine-wide) read-only schedule registry, plus the device error
// word that bounded waits set instead of trapping.
struct DScheds {
  const DSched* scheds;
  const uint32_t* chunk_off;  // word offset of each chunk in `stream`
  const uint32_t* chunk_len;  // words (multiple of 4)
  const uint32_t* stream;
  uint32_t* err;
  uint32_t fault;  // FAULT_BIT_* test switches (0 in normal operation)
};
enum : uint32_t { ERR_BIT_TMA_TIMEOUT = 1u, ERR_BIT_GRID_OVERFLOW = 2u };
// Test switch for failure detection: every executor group treats its first
// bulk-copy wait as timed out (and takes the timeout path: error word, wait
// for the copy in flight to land, leave) without a real timeout.
enum : uint32_t { FAULT_BIT_WAIT = 1u };

// Extension broadphase: hashed uniform grid, sorted form (large grids and
// the allocation-free entry point): built by a counting sort each sub-step.
// Every world with particle collisions owns a power-of-two range of
// buckets; a bucket's entries are contiguous in `sorted`.
// bucket scan tiles: 1,024 buckets (256 threads x 4 each) for grids of up to
// SCAN_SMALL_MAX buckets, else 16,384 (four sub-tiles of 1024 threads x 4)
constexpr uint32_t SCAN_SMALL_TILE = 1024;
constexpr uint32_t SCAN_LARGE_TILE = 16384;
constexpr uint32_t SCAN_SMALL_MAX = 1u << 20;
struct DGrid {
  uint32_t* count;       // nbuckets: entries per bucket (all zero between sub-steps)
  uint2* range;          // nbuckets: {first entry in sorted, count}
  uint32_t* cursor;      // entries of sorted handed out so far this sub-step
  uint2* pbr;            // per particle: (bucket, rank within bucket)
  uint4* sorted;         // cap entries: {pos.x bits, pos.y bits, cell x, cell y}
  uint32_t* err;         // device error word (ERR_BIT_*)
  uint32_t nbuckets;
  uint32_t cap;
};

// The engine's form of the same grid: no sort.  Each particle is inserted
// straight into its bucket, whose first GRID_SLOTS entries sit in fixed
// slots; later ones go to an overflow array, chained per bucket.  A
// sub-step's inserts use the cell words of parity sub & 1; that sub-step's
// collide pass clears the other parity's words for the next sub-step (and
// resets the overflow cursor).  Slots are interleaved by strip (four
// buckets): slot k of the strip's four buckets is one 64-byte run, so the
// first entries of a row of neighbour cells share a cache line.
constexpr uint32_t GRID_SLOTS = 4;
struct DSlots {
  uint2* cell;           // 2 x nbuckets (parity-major): {entries, overflow head + 1 (0: none)}
  uint4* slot;           // nbuckets x GRID_SLOTS entries {pos.x bits, pos.y bits, cell x, cell y}
  uint4* ovf;            // cap overflow entries
  uint32_t* ovf_next;    // cap: the bucket's next overflow entry + 1 (0: end)
  uint32_t* cursor;      // overflow entries handed out this sub-step
  uint32_t* err;         // device error word (ERR_BIT_*)
  uint32_t nbuckets;
  uint32_t cap;
};

}  // namespace b2d
