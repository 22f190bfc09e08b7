// planner.cpp — turns one world (the reference's Solver contents) into its
// device image: bodies, executor choice, level schedules and the world block.
//
// Level scheduling.  The reference applies links one at a time in insertion
// order (src/solver.rs:143-146), then bounds and integration per particle
// (src/solver.rs:155-158, :118-121).  Give each op the level
//   level(op) = 1 + max(level of the last earlier op touching any of its particles)
// Ops on one level touch disjoint particles, and every particle sees its ops
// in the original order, so executing level by level reproduces the
// sequential loop exactly.  A FULL schedule chains all sub-steps and link
// iterations of one Solver::update, which lets independent regions of a body
// run ahead into later passes (the critical path of a 32x32 cloth step drops
// from 4032 to ~413 levels).
#include <algorithm>
#include <array>
#include <cstdlib>
#include <cstring>
#include <numeric>

#include "engine.hpp"

namespace b2d {

static uint32_t pow2ceil(uint32_t x) {
  uint32_t p = 1;
  while (p < x) p <<= 1;
  return p;
}
static size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

bool PlanTuning::set(const std::string& k, double v) {
  if (k == "serial_width") serial_width = (float)v;
  else if (k == "t_min") t_min = (uint32_t)v;
  else if (k == "t_max") t_max = (uint32_t)v;
  else if (k == "pack_np") pack_np = (uint32_t)v;
  else if (k == "pack_nl") pack_nl = (uint32_t)v;
  else if (k == "free_chunk") free_chunk = (uint32_t)v;
  else if (k == "smem_max") smem_max = (uint32_t)v;
  else if (k == "warp_groups") warp_groups = (uint32_t)v;
  else if (k == "max_groups") max_groups = (uint32_t)v;
  else if (k == "width_per_thread") width_per_thread = (float)v;
  else if (k == "resident") resident = (uint32_t)v;
  else if (k == "res_max") res_max = (uint32_t)v;
  else if (k == "stage_frac") stage_frac = (float)v;
  else if (k == "bucket_factor") bucket_factor = (float)v;
  else if (k == "collide_thread_min") collide_thread_min = (uint32_t)v;
  else if (k == "large_max") large_max = (uint32_t)v;
  else if (k == "grid_slot_max") grid_slot_max = (uint32_t)std::min(v, 4294967295.0);
  else return false;
  return true;
}

// A round's time with tl <= 512 link threads, in 10 ns, beside a time for each
// op (measured on bodies of 840 to 4,200 particles): one to four warps a
// scheduler.
static uint32_t round_cost(uint32_t tl) {
  constexpr uint32_t ROUND[4] = {11, 13, 15, 19};
  return ROUND[(tl + 127u) / 128u - 1u];
}

uint32_t SchedRegistry::get(const uint2* links, uint32_t nl, uint32_t np, uint32_t S, uint32_t I,
                            bool full, bool group, const PlanTuning& t) {
  std::string key;
  uint32_t hdr[8] = {np, nl, S, I, (full ? 1u : 0u) | (group ? 2u : 0u), 0u, 0u, 0u};
  if (group) {
    hdr[5] = t.t_min;
    hdr[6] = t.t_max;
    std::memcpy(&hdr[7], &t.width_per_thread, 4);
  }
  key.resize(sizeof(hdr) + (size_t)nl * 8);
  std::memcpy(&key[0], hdr, sizeof(hdr));
  if (nl) std::memcpy(&key[sizeof(hdr)], links, (size_t)nl * 8);
  auto it = index.find(key);
  if (it != index.end()) return it->second;

  const uint32_t nsub = full ? S : 1u;
  const size_t total = (size_t)nsub * ((size_t)I * nl + (full ? np : 0));
  std::vector<uint32_t> last(np, 0), lvl_of, op_of;
  lvl_of.reserve(total);
  op_of.reserve(total);
  uint32_t maxl = 0;
  for (uint32_t s = 0; s < nsub; ++s) {
    for (uint32_t it2 = 0; it2 < I; ++it2) {
      for (uint32_t k = 0; k < nl; ++k) {
        const uint32_t a = links[k].x, b = links[k].y;
        const uint32_t l = std::max(last[a], last[b]) + 1;
        last[a] = l;
        last[b] = l;
        lvl_of.push_back(l);
        op_of.push_back(k);
        maxl = std::max(maxl, l);
      }
    }
    if (full) {
      for (uint32_t p = 0; p < np; ++p) {
        const uint32_t l = last[p] + 1;
        last[p] = l;
        lvl_of.push_back(l);
        op_of.push_back(OP_INTEG | p);
        maxl = std::max(maxl, l);
      }
    }
  }
  // stable counting sort by level
  std::vector<uint32_t> start(maxl + 2, 0);
  for (uint32_t l : lvl_of) start[l + 1]++;
  for (uint32_t l = 1; l <= maxl + 1; ++l) start[l] += start[l - 1];
  std::vector<uint32_t> sorted(total);
  {
    std::vector<uint32_t> fill(start.begin(), start.end());
    for (size_t i = 0; i < total; ++i) sorted[fill[lvl_of[i]]++] = op_of[i];
  }
  // a level's link ops first (its ops are independent, so their order within
  // the level is free); nlink[l] of them
  std::vector<uint32_t> nlink(maxl + 2, 0);
  uint32_t max_link = 0, max_integ = 0;
  for (uint32_t l = 1; l <= maxl; ++l) {
    const auto b = sorted.begin() + start[l], e = sorted.begin() + start[l + 1];
    const auto m = full ? std::stable_partition(b, e, [](uint32_t op) { return !(op & OP_INTEG); }) : e;
    nlink[l] = (uint32_t)(m - b);
    max_link = std::max(max_link, nlink[l]);
    max_integ = std::max(max_integ, (uint32_t)(e - m));
  }
  for (uint32_t op : sorted)  // self-check: ops name the body's links/particles
    if ((op & OP_INTEG) ? (op & ~OP_INTEG) >= np : op >= nl) std::abort();
  DSched d;
  d.chunk0 = (uint32_t)chunk_off.size();
  d.nlvl = maxl;
  d.nops = (uint32_t)total;
  d.tl = d.ti = 0;
  if (group) {
    // Threads for the link ops: the widest level's, in whole warps, within
    // the tunables; a wider level takes several rounds.  Threads for the
    // integrate ops: up to 256 (512 in a body without links, which has
    // nothing else to run); a wider round takes several turns.
    if (max_link) {
      const float avg = maxl ? (float)total / (float)maxl : 1.0f;
      const uint32_t want = pow2ceil((uint32_t)(avg / t.width_per_thread + 0.999f));
      d.tl = std::min((max_link + 31u) & ~31u, std::max(want, 32u));
      d.tl = std::min(std::max(d.tl, t.t_min), t.t_max);
      d.tl = std::min(std::max((d.tl + 31u) & ~31u, 32u), 512u);
    }
    if (max_integ) d.ti = std::min((max_integ + 31u) & ~31u, max_link ? 256u : 512u);
    if (max_link) {
      // Fewer link threads where the shorter rounds outweigh the more of them:
      // warps without an op issue a round's instructions too (round_cost).
      // 41x27 in fast order (levels of 509 to 553 links): 512
      // threads 486 rounds 126 us, 320 threads 519 rounds 111 us; 52x42: 512
      // threads 208 us, 384 threads 189 us; but 36x30 (480 to 540 links): 512
      // threads 353 rounds 101 us, 320 threads 519 rounds 109 us.
      auto cost = [&](uint32_t tl) {
        uint64_t r = 0;
        for (uint32_t l = 1; l <= maxl; ++l) r += (nlink[l] + tl - 1) / tl;
        return r * round_cost(tl);
      };
      const uint64_t now = cost(d.tl);
      uint64_t least = now - now / 20u;  // only for a gain of 5 %
      for (uint32_t tl = d.tl; tl > std::max(t.t_min, 32u);) {
        tl -= 32u;
        const uint64_t c = cost(tl);
        if (c <= least) {
          least = c;
          d.tl = tl;
        }
      }
    }
    if (d.tl + d.ti == 0) d.tl = 32;
  }
  // cut the level sequence into chunks of rounds (a level may span chunks)
  const bool narrow = np <= 65535u;
  std::vector<uint32_t> ends, chunk_ops;  // chunk_ops: op ids
  auto flush = [&]() {
    if (ends.empty()) return;
    while (stream.size() % 4) stream.push_back(0);
    chunk_off.push_back((uint32_t)stream.size());
    const size_t at = stream.size();
    stream.push_back((uint32_t)ends.size());
    stream.insert(stream.end(), ends.begin(), ends.end());
    stream.insert(stream.end(), 2, full ? (uint32_t)chunk_ops.size() * 0x10001u
                                        : (uint32_t)chunk_ops.size());
    if ((stream.size() - at) % 2) stream.push_back(0);
    if (stream.size() - at != sched_head_words((uint32_t)ends.size())) std::abort();
    for (uint32_t op : chunk_ops) {
      if (op & OP_INTEG) {
        const uint32_t p = op & ~OP_INTEG;
        stream.push_back(narrow ? p * 0x10001u : p);
        stream.push_back(0);
      } else if (narrow) {
        stream.push_back(links[op].x | (links[op].y << 16));
        stream.push_back(op);
      } else {
        stream.push_back(op);
        stream.push_back(OP_WIDE);
      }
    }
    while ((stream.size() - at) % 4) stream.push_back(0);
    chunk_len.push_back((uint32_t)(stream.size() - at));
    if (chunk_len.back() > SCHED_CHUNK_WORDS) std::abort();
    ends.clear();
    chunk_ops.clear();
  };
  // ops that still fit the open chunk beside one more round
  auto room = [&]() -> uint32_t {
    const size_t used = sched_head_words((uint32_t)ends.size() + 1) + 2 * chunk_ops.size() + 3;
    return used + 2 > SCHED_CHUNK_WORDS ? 0u : (uint32_t)(SCHED_CHUNK_WORDS - used) / 2;
  };
  for (uint32_t l = 1; l <= maxl; ++l) {
    uint32_t lk = start[l], in = start[l] + nlink[l];  // next link op, next integrate op
    const uint32_t le = in, ie = start[l + 1];
    while (lk < le || in < ie) {
      uint32_t want_l = le - lk;
      if (group && d.tl) want_l = std::min(want_l, d.tl);
      const uint32_t want = want_l + (ie - in);
      // a round that fits a chunk of its own is not split between two
      if (room() == 0 || (room() < want && !ends.empty() && group)) {
        flush();
        continue;
      }
      const uint32_t tl = std::min(want_l, room());
      const uint32_t ti = std::min(ie - in, room() - tl);
      chunk_ops.insert(chunk_ops.end(), sorted.begin() + lk, sorted.begin() + lk + tl);
      const uint32_t lend = (uint32_t)chunk_ops.size();
      chunk_ops.insert(chunk_ops.end(), sorted.begin() + in, sorted.begin() + in + ti);
      const uint32_t end = (uint32_t)chunk_ops.size();
      ends.push_back(full ? (lend | (end << 16)) : end);
      lk += tl;
      in += ti;
    }
  }
  flush();
  d.nchunks = (uint32_t)chunk_off.size() - d.chunk0;
  d.off = d.words = 0;
  if (d.nchunks) {
    d.off = chunk_off[d.chunk0];
    for (uint32_t c = d.chunk0; c + 1 < d.chunk0 + d.nchunks; ++c)  // self-check: contiguous
      if (chunk_off[c] + chunk_len[c] != chunk_off[c + 1]) std::abort();
    d.words = chunk_off.back() + chunk_len.back() - d.off;
  }
  const uint32_t id = (uint32_t)scheds.size();
  scheds.push_back(d);
  index.emplace(std::move(key), id);
  return id;
}

// CTA r of a flow body integrates particles [np*r/C, np*(r+1)/C) and solves the
// links whose first endpoint is one of them.
static void flow_owners(uint32_t np, uint32_t C, std::vector<uint32_t>& own, std::vector<uint8_t>& cta) {
  own.resize(C + 1);
  for (uint32_t r = 0; r <= C; ++r) own[r] = (uint32_t)((uint64_t)np * r / C);
  cta.resize(np);
  for (uint32_t r = 0; r < C; ++r)
    for (uint32_t p = own[r]; p < own[r + 1]; ++p) cta[p] = (uint8_t)r;
}

// The most of a CTA's {window, own particles, links} in the flow schedule over
// C CTAs, known before any of it is built.
static std::array<uint32_t, 3> flow_sizes(const uint2* links, uint32_t nl, uint32_t np, bool solves,
                                          bool integrates, uint32_t C) {
  std::vector<uint32_t> own;
  std::vector<uint8_t> cta;
  flow_owners(np, C, own, cta);
  std::vector<uint32_t> lo(own.begin(), own.end() - 1), hi(lo), count(C, 0);
  for (uint32_t r = 0; r < C; ++r) {
    if (integrates) hi[r] = own[r + 1];
    else if (solves) lo[r] = np;  // its links' particles alone
  }
  for (uint32_t k = 0; k < nl; ++k) {
    const uint32_t r = cta[links[k].x];
    ++count[r];
    if (!solves) continue;
    lo[r] = std::min(lo[r], std::min(links[k].x, links[k].y));
    hi[r] = std::max(hi[r], std::max(links[k].x, links[k].y) + 1);
  }
  std::array<uint32_t, 3> most{1, 0, 0};
  for (uint32_t r = 0; r < C; ++r) {
    if (hi[r] > lo[r]) most[0] = std::max(most[0], hi[r] - lo[r]);
    most[1] = std::max(most[1], own[r + 1] - own[r]);
    most[2] = std::max(most[2], count[r]);
  }
  return most;
}

uint32_t SchedRegistry::get_flow(const uint2* links, uint32_t nl, uint32_t np, uint32_t S, uint32_t I,
                                 bool full, uint32_t C) {
  std::string key;
  const uint32_t hdr[8] = {np, nl, S, I, (full ? 1u : 0u) | 4u, C, 0u, 0u};
  key.resize(sizeof(hdr) + (size_t)nl * 8);
  std::memcpy(&key[0], hdr, sizeof(hdr));
  if (nl) std::memcpy(&key[sizeof(hdr)], links, (size_t)nl * 8);
  auto it = index.find(key);
  if (it != index.end()) return it->second;
  if (np > 65535u || C < 2 || C > FLOW_MAX_C || np < C) return NONE;

  std::vector<uint32_t> own;
  std::vector<uint8_t> cta;
  flow_owners(np, C, own, cta);
  std::vector<uint32_t> lidx(nl);  // link -> its index among its CTA's links
  std::vector<std::vector<uint32_t>> mine(C);
  for (uint32_t k = 0; k < nl; ++k) {
    std::vector<uint32_t>& m = mine[cta[links[k].x]];
    lidx[k] = (uint32_t)m.size();
    if (m.size() > 65535u) return NONE;
    m.push_back(k);
  }
  // ops in sequence, with their levels; of each op, where its particles go next
  struct Op { uint32_t id, level; uint8_t cta, to[2]; };
  const uint32_t nsub = full ? S : 1u;
  std::vector<Op> seq;
  seq.reserve((size_t)nsub * ((size_t)I * nl + (full ? np : 0)));
  struct Use { uint32_t op; uint8_t end; };  // a particle's latest use
  std::vector<Use> last(np, Use{NONE, 0});
  std::vector<uint32_t> depth(np, 0), first(np, NONE), lo(C, NONE), hi(C, 0);
  std::vector<std::vector<uint32_t>> expect(C);
  uint32_t nlvl = 0;
  auto use = [&](uint32_t p, uint32_t op, uint8_t end) {
    Op& o = seq[op];
    lo[o.cta] = std::min(lo[o.cta], p);
    hi[o.cta] = std::max(hi[o.cta], p + 1);
    const Use u = last[p];
    if (u.op == NONE) {
      first[p] = o.cta;
    } else if (seq[u.op].cta != o.cta) {
      const uint32_t d = std::min(o.level - seq[u.op].level, FLOW_AHEAD);
      seq[u.op].to[u.end] = (uint8_t)(1u | (o.cta << 1) | ((d - 1u) << 4));
      std::vector<uint32_t>& e = expect[o.cta];
      const uint32_t at = seq[u.op].level + d;
      if (e.size() <= at) e.resize(at + 64, 0);
      ++e[at];
    }
    last[p] = Use{op, end};
    depth[p] = o.level + 1;
    nlvl = std::max(nlvl, o.level + 1);
  };
  for (uint32_t s = 0; s < nsub; ++s) {
    for (uint32_t it2 = 0; it2 < I; ++it2)
      for (uint32_t k = 0; k < nl; ++k) {
        const uint32_t a = links[k].x, b = links[k].y, op = (uint32_t)seq.size();
        seq.push_back(Op{k, std::max(depth[a], depth[b]), cta[a], {0, 0}});
        use(a, op, 0);
        use(b, op, 1);
      }
    if (full)
      for (uint32_t p = 0; p < np; ++p) {
        seq.push_back(Op{OP_INTEG | p, depth[p], cta[p], {0, 0}});
        use(p, (uint32_t)seq.size() - 1, 0);
      }
  }
  // by CTA, level, and kind: links that send, other links, integrate ops
  auto kind = [](const Op& o) { return o.id & OP_INTEG ? 2u : (o.to[0] | o.to[1]) & 1u ? 0u : 1u; };
  std::vector<uint32_t> count((size_t)C * nlvl * 3 + 1, 0);
  auto bin = [&](const Op& o) { return ((size_t)o.cta * nlvl + o.level) * 3 + kind(o); };
  for (const Op& o : seq) ++count[bin(o) + 1];
  for (size_t i = 1; i < count.size(); ++i) count[i] += count[i - 1];
  std::vector<uint32_t> order(seq.size());
  {
    std::vector<uint32_t> at(count.begin(), count.end() - 1);
    for (uint32_t i = 0; i < seq.size(); ++i) order[at[bin(seq[i])]++] = i;
  }
  uint32_t max_link = 0, max_integ = 0;
  for (size_t g = 0; g < (size_t)C * nlvl; ++g) {
    max_link = std::max(max_link, count[3 * g + 2] - count[3 * g]);
    max_integ = std::max(max_integ, count[3 * g + 3] - count[3 * g + 2]);
  }
  DSched d{};
  d.nlvl = nlvl;
  d.nops = (uint32_t)seq.size();
  d.ti = max_integ ? std::min((max_integ + 31u) & ~31u, 256u) : 0u;
  // Link threads as in get(), over the widest CTA of each level: 100x100 over
  // seven CTAs has 576 to 616 links in the widest one on 445 of 685 levels: two
  // rounds of 512 threads 526 us an update, one of 640 519 us, two of 320
  // 495 us.
  d.tl = std::min(std::max((max_link + 31u) & ~31u, 32u), 512u);
  std::vector<uint32_t> widest(nlvl, 0);
  for (uint32_t r = 0; r < C; ++r)
    for (uint32_t l = 0; l < nlvl; ++l) {
      const size_t g = (size_t)r * nlvl + l;
      widest[l] = std::max(widest[l], count[3 * g + 2] - count[3 * g]);
    }
  auto cost = [&](uint32_t tl) {
    uint64_t n = 0;
    for (uint32_t w : widest) n += (w + tl - 1) / tl;
    return n * round_cost(tl);
  };
  for (uint32_t tl = d.tl; tl >= 32u; tl -= 32u)
    if (cost(tl) < cost(d.tl)) d.tl = tl;
  d.chunk0 = (uint32_t)chunk_off.size();
  std::vector<uint32_t> rec((size_t)C * FLOW_REC_WORDS, 0);
  for (uint32_t r = 0; r < C; ++r) {
    uint32_t* R = &rec[(size_t)r * FLOW_REC_WORDS];
    if (lo[r] == NONE) lo[r] = own[r], hi[r] = own[r] + 1;
    R[FR_CHUNK0] = (uint32_t)chunk_off.size();
    R[FR_LO] = lo[r];
    R[FR_WINDOW] = hi[r] - lo[r];
    R[FR_OWN0] = own[r];
    R[FR_OWN1] = own[r + 1];
    std::vector<uint32_t> words, ops;  // of the open chunk: rounds; op indices in seq
    auto flush = [&](uint32_t next_level) {
      while (stream.size() % 4) stream.push_back(0);
      chunk_off.push_back((uint32_t)stream.size());
      const size_t at = stream.size();
      stream.push_back((uint32_t)words.size());
      stream.insert(stream.end(), words.begin(), words.end());
      const uint32_t end = (uint32_t)ops.size();
      stream.insert(stream.end(), 2, end | (end << 11) | ((next_level % 32u) << 22));
      if ((stream.size() - at) % 2) stream.push_back(0);
      for (uint32_t i : ops) {
        const Op& o = seq[i];
        if (o.id & OP_INTEG) {
          stream.push_back((o.id & ~OP_INTEG) * 0x10001u);
          stream.push_back((uint32_t)o.to[0] << 16);
        } else {
          stream.push_back(links[o.id].x | (links[o.id].y << 16));
          stream.push_back(lidx[o.id] | ((uint32_t)o.to[0] << 16) | ((uint32_t)o.to[1] << 23));
        }
      }
      stream.push_back(lo[r] * 0x10001u);
      stream.push_back(0);
      while ((stream.size() - at) % 4) stream.push_back(0);
      chunk_len.push_back((uint32_t)(stream.size() - at));
      if (chunk_len.back() > SCHED_CHUNK_WORDS) std::abort();
      words.clear();
      ops.clear();
    };
    auto room = [&]() -> uint32_t {  // ops that fit beside one more round and the last op
      const size_t used = sched_head_words((uint32_t)words.size() + 1) + 2 * ops.size() + 2 + 3;
      return used + 2 > SCHED_CHUNK_WORDS ? 0u : (uint32_t)(SCHED_CHUNK_WORDS - used) / 2;
    };
    for (uint32_t l = 0; l < nlvl; ++l) {
      const size_t g = (size_t)r * nlvl + l;
      uint32_t lk = count[3 * g], in = count[3 * g + 2];
      const uint32_t le = in, ie = count[3 * g + 3];
      do {  // a level without ops here is an empty round
        const uint32_t want_l = std::min(le - lk, d.tl), want = want_l + (ie - in);
        if (room() < std::max(want, 1u) && !words.empty()) flush(l);
        const uint32_t tl = std::min(want_l, room()), ti = std::min(ie - in, room() - tl);
        ops.insert(ops.end(), order.begin() + lk, order.begin() + lk + tl);
        const uint32_t lend = (uint32_t)ops.size();
        ops.insert(ops.end(), order.begin() + in, order.begin() + in + ti);
        words.push_back(lend | ((uint32_t)ops.size() << 11) | ((l % 32u) << 22));
        lk += tl;
        in += ti;
      } while (lk < le || in < ie);
    }
    flush(nlvl);
    R[FR_NCHUNKS] = (uint32_t)chunk_off.size() - R[FR_CHUNK0];
  }
  d.nchunks = (uint32_t)chunk_off.size() - d.chunk0;
  auto list = [&](const std::vector<uint32_t>& v, uint32_t* at, uint32_t* n) {
    *at = (uint32_t)stream.size();
    *n = (uint32_t)v.size();
    stream.insert(stream.end(), v.begin(), v.end());
  };
  for (uint32_t r = 0; r < C; ++r) {
    uint32_t* R = &rec[(size_t)r * FLOW_REC_WORDS];
    list(mine[r], &R[FR_LINKS], &R[FR_NLINKS]);
    std::vector<uint32_t> load, store;
    for (uint32_t p = 0; p < np; ++p) {
      if (first[p] == r) load.push_back(p);
      if (first[p] != NONE && seq[last[p].op].cta == r) store.push_back(p);
    }
    list(load, &R[FR_LOAD], &R[FR_NLOAD]);
    list(store, &R[FR_STORE], &R[FR_NSTORE]);
    expect[r].resize(nlvl, 0);
    list(expect[r], &R[FR_EXPECT], &R[FR_NLEVELS]);
  }
  while (stream.size() % 4) stream.push_back(0);
  d.off = (uint32_t)stream.size();
  d.words = (uint32_t)rec.size();
  stream.insert(stream.end(), rec.begin(), rec.end());
  const uint32_t id = (uint32_t)scheds.size();
  scheds.push_back(d);
  index.emplace(std::move(key), id);
  return id;
}

// Bounds check of a finished image: every index a kernel dereferences must
// land inside the world's arrays.  Runs on every plan (linear in the size of
// the world); a failure is a planner bug and stops the world from reaching
// the GPU.
static bool check_image(const WorldImage& im, const SchedRegistry& reg, std::string* why) {
  auto bad = [&](const std::string& m) {
    if (why) *why = "internal planner check failed: " + m;
    return false;
  };
  const DWorld& P = im.params;
  if (im.pos.size() != P.np || im.prev.size() != P.np) return bad("particle arrays");
  if (im.bodies.size() != P.nb) return bad("body count");
  for (const DBody& B : im.bodies) {
    if ((size_t)B.i0 + B.np > im.bidx.size()) return bad("body particle range");
    const bool serial = (B.flags & BODY_SERIAL) != 0u;
    if ((size_t)B.l0 + B.nl > (serial ? im.lrec.size() : im.lab.size()) ||
        im.lab.size() != im.lrest.size() || im.lab.size() != im.lstiff.size())
      return bad("body link range");
    for (uint32_t i = 0; i < B.np; ++i)
      if (im.bidx[B.i0 + i] >= P.np) return bad("body particle index");
    if (B.first != NO_FIRST &&
        ((size_t)B.first + B.np > P.np || (B.np && im.bidx[B.i0] != B.first)))
      return bad("body first particle");
    const uint32_t lim = B.local ? B.np : P.np;
    for (uint32_t k = 0; k < B.nl; ++k) {
      const uint2 e = serial ? record_ends(im.lrec[B.l0 + k], B.flags & BODY_CARRY) : im.lab[B.l0 + k];
      if (e.x >= lim || e.y >= lim || e.x == e.y) return bad("link endpoint");
    }
  }
  for (const GroupBody& g : im.groups) {
    if (g.body >= im.bodies.size()) return bad("group body id");
    const DBody& B = im.bodies[g.body];
    if (B.sched >= reg.scheds.size()) return bad("schedule id");
    const DSched& S = reg.scheds[B.sched];
    if ((size_t)S.chunk0 + S.nchunks > reg.chunk_off.size() ||
        (size_t)S.off + S.words > reg.stream.size())
      return bad("schedule range");
    if (g.smem && (!B.local || B.np > 65535u)) return bad("shared-memory body needs local links");
    if (g.flow_pos) {  // the flow executor's records
      if (g.smem || !B.local || g.large_c < 2 || g.large_c > FLOW_MAX_C || B.np > 65535u ||
          S.words != g.large_c * FLOW_REC_WORDS || g.T != S.tl + S.ti + 32u || S.tl > 512u ||
          S.ti > 256u)
        return bad("flow executor layout");
      for (uint32_t r = 0; r < g.large_c; ++r) {
        const uint32_t* R = &reg.stream[S.off + r * FLOW_REC_WORDS];
        if ((size_t)R[FR_CHUNK0] + R[FR_NCHUNKS] > reg.chunk_off.size() ||
            R[FR_LO] + R[FR_WINDOW] > B.np || 8u * R[FR_WINDOW] > g.flow_pos || R[FR_OWN1] > B.np ||
            (!im.ext && 8u * (R[FR_OWN1] - R[FR_OWN0]) > g.flow_prev) ||
            (B.flags & BODY_UNIT ? 4u : 8u) * R[FR_NLINKS] > g.flow_rest || R[FR_NLEVELS] != S.nlvl)
          return bad("flow executor record");
        for (uint32_t f : {FR_LINKS, FR_LOAD, FR_STORE, FR_EXPECT})
          if ((size_t)R[f] + R[f + 1] > reg.stream.size()) return bad("flow executor list");
        for (uint32_t i = 0; i < R[FR_NLINKS]; ++i)
          if (reg.stream[R[FR_LINKS] + i] >= B.nl) return bad("flow executor link");
        for (uint32_t f : {FR_LOAD, FR_STORE})
          for (uint32_t i = 0; i < R[f + 1]; ++i)
            if (reg.stream[R[f] + i] - R[FR_LO] >= R[FR_WINDOW]) return bad("flow executor particle");
      }
    } else if (g.large_c && (g.smem || !B.local || g.large_c > 16u || g.log2per > 14u ||
                             (size_t)g.large_c << g.log2per < B.np || g.T > 1024u))
      return bad("large-body executor layout");
    if (g.res && (!g.smem || g.res != S.words * 4u)) return bad("resident schedule size");
    if (g.T < 32 || g.T % 32) return bad("group size");
    if (g.smem && (S.tl + S.ti != g.T || S.tl % 32)) return bad("group threads");
    if (!g.large_c && g.T > group_threads_max(!im.ext)) return bad("group threads");
  }
  for (uint32_t b : im.serials) {
    if (b >= im.bodies.size() || !im.bodies[b].local || !(im.bodies[b].flags & BODY_SERIAL))
      return bad("serial body");
    const DBody& B = im.bodies[b];
    if (B.sched && (B.sched >= B.nl || B.nl - B.sched < (B.flags >> BODY_LAG_SHIFT)))
      return bad("serial body halves");
  }
  if (im.cpos.size() != P.nc || im.crad.size() != P.nc) return bad("circle arrays");
  for (const uint2& e : im.clab)
    if (e.x >= P.nc || e.y >= P.nc) return bad("circle link");
  if (im.polys.size() != P.ng || im.pcenter.size() != P.ng) return bad("polygon arrays");
  for (const DPoly& g : im.polys) {
    if ((size_t)g.v0 + g.nv > im.vpos.size()) return bad("polygon vertex range");
    if ((size_t)g.l0 + g.nl > im.plab.size()) return bad("polygon link range");
    for (uint32_t k = 0; k < g.nl; ++k) {
      const uint2 e = im.plab[g.l0 + k];
      if (e.x >= g.nv || e.y >= g.nv) return bad("polygon link endpoint");
    }
  }
  const size_t nst = P.ng >= 2 ? (size_t)P.ng * (P.ng - 1) + 1 : 0;
  if (im.stage_off.size() != nst) return bad("polygon stage table");
  if (im.stage_pr.size() != (nst ? nst - 1 : 0)) return bad("polygon stage pairs");
  for (uint32_t v : im.stage_pr)
    if ((v & 0xFFFFu) >= P.ng || (v >> 16) >= P.ng) return bad("polygon stage pair");
  for (size_t i = 1; i < nst; ++i)
    if (im.stage_off[i] < im.stage_off[i - 1]) return bad("polygon stage order");
  return true;
}

namespace {
struct Comp {
  std::vector<uint32_t> parts;  // ascending world indices
  std::vector<uint32_t> links;  // world link ids in execution order
};

// Levels of one pass over the component's links, and how many a second pass
// adds (0 where the first pass alone is `enough` wide).  A rope's second pass
// starts two levels behind its first, a ring's only once the spokes have moved
// the rim again.
struct PassDepth { uint32_t first, more; };
PassDepth pass_depth(const WorldHost& w, const Comp& c, float enough, std::vector<uint32_t>& last) {
  uint32_t depth[2] = {0, 0};
  for (int pass = 0; pass < 2; ++pass) {
    depth[pass] = depth[0];
    if (pass && (float)c.links.size() / (float)std::max(depth[0], 1u) >= enough) break;
    for (uint32_t k : c.links) {
      const uint32_t a = (uint32_t)w.particle_links[k].particle_a;
      const uint32_t b = (uint32_t)w.particle_links[k].particle_b;
      const uint32_t l = std::max(last[a], last[b]) + 1;
      last[a] = l;
      last[b] = l;
      depth[pass] = std::max(depth[pass], l);
    }
  }
  for (uint32_t k : c.links) {
    last[w.particle_links[k].particle_a] = 0;
    last[w.particle_links[k].particle_b] = 0;
  }
  return PassDepth{depth[0], depth[1] - depth[0]};
}
// Whether the second half of a serial body's links can run beside the first
// half of the next pass, a lag behind it: step j solves link j of the second
// half and link j - lag of the next first half; a particle is integrated a step
// after the link that moves it last, and read a step before its link.  So every
// particle of first-half link i must have been moved for the last time in the
// pass by step i + lag - 3, and every particle must be moved by some link of the second half.  A link integrates one particle; only the last, which
// moves both of its particles last, has a step more for the other.  Taken when
// the lag is at most a quarter of the half: then B.sched is the first half's
// length, the lag is in B.flags, and the last link of the pass that moves a
// particle marks it (LINK_FINAL).
void split_chain(DBody& B, uint4* ab) {
  B.sched = 0;
  const uint32_t m = B.nl / 2, nb = B.nl - m;
  if (m < 8) return;
  constexpr uint32_t NONE = 0xFFFFFFFFu;
  std::vector<uint32_t> last(B.np, NONE);  // the particle's last link in the second half
  for (uint32_t j = 0; j < nb; ++j) last[ab[m + j].x] = last[ab[m + j].y] = j;
  for (uint32_t l : last)
    if (l == NONE) return;
  for (uint32_t j = 0; j + 1 < nb; ++j)
    if (last[ab[m + j].x] == j && last[ab[m + j].y] == j) return;
  const uint4 end = ab[B.nl - 1];  // one of its particles is integrated a step after it
  uint32_t lag = 1;
  for (uint32_t i = 0; i < m; ++i) {
    uint32_t l = std::max(last[ab[i].x], last[ab[i].y]) + 3u;
    if (ab[i].x == end.x || ab[i].y == end.x || ab[i].x == end.y || ab[i].y == end.y) l = nb + 3u;
    if (l > i) lag = std::max(lag, l - i);
    if (lag > nb / 4) return;
  }
  for (uint32_t p = 0; p < B.np; ++p) {
    uint4& e = ab[m + last[p]];
    (e.x == p ? e.x : e.y) |= LINK_FINAL;
  }
  B.sched = m;
  B.flags |= lag << BODY_LAG_SHIFT;
}
// Whether each half's consecutive links share exactly one particle; then the
// records say which one is handed on (LINK_SWAPPED, LINK_KEEP).
void carry_chain(DBody& B, uint4* ab) {
  if (B.np > LINK_INDEX) return;
  std::vector<uint32_t> on(B.nl);  // the endpoint that link k takes from the link before
  auto has = [&](uint32_t k, uint32_t p) {
    return (ab[k].x & LINK_INDEX) == p || (ab[k].y & LINK_INDEX) == p;
  };
  for (uint32_t half = 0; half < 2; ++half) {
    const uint32_t k0 = half ? B.sched : 0u, k1 = half ? B.nl : B.sched;
    for (uint32_t k = k0; k < k1; ++k) {
      const uint32_t x = ab[k].x & LINK_INDEX, y = ab[k].y & LINK_INDEX;
      if (k + 1 < k1) {
        if (has(k + 1, x) == has(k + 1, y)) return;
        on[k + 1] = has(k + 1, x) ? x : y;
      }
      if (k == k0) on[k] = k + 1 < k1 && on[k + 1] == x ? y : x;
    }
  }
  for (uint32_t k = 0; k < B.nl; ++k) {
    const bool end = k + 1 == B.nl || k + 1 == B.sched;
    const bool keep = end || on[k + 1] == on[k];
    if ((ab[k].x & LINK_INDEX) == on[k]) {
      std::swap(ab[k].x, ab[k].y);
      ab[k].x |= LINK_SWAPPED;
    }
    if (keep) ab[k].y |= LINK_KEEP;
  }
  B.flags |= BODY_CARRY;
}
}  // namespace

int plan_world(const WorldHost& w, const PlanTuning& tune, SchedRegistry& reg, WorldImage& im,
               std::string* why) {
  int st = validate_world(w, why);
  if (st != OK) return st;
  const size_t np64 = w.particles.size();
  if (np64 >= 0x7FFFFFFFull || w.particle_links.size() >= 0x7FFFFFFFull) {
    if (why) *why = "world too large for 32-bit indices";
    return ERR_ARG;
  }
  const uint32_t np = (uint32_t)np64;
  const uint32_t nl = (uint32_t)w.particle_links.size();
  im = WorldImage();
  DWorld& P = im.params;
  std::memset(&P, 0, sizeof(P));
  P.gx = 0.0f + w.gravity.x;  // acc = 0 + g at integrate time (src/particle.rs:52-54)
  P.gy = 0.0f + w.gravity.y;
  P.bx = w.bounds.pos.x;
  P.by = w.bounds.pos.y;
  P.bw = w.bounds.size.x;
  P.bh = w.bounds.size.y;
  P.radius = w.particle_radius;
  P.cell = w.grid_cell;
  P.icell = pow2_reciprocal(w.grid_cell);
  P.S = w.sub_steps;
  P.I = w.link_iters;
  P.flags = w.collide & (COLLIDE_PP | COLLIDE_PC | COLLIDE_PPOLY);
  P.np = np;
  P.nc = (uint32_t)w.circles.size();
  P.ncl = (uint32_t)w.circle_links.size();
  P.ng = (uint32_t)w.polygons.size();
  im.ext = P.flags != 0;
  const bool full = !im.ext;

  im.pos.resize(np);
  im.prev.resize(np);
  for (uint32_t i = 0; i < np; ++i) {
    im.pos[i] = make_float2(w.particles[i].pos.x, w.particles[i].pos.y);
    im.prev[i] = make_float2(w.particles[i].prev_pos.x, w.particles[i].prev_pos.y);
  }

  // link execution order: insertion order, or colour-major in fast mode
  std::vector<uint32_t> order(nl);
  std::iota(order.begin(), order.end(), 0u);
  if (w.mode == MODE_FAST) {
    order = colour_link_order(w, &im.stats.colours);
    im.link_order = order;
  }

  // connected components (union-find over links)
  std::vector<uint32_t> parent(np);
  std::iota(parent.begin(), parent.end(), 0u);
  auto find = [&](uint32_t x) {
    while (parent[x] != x) {
      parent[x] = parent[parent[x]];
      x = parent[x];
    }
    return x;
  };
  for (uint32_t k = 0; k < nl; ++k) {
    uint32_t a = find((uint32_t)w.particle_links[k].particle_a);
    uint32_t b = find((uint32_t)w.particle_links[k].particle_b);
    if (a != b) parent[std::max(a, b)] = std::min(a, b);
  }
  std::vector<int64_t> comp_of_root(np, -1);
  std::vector<Comp> comps;
  std::vector<uint32_t> comp_of(np);
  for (uint32_t i = 0; i < np; ++i) {
    const uint32_t r = find(i);
    if (comp_of_root[r] < 0) {
      comp_of_root[r] = (int64_t)comps.size();
      comps.emplace_back();
    }
    comp_of[i] = (uint32_t)comp_of_root[r];
    comps[comp_of[i]].parts.push_back(i);
  }
  for (uint32_t k : order) comps[comp_of[w.particle_links[k].particle_a]].links.push_back(k);

  std::vector<uint32_t> last(np, 0), local(np, 0);
  std::vector<uint32_t> free_parts;
  std::vector<const Comp*> pack;
  uint32_t pack_np = 0, pack_nl = 0;

  // The executor of a group body, chosen by its size with stiffness (a body of
  // unit stiffness takes less): one CTA's shared memory; over that the flow
  // executor, over as many CTAs as give each ~200 ops a level, at least as many
  // as hold it; failing that (more than 65,535 particles, or too much for
  // large_max CTAs) the large-body executor, which keeps its positions (and
  // prev) in the shared memory of a cluster of up to large_max CTAs, at most
  // 128 KB each (8,192 particles whole-step, 16,384 for link passes), with link
  // parameters and schedule read through the caches; beyond that the group
  // executor from global memory.
  struct Place {
    bool smem;
    uint32_t flow_c, flow[3];    // CTAs; bytes of positions, prev and link parameters in each
    uint32_t large_c, log2per;
  };
  auto fits_cta = [&](size_t n, size_t links) {
    return align16((full ? 16u : 8u) * n + 8u * links) <= tune.smem_max && n <= 65535u;
  };
  auto place = [&](const uint2* loc, uint32_t n, uint32_t links, bool unit, uint32_t pass_levels) {
    Place at{};
    const size_t state = (full ? 16u : 8u) * (size_t)n;
    at.smem = fits_cta(n, links);
    if (at.smem) return at;
    if (tune.large_max >= 2 && n <= 65535u) {
      const double wide = (double)links / std::max((double)pass_levels, 1.0) *
                          (full ? (double)P.S * P.I : P.I);
      const uint32_t most = std::min(tune.large_max, FLOW_MAX_C);
      uint32_t c = (uint32_t)std::min(std::max(wide / 400.0, 2.0), (double)FLOW_MAX_C);
      for (c = std::min(c, most); c <= most && c <= n; ++c) {
        // (what it takes at the least, and then exactly)
        const uint32_t per_link = unit ? 4u : 8u;
        const size_t least = (state + per_link * (size_t)links) / c;
        if (least + FLOW_TAIL_BYTES + STREAM_BUFFERS > tune.res_max) continue;
        const auto most_of = flow_sizes(loc, links, n, P.I > 0 && (!full || P.S > 0),
                                        full && P.S > 0, c);
        const size_t need[3] = {align16(8 * (size_t)most_of[0]), full ? align16(8 * (size_t)most_of[1]) : 0,
                                align16(per_link * (size_t)most_of[2])};
        if (need[0] + need[1] + need[2] + FLOW_TAIL_BYTES + STREAM_BUFFERS > tune.res_max) continue;
        at.flow_c = c;
        for (int k = 0; k < 3; ++k) at.flow[k] = (uint32_t)need[k];
        return at;
      }
    }
    if (tune.large_max > 0 && n > 0) {
      const uint32_t cap_log2 = full ? 13u : 14u;
      uint32_t l2 = 0;
      while (l2 < cap_log2 && (1u << l2) < n) ++l2;
      const uint32_t c = (n + (1u << l2) - 1u) >> l2;
      if (c <= tune.large_max) {
        at.large_c = c;
        at.log2per = l2;
      }
    }
    return at;
  };

  struct Item { uint2 e; float rest, stiff; uint32_t level; };
  std::vector<Item> seq;                // emit_group's, kept between bodies
  std::vector<uint32_t> depth, at;
  auto emit_group = [&](const std::vector<const Comp*>& cs) {
    DBody B{};
    B.i0 = (uint32_t)im.bidx.size();
    B.l0 = (uint32_t)im.lab.size();
    uint32_t n = 0;
    for (const Comp* c : cs)
      for (uint32_t p : c->parts) {
        local[p] = n++;
        im.bidx.push_back(p);
      }
    B.np = n;
    // The links sorted by their level in one pass (links of one level share no
    // particle, and each particle still meets its links in order, so this is
    // the same sequence): the links of a schedule round then sit in a few
    // consecutive runs, and so do the rest lengths that a warp loads together.
    seq.clear();
    depth.assign(n, 0);
    at.assign(1, 0);
    for (const Comp* c : cs)
      for (uint32_t k : c->links) {
        const Link& L = w.particle_links[k];
        const uint32_t a = local[L.particle_a], b = local[L.particle_b];
        const uint32_t l = std::max(depth[a], depth[b]) + 1;
        depth[a] = depth[b] = l;
        if (l == at.size()) at.push_back(0);
        ++at[l];
        seq.push_back(Item{make_uint2(a, b), L.target_distance, L.stiffness, l - 1});
      }
    for (size_t l = 1; l < at.size(); ++l) at[l] += at[l - 1];
    std::vector<uint2> loc(seq.size());
    im.lrest.resize(B.l0 + seq.size());
    im.lstiff.resize(B.l0 + seq.size());
    B.nl = (uint32_t)seq.size();
    B.flags = BODY_UNIT | BODY_RANGE;
    for (const Item& it : seq) {
      const uint32_t i = at[it.level]++;
      loc[i] = it.e;
      im.lrest[B.l0 + i] = it.rest;
      im.lstiff[B.l0 + i] = it.stiff;
      if (it.stiff != 1.0f) B.flags &= ~BODY_UNIT;
      if (!(it.rest < 0x1p100f && it.rest > -0x1p100f)) B.flags &= ~BODY_RANGE;
    }
    const bool unit = (B.flags & BODY_UNIT) != 0u;
    const Place pl = place(loc.data(), B.np, B.nl, unit, (uint32_t)at.size() - 1u);
    const bool smem = pl.smem;
    const size_t region = align16((full ? 16u : 8u) * (size_t)B.np + (unit ? 4u : 8u) * (size_t)B.nl);
    if (pl.flow_c) B.sched = reg.get_flow(loc.data(), B.nl, B.np, P.S, P.I, full, pl.flow_c);
    else B.sched = reg.get(loc.data(), B.nl, B.np, P.S, P.I, full, smem, tune);
    if (B.sched == SchedRegistry::NONE) std::abort();  // place() chose what a schedule can hold
    const DSched& S = reg.scheds[B.sched];
    const float avg = S.nlvl ? (float)S.nops / (float)S.nlvl : 1.0f;
    uint32_t T = pow2ceil((uint32_t)(avg / tune.width_per_thread + 0.999f));
    T = std::min(std::min(std::max(T, tune.t_min), tune.t_max), group_threads_max(full));
    if (smem || pl.flow_c) T = S.tl + S.ti;
    // the whole schedule resident in shared memory when it fits beside the body
    uint32_t res = 0;
    if (smem && tune.resident) {
      const size_t sb = (size_t)S.words * 4u;
      if (region + sb + GROUP_TAIL_BYTES <= tune.res_max)
        res = (uint32_t)sb;
    }
    uint32_t large_c = pl.large_c, TL = T;
    if (large_c) {
      const float w = avg / (tune.width_per_thread * (float)large_c);
      TL = std::min<uint32_t>(1024u, std::max<uint32_t>(64u, pow2ceil((uint32_t)(w + 0.999f))));
    } else if (pl.flow_c) {
      large_c = pl.flow_c;
      TL = T + 32;  // and the control warp
    }
    const bool local = smem || large_c > 0;
    B.local = local ? 1u : 0u;
    for (size_t i = 0; i < loc.size(); ++i) {
      if (local) im.lab.push_back(loc[i]);
      else im.lab.push_back(make_uint2(im.bidx[B.i0 + loc[i].x], im.bidx[B.i0 + loc[i].y]));
    }
    const uint32_t id = (uint32_t)im.bodies.size();
    im.bodies.push_back(B);
    GroupBody gbody{id, large_c ? TL : T, smem ? (uint32_t)region : 0u, res, smem};
    gbody.large_c = large_c;
    gbody.log2per = pl.log2per;
    gbody.flow_pos = pl.flow[0];
    gbody.flow_prev = pl.flow[1];
    gbody.flow_rest = pl.flow[2];
    im.groups.push_back(gbody);
    im.stats.group_bodies++;
    if (large_c) im.stats.large_bodies++;
    else if (!smem) im.stats.global_bodies++;
    im.stats.levels += S.nlvl;
    im.stats.ops += S.nops;
  };
  auto flush_pack = [&]() {
    if (!pack.empty()) emit_group(pack);
    pack.clear();
    pack_np = pack_nl = 0;
  };

  // whether the large-body executor would run a component by levels
  auto to_large = [&](const Comp& c, uint32_t pass_levels) {
    if (fits_cta(c.parts.size(), c.links.size())) return false;
    std::vector<uint2> loc;
    loc.reserve(c.links.size());
    for (size_t i = 0; i < c.parts.size(); ++i) local[c.parts[i]] = (uint32_t)i;
    bool unit = true;
    for (uint32_t k : c.links) {
      const Link& L = w.particle_links[k];
      loc.push_back(make_uint2(local[L.particle_a], local[L.particle_b]));
      unit &= L.stiffness == 1.0f;
    }
    return place(loc.data(), (uint32_t)c.parts.size(), (uint32_t)loc.size(), unit, pass_levels).large_c != 0u;
  };

  for (const Comp& c : comps) {
    if (c.links.empty()) {
      free_parts.push_back(c.parts[0]);
      continue;
    }
    // Serial or by levels: a body whose single pass is narrow may still be wide
    // over the passes its schedule chains, which start behind one another.
    // Measured on 24 ropes of 200 particles (one pass 1 wide, the 8 x 4 passes
    // of an update ~29): 1,710 us a pass replayed by one thread each, 60 us by
    // levels.  Rings of a hub and spokes stay below 3 (the next pass's rim
    // runs beside this pass's spokes) and run serially.  3 is near the crossing
    // on every executor but one (2 x 1 passes, width 4, serially and by levels:
    // ropes of 11,000 and 30,000 on the flow executor 6.8 and 3.4 ms, 19.8 and
    // 9.3; of 70,000 from global memory 45.9 and 39.5): a level of the
    // large-body executor costs 1.1 us, and in its link passes a rope of 70,000
    // takes 52.7 ms serially and 79.6 by levels at width 4, 79.2 and 79.8 at 6,
    // 105.7 and 79.9 at 8, one with braces 144.6 and 159.9 at 6, 192.9 and
    // 160.6 at 8.  So it takes chains from 7.
    const PassDepth pd = pass_depth(w, c, tune.serial_width, last);
    const double passes = full ? (double)P.S * P.I : (double)P.I;
    const double ops = passes * (double)c.links.size() + (full ? (double)P.S * c.parts.size() : 0.0);
    const double levels = (double)pd.first + (passes - 1.0) * pd.more + (full ? (double)P.S : 0.0);
    const double width = (double)c.links.size() / (double)std::max(pd.first, 1u);
    const double many = ops / std::max(levels, 1.0);
    if (width < tune.serial_width &&
        (many < 1.5 * tune.serial_width ||
         (many < 3.5 * tune.serial_width && to_large(c, pd.first)))) {
      DBody B{};
      B.i0 = (uint32_t)im.bidx.size();
      B.np = (uint32_t)c.parts.size();
      B.l0 = (uint32_t)im.lrec.size();
      B.nl = (uint32_t)c.links.size();
      B.local = 1;  // body-local endpoints: index into the body's particle list
      uint32_t nloc = 0;
      for (uint32_t p : c.parts) {
        local[p] = nloc++;
        im.bidx.push_back(p);
      }
      B.flags = BODY_SERIAL | BODY_RANGE;
      for (uint32_t k : c.links) {
        const Link& L = w.particle_links[k];
        uint32_t rs[2];
        std::memcpy(&rs[0], &L.target_distance, 4);
        std::memcpy(&rs[1], &L.stiffness, 4);
        im.lrec.push_back(make_uint4(local[L.particle_a], local[L.particle_b], rs[0], rs[1]));
        if (!(L.target_distance < 0x1p100f && L.target_distance > -0x1p100f)) B.flags &= ~BODY_RANGE;
      }
      split_chain(B, &im.lrec[B.l0]);
      carry_chain(B, &im.lrec[B.l0]);
      im.serials.push_back((uint32_t)im.bodies.size());
      im.bodies.push_back(B);
      im.stats.serial_bodies++;
      continue;
    }
    const uint32_t cn = (uint32_t)c.parts.size(), cl = (uint32_t)c.links.size();
    if (!pack.empty() && (pack_np + cn > tune.pack_np || pack_nl + cl > tune.pack_nl)) flush_pack();
    pack.push_back(&c);
    pack_np += cn;
    pack_nl += cl;
  }
  flush_pack();
  // link-free particles: integrate-only bodies (the extension pipeline
  // integrates every particle in its collide pass instead)
  if (full) {
    for (size_t i = 0; i < free_parts.size(); i += tune.free_chunk) {
      std::vector<Comp> chunk(1);
      const size_t e = std::min(free_parts.size(), i + tune.free_chunk);
      chunk[0].parts.assign(free_parts.begin() + i, free_parts.begin() + e);
      std::vector<const Comp*> cs{&chunk[0]};
      emit_group(cs);
    }
  }
  P.nb = (uint32_t)im.bodies.size();
  im.stats.bodies = P.nb;
  // particle collisions with every particle in a shared-memory group body:
  // the link executor counts them into the grid (GRID_IN_LINKS)
  if ((P.flags & COLLIDE_PP) && free_parts.empty() && im.serials.empty() && np > 0) {
    bool all_smem = true;
    for (const GroupBody& gb : im.groups) all_smem = all_smem && gb.smem;
    if (all_smem) P.flags |= GRID_IN_LINKS;
  }

  // circles (src/circle.rs:4-8) and circle links
  for (const Circle& c : w.circles) {
    im.cpos.push_back(make_float2(c.point.pos.x, c.point.pos.y));
    im.cprev.push_back(make_float2(c.point.prev_pos.x, c.point.prev_pos.y));
    im.cacc.push_back(make_float2(c.point.acc.x, c.point.acc.y));
    im.crad.push_back(c.radius);
    im.cstatic.push_back(c.is_static ? 1u : 0u);
  }
  for (const Link& l : w.circle_links) {
    im.clab.push_back(make_uint2((uint32_t)l.particle_a, (uint32_t)l.particle_b));
    im.clrest.push_back(l.target_distance);
  }
  // polygons (src/polygon.rs:7-14)
  for (const Polygon& g : w.polygons) {
    DPoly d{};
    d.v0 = (uint32_t)im.vpos.size();
    d.nv = (uint32_t)g.particles.size();
    d.l0 = (uint32_t)im.plab.size();
    d.nl = (uint32_t)g.particle_links.size();
    d.is_static = g.is_static ? 1u : 0u;
    for (const Particle& v : g.particles) {
      im.vpos.push_back(make_float2(v.pos.x, v.pos.y));
      im.vprev.push_back(make_float2(v.prev_pos.x, v.prev_pos.y));
      im.vacc.push_back(make_float2(v.acc.x, v.acc.y));
    }
    for (const Link& l : g.particle_links) {
      im.plab.push_back(make_uint2((uint32_t)l.particle_a, (uint32_t)l.particle_b));
      im.plrest.push_back(l.target_distance);
    }
    im.pcenter.push_back(make_float2(g.center.x, g.center.y));
    im.polys.push_back(d);
  }
  // polygon pair stages: (i,j) then (j,i) for pairs i<j in row-major order
  if (P.ng >= 2) {
    uint32_t acc = 0;
    if (P.ng > 65535u) {
      if (why) *why = "at most 65535 polygons per world";
      return ERR_ARG;
    }
    for (uint32_t i = 0; i < P.ng; ++i)
      for (uint32_t j = i + 1; j < P.ng; ++j) {
        im.stage_off.push_back(acc);
        im.stage_pr.push_back(i | (j << 16));
        acc += im.polys[i].nv * im.polys[j].nv;
        im.stage_off.push_back(acc);
        im.stage_pr.push_back(j | (i << 16));
        acc += im.polys[j].nv * im.polys[i].nv;
      }
    im.stage_off.push_back(acc);
  }
  for (DBody& B : im.bodies) {  // contiguous particle lists load without bidx
    B.first = B.np ? im.bidx[B.i0] : NO_FIRST;
    for (uint32_t i = 1; i < B.np && B.first != NO_FIRST; ++i)
      if (im.bidx[B.i0 + i] != B.first + i) B.first = NO_FIRST;
  }
  if (!check_image(im, reg, why)) return ERR_STATE;
  return OK;
}

BlockLayout layout_of(const WorldImage& im) {
  BlockLayout L;
  size_t o = 0;
  auto seg = [&](size_t bytes) {
    size_t at = o;
    o = align16(o + bytes);
    return at;
  };
  const size_t np = im.pos.size(), nc = im.cpos.size(), nv = im.vpos.size(),
               ng = im.polys.size();
  // the state prefix is one contiguous run of float2
  L.o_pos = 0;
  L.o_prev = L.o_pos + 8 * np;
  L.o_cpos = L.o_prev + 8 * np;
  L.o_cprev = L.o_cpos + 8 * nc;
  L.o_cacc = L.o_cprev + 8 * nc;
  L.o_vpos = L.o_cacc + 8 * nc;
  L.o_vprev = L.o_vpos + 8 * nv;
  L.o_vacc = L.o_vprev + 8 * nv;
  L.o_pcenter = L.o_vacc + 8 * nv;
  L.state_bytes = L.o_pcenter + 8 * ng;
  o = align16(L.state_bytes);
  L.o_pos1 = seg(8 * np);
  L.o_bidx = seg(4 * im.bidx.size());
  L.o_bodies = seg(sizeof(DBody) * im.bodies.size());
  L.o_lab = seg(8 * im.lab.size());
  L.o_lrest = seg(4 * im.lrest.size());
  L.o_lstiff = seg(4 * im.lstiff.size());
  L.o_lrec = seg(16 * im.lrec.size());
  L.o_crad = seg(4 * nc);
  L.o_cstatic = seg(4 * nc);
  L.o_clab = seg(8 * im.clab.size());
  L.o_clrest = seg(4 * im.clrest.size());
  L.o_polys = seg(sizeof(DPoly) * ng);
  L.o_paabb = seg(16 * ng);
  L.o_plab = seg(8 * im.plab.size());
  L.o_plrest = seg(4 * im.plrest.size());
  L.o_stage = seg(4 * im.stage_off.size());
  L.o_stage_pr = seg(4 * im.stage_pr.size());
  L.total = std::max<size_t>(o, 16);
  return L;
}

void write_block(const WorldImage& im, const BlockLayout& L, unsigned char* dst) {
  std::memset(dst, 0, L.total);
  auto put = [&](size_t off, const void* src, size_t bytes) {
    if (bytes) std::memcpy(dst + off, src, bytes);
  };
  put(L.o_pos, im.pos.data(), 8 * im.pos.size());
  put(L.o_prev, im.prev.data(), 8 * im.prev.size());
  put(L.o_cpos, im.cpos.data(), 8 * im.cpos.size());
  put(L.o_cprev, im.cprev.data(), 8 * im.cprev.size());
  put(L.o_cacc, im.cacc.data(), 8 * im.cacc.size());
  put(L.o_vpos, im.vpos.data(), 8 * im.vpos.size());
  put(L.o_vprev, im.vprev.data(), 8 * im.vprev.size());
  put(L.o_vacc, im.vacc.data(), 8 * im.vacc.size());
  put(L.o_pcenter, im.pcenter.data(), 8 * im.pcenter.size());
  put(L.o_pos1, im.pos.data(), 8 * im.pos.size());
  put(L.o_bidx, im.bidx.data(), 4 * im.bidx.size());
  put(L.o_bodies, im.bodies.data(), sizeof(DBody) * im.bodies.size());
  put(L.o_lab, im.lab.data(), 8 * im.lab.size());
  put(L.o_lrest, im.lrest.data(), 4 * im.lrest.size());
  put(L.o_lstiff, im.lstiff.data(), 4 * im.lstiff.size());
  put(L.o_lrec, im.lrec.data(), 16 * im.lrec.size());
  put(L.o_crad, im.crad.data(), 4 * im.crad.size());
  put(L.o_cstatic, im.cstatic.data(), 4 * im.cstatic.size());
  put(L.o_clab, im.clab.data(), 8 * im.clab.size());
  put(L.o_clrest, im.clrest.data(), 4 * im.clrest.size());
  put(L.o_polys, im.polys.data(), sizeof(DPoly) * im.polys.size());
  put(L.o_plab, im.plab.data(), 8 * im.plab.size());
  put(L.o_plrest, im.plrest.data(), 4 * im.plrest.size());
  put(L.o_stage, im.stage_off.data(), 4 * im.stage_off.size());
  put(L.o_stage_pr, im.stage_pr.data(), 4 * im.stage_pr.size());
}

}  // namespace b2d
