"""The schedules that planning a world leaves in the registry, which all go to
the device: one for a body, whatever executors were considered for it."""
import shutil
import subprocess

import pytest

# usage: plan W H SCATTER COLLIDE SUB_STEPS LINK_ITERS LARGE_MAX -> schedules, kind, CTAs
PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <random>
#include "engine.hpp"
int main(int, char** v) {
  using namespace b2d;
  auto arg = [&](int i) { return (uint32_t)std::atoi(v[i]); };
  const uint32_t w = arg(1), h = arg(2), n = w * h;
  std::vector<uint32_t> id(n);
  std::iota(id.begin(), id.end(), 0u);
  if (arg(3)) std::shuffle(id.begin(), id.end(), std::mt19937(7));
  WorldHost W;
  W.particles.resize(n);
  for (uint32_t i = 0; i < n; ++i) {
    const Vec2 p{(float)(i % w), (float)(i / w)};
    W.particles[id[i]] = Particle{p, p, {0, 0}};
  }
  auto link = [&](uint32_t a, uint32_t b) {
    W.particle_links.push_back(Link{std::min(id[a], id[b]), std::max(id[a], id[b]), 1.0f, 1.0f});
  };
  for (uint32_t y = 0; y < h; ++y)
    for (uint32_t x = 0; x < w; ++x) {
      if (x + 1 < w) link(y * w + x, y * w + x + 1);
      if (y + 1 < h) link(y * w + x, y * w + x + w);
      if (x + 1 < w && y + 1 < h) link(y * w + x, y * w + x + w + 1);
    }
  W.collide = arg(4);
  W.sub_steps = arg(5);
  W.link_iters = arg(6);
  PlanTuning t;
  t.large_max = arg(7);
  t.serial_width = 0.0f;
  SchedRegistry reg;
  WorldImage im;
  std::string why;
  if (plan_world(W, t, reg, im, &why) != OK) { std::printf("failed: %s\n", why.c_str()); return 1; }
  const GroupBody& g = im.groups.at(0);
  std::printf("%zu %s %u\n", reg.scheds.size(),
              g.flow_pos ? "flow" : g.large_c ? "large" : g.smem ? "group" : "global", g.large_c);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    from bendy2d_gb300 import build as b
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    inc = [f"-I{p}" for p in (b.CSRC, b.PKG.parent / "include", b.CUDA_HOME / "include")]
    subprocess.run(["g++", "-O1", "-std=c++17", *inc, str(d / "plan.cpp"), str(b.CSRC / "planner.cpp"),
                    str(b.CSRC / "host.cpp"), "-o", str(d / "plan")], check=True)

    def run(*args):
        r = subprocess.run([str(d / "plan"), *map(str, args)], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
        n, kind, ctas = r.stdout.split()
        return int(n), kind, int(ctas)
    return run


@pytest.mark.parametrize("case,kind,ctas", [
    # w, h, scatter, collide, sub_steps, link_iters, large_max
    ((100, 100, 0, 0, 8, 4, 8), "flow", None),
    ((100, 100, 1, 0, 2, 4, 8), "flow", None),
    ((140, 140, 1, 0, 2, 2, 8), "large", 3),
    ((200, 200, 1, 1, 2, 4, 8), "large", 3),
    ((140, 140, 1, 0, 2, 2, 2), "global", 0),
    ((260, 260, 0, 1, 1, 1, 8), "large", 5),
    ((30, 30, 0, 0, 2, 2, 8), "group", 0),
    ((100, 100, 0, 1, 2, 0, 8), "flow", 2),  # no link iterations
    ((120, 120, 0, 0, 2, 0, 8), "flow", 3),
])
def test_one_schedule_a_body(plan, case, kind, ctas):
    n, got, c = plan(*case)
    assert (n, got) == (1, kind)
    assert ctas is None or c == ctas


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("scatter", [0, 1])
@pytest.mark.parametrize("link_iters", [0, 1, 3])
@pytest.mark.parametrize("w,h", [(75, 75), (91, 83), (128, 97), (211, 60), (3, 9000), (9000, 3)])
def test_sizes_known_before_a_schedule_is_built_hold_it(plan, w, h, link_iters, scatter, collide):
    """The image check compares every CTA of the schedule with them."""
    for large_max in (2, 5, 8):
        plan(w, h, scatter, collide, 1, link_iters, large_max)
