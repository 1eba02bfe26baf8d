"""Host checks of rules that decide which path a call takes: the functions of common.cuh that the kernels and their launchers share,
compiled with g++ and compared with the property they stand for."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"
pytestmark = pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INC), reason="needs g++ and the CUDA headers")


def _run(tmp_path, source):
    src = tmp_path / "check.cpp"
    src.write_text(source)
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.check_call([gxx, "-O1", "-std=c++17", "-x", "c++", str(src), "-o", str(tmp_path / "check"), "-I", os.path.join(ROOT, "pytorch-vulkan_b200", "csrc"),
                           "-I", os.path.join(ROOT, "include"), "-I", CUDA_INC])
    out = subprocess.run([str(tmp_path / "check")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout


def test_channel_quads_are_aligned_in_every_group(tmp_path):
    """Every address that a 16-byte load of a channels-last view would use, over groups whose channel count is no multiple of four and pixels
    that are padded, offset or sliced: the rule may only say yes where all of them are whole 16-byte pieces, and says it for whole layers."""
    out = _run(tmp_path, r"""
#include <cstdio>
#include "common.cuh"
int main() {
  int yes = 0, wrong = 0, missed = 0;
  for (int groups = 1; groups <= 3; ++groups)
    for (int per = 30; per <= 68; ++per)
      for (int pad = 0; pad <= 4; ++pad)
        for (int offset = 0; offset <= 4; ++offset) {
          const long long pixel = (long long)groups * per + pad, row = 5 * pixel, image = 3 * row;
          const b200::View4 v{reinterpret_cast<const float*>(4096) + offset, image, 1, row, pixel};
          bool aligned = true;
          for (int n = 0; n < 2; ++n)
            for (int x = 0; x < 3; ++x)
              for (int g = 0; g < groups; ++g)
                for (int c = 0; c < 8; c += 4)
                  aligned &= reinterpret_cast<uintptr_t>(v.ptr + n * v.s0 + n * v.s2 + x * v.s3 + (long long)g * per + c) % 16 == 0;
          const bool said = b200::channel_quads_aligned(v, per, groups);
          yes += said;
          wrong += said && !aligned;
          missed += !said && aligned;
        }
  printf("%d %d %d\n", yes, wrong, missed);
  return wrong != 0 || missed != 0 || yes == 0;
}
""")
    assert int(out.split()[1]) == 0


CLUSTER_SOURCES = ("reduce.cu", "batch_norm.cu", "group_norm.cu", "norm_resident.cuh", "conv_tc_small.cu")


def _functions(name):
    """(name, body) of the kernels and device functions of a source file that hold or reach a store into another CTA's shared memory."""
    import re
    with open(os.path.join(ROOT, "pytorch-vulkan_b200", "csrc", name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for m in re.finditer(r"\n__(?:global|device)__[^;{]*?\b(\w+)\([^;{]*\)\s*\{", text):
        end = text.find("\n}", m.end())
        yield m.group(1), m.group(0).startswith("\n__global__"), text[m.end():end]


def test_clusters_wait_until_every_cta_has_started():
    """CUDA allows access to another CTA's shared memory only once that CTA runs.  In every kernel that reaches such a store, all threads
    announce themselves before anything else, and wait for the other CTAs before the first store."""
    waits_itself = {"row_moments"}          # holds the wait ahead of its first sum
    checked = 0
    for name in CLUSTER_SOURCES:
        for function, kernel, body in _functions(name):
            stores = [body.find(w) for w in ("map_shared_rank", "cluster_sum(", "row_moments<", "st_remote(") if w in body]
            if not stores or function == "cluster_sum":
                continue
            waited, first = body.find("cluster_wait_started()"), min(stores)
            inside = any(f + "<" in body and body.find(f + "<") == first for f in waits_itself)
            assert inside or 0 <= waited < first, f"{name}: {function} stores into another CTA before it knows that it runs"
            if kernel:
                announced = body.find("cluster_announce()")
                assert 0 <= announced < body.find("wait_previous()"), f"{name}: {function} does not announce itself first"
                checked += 1
    assert checked == 7


def test_norm_rank_plans_hold_their_rows(tmp_path):
    """Every plan for a row that stays resident gives its threads all units (no more than `most` each, no rank empty for want of units), widens
    only as far as all CTAs run at once, and the rows that the resident kernels took at a loss stream: forward passes of single values over
    several waves of wide clusters."""
    _run(tmp_path, r"""
#include <cstdio>
#include <initializer_list>
#include "norm_plan.cuh"
using namespace b200::nres;
int main() {
  int wrong = 0, resident = 0, streams = 0;
  const int sms = 148;
  for (int most : {4, 8, 16})
    for (long long units = 1; units < 80000; units = units * 9 / 8 + 1)
      for (long long rows = 1; rows < 5000; rows = rows * 3 / 2 + 1) {
        const RankPlan p = plan_ranks(units, rows, most, sms);
        const long long holds = 256ll * most;
        if (units > 16 * holds) { wrong += p.ranks != 0; continue; }
        wrong += p.ranks < 1 || p.ranks > 16 || (units + p.ranks - 1) / p.ranks > holds || p.need != (units + holds - 1) / holds;
        if (p.ranks != p.need) wrong += p.ranks > 8 || rows * p.ranks > 4 * sms || units <= p.ranks / 2 * 512;
        for (int vec : {1, 4})
          for (int backward = 0; backward < 2; ++backward)
            for (long long plane : {49, 225, 900, 3136}) {
              const bool b = batch_norm_resident(p, vec, plane, backward), g = group_norm_resident(p, vec, plane, backward, rows <= 3 * sms);
              (b ? resident : streams) += 1;
              if (p.waves <= 1.0 || vec == 4 || backward) wrong += !b || !g;
              else if (p.need > 8 && p.waves > 4.0) wrong += b || g;
              else if (p.need > 4 && p.waves > 2.0 && plane > 256) wrong += b || (p.need <= 8 && g);
            }
      }
  printf("%d %d %d\n", wrong, resident, streams);
  return wrong != 0 || resident == 0 || streams == 0;
}
""")


def test_plan_table_holds_a_network(tmp_path):
    """The layers of ResNet-50, forward and dInput: every plan is made once, whatever the batch, and kept through the following steps; more
    layers than the table has places still get plans of their own."""
    _run(tmp_path, r"""
#include <cstdio>
#include <vector>
#include "plan_cache.cuh"
namespace b200 { int sm_count() { return 148; } }
using namespace b200;
static ConvGeom layer(int n, int cin, int cout, int hw, int k, int s) {
  const int p = (k - 1) / 2, o = (hw + 2 * p - k) / s + 1;
  return ConvGeom{n, cin, cout, hw, hw, k, k, o, o, s, s, p, p, 1, 1, 1, cin, cout};
}
int main() {
  int wrong = 0;
  for (int n : {1, 2, 8, 32, 64, 100, 256}) {
    std::vector<ConvGeom> net{layer(n, 3, 64, 224, 7, 2)};
    const int blocks[] = {3, 4, 6, 3};
    int cin = 64, hw = 56;
    for (int stage = 0; stage < 4; ++stage)
      for (int b = 0; b < blocks[stage]; ++b) {
        const int width = 64 << stage, s = stage > 0 && b == 0 ? 2 : 1;
        net.push_back(layer(n, cin, width, hw, 1, 1));
        net.push_back(layer(n, width, width, hw, 3, s));
        if (b == 0) net.push_back(layer(n, cin, 4 * width, hw, 1, s));
        hw /= s;
        net.push_back(layer(n, width, 4 * width, hw, 1, 1));
        cin = 4 * width;
      }
    PlanCache<int> cache;
    int made = 0, first = 0;
    for (int step = 0; step < 4; ++step) {
      for (size_t i = 0; i < net.size(); ++i)
        for (int is_dx = 0; is_dx < 2; ++is_dx) {
          const int want = net[i].cin * 100000 + net[i].cout * 20 + net[i].h + 7 * net[i].kh + 3 * net[i].sh + is_dx;
          wrong += cache.get(net[i], is_dx, [&] { ++made; return want; }) != want;
        }
      if (step == 0) first = made;
    }
    printf("batch %d: %d layers, %d plans made\n", n, (int)net.size(), made);
    wrong += made != first;
  }
  PlanCache<int> cache;
  for (int step = 0; step < 2; ++step)
    for (int i = 1; i < 5000; ++i) wrong += cache.get(layer(1, i, 16, 8, 3, 1), 0, [&] { return i; }) != i;
  return wrong != 0;
}
""")


@pytest.mark.parametrize("n,cin,cout,hw,k,tc", [(3, 3, 119, 8, 1, False), (2, 8, 117, 15, 1, False), (3, 6, 103, 17, 1, True), (9, 8, 60, 8, 1, True),
                                                (2, 15, 119, 13, 1, True), (1, 1, 80, 29, 3, False), (1, 1, 80, 30, 3, True), (8, 3, 64, 16, 3, True)])
def test_forward_passes_of_a_few_products_stay_on_the_cuda_cores(n, cin, cout, hw, k, tc):
    import b200conv
    p = b200conv.geometry((n, cin, hw, hw), cout, (k, k), padding=(k // 2, k // 2))
    chosen = b200conv.select(p, b200conv.PHASE_FORWARD)
    assert (chosen == b200conv.ALGO_TC) == tc
    assert b200conv.select(p, b200conv.PHASE_FORWARD, b200conv.ALGO_TC) == b200conv.ALGO_TC      # still there when asked for
