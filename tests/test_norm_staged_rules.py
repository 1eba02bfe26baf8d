"""Host rules of the group-norm rows in a cluster's shared memory: the order of announcements and remote stores, and plans that hold their rows."""
import test_host_rules as rules


def test_staged_clusters_wait_until_every_cta_has_started():
    kernels = 0
    for function, kernel, body in rules._functions("group_norm_staged.cuh"):
        first = min(body.find(w) for w in ("map_shared_rank", "row_moments<") if w in body)
        assert body.find("row_moments<") == first or 0 <= body.find("cluster_wait_started()") < first, function
        assert 0 <= body.find("cluster_announce()") < body.find("wait_previous()"), function
        kernels += kernel
    assert kernels == 2


def test_staged_plans_hold_their_rows(tmp_path):
    rules._run(tmp_path, r"""
#include <cstdio>
#include <initializer_list>
#include "norm_plan.cuh"
using namespace b200::nres;
int main() {
  int wrong = 0, held = 0;
  for (int bytes : {4, 8, 16, 32})
    for (int quarter : {46 * 1024, 54 * 1024})
      for (long long units = 1; units < 500000; units += 1 + units / 97) {
        const StagedPlan p = plan_staged(units, bytes, quarter);
        if (!p.ranks) {
          if (units * bytes <= 15ll * PLAN_STAGED_BYTES) ++wrong;       // sixteen shares, less their rounding
          continue;
        }
        ++held;
        const long long per = (units + p.ranks - 1) / p.ranks;
        if (p.ranks > PLAN_MAX_RANKS || per > (long long)p.units * PLAN_THREADS || (long long)p.units * PLAN_THREADS * bytes > PLAN_STAGED_BYTES) ++wrong;
        if (p.ranks < PLAN_MAX_RANKS && (long long)p.units * PLAN_THREADS * bytes > quarter) ++wrong;
      }
  printf("%d %d\n", wrong, held);
  return wrong != 0 || held < 1000;
}
""")
