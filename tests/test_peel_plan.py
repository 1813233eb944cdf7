"""The batched peel's host-side plan: what a launch over several graphs needs,
asked of the library itself by a small program (tests/native/plan_check.cpp)."""
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "pargridcpu_b200")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "plan_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(os.path.dirname(PKG), "include"),
                    "-I", "/usr/local/cuda/include", os.path.join(HERE, "native", "plan_check.cpp"),
                    "-o", exe, "-L", PKG, "-lfirmcore", f"-Wl,-rpath,{PKG}"], check=True)

    def run(what, late, graphs, **env):
        args = [exe, what, str(int(late))] + [",".join(str(x) for x in g) for g in graphs]
        out = subprocess.run(args, check=True, capture_output=True, text=True,
                             env=dict(os.environ, **{k: str(v) for k, v in env.items()}))
        return [int(x) for x in out.stdout.split()]

    return run


# nodes, layers, directed entries, largest layer degree
ONE_LAYER = (1000, 1, 6000, 90)
MANY_LAYERS = (60_000, 24, 9_000_000, 4000)


@pytest.mark.parametrize("env", [{}, {"FC_PEEL_LATE": 0}])
def test_packing_does_not_depend_on_which_graph_is_first(plan, env):
    """Without the late form a launch of a one-layer graph and a many-layer one
    packs columns, in either order."""
    late = bool(env)
    first = plan("scratch", late, [ONE_LAYER] + 4 * [MANY_LAYERS], **env)[0]
    last = plan("scratch", late, 4 * [MANY_LAYERS] + [ONE_LAYER], **env)[0]
    alone = plan("scratch", late, 4 * [MANY_LAYERS], **env)[0]
    assert abs(first - last) <= 64 << 10  # places are rounded to 256 bytes
    assert first < 1.1 * alone


MIXES = {
    # a launch's planes are as many as its widest graph's
    "wide_beside_hubs": [(2_000_000, 12, 40_000_000, 100_000), (2000, 24, 60_000, 200)],
    "wide_beside_two_million": [(2_000_000, 4, 40_000_000, 5000), (2000, 24, 60_000, 200)],
    "wide_beside_small": 4 * [(60_000, 4, 1_000_000, 900)] + [(2000, 24, 60_000, 200)],
    "wide_beside_many": 15 * [(60_000, 4, 1_000_000, 900)] + [(1000, 28, 60_000, 200)],
    # graphs that alone start in the late form, more nodes than it takes
    "past_its_nodes": 32 * [(60_000, 12, 3_000_000, 900)],
    "one_layer_first": [(1000, 1, 6000, 90)] + 12 * [MANY_LAYERS],
    "many_layers_between": [(900, 6, 9000, 50), (50, 600, 60_000, 40), (900, 6, 9000, 50)],
    # counters of hubs on lines of their own, or not, as the degrees turn out
    "hubs_unknown": [(70_000, 28, 40_000_000, 69_000), (70_000, 4, 9_000_000, 60_000)],
}


@pytest.mark.parametrize("name", sorted(MIXES))
def test_admission_charges_what_a_batch_takes(plan, name):
    """A server charges a batch's scratch before the graphs are on the device,
    where their degrees are known: it must cover what the launches then take."""
    charged, lean, taken, joined = plan("admit", 150 * 10**9, MIXES[name])
    assert not lean and joined == len(MIXES[name])
    assert charged >= taken


@pytest.mark.parametrize("seed", range(6))
def test_admission_charges_what_a_random_batch_takes(plan, seed):
    rng = np.random.default_rng(seed)
    mix = []
    for _ in range(int(rng.integers(2, 20))):
        n = int(10 ** rng.uniform(2, 6.2))
        L = int(rng.integers(1, 30))
        entries = int(n * L * rng.uniform(0.5, 20))
        mix.append((n, L, entries, int(rng.uniform(0, 1) ** 3 * (n - 1))))
    charged, _, taken, joined = plan("admit", 150 * 10**9, mix)
    assert charged >= taken and joined == len(mix)


def test_a_request_that_does_not_fit_does_not_change_the_batch(plan):
    """A graph that only fits the budget without the late form, and one that
    does not fit at all, leave the late form to a batch that has begun; the
    first goes without it when it begins one."""
    small, large, huge = (900, 6, 9000, 50), (300_000, 12, 60_000_000, 900), \
        (3_000_000, 12, 600_000_000, 900)
    with_late = plan("scratch", 1, [large])[0]
    without = plan("scratch", 0, [large])[0]
    assert without < with_late
    budget = (without + with_late) // 2
    charged, lean, taken, joined = plan("admit", budget, [small, large, huge, small])
    assert (lean, joined) == (0, 2) and charged == taken
    charged, lean, taken, joined = plan("admit", budget, [large, small])
    assert (lean, joined) == (1, 1) and charged >= taken


@pytest.mark.parametrize("graph", [(100_000_000, 4, 400_000_000, 500),
                                   (2_600_000, 24, 96_000_000, 5000),
                                   (9_000_000, 60, 900_000_000, 5000),
                                   (60_000, 33_000, 200_000_000, 500),
                                   (2_400_000, 4, 68_000_000, 900_000),
                                   (3000, 1, 20_000, 50)])
@pytest.mark.parametrize("mb", [64, 4096])
def test_column_groups_keep_their_budget(plan, graph, mb):
    """A group is one column, or its scratch is within the budget and as many
    columns as fit it."""
    cols, bytes_, more = plan("group", 0, [graph], FC_PEEL_GROUP_MB=mb)
    assert 1 <= cols <= graph[1]
    assert cols == 1 or bytes_ <= mb << 20
    assert cols == graph[1] or more > mb << 20 or (cols + 1) * graph[0] >= 1 << 32
