"""The batched peel's host-side plan: what a launch over several graphs needs,
asked of the library itself by a small program (tests/native/plan_check.cpp)."""
import os
import subprocess

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
