"""The shared-memory limit of a kernel when worlds on several threads launch it with
different sizes (csrc/smem_limit.cuh): no launch finds it below its own size."""
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "physecs_gb300", "csrc")


def test_limit_is_never_lowered(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "check_smem_limit")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(HERE, "limits", "check_smem_limit.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_worlds_of_many_sizes_on_threads(gpu_lib):
    from physecs_gb300 import scenes
    from physecs_gb300.api import World
    sizes = [40, 3900, 200, 2000, 900, 3000, 500, 1300]
    ss = [scenes.batch_scene(60 + i, n_bodies=n) for i, n in enumerate(sizes)]
    out, errors = [None] * len(ss), []

    def run(i, into):
        try:
            w = World([ss[i]])
            w.step(frames=2)
            w.synchronize()
            into[i] = w.read_bodies()
            w.close()
        except Exception as e:  # noqa: BLE001 - reported by the test
            errors.append((i, e))

    threads = [threading.Thread(target=run, args=(i, out)) for i in range(len(ss))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    alone = [None] * len(ss)
    for i in range(len(ss)):
        run(i, alone)
    assert not errors
    for a, b in zip(out, alone):
        for k in b:
            assert np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32)), k
