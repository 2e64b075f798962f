"""Transfer lists of several scenes, built by several threads on one context: the scenes'
leaves and triangles ask for different amounts of shared memory."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_with_scenes_of_their_own(gpu_ctx):
    from test_gpu_transfer_tiles import _env, _same
    from vrad_gb300 import scenes

    made = [(_env(gpu_ctx, scenes.lit_scene(40 + i, n_faces=n, spacing=96.0, n_point=1, n_spot=1)),
             scenes.transfer_directions(k)) for i, (n, k) in enumerate([(6, 256), (900, 512), (60, 128), (2500, 256)])]
    want = [env.get_transfers(leaves, env.make_transfers(dirs)) for (env, leaves), dirs in made]
    wrong = []

    def build(i):
        (env, leaves), dirs = made[i]
        try:
            for _ in range(60):
                if not _same(env.get_transfers(leaves, env.make_transfers(dirs)), want[i]):
                    wrong.append(f"scene {i}: other lists")
        except Exception as e:
            wrong.append(f"scene {i}: {e}")

    threads = [threading.Thread(target=build, args=(i,)) for i in range(len(made))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong and all(len(w[1]) > 0 for w in want[1:])
