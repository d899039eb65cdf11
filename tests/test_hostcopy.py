"""Large copies between pageable host fields and the device (csrc/hostcopy.cuh) on
the CPU, against a fake of the CUDA runtime calls that it makes: whole at every
size, the caller's current device left alone, several threads and devices at
once, errors returned, the pinned set made when it pays and given back.  On the
GPU: whole fields through it."""
import os
import subprocess
import threading

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_hostcopy(tmp_path):
    exe = str(tmp_path / "hostcopy_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-Wall", "-pthread", "-I",
                    os.path.join(HERE, "fake_cuda"), "-x", "c++",
                    os.path.join(HERE, "fake_cuda", "hostcopy_check.cc"), "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr


@pytest.mark.gpu
def test_fields_cross_the_bus_whole_again_and_again(engine_mod):
    """A field of 28.7 MB (14 chunks and a part of one) up and down until copies go
    through the pinned buffers and after; then two threads with an engine each."""
    P = engine_mod
    L, N = (8, 8, 8, 12), 8
    rng = np.random.default_rng(9)
    fields = [rng.normal(size=(int(np.prod(L)), 4, P.series_len(N))) for _ in range(2)]
    with P.NsptEngine(L, N) as e, P.NsptEngine(L, N) as f:
        for rep in range(4):
            a = fields[rep % 2]
            e.upload(a)
            assert np.array_equal(e.download(), a)
        whole = [0, 0]

        def copies(k, engine):
            for _ in range(6):
                engine.upload(fields[k])
                whole[k] += np.array_equal(engine.download(), fields[k])

        threads = [threading.Thread(target=copies, args=(k, g)) for k, g in enumerate((e, f))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert whole == [6, 6]
