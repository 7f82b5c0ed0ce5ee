"""Device memory of the calls that take host arrays, against a CUDA runtime for the CPU
(fake_cudart.c) that counts allocations, copies and waits and fails a chosen one. Each
test is a process of its own, since the runtime has to be in place before the library
is loaded."""

import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PRELUDE = r'''
import ctypes, json, sys
import numpy as np
import lambda_b200 as lb

rt = ctypes.CDLL(sys.argv[1])
MALLOC, FREE, HOST_ALLOC, COPY_IN, LAUNCH, SYNC = range(6)
scene = lb.HostScene.parse(sys.argv[2])
ctx = lb.Context(0)
ctx.upload(scene)


def rays(n):
    return np.ones((n, 6), np.float32)


def shadow(n):
    pick = np.zeros(n, np.int64)
    return ctx.trace_shadow(rays(n), scene.light_instances[pick], scene.light_objects[pick])


def films(n):
    return np.ones((n, 5), np.float32)


calls = {
    "closest": lambda n: ctx.trace_closest(rays(n)),
    "shadow": shadow,
    "film": lambda n: ctx.thinfilm_exact(films(n)),
    "film_fp64": lambda n: ctx.thinfilm_fp64(films(n)),
}


def counted(call):
    """Allocations and frees of a call, and whether it raised out of memory."""
    rt.fake_reset()
    try:
        call()
        error = ""
    except lb.LambdaError as e:
        error = str(e)
    return rt.fake_count(MALLOC), rt.fake_count(FREE), error


'''


@pytest.fixture(scope="module")
def on_cpu(tmp_path_factory):
    """Runs a script over the prelude and returns what it prints last, as JSON."""
    d = tmp_path_factory.mktemp("fake")
    so = d / "fake_cudart.so"
    subprocess.run(["gcc", "-std=c11", "-O1", "-shared", "-fPIC", "-I", os.path.join(CUDA, "include"),
                    "-include", "vector_types.h", os.path.join(ROOT, "tests", "fake_cudart.c"), "-o", str(so)], check=True)

    def run(script):
        r = subprocess.run([sys.executable, "-c", PRELUDE + script, str(so),
                            os.path.join(ROOT, "tests", "golden", "scenes", "cornell.lrd")],
                           env=dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT), cwd=ROOT, capture_output=True,
                           text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return json.loads(r.stdout.splitlines()[-1])

    return run


@pytest.mark.parametrize("name", ["closest", "shadow", "film", "film_fp64"])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6])
def test_a_failed_allocation_is_not_reported_by_a_later_call(on_cpu, name, k):
    """Whichever allocation of a first call fails, the call says so or does without it, no
    error is left in the runtime, and the next call works."""
    got = on_cpu(f'''
rt.fake_fail_malloc({k})
first = counted(lambda: calls["{name}"](1000))
rt.fake_fail_malloc(0)
left = rt.fake_pending()
second = counted(lambda: calls["{name}"](1000))
print(json.dumps([first, left, second]))
''')
    first, left, second = got
    assert first[2] == "" or "OUT_OF_MEMORY" in first[2]
    assert left == 0 and second[2] == ""


@pytest.mark.parametrize("name", ["closest", "shadow", "film", "film_fp64"])
def test_a_call_allocates_its_staging_once(on_cpu, name):
    """The first call makes one allocation for all its arrays and frees none; calls that fit
    make none; a larger one replaces it. One that is larger than the kept memory (64 MB)
    allocates once for itself."""
    got = on_cpu(f'''
call = calls["{name}"]
small = [counted(lambda: call(n)) for n in (1000, 1000, 10)]
grown = [counted(lambda: call(n)) for n in (20_000, 20_000, 1000)]
large = [counted(lambda: call(n)) for n in (2_000_000, 2_000_000, 1000)]
print(json.dumps([small, grown, large]))
''')
    small, grown, large = got
    assert small == [[1, 0, ""], [0, 0, ""], [0, 0, ""]]
    assert grown == [[1, 1, ""], [0, 0, ""], [0, 0, ""]]
    assert large == [[1, 1, ""], [1, 1, ""], [0, 0, ""]]


def test_a_large_call_takes_the_kept_memory_where_there_is_no_other(on_cpu):
    got = on_cpu('''
counted(lambda: calls["film"](1000))
rt.fake_fail_malloc(1)
print(json.dumps([counted(lambda: calls["film"](2_000_000)), rt.fake_pending(), counted(lambda: calls["film"](1000))]))
''')
    assert got == [[2, 2, ""], 0, [1, 0, ""]]


@pytest.mark.parametrize("name", ["closest", "shadow", "film", "film_fp64"])
def test_a_call_that_fails_waits_for_its_copies(on_cpu, name):
    """A call whose launch fails returns only once the copies from the caller's arrays are
    done: the caller may free page-locked arrays, which copy behind its back."""
    got = on_cpu(f'''
counted(lambda: calls["{name}"](1000))
rt.fake_fail_launch(1)
failed = counted(lambda: calls["{name}"](1000))
waited = rt.fake_copies_waited_for()
print(json.dumps([failed, waited, counted(lambda: calls["{name}"](1000))]))
''')
    failed, waited, after = got
    assert "LAMBDA_ERR_CUDA" in failed[2] and after == [0, 0, ""]
    assert waited == 1
