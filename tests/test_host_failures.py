"""The library's host side when a call of the CUDA runtime fails or a kernel
reports an error, on the CPU: the library runs in a child process over a
stand-in runtime (fake_cudart.cpp), whose kernels do nothing and whose failures
are set by the test.
"""
import os
import subprocess
import sys

import pytest

import rodgpu

HERE = os.path.dirname(os.path.abspath(__file__))

SETUP = """
import ctypes
import numpy as np
import rodgpu

fake = ctypes.CDLL({fake!r})
fake.fake_launches.restype = ctypes.c_longlong
fake.fake_uploads.restype = ctypes.c_size_t
fake.fake_uploads.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
ERR = dict(contacts=1, lists=2, history=8, timeout=16)
N = 50
rng = np.random.default_rng(1)
X, Q, Z = rng.uniform(-1, 1, (N, 3)), np.tile([1.0, 0, 0, 0], (N, 1)), np.zeros((N, 3))


def system(model):
    s = rodgpu.System(rodgpu.default_config(n_bodies=N, model=model, dt=1e-4))
    s.set_bodies(np.full(N, 0.05), np.full(N, 0.5), np.ones(N), np.ones((N, 3)))
    s.set_state(X, Q, Z, Z)
    return s


def uploads():
    buf = ctypes.create_string_buffer(1 << 20)
    n = fake.fake_uploads(buf, len(buf))
    assert n <= len(buf)
    return buf.raw[:n]


def code(call, *a):
    try:
        call(*a)
    except rodgpu.RgError as e:
        return rodgpu.STATUS[e.code]
    return "ok"

"""


@pytest.fixture(scope="module")
def run_child(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I/usr/local/cuda/include", "-o", out,
                    os.path.join(HERE, "fake_cudart.cpp")], check=True)

    def run(body):
        env = dict(os.environ, LD_PRELOAD=out, PYTHONPATH=rodgpu.PKG)
        r = subprocess.run([sys.executable, "-c", SETUP.format(fake=out) + body], env=env, capture_output=True,
                           text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr

    return run


@pytest.mark.parametrize("model", ["hertz-mindlin", "harmonic"])
@pytest.mark.parametrize("call", ["s.step, 4", "s.compute_forces"])
@pytest.mark.parametrize("failure", ["fake.fake_fail_launches(1)", "fake.fake_next_error(ERR['timeout'])"])
def test_contacts_of_a_failed_call_are_not_used(run_child, model, call, failure):
    # What the next step uploads (control words, then the kernel's view with
    # the flag that says which contacts are current) is what a step after a
    # new state uploads, byte for byte: the failed call left nothing.
    run_child(f"""
s = system({model!r})
s.detect(0.0)        # names the error word
s.set_state(X, Q, Z, Z)
uploads()
s.step(3)
first = uploads()
s.step(2)
assert uploads() != first          # contacts of the call before are used
s.set_state(X, Q, Z, Z)
uploads()
s.step(3)
assert uploads() == first
s.set_state(X, Q, Z, Z)
{failure}
assert code({call}) in ("CUDA error", "device wait timed out")
uploads()
s.step(3)
assert uploads() == first
""")


@pytest.mark.parametrize("model", ["nsc", "hertz-mindlin", "harmonic"])
def test_every_device_allows_the_shared_memory_of_the_step(run_child, model):
    # the limit on dynamic shared memory belongs to a device, not to the process
    run_child(f"""
for device in (0, 1, 0):
    fake.fake_set_device(device)
    s = system({model!r})
    s.step(2)
    if {model!r} != "nsc":
        s.compute_forces()
    s.close()
assert fake.fake_smem_refused() == 0
""")


@pytest.mark.parametrize("model,bit", [("hertz-mindlin", "contacts"), ("harmonic", "lists"), ("nsc", "contacts")])
def test_a_handle_without_buffers_asks_for_its_bodies(run_child, model, bit):
    # the larger buffers cannot be allocated: no kernel may run on the handle
    # until its bodies are set again
    run_child(f"""
seen = 0
for left in range(0, 60):
    s = system({model!r})
    s.detect(0.0)
    s.step(1)
    fake.fake_next_error(ERR[{bit!r}])
    fake.fake_fail_malloc_after(left)
    first = code(s.step, 1)
    fake.fake_fail_malloc_after(-1)
    if first == "ok":
        s.close()
        break
    n = fake.fake_launches()
    if first == "capacity exceeded":
        seen += 1
        assert code(s.step, 1) == code(s.detect, 0.0) == "call out of order"
        if {model!r} != "nsc":
            assert code(s.compute_forces) == "call out of order"
        assert fake.fake_launches() == n
        s.set_bodies(np.full(N, 0.05), np.full(N, 0.5), np.ones(N), np.ones((N, 3)))
    else:  # the buffers are there, the snapshot's are not
        assert first == "CUDA error", first
    assert code(s.step, 1) == "ok" and fake.fake_launches() > n
    s.close()
assert seen > 1
""")


def test_a_batch_asks_again_for_what_its_first_step_did_not_get(run_child):
    # the tables of the Verlet members' launch are allocated by the first
    # step; a step that got only some of them leaves the others to the next
    run_child("""
cut = 0
for left in range(0, 200):
    b = rodgpu.Batch([rodgpu.default_config(n_bodies=N, model=m, dt=1e-4) for m in ("hertz-mindlin", "harmonic")])
    for k in range(2):
        b.set_bodies(k, np.full(N, 0.05), np.full(N, 0.5), np.ones(N), np.ones((N, 3)))
        b.set_state(k, X, Q, Z, Z)
    fake.fake_fail_malloc_after(left)
    try:
        b.step(1)
        done = True
    except rodgpu.RgError as e:
        done = False
        if "Verlet launch" in str(e):
            cut += 1
            fake.fake_fail_malloc_after(-1)
            assert code(b.step, 1) == "ok"
    fake.fake_fail_malloc_after(-1)
    b.close()
    if done:
        break
assert cut == 4, cut
""")
