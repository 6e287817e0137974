"""The exchange of scalars in the persistent CG kernel (csrc/efe_pcg_slots.cuh) under every order its CTAs can run in:
two CTAs of two warps, a warp per value, each epoch as efe_pcg.cu runs it: post the value, (warp 0) count the CTA's
arrival, wait for all arrivals, read all CTAs' slots of the value, the CTA's own barrier.  No warp may find a slot that
already belongs to a later epoch: it would wait for its own for ever."""

import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CTAS, WARPS, EPOCHS = 2, 2, 4


@pytest.fixture(scope="module")
def slots(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("slots")
    src = d / "slots.cpp"
    src.write_text('#include "efe_pcg_slots.cuh"\n'
                   'extern "C" int slot(unsigned e, int k, int grid) { return efe::pcg_slot(e, k, grid); }\n'
                   'extern "C" int slots(int grid) { return efe::pcg_slots(grid); }\n'
                   'extern "C" int sums() { return efe::PCG_SUMS; }\n'
                   'extern "C" int doubles() { return efe::PCG_SLOT_DOUBLES; }\n')  # fmt: skip
    lib = d / "slots.so"
    subprocess.run([gxx, "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "edelweissfe_gb300", "csrc"), str(src),
                    "-o", str(lib)], check=True)  # fmt: skip
    return ctypes.CDLL(str(lib))


def test_slots_of_one_epoch_are_distinct_and_inside(slots):
    for grid in (1, 2, 152, 512):
        used = [slots.slot(e, k, grid) + i for e in (1, 2) for k in range(slots.sums()) for i in range(grid)]
        assert min(used) >= 0 and max(used) < slots.slots(grid) and len(set(used)) == len(used)
    from edelweissfe_gb300 import _lib as L

    assert 8 + slots.slots(512) * slots.doubles() <= L.EFE_PCG_WORK_DOUBLES


def test_no_order_of_the_ctas_loses_a_slot(slots):
    # a warp's steps in one epoch: 0 post, 1 arrive (warp 0), 2 wait for all arrivals, 3 .. read CTA 0, 1, ...;
    # then the CTA's barrier
    last = 3 + CTAS
    index = {(e, k): slots.slot(e, k, CTAS) for e in range(1, EPOCHS + 1) for k in range(WARPS)}
    start = ((1, 0),) * (CTAS * WARPS), (0,) * slots.slots(CTAS), 0  # (epoch, step) per warp, tags, arrivals
    seen, stack, ends = {start}, [start], 0
    while stack:
        warps, tags, arrivals = stack.pop()
        moved = False
        for w, (e, step) in enumerate(warps):
            cta, k = divmod(w, WARPS)
            t, n = tags, arrivals
            if e > EPOCHS:
                continue
            if step == 0:
                i = index[e, k] + cta
                t = t[:i] + (e,) + t[i + 1 :]
                nxt = (e, 1 if k == 0 else 2)
            elif step == 1:
                n, nxt = n + 1, (e, 2)
            elif step == 2:
                if n < e * CTAS:
                    continue
                nxt = (e, 3)
            elif step < last:
                tag = t[index[e, k] + step - 3]
                assert tag <= e, f"epoch {e}: the slot of CTA {step - 3} already belongs to epoch {tag}"
                if tag < e:
                    continue
                nxt = (e, step + 1)
            else:  # the CTA's barrier: all its warps are done with the epoch
                own = warps[cta * WARPS : (cta + 1) * WARPS]
                if any(x < (e, last) for x in own):
                    continue
                nxt = (e + 1, 0)
            state = warps[:w] + (nxt,) + warps[w + 1 :], t, n
            moved = True
            if state not in seen:
                seen.add(state)
                stack.append(state)
        if not moved:
            ends += 1
            assert all(e > EPOCHS for e, _ in warps), f"stuck: {warps}"
    assert ends == 1
