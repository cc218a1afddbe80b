"""Transfers between host and device memory (fm_staging.cu) on the CPU, with the CUDA calls
replaced (staging_paths.cu, fake_cuda.cpp): which memory goes through the pinned ring, and what happens
when the ring or its threads cannot be had."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from fumeng_b200 import build

ROOT = Path(__file__).resolve().parents[1]
INVALID_VALUE = 1   # cudaErrorInvalidValue


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("staging")
    fake, exe = tmp / "fake_cuda.o", tmp / "staging_paths"
    cuda = Path(build.NVCC).resolve().parents[1] / "include"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(cuda), "-c", str(ROOT / "tests" / "fake_cuda.cpp"), "-o", str(fake)],
                   check=True, capture_output=True)
    subprocess.run([build.NVCC, *build.ARCH, "-O1", "-std=c++17", "-I", str(ROOT / "include"), "-cudart", "none",
                    str(ROOT / "tests" / "staging_paths.cu"), str(fake), "-o", str(exe), "-ldl", "-lpthread",
                    "-Xlinker", "-export-dynamic"], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    return {l.split()[0]: l.split()[1:] for l in out.stdout.splitlines()}


def _trip(lines, name):
    """(errors in and out, contents, [direct copies, ring used] in and out)."""
    e1, e2, same, a, b, c, d = lines[name]
    assert (int(e1), int(e2), same) == (0, 0, "same"), lines[name]
    return (int(a), int(b)), (int(c), int(d))


def test_pageable_memory_goes_through_the_ring_from_a_chunk_on(lines):
    assert _trip(lines, "small") == ((2, 0), (2, 0))
    assert _trip(lines, "pageable") == ((0, 1), (0, 1))


def test_page_locked_memory_is_copied_directly(lines):
    # the third array is pageable: large enough for the ring ...
    assert _trip(lines, "locked") == ((2, 1), (2, 1))
    # ... or not, beside arrays that would make up a chunk with it
    assert _trip(lines, "locked_small_rest") == ((3, 0), (3, 0))


def test_device_memory_in_place_of_host_memory_is_an_error(lines):
    assert [int(v) for v in lines["device"]] == [INVALID_VALUE, INVALID_VALUE]


def test_without_page_locked_memory_for_the_ring_the_copies_are_plain(lines):
    assert _trip(lines, "no_ring") == ((3, 0), (3, 0))


@pytest.mark.parametrize("name", ["no_threads", "two_threads"])
def test_fewer_copy_threads_than_asked_for(lines, name):
    assert _trip(lines, name) == ((0, 1), (0, 1))


@pytest.mark.gpu
def test_page_locked_arrays_give_the_same_results(ctx):
    import torch

    from fumeng_b200 import synth
    n = 300000   # 9.6 MB of rays
    rays = synth.random_rays(np.random.default_rng(1), n, (-1.5, -1.5, -1.5), (1.5, 1.5, 1.5))
    locked = torch.empty(n, 8).pin_memory()
    locked.copy_(torch.from_numpy(rays))
    obj, t = torch.empty(n, dtype=torch.int32).pin_memory(), torch.empty(n).pin_memory()
    scene = ctx.create_scene(synth.hit_scene(5, level=4, spheres=6).to_desc())
    try:
        want = scene.trace_closest(rays)
        ctx.check(ctx.lib.fm_trace_closest(ctx.h, scene.h, locked.data_ptr(), n, obj.data_ptr(), t.data_ptr(), 0))
    finally:
        scene.destroy()
    assert np.array_equal(obj.numpy(), want[0]) and np.array_equal(t.numpy(), want[1])
