"""The symmetric kernels' schedule on the CPU: the functions the kernels run
(csrc/symplan.h, plain C++) are compiled with the host compiler and every CTA's
tiles and slots are followed.  Every pair of blocks is met once, every (slot,
row) has one writer, and every counted slot is written; from one body to
systems of several sub-blocks per block and of fewer than 128 slots."""
import ctypes as C
import os
import random
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "n-body-code_b200", "csrc")
BUILD = os.path.join(HERE, "_build")

# (rows of a CTA, bodies of a tile) of the FP64, near/far, VJP and potential kernels
KERNELS = [(256, 32), (512, 32), (256, 64), (512, 128)]


@pytest.fixture(scope="module")
def lib():
    os.makedirs(BUILD, exist_ok=True)
    so = os.path.join(BUILD, "sym_schedule_check.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", CSRC, "-o", so,
                    os.path.join(HERE, "sym_schedule_check.cpp")], check=True)
    L = C.CDLL(so)
    for f in (L.check_schedule, L.check_plan):
        f.restype = C.c_char_p
    return L


def sizes(rows, rng):
    """Edges of tiles, blocks and sub-blocks, and drawn ones."""
    edge = [k * rows + d for k in (1, 2, 3, 4, 7, 8, 127, 128, 129, 255, 256, 257) for d in (-1, 0, 1)]
    return [1, 2, 31, 33, 63, 65, 127, 129] + edge + [rng.randrange(1, 200000) for _ in range(12)]


@pytest.mark.parametrize("rows,tj", KERNELS)
def test_every_pair_once_and_one_writer_per_slot(lib, rows, tj):
    rng = random.Random(rows + tj)
    for n in sizes(rows, rng):
        for S in sorted({1, 2, 3, rng.randrange(1, 65), 64}):
            bad = lib.check_schedule(rows, tj, n, S)
            assert bad is None, (n, S, bad)


@pytest.mark.parametrize("rows,tj", [(512, 32), (512, 128)])
@pytest.mark.parametrize("n", [1_398_101, 1_398_102, 1_500_001, 2_900_003, 5_600_000, 20_000_003])
def test_systems_with_fewer_slots(lib, rows, tj, n):
    """8 GiB of slots bound the blocks from 1.4e6 bodies, 32 slots are the least."""
    limit = lib.slot_limit(n)
    assert limit == (128 if n <= 1_398_101 else max(32, int(8.0 * 2 ** 30 / (48.0 * n))))
    assert lib.blocks(rows, n) <= limit and lib.sub_blocks(rows, n) > 1
    for S in (1, 5, limit // 2):
        bad = lib.check_schedule(rows, tj, n, S)
        assert bad is None, (S, bad)


@pytest.mark.parametrize("rows,tj", KERNELS)
@pytest.mark.parametrize("fp64", [0, 1])
def test_plans(lib, rows, tj, fp64):
    rng = random.Random(5)
    for n in sizes(rows, rng) + [262144, 1_500_001, 20_000_003]:
        bad = lib.check_plan(rows, tj, n, int(rows == 512), fp64)
        assert bad is None, (n, bad)
