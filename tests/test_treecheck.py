"""The device's check of a newly built TLAS (csrc/st_treecheck.h), run on the host over whole and damaged
trees: it accepts what st_validate_bvh accepts, where every node is reached, and reads nothing outside
the arrays (the program is built with the address sanitizer)."""
import os
import subprocess

import numpy as np
import pytest

import oracle
from slimtracin_b200 import api, build, structs as S
from tests.test_abi import _chain

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("treecheck") / "treecheck")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all"]
                   + sum([["-I", d] for d in build.INCLUDES], []) + [os.path.join(HERE, "treecheck.cpp"), "-o", exe], check=True)
    return exe


def tree(rng, n):
    boxes = rng.uniform(-1, 1, (n, 3))
    boxes = np.concatenate([boxes, boxes + 0.1], 1).astype(np.float32)
    codes, order, leaf = (np.zeros(n, np.uint32) for _ in range(3))
    nodes, info = np.zeros(2 * n, dtype=S.BVHNODE_DT), np.zeros(2, np.uint32)
    oracle.restatement().orc_lbvh30(boxes.ctypes.data, n, int(rng.integers(1, 4)), codes.ctypes.data, order.ctypes.data,
                                    nodes.ctypes.data, leaf.ctypes.data, info.ctypes.data)
    return nodes, (int(info[0]) - 1) // 2


def expected(L, nodes, count, n):
    if L.st_validate_bvh(nodes.ctypes.data, count, n, 1) != api.ST_OK:
        return False
    reached, stack = 0, [0]
    while stack:
        k = stack.pop()
        reached += 1
        if not nodes["child_count"][k]:
            stack += [int(nodes["first_child_id"][k]), int(nodes["first_child_id"][k]) + 1]
    return reached == count


def test_device_check_of_a_tree_equals_the_host_check(program):
    L = api.lib()
    rng = np.random.default_rng(5)
    cases, want = [], []

    def case(nodes, pairs, n):
        padded = np.zeros(2 * n, dtype=S.BVHNODE_DT)
        padded[:len(nodes)] = nodes[:2 * n]
        before = rng.integers(0, 2 * n + 2, n).astype(np.uint32)
        cases.append(np.array([n, pairs], np.uint32).tobytes() + padded.tobytes() + before.tobytes())
        count = 1 + 2 * min(pairs, n - 1)
        want.append(pairs < n and expected(L, padded, count, n))

    for depth in (1, 5, 61, 62, 63, 64, 200):
        nodes, n = _chain(depth)
        case(nodes, depth, n)
    for _ in range(3000):
        n = int(rng.integers(1, 40))
        nodes, pairs = tree(rng, n)
        case(nodes, pairs, n)
        for _ in range(int(rng.integers(0, 3))):         # damaged: links, counts, the number of pairs
            k = int(rng.integers(0, 1 + 2 * pairs))
            values = [0, 1, 2, k, int(rng.integers(0, 2 * n + 2)), 2 * pairs - 1, 2 * pairs, 2 * n - 1, n, 2 ** 31, 2 ** 32 - 1, 2 ** 32 - 2]
            if rng.integers(0, 3):
                nodes["first_child_id"][k] = values[int(rng.integers(0, len(values)))] % 2 ** 32
            else:
                nodes["child_count"][k] = values[int(rng.integers(0, len(values)))] % 65536
            case(nodes, pairs, n)
        case(nodes, int(rng.choice([0, pairs + 1, max(pairs, 1) - 1, n, 2 ** 32 - 1])), n)
    assert 1000 < sum(want) < len(want) - 1000
    got = subprocess.run([program], input=b"".join(cases), capture_output=True, check=True).stdout.decode().split()
    assert got == [f"{int(w)}{int(w)}" for w in want]
