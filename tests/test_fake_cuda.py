"""What the library does when a CUDA call is refused or memory is short, on a stand-in for the CUDA
runtime (tests/fake_cuda) linked with the library's own host code: no GPU, and nothing on one, fails."""
import os
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

from slimtracin_b200 import build

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fake_cuda")
LIBRARY = ["st_api", "st_bvh", "st_sah", "st_stage", "st_texture", "st_io", "st_obj"]
DRIVERS = ["ingest.cpp", "stage.cu"]


@pytest.fixture(scope="module")
def drivers(tmp_path_factory):
    """The driver programs: the library's host code, one driver and the stand-in runtime each."""
    out = tmp_path_factory.mktemp("fake_cuda")
    flags = ["-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false", "-Xcompiler", "-fPIC"]
    flags += sum([["-I", d] for d in build.INCLUDES + [HERE]], [])

    def compile_one(src):
        obj = str(out / (os.path.basename(src).rsplit(".", 1)[0] + ".o"))
        subprocess.run([build._nvcc()] + flags + ["-c", src, "-o", obj], check=True)
        return obj

    sources = [os.path.join(build.CSRC, f + ".cu") for f in LIBRARY]
    sources += [os.path.join(HERE, f) for f in ["runtime.cpp"] + DRIVERS]
    with ThreadPoolExecutor(os.cpu_count() or 1) as pool:
        objs = dict(zip([os.path.basename(s).rsplit(".", 1)[0] for s in sources], pool.map(compile_one, sources)))
    # what the drivers never reach (rendering, graphs) is left out, and unresolved
    subprocess.run(["g++", "-shared", "-o", str(out / "library.so"), objs["runtime"]] + [objs[f] for f in LIBRARY]
                   + ["-lpthread", "-Wl,-z,lazy"], check=True)
    for d in [f.split(".")[0] for f in DRIVERS]:
        subprocess.run(["g++", "-o", str(out / d), objs[d], str(out / "library.so"), "-lpthread", "-rdynamic", "-Wl,-z,lazy",
                        "-Wl,--allow-shlib-undefined"], check=True)
    return out


def run(drivers, name, *args):
    p = subprocess.run([str(drivers / name), *args], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, (p.returncode, p.stdout, p.stderr)


@pytest.mark.parametrize("kernel,must_not_follow", [("check_indices_kernel", "tri_aabbs_kernel"), ("tri_aabbs_kernel", "tri_records_kernel"),
                                                    ("tri_records_kernel", "")])
def test_refused_launch_fails_the_mesh_build(drivers, kernel, must_not_follow):
    """Above all that of the check on which the reads through the mesh's indices rely."""
    run(drivers, "ingest", "refused_launch", kernel, must_not_follow)


def test_page_locked_copies_make_no_slots(drivers):
    run(drivers, "stage", "locked_only")


def test_copies_keep_an_earlier_error(drivers):
    run(drivers, "stage", "keeps_errors")


@pytest.mark.parametrize("direction", ["to_host", "to_device"])
def test_a_refused_copy_leaves_none_in_flight(drivers, direction):
    run(drivers, "stage", "refused_copies", direction)


def test_copies_without_memory_or_threads(drivers):
    run(drivers, "stage", "no_resources")


def test_a_refused_allocation_fails_no_later_call(drivers):
    run(drivers, "ingest", "refused_allocation")


def test_trees_with_more_nodes_than_items_allow_are_refused(drivers):
    """The arrays of a scene hold 2n nodes and n pairs of children for n primitives or triangles."""
    run(drivers, "ingest", "oversized_trees")


def test_transient_memory_is_within_the_budget(drivers):
    run(drivers, "ingest", "budget")


def test_kept_memory_goes_back_before_a_call_is_refused(drivers):
    run(drivers, "ingest", "kept_memory")


def test_tlas_updates_page_lock_what_they_use(drivers):
    run(drivers, "ingest", "update_staging")


def test_serving_that_cannot_start_holds_nothing(drivers):
    run(drivers, "ingest", "refused_serving")
