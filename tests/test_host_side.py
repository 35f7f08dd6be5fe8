"""The library's host side on the CPU: all of its objects linked with a stand-in for the
CUDA runtime (host_side/fake_cuda.cpp: two devices, kernels that do nothing, and a record
of what the library asks for), one driver program per property."""
import importlib
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SIDE = os.path.join(HERE, "host_side")


@pytest.fixture(scope="module")
def objects(tmp_path_factory):
    b = importlib.import_module("cfgable-matmul_b200.build")
    b.build()
    tmp = tmp_path_factory.mktemp("host_side")
    inc = os.path.join(os.path.dirname(os.path.dirname(b.nvcc())), "include")
    fake = str(tmp / "fake_cuda.o")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", inc, "-c", os.path.join(SIDE, "fake_cuda.cpp"),
                    "-o", fake], check=True)
    objs = [os.path.join(b.BUILD, f[:-3] + ".o") for f in sorted(os.listdir(b.CSRC))
            if f.endswith(".cu")]
    return tmp, inc, [fake] + objs


def drive(objects, name, timeout=120):
    tmp, inc, objs = objects
    exe = str(tmp / name)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", inc, os.path.join(SIDE, name + ".cpp"),
                    "-o", exe] + objs + ["-lpthread"], check=True)
    r = subprocess.run([exe], timeout=timeout, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


def test_plan_memory_is_not_freed_under_running_work(objects):
    drive(objects, "plan_memory")


def test_each_device_grants_the_matching_its_shared_memory(objects):
    drive(objects, "pair_device")


def test_masked_gemm_takes_the_widest_block(objects):
    drive(objects, "wide_block")


def test_no_exception_leaves_a_host_call(objects):
    drive(objects, "no_memory")


def test_devices_do_not_wait_for_one_another(objects):
    drive(objects, "two_devices")


def test_a_failed_allocation_does_not_fail_the_next_call(objects):
    drive(objects, "after_failure")


def test_fock_items_are_counted_in_64_bits(objects):
    drive(objects, "fock_share")


def test_form_of_split_calls_and_plans(objects):
    drive(objects, "split_form")


def test_host_calls_read_few_error_words(objects):
    drive(objects, "wait_words")


def test_residues_by_rows_are_formed_aside(objects):
    drive(objects, "residue_streams")


def test_forms_of_the_masked_gemm(objects):
    drive(objects, "masked_forms")
