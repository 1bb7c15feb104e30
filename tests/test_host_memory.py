"""CPU tests of the memory that the library shares between calls (csrc/device_pool.cu, csrc/host_copy.cu), compiled with
g++ against a fake CUDA runtime (fake_cudart.h) whose streams can be stuck."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "icdm-2021_mascot_b200", "csrc")


def compile_check(tmp_path_factory, name, sources):
    exe = str(tmp_path_factory.mktemp(name) / name)
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", CSRC, "-I", cuda, "-x", "c++", os.path.join(ROOT, "tests", name + ".cpp")]
                          + [os.path.join(CSRC, s) for s in sources] + ["-o", exe, "-lpthread"])
    return exe


@pytest.fixture(scope="module")
def shard_timeout_check(tmp_path_factory):
    return compile_check(tmp_path_factory, "shard_timeout_check", ["shard.cu", "device_pool.cu"])


@pytest.mark.parametrize("n_test,gpus", [(5000, 1), (5000, 2), (512 * 20000, 1), (512 * 20000, 2)])
def test_sums_of_an_abandoned_evaluation_go_to_nobody_else(shard_timeout_check, n_test, gpus):
    """The all-gather in front of the evaluation kernel never ends: the call gives up after its limit, and the memory that the
    queued kernel will write into - a pinned block or device memory - is neither freed nor handed out until it has run."""
    out = subprocess.run([shard_timeout_check, "gather", str(n_test), str(gpus)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
    lines = out.stdout.splitlines()
    assert lines[1] == "hung rc -6"
    assert lines[2] == "given away 0 alive 1" and lines[3] == "kept by a release 1"
    assert lines[4] == "left pinned 0" and lines[5] == "left device 0"


def test_sharded_evaluation_reads_its_result_after_the_bounded_wait(shard_timeout_check):
    """The sum over the ranks never ends: a copy into pageable memory queued behind it would wait for good."""
    out = subprocess.run([shard_timeout_check, "reduce", "5000", "2"], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.splitlines()[1] == "hung rc -6", out.stdout


@pytest.fixture(scope="module")
def host_cores_check(tmp_path_factory):
    return compile_check(tmp_path_factory, "host_cores_check", [])


@pytest.mark.parametrize("files,quota", [
    ({}, 0),
    ({"proc/self/cgroup": "0::/\n", "sys/fs/cgroup/cpu.max": "max 100000\n"}, 0),
    ({"proc/self/cgroup": "0::/\n", "sys/fs/cgroup/cpu.max": "250000 100000\n"}, 2.5),
    ({"proc/self/cgroup": "0::/a/b\n", "sys/fs/cgroup/a/cpu.max": "100000 100000\n", "sys/fs/cgroup/a/b/cpu.max": "300000 100000\n"}, 1),
    ({"proc/self/cgroup": "0::/host/only\n", "sys/fs/cgroup/cpu.max": "50000 100000\n"}, 0.5),
    ({"proc/self/cgroup": "4:memory:/x\n3:cpu,cpuacct:/x\n", "sys/fs/cgroup/cpu/x/cpu.cfs_quota_us": "-1\n", "sys/fs/cgroup/cpu/x/cpu.cfs_period_us": "100000\n"}, 0),
    ({"proc/self/cgroup": "3:cpuset:/y\n2:cpuacct,cpu:/x/y/\n", "sys/fs/cgroup/cpu/x/cpu.cfs_quota_us": "400000\n", "sys/fs/cgroup/cpu/x/cpu.cfs_period_us": "200000\n"}, 2),
    ({"proc/self/cgroup": "no colon\n0::\n", "sys/fs/cgroup/cpu.max": "\n"}, 0),
])
def test_copy_threads_follow_a_cpu_quota(host_cores_check, tmp_path, files, quota):
    for name, text in files.items():
        (tmp_path / name).parent.mkdir(parents=True, exist_ok=True)
        (tmp_path / name).write_text(text)
    found, cores = subprocess.run([host_cores_check, str(tmp_path)], capture_output=True, text=True, check=True).stdout.split()
    have = len(os.sched_getaffinity(0))
    assert float(found) == quota
    assert int(cores) == (have if quota == 0 else max(1, min(have, int(quota))))
