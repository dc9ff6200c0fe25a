"""The rules that pick multi-RW kernels, at sizes where the choices were measured to
differ (CPU only: grass_b200/csrc/launch_rules.h is plain C++)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    """rule("expression"): its value as an integer."""
    tmp = tmp_path_factory.mktemp("rules")

    def value(expression):
        src, exe = tmp / "rule.cpp", tmp / "rule"
        src.write_text('#include <stdio.h>\n#include "launch_rules.h"\nusing namespace grass;\n'
                       f'int main() {{ printf("%lld", (long long)({expression})); }}\n')
        subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "grass_b200", "csrc"),
                        "-o", str(exe), str(src)], check=True)
        return int(subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout)
    return value


@pytest.mark.parametrize("samples,walkers,threads", [
    (1, 80, 128), (8192, 80, 128), (148, 160, 160), (8192, 160, 160), (148, 257, 288), (149, 257, 160), (8192, 512, 160),
    (1, 512, 512), (1, 513, 544), (8192, 2000, 1024)])
def test_threads_of_a_continuous_time_sample(rule, samples, walkers, threads):
    assert rule(f"mrw_block_threads({samples}, {walkers}, true, 148)") == threads


@pytest.mark.parametrize("samples,walkers,steps,blocks", [
    (1, 80, 100, False), (148, 80, 300, True), (600, 80, 300, False), (600, 80, 1024, True), (2000, 80, 1024, False),
    (148, 1000, 300, True), (148, 1000, 511, True), (300, 1000, 500, False), (600, 1000, 3000, True),
    (2000, 1000, 3000, False), (300, 2000, 2000, True), (600, 2000, 10000, True), (8192, 2000, 10000, False),
    (148, 8, 500, False), (1, 1, 5000, False), (600, 1, 1024, False)])
def test_uniform_samples_as_blocks_or_warps(rule, samples, walkers, steps, blocks):
    threads = rule(f"mrw_block_threads({samples}, {walkers}, false, 148)")
    resident = 148 * (65536 // (120 * threads))  # (120 registers a thread)
    assert rule(f"mrw_uniform_by_blocks({samples}, {walkers}, {steps}, {threads}, {resident})") == blocks


@pytest.mark.parametrize("samples,walkers,steps,groups,warps,by_groups", [
    (1, 80, 100, 15000, 4736, True), (8192, 160, 100, 8288, 4736, True), (8192, 192, 100, 8288, 4736, True),
    (3000, 192, 100, 8288, 4736, False), (8192, 208, 100, 7104, 4736, False), (7000, 208, 100, 7104, 4736, True),
    (148, 256, 100, 5920, 4736, False), (1, 256, 100, 5920, 4736, True), (12000, 192, 5, 8288, 4736, False), (12000, 192, 50, 8288, 4736, True)])
def test_degree_samples_as_groups_or_warps(rule, samples, walkers, steps, groups, warps, by_groups):
    assert rule(f"mrw_degree_by_groups({samples}, {walkers}, {steps}, {groups}, {warps})") == by_groups


@pytest.mark.parametrize("samples,walkers,threads", [
    (1, 8, 128), (296, 80, 128), (296, 300, 320), (296, 2000, 512), (297, 300, 160), (297, 2000, 256), (10000, 20, 128)])
def test_threads_of_a_batch_sample(rule, samples, walkers, threads):
    assert rule(f"batch_block_threads({samples}, {walkers}, 148)") == threads
