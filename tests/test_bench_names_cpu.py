"""Kernels that the bench and the committed traffic figures name are kernels of the library's sources, and the GDN stage table adds
the seven intervals of cssm_gdn_forward_timed up without losing one."""
import glob
import json
import os
import re
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def _kernels():
    names = set()
    for f in glob.glob(os.path.join(ROOT, "cssm_b200", "csrc", "*.cu")):
        with open(f) as h:
            for head in re.findall(r"__global__\s+void\s+(.{0,200})", h.read(), flags=re.S):
                head = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", head)
                names.add(re.match(r"\s*(\w+)\s*\(", head).group(1))
    return names


def test_named_kernels_exist():
    import bench
    have = _kernels()
    for gdn in (False, True):
        for H in (28, 32, 64):
            assert bench.spectral_kernel(gdn, H) in have, bench.spectral_kernel(gdn, H)


def test_32x32_gdn_name_is_the_kernel_that_is_launched():
    import bench
    with open(os.path.join(ROOT, "cssm_b200", "csrc", "gdn_spectral.cu")) as f:
        launched = re.search(r"PATH_R32 && a\.dk == 4\) return a\.static_image \? \w+\(a, st\) : launch_(\w+)\(a, st\)", f.read()).group(1)
    assert bench.spectral_kernel(True, 32) == launched
    with open(os.path.join(ROOT, "profiles", "traffic.json")) as f:
        assert f"{launched}_dram_bytes_per_head_step" in json.load(f)


def test_traffic_is_of_kernels_that_exist():
    have = _kernels()
    with open(os.path.join(ROOT, "profiles", "traffic.json")) as f:
        keys = [k for k in json.load(f) if "_dram_bytes_per_" in k and not k.startswith("cfg5")]
    assert keys
    for k in keys:
        assert k.split("_dram_bytes_per_")[0] in have, k


def test_stage_table():
    import bench
    assert len(bench.GDN_STAGES) == 7
    assert bench.GDN_JOINED["qkv_proj"] == bench.GDN_JOINED["short_convs"]
    assert len({bench.GDN_JOINED.get(n, n) for n in bench.GDN_STAGES}) == 6
