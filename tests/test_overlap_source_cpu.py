"""Kernels of a forward may be launched while the one before still runs (launch_k, csrc/common.cuh).  Read from
the sources: every kernel waits for it (pdl_sync or pdl_wait) unless it only runs when a plan is made, and in a
kernel whose warp roles wait on their own, a role does so before its first bounded wait on a barrier: that
limit is meant for the kernel's own loads, not for the rest of the kernel before."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cssm_b200", "csrc")
PLAN_TIME = {"khat_kernel", "rope_table_kernel", "tcode_kernel", "pack_wt_kernel", "pack_conv_wide_kernel", "pack_conv_kernel",
             "bn_fold_kernel", "affine_vec_kernel", "fill_kernel", "scale_cols_kernel"}


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = open(path).read()
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            start = text.index("{", text.index(")", m.end()))
            depth, i = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            yield os.path.basename(path), m.group(1), text[start:i]


def test_every_forward_kernel_waits_for_the_one_before():
    names = []
    for path, name, body in _kernels():
        names.append(name)
        assert "pdl_sync()" in body or "pdl_wait()" in body or name in PLAN_TIME, f"{path}: {name}"
    assert len(names) > 40 and "gemm_bf16_kernel" in names and "stem_conv1_mma_kernel" in names


def test_warp_roles_wait_before_their_first_barrier():
    checked = 0
    for path, name, body in _kernels():
        at = [m.start() for m in re.finditer(r"pdl_(?:sync|wait)\(\)", body)]
        roles = [m.start() for m in re.finditer(r"// =+ [^=\n]+ =+\n", body)]
        if not at or "mbar_wait" not in body or not roles or at[0] < roles[0]:
            continue                                   # one wait for all warps, ahead of the roles
        for a, b in zip(roles, roles[1:] + [len(body)]):
            role = body[a:b]
            wait = role.find("mbar_wait(")
            if wait < 0:
                continue
            own = re.search(r"pdl_(?:sync|wait)\(\)", role)
            assert own and own.start() < wait, f"{path}: {name}: {role.splitlines()[0].strip()}"
            checked += 1
    assert checked >= 4
