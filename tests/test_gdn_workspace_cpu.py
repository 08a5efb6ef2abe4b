"""Scratch that cssm_gdn_workspace_bytes asks for: none for states that a kernel keeps in registers (32x32 planes, key dim 4), none for gate
planes that are never written (channel gates multiplied where k and v lie: 64 channels, planes of whole 128-pixel tiles)."""
import ctypes as C

import pytest

from cssm_b200 import _lib
from cssm_b200.modules import GatedDeltaNetCSSM


def _lib_built():
    import os
    if not os.path.exists(_lib.LIB_PATH):
        from cssm_b200 import build
        build.build()
    return _lib.lib()


def _expected(B, T, H, W, Cc, dk, gate):
    up = lambda n: (n + 255) // 256 * 256
    BT, HW, NB, nh, chan = B * T, H * W, H * (W // 2 + 1), Cc // dk, gate == "channel"
    n = up(BT * 3 * Cc * HW * 4) + up(BT * Cc * HW * 4) + up(BT * H * Cc * 4) + up(BT * (nh if chan else 1) * NB * 8) + up(BT * HW * 8)
    if chan and not (Cc == 64 and HW % 128 == 0):
        n += up(BT * 2 * Cc * HW * 4)
    if not (H == W == 32 and dk == 4):
        n += up(B * nh * dk * dk * NB * 8)
    return n


@pytest.mark.parametrize("gate", ["factored", "channel"])
@pytest.mark.parametrize("B,T,H,W,Cc,dk", [(3, 2, 32, 32, 64, 4), (3, 2, 32, 32, 64, 2), (2, 5, 32, 32, 32, 4), (2, 3, 64, 64, 64, 4), (2, 3, 16, 16, 64, 4),
                                           (1, 2, 28, 28, 64, 2)])
def test_workspace_bytes(gate, B, T, H, W, Cc, dk):
    L = _lib_built()
    m = GatedDeltaNetCSSM(channels=Cc, delta_key_dim=dk, kernel_size=3, gate_type=gate, rope_mode="none", qkv_conv_size=1)
    d = m._desc((B, T, H, W, Cc))
    assert L.cssm_gdn_workspace_bytes(C.byref(d)) == _expected(B, T, H, W, Cc, dk, gate)
