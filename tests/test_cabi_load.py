"""The C-ABI library loads without a GPU and exports every declared symbol;
host-only entry points behave; argument errors are reported before any launch."""
import ctypes as C
import re
from pathlib import Path

import pytest
import torch

from gemmallm_b200 import _cabi
from gemmallm_b200._cabi import lib

HEADER = Path(__file__).resolve().parent.parent / "include" / "moe_b200.h"


def declared_symbols():
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return sorted(set(re.findall(r"\b(moe_b200_\w+)\s*\(", text)))


def test_every_declared_symbol_is_exported_and_bound():
    names = declared_symbols()
    assert len(names) >= 14
    raw = C.CDLL(str(_cabi.LIB_PATH))
    for n in names:
        assert hasattr(raw, n), f"{n} declared in moe_b200.h but not exported"
        assert n in _cabi.SIGNATURES, f"{n} has no ctypes signature"
    assert set(_cabi.SIGNATURES) == set(names)


def test_version_and_sizes():
    assert lib.moe_b200_version() == _cabi.ABI_VERSION
    n = _cabi.workspace_bytes(16384, 1024, 4096, 8, 2, _cabi.BF16)
    # perm + y (N*k*d) and h (N*k*f) dominate
    assert n > 2 * 16384 * (2 * 1024 + 4096) * 2
    lay = _cabi.workspace_layout(16384, 1024, 4096, 8, 2, _cabi.BF16)
    assert list(lay) == list(_cabi.WS_NAMES)
    offs = list(lay.values())
    assert offs == sorted(offs) and all(o % 1024 == 0 for o in offs)
    assert lib.moe_b200_plan_bytes(8) >= 4 * 8 * 8 + 2 * 8 * 128
    assert lib.moe_b200_router_blocks(65) == 2
    assert lib.moe_b200_decode_splits(4096) == 8 and lib.moe_b200_decode_splits(128) == 1
    assert lib.moe_b200_decode_max_rows() == 256
    assert lib.moe_b200_dispatch_scratch_bytes(1000, 8, 2) > 0


def test_version_goes_with_the_plan_and_the_training_workspace():
    """A caller built against another layout of a plan, or against other contents of GU and MASK or of the forward's PSUM_PART,
    PERM, H and Y, sees another version."""
    maps = [(lib.moe_b200_plan_bytes(E) - (32 * E + 127) // 128 * 128) / (128 * E) for E in (1, 8, 256)]
    assert (lib.moe_b200_version(), maps) == (4, [5, 5, 5])
    assert re.search(r"ABI_VERSION 4\b", HEADER.read_text())


def test_bad_shapes_are_rejected_on_the_host():
    assert lib.moe_b200_workspace_bytes(16, 1020, 4096, 8, 2, _cabi.BF16) == 0   # d % 8
    assert lib.moe_b200_workspace_bytes(16, 1024, 4096, 300, 2, _cabi.BF16) == 0  # E > 256
    assert lib.moe_b200_workspace_bytes(16, 1024, 4096, 8, 9, _cabi.BF16) == 0    # k > 8
    assert lib.moe_b200_workspace_bytes(16, 1024, 4096, 2, 3, _cabi.BF16) == 0    # k > E
    assert lib.moe_b200_workspace_bytes(16, 1024, 4096, 8, 2, 7) == 0             # dtype
    assert b"dtype" in lib.moe_b200_last_error_string()
    # NULL workspace: error code, nothing launched
    rc = lib.moe_b200_forward(None, None, None, None, None, None, None, 0.0, 16, 1024, 4096, 8, 2, _cabi.BF16, 0,
                              None, 0, None, None)
    assert rc == -1
    # misaligned workspace
    rc = lib.moe_b200_forward(None, None, None, None, None, None, None, 0.0, 16, 1024, 4096, 8, 2, _cabi.BF16, 0,
                              8, 1 << 40, None, None)
    assert rc == -3


def test_small_and_mid_size_entry_points_check_their_arguments():
    """The weight-streaming entry points reject what they cannot run before any launch."""
    a = 1 << 20     # any non-NULL, 16-byte aligned address: nothing is dereferenced on these paths
    # routing-independent kernel: N <= 128, E <= 32
    rc = lib.moe_b200_experts_decode_spec(a, a, a, a, 129, 2, 1024, 4096, 8, a, a, a, a, None)
    assert rc == -7 and b"128" in lib.moe_b200_last_error_string()
    rc = lib.moe_b200_experts_decode_spec(a, a, a, a, 64, 2, 1024, 4096, 33, a, a, a, a, None)
    assert rc == -7
    rc = lib.moe_b200_experts_decode_spec(a, None, a, a, 64, 2, 1024, 4096, 8, a, a, a, a, None)
    assert rc == -1
    # sorted-rows kernel: K ranges within [1, 8] and not more than there are 64-wide K blocks
    assert lib.moe_b200_experts_rows(a, a, a, 512, 1024, 4096, 8, 9, a, a, a, a, None) == -2
    assert lib.moe_b200_experts_rows(a, a, a, 512, 1024, 64, 8, 2, a, a, a, a, None) == -2
    assert lib.moe_b200_experts_rows(a, a, a, 512, 1024, 4096, 8, 4, a, a, None, a, None) == -1
    assert lib.moe_b200_experts_rows(a + 8, a, a, 512, 1024, 4096, 8, 4, a, a, a, a, None) == -3
    # both products in one launch: any number of rows, no NULL buffer, aligned rows
    mid = lambda M=512, d=1024, x=a, y=a: lib.moe_b200_experts_mid(x, a, a, M, d, 4096, 8, a, y, a, a, None)
    assert (mid(M=0), mid(M=-1), mid(d=1020), mid(y=None), mid(x=a + 8), mid(y=a + 4)) == (0, -2, -2, -1, -3, -3)
    # one counter per row block: far too many rows
    assert lib.moe_b200_experts_rows(a, a, a, 1 << 20, 1024, 4096, 8, 4, a, a, a, a, None) == -7
    # sizes the forward uses
    assert lib.moe_b200_decode_spec_rows(1) == 16 and lib.moe_b200_decode_spec_rows(65) == 128
    assert lib.moe_b200_rows_splits(1024, 1024, 4096, 8) == 4
    assert 1 <= lib.moe_b200_rows_splits(1024, 4096, 256, 8) <= 4 // 8 + 1
    # shared-work front: token limit
    assert lib.moe_b200_front_small_split(a, a, a, 2049, 1024, 8, 2, _cabi.BF16, *([a] * 12), None) == -7
    assert lib.moe_b200_front_exchange_ints(512, 8, 2) == 32 * 2 * 8 + 32 * 8
    # the single-launch kernels' fused entry point: row limit
    assert lib.moe_b200_experts_decode_fused(a, a, a, 257, 1024, 4096, 8, a, a, a, a, None) == -2
    # the one-launch block: one to eight tokens, at most 32 experts, no NULL output, aligned rows
    tiny = lambda N, d, f, E, k, x=a, out=a: lib.moe_b200_decode_tiny(
        x, a, a, a, None, N, d, f, E, k, a, a, a, a, a, a, a, a, a, a, out, a, None)
    assert tiny(9, 1024, 4096, 8, 2) == -7 and b"N <= 8" in lib.moe_b200_last_error_string()
    assert tiny(4, 1024, 4096, 33, 2) == -7
    assert tiny(4, 1024, 4096, 8, 2, out=None) == -1
    assert tiny(4, 1024, 4096, 8, 2, x=a + 8) == -3


@pytest.mark.skipif(torch.cuda.is_available(), reason="no address here is one of a device")
@pytest.mark.parametrize("N,E,k,dtype", [(512, 8, 2, _cabi.F32), (2048, 8, 2, _cabi.F32), (1, 8, 2, _cabi.F32),
                                         (1, 8, 2, _cabi.BF16), (48, 8, 2, _cabi.BF16), (300, 8, 2, _cabi.BF16),
                                         (1500, 8, 2, _cabi.BF16), (20, 64, 2, _cabi.BF16)])
@pytest.mark.parametrize("norm", [False, True])
def test_rows_and_router_weights_off_a_16_byte_boundary_are_refused_before_any_launch(N, E, k, dtype, norm):
    """The small calls' kernels read both 16 bytes at a time: an error of the host's checks, not of CUDA, comes back."""
    a = 1 << 20
    ws = _cabi.workspace_bytes(N, 64, 128, E, k, dtype)
    call = lambda x, wg: lib.moe_b200_forward(x, wg, a, a, None, a if norm else None, a if norm else None, 1e-5, N, 64, 128,
                                              E, k, dtype, 0, a, ws, a, None)
    for off in (4, 8):
        assert call(a + off, a) == -3 and b"16-byte" in lib.moe_b200_last_error_string()
    # (with a LayerNorm folded in, the large calls' kernels read the weights an element at a time: not refused there)
    if E <= 32 and not (norm and dtype == _cabi.F32):
        assert call(a, a + 4) == -3 and b"16-byte" in lib.moe_b200_last_error_string()


def test_which_calls_compute_both_products_in_one_launch():
    """Its lines, and the calls with few tiles of a long down product, which stay with the kernels that split its K."""
    one = lib.moe_b200_one_launch
    # the workloads' shapes, from 96 rows an expert to 2048
    for d, f, E in ((1024, 4096, 8), (512, 2048, 8), (2048, 1408, 8), (1024, 512, 4), (4096, 1024, 32)):
        assert [one(r, d, f, E) for r in (96 * E - 1, 96 * E, 512 * E, 2048 * E, 2048 * E + 1)] == [0, 1, 1, 1, 0]
    assert [one(r, 1024, 4096, 2) for r in (1535, 1536, 4096, 4097)] == [0, 1, 1, 0]
    # down products of 128 steps of K in 3 to 16 tiles: 68 us against 45 to 52 of the streaming kernel, and K in ranges there
    assert [one(M, 256, 8192, E) for M, E in ((288, 3), (768, 3), (768, 8), (1536, 8), (1800, 1), (2048, 2), (896, 8))] == [0] * 7
    assert one(768, 512, 8192, 4) == 0 and one(1280, 1024, 8192, 8) == 1
    # one or two experts with such a product: by d
    assert [one(M, d, 8 * d, E) for d in (512, 1024) for M, E in ((1536, 2), (3000, 1), (4096, 2))] == [0] * 3 + [1] * 3
    assert one(3000, 512, 8192, 2) == 0
    # beyond 4096 rows: the epilogue's share where K of gate_and_up is short
    assert one(16384, 256, 8192, 8) == 0 and one(7680, 256, 2048, 24) == 1 and one(16384, 512, 2048, 8) == 1
    # more than 32 experts: up to 256 rows whatever the shape, and where row blocks outnumber the streaming kernel's counters
    assert [one(r, 256, 8192, 64) for r in (0, 1, 256, 257, 4096)] == [0, 1, 1, 0, 0]
    assert one(4096, 256, 8192, 200) == 1 and one(256, 1024, 4096, 32) == 0
    assert one(1024, 1020, 4096, 8) == 0 and one(1 << 31, 1024, 4096, 256) == 0      # no such call


def test_a_claimed_tile_belongs_to_the_lane_whose_role_uses_it():
    """elect.sync does not say which lane it picks: a tile that another lane claims before the roles part would be lost, and a
    kernel whose blocks wait for its rows with it. Read from the source: on hardware that picks lane 0 nothing shows it."""
    csrc = HEADER.parent.parent / "gemmallm_b200" / "csrc"
    claims = {}
    for src in sorted(csrc.glob("experts_*.cu")):
        text = src.read_text()
        if "if (elect_one())" in text:
            claims.update({(src.name, i): line for i, line in enumerate(text.splitlines())
                           if re.search(r"if \(.*\) *\w+ = atomicAdd\(", line)})
    assert len(claims) == 2 and all("elect_one()" in line for line in claims.values()), claims


def test_host_extension_is_rebuilt_for_another_torch(tmp_path, monkeypatch):
    """Same sources, same dates: what counts besides them is the torch it was built against."""
    from gemmallm_b200 import build
    calls = []

    def compile_(cmd, **kw):
        calls.append(cmd)
        (tmp_path / "_host.so").touch()
        return type("R", (), {"returncode": 0, "stdout": "", "stderr": ""})()
    monkeypatch.setattr(build, "OBJ", tmp_path)
    monkeypatch.setattr(build, "HOST_LIB", tmp_path / "_host.so")
    monkeypatch.setattr(build.subprocess, "run", compile_)
    for _ in range(2):
        build.build_host()
    assert len(calls) == 1
    (tmp_path / "host_torch_version").write_text("another")
    build.build_host()
    assert len(calls) == 2
