"""Rules for the CUDA sources that no compiler checks, and host code of the library that needs no GPU."""
import ctypes
import re

import pytest

from sneppx_alg_b200 import _build
from sneppx_alg_b200.ops import _lib


def _kernels(text):
    """(name, parameters, body) of the __global__ functions of a source file."""
    for m in re.finditer(r"__global__\s+void\s+(?:__cluster_dims__\([^)]*\)\s*)?(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(([^)]*)\)\s*\{", text):
        yield m.group(1), m.group(2), text[m.end():text.find("\n}\n", m.end())]


def test_kernels_that_start_early_promise_nothing_about_their_inputs():
    """A kernel that waits for its predecessor inside (griddepcontrol.wait) runs while that one still writes: a __restrict__ pointer would tell the
    compiler that nobody does, and let it load ahead of the wait. And whatever is launched that way waits."""
    waiting, launched = {}, set()
    for src in _build.cuda_sources():
        text = re.sub(r"//[^\n]*", "", src.read_text())
        for name, params, body in _kernels(text):
            if re.search(r"after_predecessor\(|griddepcontrol\.wait|griddep_wait\(\)", body):
                waiting[name] = params
        launched |= set(re.findall(r"launch_dependent\((\w+_kernel)", text))
        for m in re.finditer(r"auto run = \[&\]\(auto kern[^{]*\{\s*launch_dependent\(kern", text):
            launched |= set(re.findall(r"run\((\w+_kernel)", text[m.end():m.end() + 2000].split('\nextern "C"')[0]))
    assert {"rmsnorm_fwd_kernel", "rmsnorm_fwd_long_kernel", "glu_fwd_kernel", "paged_merge_kernel", "kv_append_vec8_kernel", "paged_decode_tc_kernel"} <= launched
    assert {"gemm_skinny_kernel", "gemm_dq_kernel", "mamba_step_kernel"} <= set(waiting) and launched <= set(waiting)
    assert not [n for n, params in waiting.items() if "__restrict__" in params]


def test_entry_points_are_declared_in_one_place():
    """C linkage: a declaration beside a caller would link to whatever has the name. What one source calls of another is in the header that both include."""
    for src in _build.cuda_sources():
        text = src.read_text()
        assert not re.findall(r'^extern "C"[^{;]*;', text, re.M), src.name
        for block in re.findall(r'^extern "C" \{(.*?)^\}', text, re.M | re.S):
            assert not re.findall(r"^\w[^{};()]*\([^{}()]*\);", block, re.M), src.name


def test_ssd_output_stage_waits_for_the_tile_that_its_epilogue_reads():
    """The epilogue warps read x from shared memory that TMA filled: they wait for that transfer's barrier themselves, not only for the product's."""
    text = (_build.CSRC / "ssd_fwd.cu").read_text()
    body = next(body for name, _, body in _kernels(text) if name == "ssd_chunk_fwd_kernel")
    epilogue = body[body.index("epilogue of this head"):]
    assert epilogue.index("mbar_wait_warp(&xh_full[grp], n & 1") < epilogue.index("const uint8_t* xrow = sX")


@pytest.mark.parametrize("B,L,H,P,G,N,Q", [(1, 8192, 80, 64, 8, 128, 128), (4, 8192, 80, 64, 8, 128, 128), (4, 500, 24, 64, 1, 128, 128), (1, 4096, 16, 128, 1, 64, 128),
                                           (2, 60, 8, 64, 2, 64, 64)])
def test_mixer_scratch_is_used_again(B, L, H, P, G, N, Q):
    """The backward of the mixer as one call takes no more scratch than its stages one by one hold while they work on the Q x Q matrices, where
    they hold the most: dy, dye, dxw and dy by heads; dM, M and dG; the chunk states' gradients in 32 and 16 bits; dB, dC, C B^T, B and C by
    group; eight vectors. Every buffer is rounded up to 256 bytes."""
    nc = (L + Q - 1) // Q
    n, vec = B * nc * G, B * nc * Q * H
    held = 4 * vec * P * 2 + 3 * vec * Q * 2 + vec // Q * P * N * 6 + n * Q * (2 * N * 4 + Q * 4 + 2 * N * 2) + 8 * vec * 4
    size = _lib.lib().sx_mixer_workspace
    size.restype = ctypes.c_longlong
    a = _lib.SxMixerArgs()
    a.B, a.L, a.H, a.P, a.G, a.N, a.Q, a.K, a.fused = B, L, H, P, G, N, Q, 4, int((Q, N, P) == (128, 128, 64))
    back, forward = size(ctypes.byref(a), 1), size(ctypes.byref(a), 0)
    assert 0 < forward < back <= held + 40 * 256, (back, held)


@pytest.mark.parametrize("B,L,C", [(512, 1, 7168), (512, 7, 7168), (4096, 3, 256), (64, 64, 4096), (40, 130, 3584), (1, 8192, 7168), (4, 500, 1792), (1, 1, 64)])
def test_conv1d_backward_takes_a_partial_row_for_512_positions(B, L, C):
    """Runs of 64 positions are counted by what the sequences hold: 32 runs of 16 a partial row, or as many rows as make one wave of four CTAs an SM."""
    parts = _lib.lib().sx_conv1d_bwd_parts(B, L, C)
    runs, wave = B * ((L + 15) // 16), 148 * 4 // ((C // 2 + 31) // 32)
    assert 1 <= parts <= max((runs + 31) // 32, wave, 1)
