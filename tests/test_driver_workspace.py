"""The workspace that the C++ driver of a forward pass asks for, over the sizes of models: a walk on the host over the path of
a step that launches nothing, so no GPU is needed (the library is compiled if it is not there)."""

import ctypes as C

import pytest


@pytest.fixture(scope="module")
def lib():
    from quantinfer_b200.csrc.build import library_path

    lib = C.CDLL(str(library_path()))
    lib.qi_last_error.restype = C.c_char_p
    lib.qi_forward_workspace_bytes.restype = C.c_longlong
    return lib


def _bytes(lib, hidden, ff, n, dtype, heads=16, kv=4, layers=2, vocab=1000):
    """qi_forward_workspace_bytes of a step of `n` tokens: one prompt, or n requests' single tokens when n < 0. Addresses are never
    followed."""
    from quantinfer_b200.engine.native import _Block, _Call, _Linear, _ModelDesc, _Step

    somewhere, d = 4096, 128
    lin = lambda out, inp: _Linear(somewhere, dtype, out, inp)  # noqa: E731
    block = _Block(somewhere, somewhere, 1e-6, 1e-6, lin((heads + 2 * kv) * d, hidden), lin(hidden, heads * d), lin(2 * ff, hidden), lin(hidden, ff),
                   somewhere, somewhere, somewhere, somewhere, 1e-6, d ** -0.5, heads, kv, d, 0, d, 4096, 0, 0)
    blocks, calls = (_Block * layers)(*[block] * layers), (_Call * layers)(*[_Call(i, 0, 1, 64, 100, somewhere, somewhere) for i in range(layers)])
    desc = _ModelDesc(blocks, calls, layers, layers, dtype, hidden, vocab, somewhere, dtype, 1e-6, somewhere, lin(vocab, hidden), somewhere)
    decode, n = n < 0, abs(n)
    step = _Step(n, n if decode else 1, n if decode else 1, int(decode), 2048, 0 if decode else -(-n // 128), 0, 0, *[somewhere] * 9)
    step.block_tables[0], step.max_blocks[0] = somewhere, 64
    return int(lib.qi_forward_workspace_bytes(C.byref(desc), C.byref(step)))


FLOAT32, BFLOAT16 = 0, 1
# widths and feed-forwards of models in use, some with a down projection cut along K into many parts
SIZES = [(2048, 8192), (1536, 8960), (1024, 5120), (896, 4864), (3072, 24576), (2048, 16384), (4096, 12288), (2560, 9728), (64, 128), (5120, 17408)]


@pytest.mark.parametrize("dtype", [FLOAT32, BFLOAT16])
@pytest.mark.parametrize("hidden, ff", SIZES)
@pytest.mark.parametrize("n", [1, -1, -8, 201, 2048])
def test_every_size_has_a_workspace(lib, hidden, ff, n, dtype):
    got = _bytes(lib, hidden, ff, n, dtype)
    assert got > 0, (got, lib.qi_last_error())


def test_long_float32_prompts_do_not_keep_partial_sums_of_every_row(lib):
    """8,001 tokens through two layers of 4,096 x 12,288 in float32: the layer's own tensors (residual stream, q/k/v, gate and up and their
    product, two outputs: about 2.4 GB) and a workspace that no longer grows with the tokens."""
    assert _bytes(lib, 4096, 12288, 8001, FLOAT32, heads=32, kv=8) < 3.2e9
