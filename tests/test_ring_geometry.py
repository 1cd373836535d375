"""Operand rings of successive projections on one worker, on the CPU: the copy and MMA cursors run on from one GEMM
instruction to the next while the ring's key stays the same, so equal keys have to mean equal rings."""
import ctypes as C

import pytest

from native_pi0 import _native
from native_pi0.program import LinearWork, spread_streams

NVFP4, BF16, FP8 = 0, 1, 2
DATA_BYTES = 216 * 1024


@pytest.fixture(scope="module")
def ring():
    _native.build()
    lib = _native.load()

    def geometry(operands, rows, block_n):
        stride, stages, key = C.c_int(), C.c_int(), C.c_uint()
        assert lib.gemm_ring_geometry(operands, rows, block_n, C.byref(stride), C.byref(stages), C.byref(key)) == 0
        return stride.value, stages.value, key.value

    return geometry


def test_equal_keys_are_equal_rings(ring):
    rings = {}
    for operands in (NVFP4, BF16, FP8):
        for rows in list(range(1, 130)) + [256, 768]:
            for block_n in (128, 64, 32):
                stride, stages, key = ring(operands, rows, block_n)
                assert 3 <= stages <= (5 if operands == NVFP4 else 8) and stages * stride <= DATA_BYTES
                assert rings.setdefault(key, (stride, stages)) == (stride, stages), (operands, rows, block_n)
    # one slot size does come in two depths: the size alone is no key
    assert len({stride for stride, _ in rings.values()}) < len(rings)


@pytest.mark.parametrize("dense", [{"qkv"}, {"qkv", "gate_up"}, {"down"}, {"o_proj", "down"}, {"qkv", "o_proj", "gate_up", "down"}])
@pytest.mark.parametrize("actions", [7, 15, 31, 50, 55, 56, 60, 63, 100])
def test_cursors_stay_inside_the_ring_of_a_mixed_expert(ring, actions, dense):
    """The slots that every worker's cursors visit in three steps of a four-layer action expert whose operand formats are
    mixed, replayed from the instruction streams."""
    k = {"qkv": 1024, "o_proj": 2048, "gate_up": 1024, "down": 4096}
    n = {"qkv": 2560, "o_proj": 1024, "gate_up": 8192, "down": 1024}
    width = {op: (64 if op in ("qkv", "gate_up") else 32) if op in dense else {"qkv": 64, "o_proj": 32, "gate_up": 128, "down": 32}[op] for op in k}
    chain = ["qkv", "attention", "o_proj", "gate_up", "down"] * 12
    tiles = [104 if op == "attention" else n[op] // width[op] for op in chain]
    code = spread_streams([LinearWork(t, k.get(op, 1024)) for t, op in zip(tiles, chain)], 148, [[i - 1, -1, -1, -1] for i in range(len(chain))], chain)
    for worker in range(code.shape[0]):
        cursor, last = 0, None
        for opcode, stage, _, count in code[worker, :, :4].tolist():
            op = chain[stage]
            if opcode == 0 or op == "attention":
                continue
            _, stages, key = ring(BF16 if op in dense else NVFP4, actions + 1, width[op])
            if key != last:
                cursor, last = 0, key
            slots = -(-k[op] * (4 if op in dense else 1) // 512)            # 256 bytes of every operand row per slot
            for _ in range(count * slots):
                assert cursor < stages, (worker, stage, op)
                cursor = 0 if cursor + 1 == stages else cursor + 1


def test_wide_tiles_have_rings_that_fit(ring):
    """192-wide NVFP4 tiles: slots that fit, and a key that no other ring shares."""
    for rows in (1, 64, 65, 128, 768):
        stride, stages, key = ring(NVFP4, rows, 192)
        assert 2 <= stages <= 5 and stages * stride <= DATA_BYTES and stride % 1024 == 0
        for operands in (NVFP4, BF16, FP8):
            for other in (1, 64, 65, 128, 768):
                for width in (128, 64, 32):
                    assert ring(operands, other, width)[2] != key or ring(operands, other, width)[:2] == (stride, stages)


@pytest.mark.parametrize("rows,blocks", [(384, 4), (768, 72), (4608, 8)])
def test_scales_of_wide_tiles(rows, blocks):
    """Row r of 192-wide tile t, block b, lies where two standard atoms of 128 rows hold it; the rest is zero."""
    import numpy as np
    import torch
    from native_pi0.primitives import wide_tile_scales
    from native_pi0.quantization import scale_offsets
    standard = torch.from_numpy(np.random.default_rng(rows).integers(1, 255, size=rows * blocks, dtype=np.uint8))
    wide = wide_tile_scales(standard, rows, blocks).numpy()
    matrix = standard.numpy()[scale_offsets(rows, blocks)].reshape(rows, blocks)
    assert wide.size == rows // 192 * (blocks // 4) * 1024
    r, b = np.meshgrid(np.arange(rows), np.arange(blocks), indexing="ij")
    inside = r % 192
    where = ((r // 192 * (blocks // 4) + b // 4) * 2 + inside // 128) * 512 + inside % 32 * 16 + inside % 128 // 32 * 4 + b % 4
    np.testing.assert_array_equal(wide[where], matrix)
    wide[where] = 0
    assert not wide.any()
