"""Channel and block outliers and fills at the counts where their selections
change form (256, 512 and 1024 channels to a warp; 256, 1024 and 2048 blocks to
four warps; a block of threads above), with equal, few and spread values,
against the oracle."""
import numpy as np
import pytest


def check(oracle, x, nbits, block, threshold):
    from pulsarsr_gb300 import fbank, rfi, synth
    raw = synth.header_bytes(x.shape[1], nbits, 64e-6, 1500.0, -0.1) + \
        synth.pack(x.astype(np.float32), nbits)
    fb = fbank.decode(raw)
    m = rfi.mask(fb, block, threshold)
    _, d = oracle.decode(raw)
    od, om = oracle.rfi_mask(d, block, threshold)
    assert m.channels == [int(c) for c in om["channels"]]
    assert m.blocks == [int(b) for b in om["blocks"]]
    assert fb.data.tobytes() == np.ascontiguousarray(od).tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("nch", [1, 2, 31, 256, 257, 512, 513, 1024, 1025])
@pytest.mark.parametrize("kind", ["spread", "few", "equal"])
def test_channel_counts(gpu, oracle, nch, kind):
    rng = np.random.default_rng(nch)
    x = {"spread": rng.integers(0, 256, (70, nch)), "few": rng.integers(0, 2, (70, nch)),
         "equal": np.full((70, nch), 7)}[kind]
    x[:, nch // 3] = 255
    check(oracle, x, 8, 9, 3.0)


@pytest.mark.gpu
@pytest.mark.parametrize("nblocks", [1, 2, 256, 257, 1023, 1024, 1025, 2048, 2049])
@pytest.mark.parametrize("nbits", [8, 32])
def test_block_counts(gpu, oracle, nblocks, nbits):
    rng = np.random.default_rng(nblocks)
    block = 33  # rows of blocks that start at every byte of a 16-byte word
    x = rng.normal(100, 9, (nblocks * block - 5, 3)).round(0 if nbits == 8 else 3)
    x[block * (nblocks // 2):block * (nblocks // 2) + block] += 60
    check(oracle, x, nbits, block, 4.0)
