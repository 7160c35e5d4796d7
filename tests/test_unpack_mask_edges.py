"""Unpacking and masking at the edges of their tiles, against the oracle:
channel counts around 4 and 128 and odd bit offsets (rows that start inside a
byte), lengths around 128, blocks of one sample to the whole observation,
and more blocks than one warp ranks (2048)."""
import numpy as np
import pytest


def payload(nch, nbits, ns, seed):
    from pulsarsr_gb300 import synth
    rng = np.random.default_rng(seed)
    top = {1: 2, 2: 4, 4: 16, 8: 256, 16: 65536}.get(nbits)
    x = rng.integers(0, top, (ns, nch)) if top else rng.normal(5.0, 2.0, (ns, nch))
    if nbits < 8:  # one little-endian bit stream, padded to whole bytes
        bits = ((x.reshape(-1, 1) >> np.arange(nbits)) & 1).astype(np.uint8).reshape(-1)
        data = np.packbits(bits, bitorder="little").tobytes()
    else:
        data = synth.pack(x, nbits)
    return synth.header_bytes(nch, nbits, 64e-6, 1500.0, -0.5) + data, x


@pytest.mark.gpu
@pytest.mark.parametrize("nbits", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("nch", [1, 3, 4, 5, 31, 127, 128, 129, 260])
def test_unpack_edges(gpu, nbits, nch):
    from pulsarsr_gb300 import fbank
    for ns in (8, 120, 128, 136, 1000):  # multiples of 8: every row set fills whole bytes
        raw, x = payload(nch, nbits, ns, nch * 1000 + ns)
        fb = fbank.decode(raw)
        assert np.array_equal(fb.data, x.T.astype(np.float32)), ns


@pytest.mark.gpu
@pytest.mark.parametrize("nbits,nch,ns,block", [(8, 5, 9000, 1), (8, 5, 9000, 2), (4, 8, 5000, 2), (8, 33, 5003, 7),
                                                (8, 4, 3000, 3000), (8, 4, 3000, 9999),
                                                (16, 6, 4100, 2), (16, 9, 4097, 300),
                                                (32, 6, 6000, 2), (8, 2100, 700, 64)])
def test_mask_edges(gpu, oracle, nbits, nch, ns, block):
    from pulsarsr_gb300 import fbank, rfi
    raw, x = payload(nch, nbits, ns // 8 * 8, 5)
    x[3 * block:4 * block] = 0  # a block and a channel that stand out
    x[:, nch // 2] = 0
    from pulsarsr_gb300 import synth
    raw = synth.header_bytes(nch, nbits, 64e-6, 1500.0, -0.5) + synth.pack(x, nbits)
    fb = fbank.decode(raw)
    m = rfi.mask(fb, block, 6.0)
    _, d = oracle.decode(raw)
    od, om = oracle.rfi_mask(d, block, 6.0)
    assert m.channels == [int(c) for c in om["channels"]]
    assert m.blocks == [int(b) for b in om["blocks"]]
    assert m.masked_fraction == om["masked_fraction"]
    assert fb.data.tobytes() == np.ascontiguousarray(od).tobytes()
