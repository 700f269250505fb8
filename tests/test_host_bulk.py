"""Files whose arrays are long enough to be read and decoded by several threads (bulk.c): every precision, counts that are no
multiple of anything, any number of threads, and files that end early."""
import numpy as np
import pytest

TOPOLOGY = [1033, 1117, 3]
COUNTS = [1033 * 1117, 1117 * 3]


def build(spg):
    net = spg.Network.build(TOPOLOGY, [spg.abi.ACT_RELU, spg.abi.ACT_SOFTMAX], spg.abi.WEIGHT_INITIALIZATION_NONE)
    rng = np.random.default_rng(4)
    net.weights[:] = rng.standard_normal(sum(COUNTS), dtype=np.float32)
    net.biases[:] = rng.standard_normal(sum(TOPOLOGY[1:]), dtype=np.float32)
    return net


def decode(raw, count, name):
    """The array at the front of `raw` and the bytes it takes, by the format's definition, in float32 step by step."""
    if name == "fp32":
        return np.frombuffer(raw, np.float32, count), 4 * count
    if name == "fp16":
        return np.frombuffer(raw, np.float16, count).astype(np.float32), 2 * count
    if name == "bf16":
        return (np.frombuffer(raw, np.uint16, count).astype(np.uint32) << 16).view(np.float32), 2 * count
    amax = np.frombuffer(raw, np.float32, 1)[0]
    bits, top = {"int8": (8, 127), "int4": (4, 7), "int2": (2, 1)}[name]
    packed = np.frombuffer(raw, np.uint8, (count * bits + 7) // 8, 4)
    q = ((packed[:, None] >> (np.arange(8 // bits, dtype=np.uint8) * bits)) & ((1 << bits) - 1)).reshape(-1)[:count].astype(np.int32)
    q = np.where(q >= 1 << (bits - 1), q - (1 << bits), q)
    return (q.astype(np.float32) / np.float32(top)) * amax, 4 + len(packed)


@pytest.mark.parametrize("name", ["fp32", "fp16", "bf16", "int8", "int4", "int2"])
@pytest.mark.parametrize("threads", ["1", "3", "16", ""])
def test_arrays_read_by_several_threads(spg, tmp_path, monkeypatch, name, threads):
    monkeypatch.setenv("SPINGALETT_STAGE_THREADS", threads)
    path = str(tmp_path / "net.nn")
    build(spg).save(path, spg.abi.PRECISION_NAMES[name])
    raw = open(path, "rb").read()
    net = spg.Network.load(path)
    # arrays lie at the end of the file in the order W b W b
    arrays = [COUNTS[0], TOPOLOGY[1], COUNTS[1], TOPOLOGY[2]]
    bits = {"fp32": 32, "fp16": 16, "bf16": 16, "int8": 8, "int4": 4, "int2": 2}[name]
    size = [(4 if bits < 16 else 0) + (c * bits + 7) // 8 for c in arrays]
    at, got = len(raw) - sum(size), []
    for c, s in zip(arrays, size):
        values, used = decode(raw[at:at + s], c, name)
        assert used == s
        got.append(values)
        at += s
    assert np.array_equal(net.weights, np.concatenate([got[0], got[2]]))
    assert np.array_equal(net.biases, np.concatenate([got[1], got[3]]))


@pytest.mark.parametrize("name", ["fp32", "int4"])
def test_a_file_that_ends_early(spg, tmp_path, name):
    """What the file holds is there, the rest is zero, and the error is reported."""
    path = str(tmp_path / "net.nn")
    build(spg).save(path, spg.abi.PRECISION_NAMES[name])
    before = spg.Network.load(path)
    raw = open(path, "rb").read()
    open(path, "wb").write(raw[:-8])
    net = spg.lib().load_spingalett(path.encode())
    assert net and spg.lib().spingalett_last_error_code() != 0
    spg.lib().spingalett_clear_error()
    after = spg.Network(net)
    assert np.array_equal(after.weights[:COUNTS[0]], before.weights[:COUNTS[0]])
    assert not after.biases[-TOPOLOGY[2]:].any()
