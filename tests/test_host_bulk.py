"""Files whose arrays are long enough to be read and decoded by several threads (bulk.c): every precision, counts that are no
multiple of anything, any number of threads, and files that end early; host batches that are staged in pieces."""
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

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


def on_fake_kernels(tmp_path, program):
    """The library's host sources and tests/c/<program>.c, with a stub for every kernel call that the program does not fake."""
    host = os.path.join(ROOT, "spingalett_b200", "csrc", "host")
    sources = [os.path.join(host, f) for f in sorted(os.listdir(host)) if f.endswith(".c")] + [os.path.join(ROOT, "tests", "c", program + ".c")]
    objs = []
    for src in sources:
        objs.append(str(tmp_path / (os.path.basename(src) + ".o")))
        subprocess.run(["gcc", "-std=c2x", "-O1", "-D_GNU_SOURCE", "-I", os.path.join(ROOT, "include"), "-I", host, "-c", src, "-o", objs[-1]], check=True)
    names = subprocess.run(["nm"] + objs, capture_output=True, text=True, check=True).stdout
    missing = set(re.findall(r" U (spgk?_\w+)", names)) - set(re.findall(r" [TtDBbCR] (spgk?_\w+)", names))
    stubs = tmp_path / "stubs.c"
    stubs.write_text("".join(f"long {name}(void) {{ return 0; }}\n" for name in sorted(missing)))
    exe = str(tmp_path / program)
    subprocess.run(["gcc", "-std=c2x", "-O1", *objs, str(stubs), "-o", exe, "-lpthread", "-ldl", "-lm"], check=True)
    return exe


def test_short_last_chunks_are_staged_whole(tmp_path):
    r = subprocess.run([on_fake_kernels(tmp_path, "staged_pieces")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "all staged\n", (r.returncode, r.stdout, r.stderr)


def test_rows_to_recompute_are_counted_from_zero(tmp_path):
    r = subprocess.run([on_fake_kernels(tmp_path, "row_count")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "every count from zero\n", (r.returncode, r.stdout, r.stderr)


def test_streamed_layers_write_operands_that_have_room(tmp_path):
    r = subprocess.run([on_fake_kernels(tmp_path, "layer_operands")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "every operand fits\n", (r.returncode, r.stdout, r.stderr)


def test_outputs_where_the_inputs_lie(tmp_path):
    r = subprocess.run([on_fake_kernels(tmp_path, "in_place")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "every call on its kernel\n", (r.returncode, r.stdout, r.stderr)


def test_weights_are_read_early_only_when_they_are_there(tmp_path):
    r = subprocess.run([on_fake_kernels(tmp_path, "ready_weights")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "only when they are there\n", (r.returncode, r.stdout, r.stderr)


def test_a_net_of_very_many_layers(tmp_path):
    r = subprocess.run([on_fake_kernels(tmp_path, "deep_net")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "every layer\n", (r.returncode, r.stdout, r.stderr)


def test_files_are_written_without_reserved_room(tmp_path):
    r = subprocess.run([on_fake_kernels(tmp_path, "save_plain"), str(tmp_path / "net.nn")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "written\n", (r.returncode, r.stdout, r.stderr)


def test_orders_of_a_training_call_without_page_locked_memory(tmp_path):
    r = subprocess.run([on_fake_kernels(tmp_path, "train_orders")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "every order\n", (r.returncode, r.stdout, r.stderr)


def test_pieces_in_use_are_not_handed_out(tmp_path):
    r = subprocess.run([on_fake_kernels(tmp_path, "pieces")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "every piece at rest\n", (r.returncode, r.stdout, r.stderr)


@pytest.mark.parametrize("asked", ["", "5"])
def test_callers_at_the_same_time_share_the_cores(tmp_path, asked):
    host, exe = os.path.join(ROOT, "spingalett_b200", "csrc", "host"), str(tmp_path / "bulk_callers")
    subprocess.run(["gcc", "-std=c2x", "-O1", "-D_GNU_SOURCE", "-I", os.path.join(ROOT, "include"), "-I", host, os.path.join(host, "spg_bulk.c"),
                    os.path.join(ROOT, "tests", "c", "bulk_callers.c"), "-o", exe, "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60, env={**os.environ, "SPINGALETT_STAGE_THREADS": asked})
    first, during, after = map(int, r.stdout.split())
    cores = os.sysconf("SC_NPROCESSORS_ONLN")
    most = int(asked) if asked else max(1, min(16, cores - cores // 4))
    assert (first, after) == (most, most)
    assert during == (most if asked else max(1, min(16, (cores - cores // 4) // 2)))
