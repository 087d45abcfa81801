"""What the native host path refuses, accepts and remembers, against what the operators promise."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).half()


def _encoder(hid, heads, ffn, S, block=32, without=()):
    """One layer with random weights (None for the names in `without`) on an all-ones mask."""
    import stof_b200
    shapes = {"Wqkv": (hid, 3 * hid), "bqkv": (3 * hid,), "Wo": (hid, hid), "bo": (hid,), "g1": (hid,), "b1": (hid,), "W1": (hid, ffn), "bi1": (ffn,),
              "W2": (ffn, hid), "bi2": (hid,), "g2": (hid,), "b2": (hid,)}
    w = {k: None if k in without else _rand(s, 90 + i, 0.1).cuda() for i, (k, s) in enumerate(shapes.items())}
    enc = stof_b200.BertEncoder([stof_b200.EncoderWeights(**w)], heads, 1e-12, block_m=block, block_n=block)
    enc.set_mask(torch.ones(1, S, S, dtype=torch.float16, device="cuda"))
    return enc


@pytest.mark.parametrize("hid,heads", [(776, 12), (1032, 16), (128, 0), (128, -2)])
def test_stack_refuses_a_hidden_size_that_its_heads_do_not_divide(hid, heads):
    """776 / 12 and 1032 / 16 leave a head size of 64, which every later check takes, and columns that no head computes."""
    import stof_b200
    with pytest.raises(stof_b200.StofError, match="heads"):
        _encoder(hid, heads, 64, 64)(_rand((1, 64, hid), 1).cuda())


def _index(S, block, band):
    import stof_b200
    from oracle import masks as om
    return stof_b200.get_sparse_storage(torch.from_numpy(om.generate_sliding_mask(1, S, band, False, np.float16)).cuda(), block, block)[1:]


def test_index_checks_hold_for_an_index_whose_plan_is_known():
    """A strided view and a view of another type with the address, version and length of an index that has been used: refused, not
    answered with the plan of the other."""
    import stof_b200
    S, block = 256, 32
    frp, fci, prp, pci, pbm, lrp, lci = _index(S, block, 40)
    q, k, v = (_rand((1, 2, S, 64), i).cuda() for i in range(3))
    base = torch.zeros(2 * prp.numel(), dtype=torch.int32, device="cuda")
    base[:prp.numel()] = prp
    plain, strided = base[:prp.numel()], base[::2]
    assert (plain.data_ptr(), plain._version, plain.numel()) == (strided.data_ptr(), strided._version, strided.numel())
    for _ in range(3):                                   # decided, and remembered by the native side, at the second use
        stof_b200.block_attention(q, k, v, torch.empty_like(q), frp, fci, plain, pci, pbm, lrp, lci, block, block)
    for other in (strided, plain.view(torch.float32)):
        with pytest.raises(stof_b200.StofError, match="contiguous int32"):
            stof_b200.block_attention(q, k, v, torch.empty_like(q), frp, fci, other, pci, pbm, lrp, lci, block, block)


SLOW_LIBRARY = """
#include <stddef.h>
#include <unistd.h>
const char* stof_last_error(void) { return ""; }
size_t stof_mask_workspace_bytes(int s, int bm, int bn) { return 4096; }
int stof_mask_classify_notify() { usleep(200000); return -2; }
int stof_mask_fill() { usleep(200000); return 0; }
int stof_block_attn() { usleep(200000); return 0; }
int stof_block_attn_scheduled() { usleep(200000); return 0; }
int stof_gemm_bias_act() { usleep(200000); return 0; }
int stof_gemm_bias_residual_layernorm() { usleep(200000); return 0; }
int stof_bias_residual_layernorm() { usleep(200000); return 0; }
"""


def test_python_threads_run_while_the_library_is_in_a_call(tmp_path, monkeypatch):
    """The native path bound to a library whose calls take 0.2 s, as a launch does that finds the queue full: another Python thread gets on."""
    import subprocess
    import threading
    import time
    import stof_b200
    from stof_b200 import _lib
    source, library = tmp_path / "slow.c", tmp_path / "slow.so"
    source.write_text(SLOW_LIBRARY)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-w", "-o", str(library), str(source)])
    x, w = _rand((8, 64), 1).cuda(), _rand((64, 64), 2).cuda()
    idx, (q, k, v) = _index(256, 32, 40), (_rand((1, 2, 256, 64), i).cuda() for i in range(3))
    mask = torch.ones(1, 64, 64, device="cuda")
    out = torch.empty_like(q)
    enc, hidden = _encoder(128, 2, 256, 64), _rand((1, 64, 128), 3).cuda()
    enc(hidden)                                          # with the use below the plan is decided
    calls = {"gemm": lambda: stof_b200.gemm_bias(x, w), "gemm_ln": lambda: stof_b200.gemm_bias_residual_layernorm(x, w, None, None, None, None, 1e-5),
             "layernorm": lambda: stof_b200.bias_residual_layernorm(x), "attention": lambda: stof_b200.block_attention(q, k, v, out, *idx, 32, 32),
             "compaction": lambda: stof_b200.get_sparse_storage(mask, 64, 64), "stack": lambda: enc(hidden)}
    for f in calls.values():
        f()
    ticks, stop = [0], threading.Event()

    def tick():
        while not stop.is_set():
            ticks[0] += 1
            time.sleep(0.001)

    other = threading.Thread(target=tick)
    try:
        with monkeypatch.context() as patch:
            patch.setattr(_lib, "_LIB_PATH", str(library))
            patch.setattr(_lib, "_native", None)
            _lib.native()
            other.start()
            for name, f in calls.items():
                before = ticks[0]
                try:
                    f()
                except stof_b200.StofError:
                    assert name == "compaction"              # its stand-in reports a failure, as nothing writes the counts
                assert ticks[0] - before >= 20, name
    finally:
        stop.set()
        other.join()
        _lib._native = None
        _lib.native()
    assert (stof_b200.gemm_bias(x, w).float() - (x.float() @ w.float())).abs().max() < 0.1


@pytest.mark.parametrize("fuse", [True, False])
def test_stack_without_biases_and_affine(fuse):
    """Layers whose bias, gamma and beta are None (T5 has no biases) give what zeros and ones give."""
    from stof_b200 import EncoderWeights
    hid, x = 128, _rand((2, 64, 128), 5).cuda()
    names = ("bqkv", "bo", "bi1", "bi2", "g1", "b1", "g2", "b2")
    enc, same = _encoder(hid, 2, 256, 64, without=names), _encoder(hid, 2, 256, 64)
    enc.fuse_layernorm = same.fuse_layernorm = fuse
    w = {k: getattr(enc.layers[0], k) for k in EncoderWeights.__dataclass_fields__}
    for name in names:
        w[name] = torch.full_like(getattr(same.layers[0], name), 1.0 if name[0] == "g" else 0.0)
    same.layers = [EncoderWeights(**w)]
    assert torch.equal(enc(x), same(x))
    w["Wo"] = None
    same.layers = [EncoderWeights(**w)]
    with pytest.raises(TypeError, match="Wo"):
        same(x)


def test_softmax_scale_has_to_be_positive():
    import stof_b200
    idx, (q, k, v) = _index(256, 32, 40), (_rand((1, 2, 256, 64), i).cuda() for i in range(3))
    for scale in (-0.125, -1.0, 0.0, float("nan")):
        with pytest.raises(stof_b200.StofError, match="positive"):
            stof_b200.block_attention(q, k, v, torch.empty_like(q), *idx, 32, 32, softmax_scale=scale)
    default = stof_b200.block_attention(q, k, v, torch.empty_like(q), *idx, 32, 32)
    assert torch.equal(stof_b200.block_attention(q, k, v, torch.empty_like(q), *idx, 32, 32, softmax_scale=0.125), default)


def test_block_sizes_that_are_whole_but_no_ints():
    import stof_b200
    idx, (q, k, v) = _index(256, 32, 40), (_rand((1, 2, 256, 64), i).cuda() for i in range(3))
    for _ in range(2):                                   # the second use may pair the halves anew, which changes the order of the sums
        want = stof_b200.block_attention(q, k, v, torch.empty_like(q), *idx, 32, 32)
    for size in (32.0, np.float64(32), np.int64(32), torch.tensor(32)):
        assert torch.equal(stof_b200.block_attention(q, k, v, torch.empty_like(q), *idx, size, size), want)
        assert torch.equal(stof_b200.block_attn_mask(q.clone(), k, v, *idx, size, size, 4), want)


@pytest.mark.parametrize("block_m,block_n", [(0, 32), (32, 0), (-32, 32)])
def test_stack_refuses_block_sizes_that_are_not_positive(block_m, block_n):
    """An index that the caller sets comes with block sizes that no compaction has looked at."""
    import stof_b200
    enc = _encoder(128, 2, 64, 64)
    enc.block_m, enc.block_n = block_m, block_n
    with pytest.raises(stof_b200.StofError, match="positive"):
        enc(_rand((1, 64, 128), 1).cuda())


def test_stack_refuses_more_state_buffers_than_it_rotates():
    import stof_b200
    enc = _encoder(128, 2, 64, 64)
    for count in (0, 5):
        enc._STATES = count
        enc._io.clear()
        with pytest.raises(stof_b200.StofError, match="buffers"):
            enc(_rand((1, 64, 128), 1).cuda())


def test_strided_index_is_refused_by_the_function_and_packed_by_the_operator():
    import stof_b200
    from ops.package_op import block_attn_mask_op
    idx, (q, k, v) = _index(256, 32, 40), (_rand((1, 2, 256, 64), i).cuda() for i in range(3))
    want = stof_b200.block_attn_mask(q.clone(), k, v, *idx, 32, 32, 4)
    strided = tuple(torch.stack((t, t), -1)[..., 0] for t in idx)
    assert not any(t.is_contiguous() for t in strided)
    with pytest.raises(stof_b200.StofError, match="contiguous int32"):
        stof_b200.block_attn_mask(q.clone(), k, v, *strided, 32, 32, 4)
    tiles = idx[:4] + strided[4:5] + idx[5:]
    assert (stof_b200.block_attn_mask(q.clone(), k, v, *tiles, 32, 32, 4).float() - want.float()).abs().max() <= 2e-3      # the plan is decided at its second use
    assert (block_attn_mask_op(q.clone(), k, v, *strided, 32, 32, 4).float() - want.float()).abs().max() <= 2e-3


def test_plan_list_gives_up_the_index_used_longest_ago(monkeypatch):
    """32 plans are remembered: a 33rd index takes the place of the one that was used longest ago, in whatever order the others were."""
    import stof_b200
    from stof_b200 import _lib, attention
    asked = []
    counting = lambda *a: asked.append(a[0].data_ptr()) or attention.plan_for_call(*a)
    q, k, v = (_rand((1, 1, 128, 64), i).cuda() for i in range(3))
    idx = [_index(128, 64, 200) for _ in range(33)]
    use = lambda i: stof_b200.block_attention(q, k, v, torch.empty_like(q), *idx[i], 64, 64)
    device = lambda n: torch.device("cuda", n)
    native = _lib.native()
    try:
        native.bind(_lib._LIB_PATH, _lib.StofError, lambda n: _lib.status_word(device(n)), lambda n, what: _lib.check_status(device(n), what), counting)
        for i in range(32):
            use(i), use(i)                               # decided at the second use
        asked.clear()
        use(0)                                           # the oldest comes to the front
        use(32), use(32)                                 # and 1 goes
        asked.clear()
        for i in (31, 0, 2):
            use(i)
        assert not asked
        use(1)
        assert asked == [idx[1][0].data_ptr()]
    finally:
        _lib._native = None
        _lib.native()


def test_stacks_of_two_threads_beside_a_thread_that_computes():
    """Two encoders on streams of their own and a Python thread that never waits: the walks, which run without the interpreter's lock,
    give what they give alone."""
    import threading
    encs, xs = [_encoder(128, 2, 256, 64) for _ in range(2)], [_rand((2, 64, 128), 30 + i).cuda() for i in range(2)]
    want = []
    for e, x in zip(encs, xs):
        e(x), e(x)
        want.append(e(x).clone())
    torch.cuda.synchronize()
    stop, wrong = threading.Event(), []

    def compute():
        n = 0
        while not stop.is_set():
            n += 1

    def walk(e, x, w):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(50):
                    if not torch.equal(e(x), w):
                        wrong.append("another result")
        except Exception as error:
            wrong.append(repr(error))

    threads = [threading.Thread(target=walk, args=a) for a in zip(encs, xs, want)]
    busy = threading.Thread(target=compute)
    busy.start()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    stop.set()
    busy.join()
    assert not wrong, wrong[:3]
