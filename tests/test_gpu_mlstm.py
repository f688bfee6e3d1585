"""Parity of the CUDA mLSTM kernels (through the C ABI) with the CPU oracle on identical seeded inputs.

Tolerances (relative L2): bf16 outputs and states <= 1e-2, fp32 mode <= 1e-4.
The bf16 oracle is "inputs rounded to bf16, arithmetic in fp32".
"""
import math

import pytest
import torch

from conftest import load_golden, rel_l2
from oracle import mlstm as O

pytestmark = pytest.mark.gpu
TOL_BF16, TOL_F32 = 1e-2, 1e-4


def _inputs(seed, B, NH, S, DQ, DV, dtype, f_mean=3.0):
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(B, NH, S, DQ, generator=g) / math.sqrt(DQ) * math.sqrt(DQ) ** 0  # N(0,1); scale applied below
    k = torch.randn(B, NH, S, DQ, generator=g)
    v = torch.randn(B, NH, S, DV, generator=g)
    i = torch.randn(B, NH, S, generator=g)
    f = torch.randn(B, NH, S, generator=g) + f_mean
    q, k, v = (t.to(dtype) for t in (q, k, v))
    return q, k, v, i, f


def _state(seed, N, NH, DQ, DV):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(N, NH, DQ, DV, generator=g), torch.randn(N, NH, DQ, generator=g), torch.randn(N, NH, 1, generator=g))


def _cuda(*ts):
    return [None if t is None else t.cuda() for t in ts]


def _check(h, st, h_ref, st_ref, tol):
    assert torch.isfinite(h.float()).all()
    assert rel_l2(h.float().cpu(), h_ref) < tol, rel_l2(h.float().cpu(), h_ref)
    for a, b, name in zip(st, st_ref, "cnm"):
        a = a.float().cpu().reshape(b.shape)
        if name == "m":
            assert torch.allclose(a, b, atol=1e-3, rtol=1e-4), (a - b).abs().max()
        else:
            assert rel_l2(a, b) < tol, (name, rel_l2(a, b))


# ------------------------------------------------------------------------------------------------ step
@pytest.mark.parametrize("dtype,tol", [(torch.float32, TOL_F32), (torch.bfloat16, TOL_BF16)])
@pytest.mark.parametrize("B,NH,DQ,DV", [(3, 2, 64, 128), (2, 8, 256, 512), (1, 1, 32, 36)])
def test_step_matches_oracle(dtype, tol, B, NH, DQ, DV):
    import xlstm_b200
    q, k, v, i, f = _inputs(1, B, NH, 1, DQ, DV, dtype, f_mean=1.0)
    c0, n0, m0 = _state(2, B, NH, DQ, DV)
    h_ref, st_ref = O.mlstm_step(q[:, :, 0], k[:, :, 0], v[:, :, 0], i, f, c0, n0, m0)
    qc, kc, vc, ic, fc, cc, nc, mc = _cuda(q[:, :, 0], k[:, :, 0], v[:, :, 0], i, f, c0.clone(), n0, m0)
    h, st = xlstm_b200.mlstm_step(qc, kc, vc, ic, fc, cc, nc, mc)
    assert st[0] is cc  # the large state is updated in place and handed back as the same object
    _check(h, st, h_ref, st_ref, tol)
    # from the zero state
    h_ref, st_ref = O.mlstm_step(q[:, :, 0], k[:, :, 0], v[:, :, 0], i, f)
    h, st = xlstm_b200.mlstm_step(qc, kc, vc, ic, fc, None, None, None)
    _check(h, st, h_ref, st_ref, tol)


def test_step_slots_and_strided_views():
    import xlstm_b200
    B, NH, DQ, DV, N = 3, 2, 64, 128, 5
    q, k, v, i, f = _inputs(3, B, NH, 1, DQ, DV, torch.bfloat16)
    c0, n0, m0 = _state(4, N, NH, DQ, DV)
    slot = torch.tensor([4, 0, 2], dtype=torch.int32)
    h_ref, st_ref = O.mlstm_step(q[:, :, 0], k[:, :, 0], v[:, :, 0], i, f, c0[slot.long()], n0[slot.long()], m0[slot.long()])
    # q,k,v as slices of one fused projection buffer (B, NH*(2DQ+DV)) -> strided (B,NH,D) views
    fused = torch.cat([q[:, :, 0].reshape(B, -1), k[:, :, 0].reshape(B, -1), v[:, :, 0].reshape(B, -1)], dim=1).cuda()
    qv = fused[:, : NH * DQ].view(B, NH, DQ)
    kv = fused[:, NH * DQ: 2 * NH * DQ].view(B, NH, DQ)
    vv = fused[:, 2 * NH * DQ:].view(B, NH, DV)
    cc, nc, mc = c0.cuda(), n0.cuda(), m0.cuda()
    h, (c, n, m) = xlstm_b200.mlstm_step(qv, kv, vv, i.cuda(), f.cuda(), cc, nc, mc, slot=slot.cuda())
    _check(h, (c[slot.long().cuda()], n[slot.long().cuda()], m[slot.long().cuda()]), h_ref, st_ref, TOL_BF16)
    untouched = torch.tensor([1, 3])
    assert torch.equal(c[untouched.cuda()].cpu(), c0[untouched]) and torch.equal(n[untouched.cuda()].cpu(), n0[untouched])


# ------------------------------------------------------------------------------------------------ recurrent
@pytest.mark.parametrize("name", ["mlstm_chunk_zero", "mlstm_chunk_init", "hf_chunk", "hf_seq"])
def test_recurrent_fp32_matches_reference_fixtures(name):
    import xlstm_b200
    g = load_golden(name)
    init = _cuda(g.get("c0"), g.get("n0"), g.get("m0"))
    h, st = xlstm_b200.mlstm_sequence(*_cuda(g["q"], g["k"], g["v"], g["i"], g["f"]), *init, kernel="recurrent")
    _check(h, st, g["h"], (g["c"], g["n"], g["m"].reshape(g["c"].shape[0], -1, 1)), TOL_F32)


def test_recurrent_fp32_config1_shape():
    """B=3, NH=4, S=256, DHQK=64, DHV=128, fp32: the cell shape of the small reference model (embedding 512, 4 heads)."""
    import xlstm_b200
    q, k, v, i, f = _inputs(5, 3, 4, 256, 64, 128, torch.float32)
    h_ref, st_ref = O.mlstm_chunkwise(q, k, v, i, f)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), kernel="auto")  # fp32 -> recurrence
    _check(h, st, h_ref, st_ref, TOL_F32)


@pytest.mark.parametrize("dtype,tol", [(torch.float32, TOL_F32), (torch.bfloat16, TOL_BF16)])
@pytest.mark.parametrize("B,NH,S,DQ,DV,with_state", [
    (1, 2, 1, 64, 128, True), (2, 1, 31, 36, 36, False), (1, 1, 32, 6, 33, True), (1, 2, 33, 100, 130, True),
    (2, 3, 69, 64, 32, False), (1, 1, 97, 260, 64, True), (1, 1, 40, 512, 40, False), (1, 1, 64, 512, 31, True)])
def test_recurrent_at_the_edges_of_its_tiles(dtype, tol, B, NH, S, DQ, DV, with_state):
    """Chunks of 32 tokens, 32 columns per thread block, features in fours, one buffer instead of two beyond 256 features."""
    import xlstm_b200
    q, k, v, i, f = _inputs(51, B, NH, S, DQ, DV, dtype)
    init = _state(52, B, NH, DQ, DV) if with_state else (None, None, None)
    h_ref, st_ref = O.mlstm_sequence(q, k, v, i, f, *init)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), *_cuda(*init), kernel="recurrent")
    _check(h, st, h_ref, st_ref, tol)


@pytest.mark.parametrize("dtype,tol", [(torch.float32, TOL_F32), (torch.bfloat16, TOL_BF16)])
@pytest.mark.parametrize("gate", [-float("inf"), -1e30, -2e6, -9e5])
@pytest.mark.parametrize("at,with_state", [((0,), True), ((31,), False), ((32,), True), ((5, 6, 21), False), ((63, 64, 95, 96), True), ((99,), False)])
def test_recurrent_forget_gates_that_reset_the_state(dtype, tol, gate, at, with_state):
    """Forget gates of -inf (f = 0 exactly) and huge negative ones, at the edges of the 32-token chunks and in a row: what is
    behind a reset depends on nothing in front of it, and the input gates there keep their precision."""
    import xlstm_b200
    q, k, v, i, f = _inputs(53, 1, 2, 100, 64, 64, dtype)
    f[:, :, list(at)] = gate
    init = _state(54, 1, 2, 64, 64) if with_state else (None, None, None)
    h_ref, st_ref = O.mlstm_sequence(q, k, v, i, f, *init)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), *_cuda(*init), kernel="recurrent")
    _check(h, st, h_ref, st_ref, tol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("at", [1, 15, 16, 31, 32, 70])
def test_recurrent_values_that_are_not_finite_stay_causal(dtype, bad, at):
    """A NaN or an infinity among the values reaches its own column from its own token on, nothing in front and no other column."""
    import xlstm_b200
    q, k, v, i, f = _inputs(55, 1, 1, 80, 64, 40, dtype)
    want, _ = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), kernel="recurrent")
    v[:, :, at, 17] = bad
    h, (c, n, m) = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), kernel="recurrent")
    keep = [x for x in range(40) if x != 17]
    tol = 2 ** -7 if dtype == torch.bfloat16 else 1e-6   # (the sums of a chunk with such a value run in another order)
    for a, b in ((h[:, :, :at], want[:, :, :at]), (h[..., keep], want[..., keep])):
        assert float((a.float() - b.float()).norm()) <= tol * float(b.float().norm())
    assert not bool(torch.isfinite(h[:, :, at, 17]).any()) and not bool(torch.isfinite(c[..., 17]).any())


# ------------------------------------------------------------------------------------------------ chunkwise (tcgen05)
@pytest.mark.parametrize("B,NH,S,DQ,DV,with_state", [
    (2, 2, 256, 64, 128, False),
    (1, 2, 150, 128, 256, True),     # 2 full chunks + 22-token tail, initial state
    (1, 1, 64, 256, 512, False),
    (2, 3, 1000, 256, 512, True),
    (1, 2, 7, 64, 128, False),       # shorter than one chunk
    (1, 2, 200, 256, 256, True),     # more feature blocks than value slices: no cluster split of the normaliser
    (1, 1, 130, 128, 512, False),    # fewer feature blocks than value slices: likewise
])
def test_chunkwise_matches_oracle(B, NH, S, DQ, DV, with_state):
    import xlstm_b200
    q, k, v, i, f = _inputs(7, B, NH, S, DQ, DV, torch.bfloat16)
    init = _state(8, B, NH, DQ, DV) if with_state else (None, None, None)
    h_ref, st_ref = O.mlstm_inference(q, k, v, i, f, *init)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), *_cuda(*init), kernel="chunkwise")
    xlstm_b200.check_device_status()
    _check(h, st, h_ref, st_ref, TOL_BF16)


@pytest.mark.parametrize("cluster,DQ,DV", [(4, 256, 512), (2, 128, 256), (2, 256, 512)])
def test_chunkwise_cluster_shared_normaliser_opt_in(cluster, DQ, DV):
    """XL_CW_CLUSTER=2|4 lets the value slices of a head share the normaliser work through a thread-block cluster
    (read once per process, hence the child process).  Same results as the default path."""
    import os, subprocess, sys
    code = (
        "import sys, torch; sys.path.insert(0, %r); sys.path.insert(0, %r)\n"
        "import xlstm_b200\n"
        "from oracle import mlstm as O\n"
        "from conftest import rel_l2\n"
        "from test_gpu_mlstm import _inputs, _state\n"
        "q, k, v, i, f = _inputs(31, 2, 2, 300, %d, %d, torch.bfloat16)\n"
        "init = _state(32, 2, 2, %d, %d)\n"
        "h_ref, st_ref = O.mlstm_inference(q, k, v, i, f, *init)\n"
        "h, st = xlstm_b200.mlstm_sequence(*[t.cuda() for t in (q, k, v, i, f)], *[t.cuda() for t in init], kernel='chunkwise')\n"
        "xlstm_b200.check_device_status()\n"
        "errs = [rel_l2(h.float().cpu(), h_ref.float())] + [rel_l2(a.cpu(), b) for a, b in zip(st, st_ref)]\n"
        "print('ERRS', errs)\n"
        "assert max(errs) < 1e-2, errs\n"
    ) % (os.path.dirname(os.path.dirname(os.path.abspath(__file__))), os.path.dirname(os.path.abspath(__file__)), DQ, DV, DQ, DV)
    env = dict(os.environ, XL_CW_CLUSTER=str(cluster))
    res = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-2000:]


@pytest.mark.parametrize("B,NH,S,DQ,DV,with_state,f_mean", [
    (1, 1, 2496, 64, 128, False, 3.0),    # 39 chunks: parts of unequal length
    (1, 2, 2000, 256, 512, True, 3.0),    # initial state, a tail chunk in the last part
    (1, 1, 4096, 128, 256, True, -2.0),   # strong decay: the states of early parts vanish
    (1, 1, 2048, 256, 128, False, 3.0),   # one value slice forms every feature block of n
    (4, 2, 3000, 64, 256, False, 3.0),    # several rows, a short tail
])
def test_chunkwise_split_into_parts_matches_oracle(B, NH, S, DQ, DV, with_state, f_mean):
    """Sizes whose documents are cut into parts: the C entry says so through the scratch it asks for."""
    import ctypes
    import xlstm_b200
    from xlstm_b200 import _lib
    p = _lib.MlstmSeqParams()
    p.B, p.NH, p.S, p.DHQK, p.DHV = B, NH, S, DQ, DV
    assert _lib.lib().xl_mlstm_chunkwise_scratch_bytes(ctypes.byref(p)) > 0
    q, k, v, i, f = _inputs(61, B, NH, S, DQ, DV, torch.bfloat16, f_mean=f_mean)
    if f_mean < 0:
        i[:, :, S // 2:] += 25.0          # the stabiliser jumps between parts
    init = _state(62, B, NH, DQ, DV) if with_state else (None, None, None)
    h_ref, st_ref = O.mlstm_inference(q, k, v, i, f, *init)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), *_cuda(*init), kernel="chunkwise")
    xlstm_b200.check_device_status()
    _check(h, st, h_ref, st_ref, TOL_BF16)


@pytest.mark.parametrize("lo,hi", [(0, 64), (0, 512), (256, 640), (900, 1000), (0, 1000)])
@pytest.mark.parametrize("with_state", [False, True])
def test_chunkwise_parts_with_masked_tokens(lo, hi, with_state):
    """Input gates of -inf (a caller's padding) over whole parts: these add nothing, and what lies in front and behind is kept.
    1000 tokens of four heads are cut into parts of a chunk or two."""
    import xlstm_b200
    q, k, v, i, f = _inputs(64, 1, 4, 1000, 64, 128, torch.bfloat16)
    i[:, :, lo:hi] = -float("inf")
    init = _state(65, 1, 4, 64, 128) if with_state else (None, None, None)
    h_ref, st_ref = O.mlstm_sequence(q, k, v, i, f, *init)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), *_cuda(*init), kernel="chunkwise")
    xlstm_b200.check_device_status()
    if hi - lo == 1000 and not with_state:
        assert all(int(torch.count_nonzero(t)) == 0 for t in (h, st[0], st[1]))
        assert rel_l2(st[2].cpu().reshape(st_ref[2].shape), st_ref[2]) < TOL_F32
    else:
        _check(h, st, h_ref, st_ref, TOL_BF16)


@pytest.mark.parametrize("S", [400, 2048])   # one block per document, and documents in parts
@pytest.mark.parametrize("DQ", [64, 128, 256])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_chunkwise_queries_that_are_not_finite_stay_in_their_document(S, DQ, bad):
    """The tile of a document's last chunk holds the next document's first tokens: a NaN or an infinity among their queries must
    not enter what the first document's tokens are computed from."""
    import xlstm_b200
    q, k, v, i, f = _cuda(*_inputs(66, 1, 8, S, DQ, 256, torch.bfloat16))
    cu = [0, 20, S]
    want, st = xlstm_b200.mlstm_sequence(q, k, v, i, f, cu_seqlens=cu, kernel="chunkwise")
    q[:, :, 30] = bad
    h, (c, n, m) = xlstm_b200.mlstm_sequence(q, k, v, i, f, cu_seqlens=cu, kernel="chunkwise")
    xlstm_b200.check_device_status()
    assert torch.equal(h[:, :, :30], want[:, :, :30]) and torch.equal(h[:, :, 31:], want[:, :, 31:])
    assert all(torch.equal(a, b) for a, b in zip((c, n, m), st))   # (no state depends on q)


@pytest.mark.parametrize("NH,S,DQ,DV", [(8, 8192, 256, 512), (16, 16384, 64, 256), (4, 4096, 128, 128), (4, 1000, 64, 128)])
@pytest.mark.parametrize("f_mean", [3.0, 0.0, -6.0, -12.0])
def test_chunkwise_part_states_against_64_bits(NH, S, DQ, DV, f_mean):
    """n and m (formed in fp32) where the final state is that of a part in the middle: it forgets at f_mean but for its last 64
    tokens, and behind it nothing is forgotten and next to nothing added.  The sums that matter span the ~50 tokens that carry
    the weight, at 2^-21.4 each (the hardware logarithm's bound): 1.8e-5.  C has weights rounded to bf16."""
    import xlstm_b200
    q, k, v, i, f = _cuda(*_inputs(67, 1, NH, S, DQ, DV, torch.bfloat16, f_mean=f_mean))
    half = S // 128 * 64
    f[:, :, half - 64:half] += 3.0 - f_mean
    f[:, :, half:] = 30.0
    i[:, :, half:] -= 40.0
    h, (c, n, m) = xlstm_b200.mlstm_sequence(q, k, v, i, f, kernel="chunkwise")
    xlstm_b200.check_device_status()
    lf = torch.nn.functional.logsigmoid(f.double())
    behind = lf.flip(-1).cumsum(-1).flip(-1) - lf
    m64 = torch.maximum((i.double() + behind).amax(-1), lf.sum(-1))
    w = torch.exp(i.double() + behind - m64[..., None])
    n64 = torch.einsum("bns,bnsd->bnd", w, k.double())
    c64 = torch.einsum("bnsd,bnse->bnde", w[..., None] * k.double(), v.double())
    assert float((m.double()[..., 0] - m64).abs().max()) <= 1.8e-5
    assert float((n.double() - n64).norm()) <= 1.8e-5 * float(n64.norm())
    assert float((c.double() - c64).norm()) <= TOL_BF16 * float(c64.norm())


def test_chunkwise_packed_documents_longer_than_a_part():
    """Packed rows with documents far above and far below the length of a part, empty ones among them."""
    import xlstm_b200
    B, NH, S, DQ, DV = 2, 1, 4096, 64, 128
    cu = [0, 1, 1, 3000, 3064, 4095, 4096, 4096 + 4096, 8192]
    q, k, v, i, f = _inputs(63, B, NH, S, DQ, DV, torch.bfloat16)
    flat = lambda t: t.transpose(0, 1).reshape(NH, B * S, *t.shape[3:])
    h_ref, st_ref = O.mlstm_packed(flat(q), flat(k), flat(v), flat(i), flat(f), cu)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), cu_seqlens=cu, kernel="chunkwise")
    xlstm_b200.check_device_status()
    _check(flat(h.cpu()), st, h_ref, st_ref, TOL_BF16)


def test_chunkwise_harsh_gates_stay_finite_and_match():
    """Forget gates around -6 (strong decay) and input gates with a wide spread exercise the stabilisers."""
    import xlstm_b200
    B, NH, S, DQ, DV = 1, 2, 320, 64, 128
    q, k, v, i, f = _inputs(9, B, NH, S, DQ, DV, torch.bfloat16, f_mean=-6.0)
    i = i * 6.0
    h_ref, st_ref = O.mlstm_inference(q, k, v, i, f)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), kernel="chunkwise")
    _check(h, st, h_ref, st_ref, TOL_BF16)


@pytest.mark.parametrize("DQ,DV", [(64, 128), (256, 512)])
@pytest.mark.parametrize("jump", [20.0, 40.0, 120.0])
def test_chunkwise_stabiliser_jumps_inside_a_chunk(jump, DQ, DV):
    """An input gate that leaps by `jump` nats in the middle of a chunk: the rows before the leap must keep their
    own scale (the kernel switches that chunk to its per-row frame), the rows after it forget the past."""
    import xlstm_b200
    B, NH, S = 1, 2, 256
    q, k, v, i, f = _inputs(21, B, NH, S, DQ, DV, torch.bfloat16)
    # a common component in q and k keeps q.n away from zero, so that h is well conditioned where only a few
    # tokens carry weight
    q = (q.float() + 1.0).to(torch.bfloat16)
    k = (k.float() + 1.0).to(torch.bfloat16)
    i = i.clone()
    i[:, :, 100:] += jump          # inside chunk 1
    i[:, 1, 200:] -= 2 * jump      # and back down inside chunk 3 for one head
    h_ref, st_ref = O.mlstm_inference(q, k, v, i, f)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), kernel="chunkwise")
    assert torch.isfinite(h.float()).all()
    _check(h, st, h_ref, st_ref, TOL_BF16)
    # the rows before the leap alone
    assert rel_l2(h[:, :, 64:100].float().cpu(), h_ref[:, :, 64:100].float()) <= TOL_BF16


def test_chunkwise_transposed_views_like_the_reference_layer():
    """q,k,v arrive as (B,S,NH*D) projections viewed as (B,NH,S,D) -- xlstm_large/model.py:415-419."""
    import xlstm_b200
    B, NH, S, DQ, DV = 2, 4, 192, 64, 128
    q, k, v, i, f = _inputs(10, B, NH, S, DQ, DV, torch.bfloat16)
    h_ref, st_ref = O.mlstm_inference(q, k, v, i, f)
    qc = q.transpose(1, 2).reshape(B, S, NH * DQ).cuda().reshape(B, S, NH, DQ).transpose(1, 2)
    kc = k.transpose(1, 2).reshape(B, S, NH * DQ).cuda().reshape(B, S, NH, DQ).transpose(1, 2)
    vc = v.transpose(1, 2).reshape(B, S, NH * DV).cuda().reshape(B, S, NH, DV).transpose(1, 2)
    ic = i.transpose(1, 2).contiguous().cuda().transpose(1, 2)
    fc = f.transpose(1, 2).contiguous().cuda().transpose(1, 2)
    assert not qc.is_contiguous()
    h, st = xlstm_b200.mlstm_sequence(qc, kc, vc, ic, fc, kernel="chunkwise")
    _check(h, st, h_ref, st_ref, TOL_BF16)


@pytest.mark.parametrize("kernel,dtype,tol", [("chunkwise", torch.bfloat16, TOL_BF16), ("recurrent", torch.float32, TOL_F32)])
def test_packed_documents_reset_state_in_kernel(kernel, dtype, tol):
    """Ragged documents packed into rows, boundaries anywhere (also inside a 64-token chunk), an empty
    document, and a document that ends exactly at a row end.  Oracle = each document alone."""
    import xlstm_b200
    B, NH, S, DQ, DV = 2, 2, 256, 64, 128
    cu = [0, 5, 5, 70, 200, 256, 256 + 64, 256 + 191, 512]
    q, k, v, i, f = _inputs(11, B, NH, S, DQ, DV, dtype)
    flat = lambda t: t.transpose(0, 1).reshape(NH, B * S, *t.shape[3:])
    h_ref, st_ref = O.mlstm_packed(flat(q), flat(k), flat(v), flat(i), flat(f), cu)
    h, st = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), cu_seqlens=cu, kernel=kernel)
    xlstm_b200.check_device_status()
    assert st[0].shape == (len(cu) - 1, NH, DQ, DV)
    _check(flat(h.cpu()), st, h_ref, st_ref, tol)


def test_chunkwise_full_size_config2_properties():
    """The benchmark shape at full size (B=4, NH=8, S=8192, DHQK=256, DHV=512, bf16: xLSTM-7B heads).  Checks:
    (1) the tensor-core kernel agrees with the on-device fp32 recurrence for one (batch, head) pair,
    (2) splitting the sequence in two calls that hand the state over gives the same result,
    (3) batch rows / heads are independent (same inputs in two rows -> identical outputs),
    (4) two full rows against the CPU oracle (h, C, n, m)."""
    import xlstm_b200
    B, NH, S, DQ, DV = 4, 8, 8192, 256, 512
    g = torch.Generator(device="cuda").manual_seed(0)
    q = (torch.randn(B, NH, S, DQ, generator=g, device="cuda") / math.sqrt(DQ)).bfloat16()
    k = (torch.randn(B, NH, S, DQ, generator=g, device="cuda") / math.sqrt(DQ)).bfloat16()
    v = torch.randn(B, NH, S, DV, generator=g, device="cuda").bfloat16()
    i = torch.randn(B, NH, S, generator=g, device="cuda")
    f = torch.randn(B, NH, S, generator=g, device="cuda") + 3.0
    q[3], k[3], v[3], i[3], f[3] = q[0], k[0], v[0], i[0], f[0]
    h, (c, n, m) = xlstm_b200.mlstm_sequence(q, k, v, i, f, kernel="chunkwise")
    xlstm_b200.check_device_status()
    assert torch.isfinite(h.float()).all() and torch.isfinite(c).all()
    assert torch.equal(h[3], h[0]) and torch.equal(c[3], c[0])
    sl = (slice(1, 2), slice(2, 3))
    hr, (cr, nr, mr) = xlstm_b200.mlstm_sequence(q[sl], k[sl], v[sl], i[sl], f[sl], kernel="recurrent")
    assert rel_l2(h[sl].float(), hr.float()) < TOL_BF16
    assert rel_l2(c[sl], cr) < TOL_BF16 and rel_l2(n[sl], nr) < TOL_BF16
    assert torch.allclose(m[sl], mr, atol=1e-3)
    half = 4096 + 37
    h1, st1 = xlstm_b200.mlstm_sequence(q[:1, :, :half], k[:1, :, :half], v[:1, :, :half], i[:1, :, :half], f[:1, :, :half], kernel="chunkwise")
    h2, st2 = xlstm_b200.mlstm_sequence(q[:1, :, half:], k[:1, :, half:], v[:1, :, half:], i[:1, :, half:], f[:1, :, half:], *st1, kernel="chunkwise")
    assert rel_l2(torch.cat([h1, h2], 2).float(), h[:1].float()) < TOL_BF16
    assert rel_l2(st2[0], c[:1]) < TOL_BF16
    # (4) against the CPU oracle directly: two full rows (all 8 heads, all 8192 tokens) of h and of the final C, n, m
    for row in (1, 2):
        h_ref, (c_ref, n_ref, m_ref) = O.mlstm_inference(q[row:row + 1].cpu(), k[row:row + 1].cpu(), v[row:row + 1].cpu(),
                                                         i[row:row + 1].cpu(), f[row:row + 1].cpu())
        _check(h[row:row + 1], (c[row:row + 1], n[row:row + 1], m[row:row + 1]), h_ref, (c_ref, n_ref, m_ref), TOL_BF16)
        # no drift along the sequence: the last 512 tokens are as close as the whole row
        assert rel_l2(h[row, :, -512:].float().cpu(), h_ref[0, :, -512:]) < TOL_BF16


def test_prefill_from_pinned_host_buffers_equals_device_call():
    """The host-buffer entry (pieces over three streams, uploads / kernels / downloads overlapped) returns what the
    device-resident call returns."""
    import xlstm_b200
    B, NH, S, DQ, DV = 3, 4, 200, 64, 128
    q, k, v, i, f = _inputs(41, B, NH, S, DQ, DV, torch.bfloat16)
    host = [t.pin_memory() for t in (q, k, v, i, f)]
    h_host = torch.empty(B, NH, S, DV, dtype=torch.bfloat16).pin_memory()
    c_host = torch.empty(B, NH, DQ, DV).pin_memory()
    n_host = torch.empty(B, NH, DQ).pin_memory()
    m_host = torch.empty(B, NH, 1).pin_memory()
    xlstm_b200.mlstm_sequence_from_host(*host, h_host, c_host, n_host, m_host)
    torch.cuda.synchronize()
    h, (c, n, m) = xlstm_b200.mlstm_sequence(*_cuda(q, k, v, i, f), kernel="chunkwise")
    assert torch.equal(h_host, h.cpu()) and torch.equal(c_host, c.cpu())
    assert torch.equal(n_host, n.cpu()) and torch.equal(m_host, m.cpu())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,NH,DQ,DV,with_slots", [(8, 8, 256, 512, False), (5, 3, 64, 128, True), (2, 2, 128, 1024, True), (3, 4, 32, 40, False)])
def test_fused_decode_cell_equals_cap_step_norm_gate(dtype, B, NH, DQ, DV, with_slots):
    """One kernel for gate soft cap + cell step + per-head norm + output gate against the three separate kernels: the
    states bit for bit (same arithmetic), the gated output up to the summation order of the norm's two sums (the thread
    blocks of a head exchange partial sums through distributed shared memory)."""
    import xlstm_b200
    from xlstm_b200 import ops
    if dtype == torch.float32 and DV > 512:
        pytest.skip("the separate norm kernel takes at most 512 fp32 columns per head")
    g = torch.Generator().manual_seed(B * 100 + NH * 10 + DV)
    rnd = lambda *shape: torch.randn(*shape, generator=g)
    q, k, v = rnd(B, NH, DQ).to(dtype).cuda(), rnd(B, NH, DQ).to(dtype).cuda(), rnd(B, NH, DV).to(dtype).cuda()
    wide = (4.0 * rnd(B, 2 * NH + 24)).to(dtype).cuda()
    gates_raw = wide[:, 8:8 + 2 * NH]                      # a column slice of a wider projection output
    bias = torch.cat([torch.zeros(NH), 3.0 + torch.zeros(NH)]).to(dtype).cuda()
    ogate, w = rnd(B, NH * DV).to(dtype).cuda(), (1.0 + 0.1 * rnd(NH * DV)).to(dtype).cuda()
    N = B + 3 if with_slots else B
    pool = [rnd(N, NH, DQ, DV).cuda(), rnd(N, NH, DQ).cuda(), rnd(N, NH, 1).cuda()]
    slot = None
    if with_slots:
        slot = torch.tensor([N - 1 - 2 * j if j % 3 != 1 else -1 for j in range(B)], dtype=torch.int32)   # every third stream inactive
    # the three kernels
    gates = ops.soft_cap(gates_raw, 15.0, out_float32=True, float32_math=True, bias=bias)
    c1 = [t.clone() for t in pool]
    h, st1 = xlstm_b200.mlstm_step(q, k, v, gates[:, :NH], gates[:, NH:], *c1, slot=slot)
    want = xlstm_b200.headnorm_gate(h[:, :, None], ogate[:, None], w)[:, 0]
    # the one kernel
    c2 = [t.clone() for t in pool]
    got, st2 = ops.mlstm_decode_cell(q, k, v, gates_raw, bias, 15.0, ogate, w, *c2, slot=slot)
    xlstm_b200.check_device_status()
    for a, b_ in zip(st1, st2):
        assert torch.equal(a, b_)
    assert got.shape == (B, NH * DV)
    d = (got.float() - want.float()).abs()
    tol = 2.0 ** -7 if dtype == torch.bfloat16 else 1e-5
    assert (d <= want.float().abs() * tol + 1e-5).all(), float(d.max())
    if with_slots:   # inactive streams: zero output, pool untouched
        idle = [j for j in range(B) if int(slot[j]) < 0]
        assert float(got[idle].float().abs().max()) == 0.0


@pytest.mark.parametrize("DQ", [64, 128, 256])
@pytest.mark.parametrize("S,off", [(33, 0), (64, 1), (70, 0)])
def test_recurrent_with_compiled_head_sizes_equals_the_general_kernel(DQ, S, off):
    """Head sizes with an instance of their own, with and without 16-byte rows.  One zero feature more takes the general
    instance: same sums, up to 1/sqrt(d), which q makes up for.  Both are fp32 sums, so TOL_F32 is far above their difference."""
    import xlstm_b200
    q, k, v, i, f = _cuda(*_inputs(61, 1, 2, S, DQ, 96, torch.float32))
    if off:   # rows that start 4 bytes past a 16-byte boundary
        q, k = (torch.cat([torch.zeros_like(t[..., :1]), t, torch.zeros_like(t[..., :3])], -1)[..., 1:DQ + 1] for t in (q, k))
    h, (c, n, m) = xlstm_b200.mlstm_sequence(q, k, v, i, f, kernel="recurrent")
    pad = lambda t: torch.cat([t, torch.zeros_like(t[..., :1])], -1)
    h1, (c1, n1, m1) = xlstm_b200.mlstm_sequence(pad(q) * ((DQ + 1) / DQ) ** 0.5, pad(k), v, i, f, kernel="recurrent")
    for a, b in ((h, h1), (c, c1[:, :, :DQ]), (n, n1[..., :DQ]), (m, m1)):
        assert float((a - b).norm()) <= TOL_F32 * float(b.norm())


def _whole_documents(q, k, v, i, f):
    """Parameters and outputs of the C entry without scratch: every row one chain."""
    import ctypes
    import xlstm_b200
    from xlstm_b200 import _lib
    B, NH, S, DQ = q.shape
    DV = v.shape[3]
    out = [torch.empty(B, NH, S, DV, dtype=torch.bfloat16, device="cuda"), torch.empty(B, NH, DQ, DV, device="cuda"),
           torch.empty(B, NH, DQ, device="cuda"), torch.empty(B, NH, 1, device="cuda")]
    p = _lib.MlstmSeqParams()
    p.B, p.NH, p.S, p.DHQK, p.DHV, p.num_docs = B, NH, S, DQ, DV, B
    p.q, p.k, p.v, p.igate, p.fgate = (t.data_ptr() for t in (q, k, v, i, f))
    p.h, p.c_out, p.n_out, p.m_out = (t.data_ptr() for t in out)
    p.status = xlstm_b200.ops.status_word("cuda").data_ptr()
    p.q_sb, p.q_sh, p.q_st = p.k_sb, p.k_sh, p.k_st = q.stride()[:3]
    p.v_sb, p.v_sh, p.v_st = p.h_sb, p.h_sh, p.h_st = v.stride()[:3]
    p.g_sb, p.g_sh, p.g_st = i.stride()
    p.eps, p.dtype = 1e-6, _lib.XL_BF16
    assert _lib.lib().xl_mlstm_chunkwise(ctypes.byref(p), torch.cuda.current_stream().cuda_stream) == 0
    return p, out


def test_host_buffer_prefill_keeps_documents_whole():
    """Pieces whose rows would be cut into parts on their own: h and the states are those of the uncut chain, bit for bit."""
    import ctypes
    import xlstm_b200
    from xlstm_b200 import _lib
    B, NH, S, DQ, DV = 2, 4, 2048, 64, 128
    q, k, v, i, f = _inputs(72, B, NH, S, DQ, DV, torch.bfloat16)
    p, want = _whole_documents(*_cuda(q, k, v, i, f))
    p.B = p.num_docs = 1
    assert _lib.lib().xl_mlstm_chunkwise_scratch_bytes(ctypes.byref(p)) > 0
    outs = [torch.empty(t.shape, dtype=t.dtype).pin_memory() for t in want]
    xlstm_b200.mlstm_sequence_from_host(*(t.pin_memory() for t in (q, k, v, i, f)), *outs)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b.cpu()) for a, b in zip(outs, want))


def test_chunkwise_without_room_for_its_scratch_keeps_documents_whole():
    """A packed row of 32768 tokens asks for 37 MB of part states.  With room for the outputs alone the call still works, and
    equals the C entry without scratch bit for bit."""
    import ctypes
    import xlstm_b200
    from xlstm_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(5)
    S, NH, DQ, DV = 32768, 8, 256, 512
    q, k, v, i, f = (torch.randn(1, NH, S, *d, generator=g, device="cuda") for d in ((DQ,), (DQ,), (DV,), (), ()))
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    cu = torch.tensor([0, S], dtype=torch.int32, device="cuda")
    p, want = _whole_documents(q, k, v, i, f)
    p.cu_seqlens = cu.data_ptr()
    assert _lib.lib().xl_mlstm_chunkwise_scratch_bytes(ctypes.byref(p)) > 32 << 20
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = [torch.empty_like(t) for t in want]   # what the outputs will take; everything else is taken now
    taken = []
    torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / torch.cuda.get_device_properties(0).total_memory)
    try:
        for size in (256 << 20, 64 << 20, 16 << 20, 4 << 20, 3 << 19):
            try:
                while True:
                    taken.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                pass
        del room
        ooms = torch.cuda.memory_stats()["num_ooms"]
        h, st = xlstm_b200.mlstm_sequence(q, k, v, i, f, cu_seqlens=cu, kernel="chunkwise")
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    xlstm_b200.check_device_status()
    assert torch.cuda.memory_stats()["num_ooms"] > ooms
    assert all(torch.equal(a, b) for a, b in zip((h, *st), want))


def test_host_vectors_are_refused_under_capture():
    """A replay would read the host buffer of the capture.  The device forms are captured."""
    import xlstm_b200
    q, k, v, i, f = _cuda(*_inputs(68, 2, 2, 64, 64, 128, torch.bfloat16))
    c, n, m = _cuda(*_state(69, 3, 2, 64, 128))
    step = lambda slot: xlstm_b200.mlstm_step(q[:, :, 0], k[:, :, 0], v[:, :, 0], i[:, :, 0], f[:, :, 0], c, n, m, slot=slot, inplace=False)
    seq = lambda cu: xlstm_b200.mlstm_sequence(q, k, v, i, f, cu_seqlens=cu)
    slot, cu = torch.tensor([2, 0], dtype=torch.int32, device="cuda"), torch.tensor([0, 20, 64, 128], dtype=torch.int32, device="cuda")
    want = step([2, 0]), seq([0, 20, 64, 128])
    torch.cuda.synchronize()
    for call in (lambda: step([2, 0]), lambda: seq([0, 20, 64, 128])):
        with pytest.raises(RuntimeError, match="CUDA graph"):
            with torch.cuda.graph(torch.cuda.CUDAGraph()):
                call()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step(slot), seq(cu)
    graph.replay()
    torch.cuda.synchronize()
    for (h, st), (h1, st1) in zip(got, want):
        assert torch.equal(h, h1) and all(torch.equal(a, b) for a, b in zip(st, st1))


def test_dimensions_of_size_one_in_front_of_the_features():
    """A step's k and v as (B,NH,1,D) slices of a sequence, a sequence's v as (B,NH,S,1,DHV)."""
    import xlstm_b200
    q, k, v, i, f = _cuda(*_inputs(70, 2, 2, 5, 64, 128, torch.bfloat16))
    c, n, m = _cuda(*_state(71, 2, 2, 64, 128))
    step = lambda k_, v_: xlstm_b200.mlstm_step(q[:, :, 0], k_, v_, i[:, :, 0], f[:, :, 0], c, n, m, inplace=False)
    (h, st), (h1, st1) = step(k[:, :, 0], v[:, :, 0]), step(k[:, :, :1], v[:, :, :1])
    assert h1.shape == h.shape and torch.equal(h, h1) and all(torch.equal(a, b) for a, b in zip(st, st1))
    (h, st), (h1, st1) = (xlstm_b200.mlstm_sequence(q, k, w, i, f) for w in (v, v[:, :, :, None]))
    assert h1.shape == h.shape and torch.equal(h, h1) and all(torch.equal(a, b) for a, b in zip(st, st1))
