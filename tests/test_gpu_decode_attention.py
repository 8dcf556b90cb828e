"""RoPE + cache write + attention of a decode step as one launch, where its split of the context can go wrong: context
lengths around the 16-token tiles and the shares of a cluster, sequences of one batch that leave shares empty, batches
too large to be split, and the result handed on as bf16 or as the quantised operand of the o projection.  Checked
through decoder_decode_step_batched on the small model against the oracle, with the bounds of its other driver cases."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import decoder_oracle as do
import fp4_oracle as o
import test_gpu_decoder as tgd
from conftest import ROOT
from gpu_util import REL_TOL_VS_ORACLE, bits_of, to_dev_bf16

pytestmark = pytest.mark.gpu

CONTEXTS = {
    "one-new": [0],                                        # nothing cached: the new token attends to itself
    "one-tile-edge": [15],
    "one-split": [511],                                    # 32 tiles over the largest cluster
    "one-split-ragged": [272],                             # 18 tiles: the last shares are short
    "uneven": [0, 1, 15, 16, 17, 62, 63, 64, 450],         # most shares of the short sequences are empty
    "few": [(11 * i) % 70 for i in range(74)],             # the last batch whose quantised result comes from two launches
    "many": [(11 * i) % 70 for i in range(75)],            # ... and the first from one
    "unsplit": [(7 * i) % 83 for i in range(230)],         # more CTAs than a split could use
}


def run_contexts(mode):
    from glm_asr_stack_b200 import engine, ops
    rng = np.random.default_rng(31)
    ws, cfg, layers, fn, (H, F, QH, KVH, HD, L) = tgd.build_toy_model(rng, 700, "plain")
    lin = tgd.oracle_linears(layers, mode)
    bs, max_blocks = 16, 33
    errs = {}
    for name, ctx in CONTEXTS.items():
        cached, n = np.array(ctx, np.int32), len(ctx)
        num_blocks = sum(c // bs + 1 for c in ctx) + 3
        pool = engine.KVPool(num_blocks, bs, L, KVH, HD, max_seqs=n, max_blocks_per_seq=max_blocks)
        perm = rng.permutation(num_blocks).tolist()
        tables = [[perm.pop() for _ in range(c // bs + 1)] for c in ctx]
        bts = engine.BlockTables(pool, tables)
        bt_np = np.full((n, max_blocks), -1, np.int32)
        for i, t in enumerate(tables):
            bt_np[i, :len(t)] = t
        kc0 = tgd.rnd_bits(rng, (L, num_blocks * bs, KVH * HD))
        vc0 = tgd.rnd_bits(rng, (L, num_blocks * bs, KVH * HD))
        pool.k.copy_(to_dev_bf16(kc0).view(pool.k.shape))
        pool.v.copy_(to_dev_bf16(vc0).view(pool.v.shape))
        hidden = tgd.rnd_bits(rng, (n, H))
        x = to_dev_bf16(hidden)
        d_lens = torch.from_numpy(cached.copy()).cuda()
        engine.decode_step(ws, cfg, pool, bts, x, d_lens, (ctypes.c_int * n)(*ctx))
        torch.cuda.synchronize()
        assert ops.status() == 0
        slots = np.array([bt_np[i, c // bs] * bs + c % bs for i, c in enumerate(ctx)], np.int64)
        kc, vc = [kc0[l].copy() for l in range(L)], [vc0[l].copy() for l in range(L)]
        want = do.decode_step(hidden, layers, fn, kc, vc, bt_np, cached, slots, QH, KVH, HD, bs, lin)
        errs[name] = o.rel_err(bits_of(x), want)
        assert errs[name] <= REL_TOL_VS_ORACLE, (name, errs)
        others = np.ones(num_blocks * bs, bool)
        others[slots] = False                              # only the new token's rows are written
        for l in range(L):
            for dev, before in ((pool.k, kc0), (pool.v, vc0)):
                assert np.array_equal(bits_of(dev[l].reshape(num_blocks * bs, -1))[others], before[l][others]), (name, l)
    return errs


@pytest.mark.parametrize("mode", ["w4a16", "all_w4a4"])
def test_decode_attention_contexts(mode):
    code = ("import sys; sys.path[:0]=[%r,%r,%r]; import test_gpu_decode_attention as t; print('RESULT', t.run_contexts(%r))"
            % (ROOT, os.path.join(ROOT, "oracle"), os.path.join(ROOT, "tests"), mode))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, **tgd.MODE_ENV[mode]), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and "RESULT" in r.stdout, r.stdout[-4000:] + r.stderr[-4000:]


# rows that attend to a token another row of the same step writes: (tokens in the cache, pages of row i are those of row j)
SHARED = {
    "consecutive": ([37, 38], {1: 0}),                     # two tokens of one sequence in one step
    "consecutive-over-a-page": ([15, 16, 200], {1: 0}),
    "same-slot-twice": ([20, 20, 50], {1: 0}),             # a batch padded with a copy of a row
    "run-of-many": ([40 + i for i in range(24)] + [9], {i: 0 for i in range(1, 24)}),
}


def run_shared(mode):
    from glm_asr_stack_b200 import engine, ops
    rng = np.random.default_rng(37)
    ws, cfg, layers, fn, (H, F, QH, KVH, HD, L) = tgd.build_toy_model(rng, 900, "plain")
    lin = tgd.oracle_linears(layers, mode)
    bs, max_blocks, num_blocks = 16, 20, 64
    errs = {}
    for name, (ctx, same) in SHARED.items():
        n, cached = len(ctx), np.array(ctx, np.int32)
        perm = rng.permutation(num_blocks).tolist()
        need = [max(c for j, c in enumerate(ctx) if same.get(j, j) == i) // bs + 1 if i not in same else 0 for i in range(n)]
        own = [[perm.pop() for _ in range(b)] for b in need]
        tables = [own[same.get(i, i)] for i in range(n)]
        kc0, vc0 = (tgd.rnd_bits(rng, (L, num_blocks * bs, KVH * HD)) for _ in range(2))
        hidden = tgd.rnd_bits(rng, (n, H))
        if name == "same-slot-twice":
            hidden[1] = hidden[0]
        bt_np = np.full((n, max_blocks), -1, np.int32)
        for i, t in enumerate(tables):
            bt_np[i, :len(t)] = t
        slots = np.array([bt_np[i, c // bs] * bs + c % bs for i, c in enumerate(ctx)], np.int64)
        kc, vc = [kc0[l].copy() for l in range(L)], [vc0[l].copy() for l in range(L)]
        want = do.decode_step(hidden, layers, fn, kc, vc, bt_np, cached, slots, QH, KVH, HD, bs, lin)
        for _ in range(5):
            pool = engine.KVPool(num_blocks, bs, L, KVH, HD, max_seqs=n, max_blocks_per_seq=max_blocks)
            bts = engine.BlockTables(pool, tables)
            pool.k.copy_(to_dev_bf16(kc0).view(pool.k.shape))
            pool.v.copy_(to_dev_bf16(vc0).view(pool.v.shape))
            x = to_dev_bf16(hidden)
            engine.decode_step(ws, cfg, pool, bts, x, torch.from_numpy(cached.copy()).cuda(), (ctypes.c_int * n)(*ctx))
            torch.cuda.synchronize()
            assert ops.status() == 0
            errs[name] = o.rel_err(bits_of(x), want)
            assert errs[name] <= REL_TOL_VS_ORACLE, (name, errs)
    return errs


@pytest.mark.parametrize("mode", ["w4a16", "all_w4a4"])
def test_rows_that_read_what_other_rows_write(mode):
    code = ("import sys; sys.path[:0]=[%r,%r,%r]; import test_gpu_decode_attention as t; print('RESULT', t.run_shared(%r))"
            % (ROOT, os.path.join(ROOT, "oracle"), os.path.join(ROOT, "tests"), mode))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, **tgd.MODE_ENV[mode]), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and "RESULT" in r.stdout, r.stdout[-4000:] + r.stderr[-4000:]


def run_setup(mode):
    """The set-up of a step in one launch (parameters for 32 or 256 rows) and its copies behind that: rows in one block, rows
    scattered over memory in any order, rows that are not 16-byte aligned.  Hidden rows, lengths and caches get equal bits."""
    from glm_asr_stack_b200 import _lib, engine, ops
    rng = np.random.default_rng(41)
    ws, cfg, layers, fn, (H, F, QH, KVH, HD, L) = tgd.build_toy_model(rng, 1100, "plain")
    bs, errs = 16, {}
    for n in (1, 32, 33, 256, 257):
        ctx = [(13 * i) % 37 for i in range(n)]
        cached, num_blocks = np.array(ctx, np.int32), sum(c // bs + 1 for c in ctx)
        perm = rng.permutation(num_blocks).tolist()
        tables = [[perm.pop() for _ in range(c // bs + 1)] for c in ctx]
        bt_np = np.full((n, 4), -1, np.int32)
        for i, t in enumerate(tables):
            bt_np[i, :len(t)] = t
        kc0, vc0 = (tgd.rnd_bits(rng, (L, num_blocks * bs, KVH * HD)) for _ in range(2))
        hidden = tgd.rnd_bits(rng, (n, H))
        order = rng.permutation(n).tolist()
        results = []
        for layout in ("block", "scattered", "unaligned"):
            pool = engine.KVPool(num_blocks, bs, L, KVH, HD, max_seqs=n, max_blocks_per_seq=4)
            bts = engine.BlockTables(pool, tables)
            pool.k.copy_(to_dev_bf16(kc0).view(pool.k.shape))
            pool.v.copy_(to_dev_bf16(vc0).view(pool.v.shape))
            off, pitch = (1, H + 3) if layout == "unaligned" else (0, H if layout == "block" else H + 64)
            at = order if layout == "scattered" else list(range(n))
            buf = torch.zeros(n * pitch + 8, dtype=torch.bfloat16, device="cuda")
            rows = [buf[off + at[i] * pitch:off + at[i] * pitch + H] for i in range(n)]
            for r, h in zip(rows, to_dev_bf16(hidden)):
                r.copy_(h)
            d_lens, h_lens = torch.from_numpy(cached.copy()).cuda(), (ctypes.c_int * n)(*ctx)
            ptrs = (ctypes.c_void_p * n)(*[r.data_ptr() for r in rows])
            _lib.load().decoder_decode_step_batched(None, ctypes.byref(ws.c), ptrs, ctypes.byref(pool.c), bts.arr,
                                                    ctypes.c_void_p(d_lens.data_ptr()), h_lens, n, None, None, ctypes.byref(cfg))
            torch.cuda.synchronize()
            assert ops.status() == 0
            assert list(h_lens) == (cached + 1).tolist() == d_lens.cpu().tolist()
            results.append((torch.stack(rows), pool.k.clone(), pool.v.clone()))
        for other in results[1:]:
            for a, b in zip(results[0], other):
                assert torch.equal(a.view(torch.int16), b.view(torch.int16)), n
        slots = np.array([bt_np[i, c // bs] * bs + c % bs for i, c in enumerate(ctx)], np.int64)
        kc, vc = [kc0[l].copy() for l in range(L)], [vc0[l].copy() for l in range(L)]
        want = do.decode_step(hidden, layers, fn, kc, vc, bt_np, cached, slots, QH, KVH, HD, bs, tgd.oracle_linears(layers, mode))
        errs[n] = o.rel_err(bits_of(results[0][0]), want)
        assert errs[n] <= REL_TOL_VS_ORACLE, errs
    return errs


@pytest.mark.parametrize("mode", ["w4a16", "all_w4a4"])
def test_step_setup_layouts(mode):
    code = ("import sys; sys.path[:0]=[%r,%r,%r]; import test_gpu_decode_attention as t; print('RESULT', t.run_setup(%r))"
            % (ROOT, os.path.join(ROOT, "oracle"), os.path.join(ROOT, "tests"), mode))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, **tgd.MODE_ENV[mode]), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and "RESULT" in r.stdout, r.stdout[-4000:] + r.stderr[-4000:]
