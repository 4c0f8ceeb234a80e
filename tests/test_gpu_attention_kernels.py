"""GPU parity of the attention kernels behind the decode and prefill entry points, at the sizes where their
work split changes: edges of row and key tiles, page holes, masks, one and several key ranges, group sizes.
Outputs must satisfy the library tolerance |x - y| <= 1e-4 + 1e-3 |y| against the CPU checker."""
import numpy as np
import pytest
import torch

import longhornai_b200 as lb
from cpu_checker import AttnCfg, Layout, best_checker
from gpu_util import assert_close, dev, host, lb_cfg, lb_layout
from test_gpu_parity import build_paged_case, poll_ok

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def chk():
    return best_checker()


def blocks(lens):
    return sum((n + 15) // 16 for n in lens) + 3


@pytest.mark.parametrize("qh,kvh,window,lens", [(8, 1, 0, [700, 16]), (20, 4, 0, [33]), (32, 2, 100, [1, 300, 128]), (4, 4, 0, [0, 65])])
def test_decode_attention_group_sizes(chk, qh, kvh, window, lens):
    """More than four query heads per KV head (several CTAs per KV head), and the single-request call."""
    rng = np.random.default_rng(qh + sum(lens))
    L, tables, pools, (k, v, ks, vs) = build_paged_case(chk, rng, len(lens), lens, qh, kvh, 128, 16, blocks(lens))
    cfg = AttnCfg(qh, kvh, 1, 128, 1, 0.0, window, 0)
    Q = rng.standard_normal((len(lens), qh, 1, 128)).astype(np.float32)
    sl = np.array(lens, np.int32)
    want = chk.paged_attention_q8_batched(Q, pools, tables, sl, cfg, L, parallel=True)
    got = lb.paged_attention_q8_batched(dev(Q), k, v, ks, vs, dev(tables), dev(sl), lb_cfg(cfg), lb_layout(L))
    assert_close(host(got), want, what="batched")
    for r, n in enumerate(lens):
        one = lb.paged_attention_q8(dev(Q[r]), k, v, ks, vs, dev(tables[r]), n, lb_cfg(cfg), lb_layout(L))
        assert_close(host(one), want[r], what=f"request {r} alone")
    poll_ok()


@pytest.mark.parametrize("qh,kvh,window,chunk,lens", [(8, 2, 0, 0, [0, 1, 8, 9, 2048]), (8, 1, 0, 0, [1500, 40]), (6, 2, 77, 0, [300]),
                                                      (4, 4, 0, 64, [130, 64])])
def test_decode_attention_fp32_pools(chk, qh, kvh, window, chunk, lens):
    rng = np.random.default_rng(qh + sum(lens))
    n, nblk = len(lens), blocks(lens)
    L = Layout(nblk, 16, kvh, 128)
    tables = np.full((n, max(1, max((x + 15) // 16 for x in lens))), -1, np.int32)
    perm, used = rng.permutation(nblk).astype(np.int32), 0
    for r, x in enumerate(lens):
        b = (x + 15) // 16
        tables[r, :b] = perm[used:used + b]; used += b
    kp = rng.standard_normal((nblk, kvh, 16, 128)).astype(np.float32)
    vp = rng.standard_normal((nblk, kvh, 16, 128)).astype(np.float32)
    Q = rng.standard_normal((n, qh, 1, 128)).astype(np.float32)
    sl = np.array(lens, np.int32)
    cfg = AttnCfg(qh, kvh, 1, 128, 1, 0.0, window, chunk)
    want = chk.paged_attention_f32_batched(Q, kp, vp, tables, sl, cfg, L)
    last = sl - 1                                               # slots after the last token may hold anything
    for r, x in enumerate(lens):
        if x % 16:
            vp[tables[r, last[r] // 16], :, x % 16:] = np.nan
            kp[tables[r, last[r] // 16], :, x % 16:] = np.nan
    got = lb.paged_attention_batched_f32(dev(Q), dev(kp), dev(vp), dev(tables), dev(sl), lb_cfg(cfg), lb_layout(L))
    assert_close(host(got), want, what="fp32 pools")
    if lens[0] > 16:                                            # a released page masks its keys
        holed = tables.copy(); holed[0, 0] = -1
        got = lb.paged_attention_batched_f32(dev(Q), dev(kp), dev(vp), dev(holed), dev(sl), lb_cfg(cfg), lb_layout(L))
        assert np.isfinite(host(got)).all()
    poll_ok()
