"""What the box-fed convolution and weight-gradient kernels ask of an SM, over every
channel count and width that they take: shared memory within a block's limit, no
more blocks of a launch on an SM than its 512 tensor memory columns serve, a stage
for every box of a row, and runs of rows that cover the image once."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SM, CTA_MAX, COLS = 228 * 1024, 227 * 1024, 512
WIDTHS = (16, 32, 48, 64, 96, 128)


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("plan") / "plan.so")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-shared", "-fPIC",
                        "-I", os.path.join(ROOT, "xbeach_gpu_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cxx", "conv_plan.cpp"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(so)


def _rows(plan):
    """(output channels, box channels, input channels, stages) of every layer the kernel over rows takes"""
    for bn in WIDTHS:
        for cin in range(16, 400, 16):
            for wc in (64, 32, 16):
                n = plan.rows_stages(bn, wc, 128, cin) if cin % wc == 0 else 0
                if n:
                    yield bn, wc, cin, n


def _wgrad(plan):
    for bn in WIDTHS:
        for wc in (32, 16):
            for nseg in range(1, 20):
                n = plan.wgrad_slots(bn, wc, nseg)
                if n:
                    yield bn, wc, n


def test_plans_fit_a_block(plan):
    rows, wg = list(_rows(plan)), list(_wgrad(plan))
    assert (32, 16, 16, 18) in rows and (64, 64, 64, 9) in rows and (32, 32, 13) in wg
    for bn, wc, cin, n in rows:
        assert 1024 + n * 256 * wc + 18 * cin * bn <= plan.rows_smem(bn, wc, cin, n) <= CTA_MAX - 1024
    for bn, wc, n in wg:
        assert 1024 + n * 512 * wc + 384 * bn <= plan.wgrad_smem(bn, wc, n) <= CTA_MAX - 512


def test_blocks_on_an_sm_fit_its_tensor_memory(plan):
    """As many blocks of a launch as an SM's shared memory holds ask for no more than
    its columns, so that none is placed there only to wait."""
    for bn, wc, cin, n in _rows(plan):
        assert SM // (plan.rows_smem(bn, wc, cin, n) + 1024) * plan.rows_cols(bn) <= COLS, (bn, wc, cin)
    for bn, wc, n in _wgrad(plan):
        assert SM // (plan.wgrad_smem(bn, wc, n) + 1024) * plan.wgrad_cols(bn) <= COLS, (bn, wc, n)


def test_layers_left_to_the_other_kernels(plan):
    """16-channel boxes with more output than input channels, beyond 32."""
    took = {(cin, bn) for bn, wc, cin, n in _rows(plan)}
    for cin, bn in ((16, 48), (16, 64), (16, 96), (16, 128), (48, 64), (48, 96), (48, 128), (80, 96), (80, 128)):
        assert (cin, bn) not in took
    for cin, bn in ((16, 16), (16, 32), (32, 128), (48, 48), (64, 128), (80, 64), (96, 32)):
        assert (cin, bn) in took


def test_a_rows_boxes_have_stages(plan):
    """All boxes of an input row are in flight together, a stage and a barrier each:
    112 and 144 input channels (21 and 27 boxes) have more than the 18 stages."""
    for bn, wc, cin, n in _rows(plan):
        assert 3 * (cin // wc) <= n <= 18, (bn, wc, cin, n)
    assert (16, 16, 80, 18) in list(_rows(plan))


@pytest.mark.parametrize("extra", [0, 1])
def test_runs_cover_every_row_once(plan, extra):
    """The runs of the blocks are the rows of all strips in order, each once, none
    empty, on at most one block per SM; and no block reads more input rows (two more
    than it writes, per strip that it touches) than runs on end would give it."""
    for sms in (1, 7, 132, 148):
        for S in (1, 2, 3, 4, 7, 8, 12, 40, 147, 148, 149, 300):
            for H in (1, 2, 3, 5, 16, 37, 100, 127, 160, 208, 256, 304, 512, 1000):
                buf = (C.c_int * (2 * sms))()
                n = plan.rows_run(S, H, sms, extra, None)
                assert 1 <= n <= sms
                plan.rows_run(S, H, sms, extra, buf)
                runs = [(buf[2 * k], buf[2 * k + 1]) for k in range(n)]
                assert runs[0][0] == 0 and runs[-1][1] == S * H
                assert all(a < b for a, b in runs) and all(p[1] == q[0] for p, q in zip(runs, runs[1:]))

                def most(rs):
                    return max(b - a + 2 * ((b - 1) // H - a // H + 1) for a, b in rs)
                per = -(-S * H // sms)
                assert most(runs) <= most([(k, min(S * H, k + per)) for k in range(0, S * H, per)])
                assert max(b - a for a, b in runs) <= per + extra
    buf = (C.c_int * 296)()
    assert plan.rows_run(2, 160, 148, 0, buf) == 108 and (buf[2], buf[3]) == (3, 6) and (buf[108], buf[109]) == (160, 163)


# 16-channel boxes where the other kernels are the faster (a first size that pays is
# beside each): too few rows a block, 16 outputs of 48 or 80 channels, wide strip edges
@pytest.mark.parametrize("bn,cin,W,H,pays", [
    (16, 16, 384, 256, 0), (16, 16, 512, 256, 0), (16, 16, 512, 336, 1), (32, 16, 240, 200, 0), (32, 16, 256, 256, 1),
    (32, 16, 320, 200, 1), (32, 16, 344, 240, 1), (16, 48, 512, 256, 0), (16, 80, 1024, 512, 0), (48, 48, 344, 240, 0),
    (48, 48, 300, 304, 0), (48, 48, 512, 256, 1), (32, 48, 192, 768, 0), (32, 80, 400, 400, 0), (32, 80, 512, 336, 1),
    (16, 32, 128, 1, 1), (128, 64, 128, 1, 1)])
def test_narrow_boxes_where_they_pay(plan, bn, cin, W, H, pays):
    assert plan.rows_pays(bn, cin, W, H * W, 148) == pays
