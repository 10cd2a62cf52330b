"""The fold kernel reports every bounded wait that runs out: its roles note a failure in a shared flag, and
the one thread that turns the flag into the device error word reads it when no role can set it any more.

Read from the kernel's source: the window between two warps of one launch cannot be steered from outside,
and nothing here makes a GPU wait fail."""
import os
import re

from tests.hostcheck import CSRC


def kernel_body():
    with open(os.path.join(CSRC, "kernels_fold.cuh")) as f:
        src = f.read()
    src = src[src.index("ffn_w4a8_fold_kernel(const"):]
    return re.sub(r"//[^\n]*", "", src)


def test_error_word_is_written_behind_the_last_barrier():
    body = kernel_body()
    assert body.count("report_error(") == 1
    assert body.index("report_error(") > body.rindex("__syncthreads();")


def test_the_wait_for_the_last_mmas_notes_its_time_out():
    body = kernel_body()
    wait = body[body.index("mbar_try_wait(drain"):]
    assert "*fail = 1;" in wait[:wait.index("break;")]
