"""Rules of the CUDA sources that no run shows: they are read as text."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _sources():
    for path in sorted(glob.glob(os.path.join(ROOT, "slhav2_b200", "csrc", "*.cu*"))):
        text = re.sub(r"/\*.*?\*/|//[^\n]*", "", open(path).read(), flags=re.S)
        yield os.path.basename(path), text


def test_only_the_models_own_arrays_are_read_through_the_non_coherent_path():
    # Kernels are launched while their predecessor on the stream still runs and wait for it on the device.  Non-coherent loads need memory that
    # nobody writes from the grid's start on: a model's arrays, complete before the model is handed out, but no argument of a call.
    models = r"^(zf|next|mp|diag|a\.z|reinterpret_cast<const float4\*>\(a\.scale\))(?!\w)"
    for name, text in _sources():
        assert "global.nc" not in text, name
        for m in re.finditer(r"__ldg\(((?:[^()]|\([^()]*\))*)", text):
            assert name == "encode.cu" and re.match(models, m.group(1)), (name, m.group(0))
        if "__ldg" in text:  # what those names point to
            for var, arrays in (("zf", "a.zf"), ("next", "zf"), ("mp", "a.p|a.pt|a.zt"), ("diag", None)):
                for d in re.finditer(r"\bconst \w+\* %s = ([^;]*);" % var, text):
                    assert arrays and re.search(r"\b(%s)\b" % arrays.replace(".", r"\."), d.group(1)), (var, d.group(0))


def test_every_kernel_that_lets_the_next_one_start_waits_for_the_one_before_it():
    for name, text in _sources():
        for m in re.finditer(r"\bdep_launch\(\);\s*(\S+)", text):
            assert m.group(1).startswith("dep_wait()"), (name, m.group(0))


def test_a_kernel_whose_answer_the_host_polls_has_met_at_a_barrier_before_it_answers():
    # The host returns on the answer: blocks that have not read the pool's counters by then would see what the caller does next.
    text = dict(_sources())["pool.cu"]
    for kernel, answer in (("enforce_step_kernel", r"\bsay\("), ("stats_kernel", r"\banswer\[8\] =")):
        body = re.search(r"\b%s\(PoolDev.*?\n}\n" % kernel, text, flags=re.S).group(0)
        assert re.search(answer, body)
        for m in re.finditer(answer, body):
            block = body[:m.start()]
            assert ".sync()" in block, (kernel, body[m.start():m.start() + 60])


def test_a_dense_call_that_is_refused_drains_the_library_s_stream():
    # Its kernels end on the check's word in the thread's scratch, which the thread's next call on another stream may write.
    text = dict(_sources())["capi_b200.cuh"]
    body = text[text.index("int32_t slha_b200_score_segments("):]
    body = body[:body.index("\n}\n")]
    refused = body[body.rindex("checked_offsets("):]
    assert "return Status" not in refused and re.search(r"sync_by_default\(c\)\) SLHA_CUDA\(cudaStreamSynchronize", refused)
