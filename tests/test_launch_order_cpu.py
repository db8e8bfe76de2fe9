"""What a launch leaves to the code. Programmatic ones: every kernel launched so
waits for its predecessor before it reads, a kernel that releases its successor
has waited itself, and the raster that clip_kernel releases finds setup's writes
by an acquire of the word that clip_kernel stored with release before releasing
it, else it waits. Any: its error is read. Read from the source: neither has
another trace."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "polyred_gb300", "csrc")
SRC = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "pr_kernels.cu")).read())


def kernels():
    out = {}
    for m in re.finditer(r"__global__[^;{]*?(\w+_kernel)\(", SRC):
        at = SRC.index("{", m.end())
        depth, end = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(SRC[end], 0)
            end += 1
        out[m.group(1)] = SRC[at:end]
    return out


BODY = kernels()


def test_every_overlapped_kernel_waits():
    overlapped = set(re.findall(r"launch\((?:true|overlap),\s*(\w+_kernel)", SRC)) | {"shade_kernel"}
    assert len(overlapped) >= 11
    for k in overlapped:
        assert "after_previous()" in BODY[k], k


def test_no_kernel_releases_before_its_own_wait():
    full_order = {"pass_init_kernel", "noalloc_init_kernel"}
    for k in full_order:
        assert not re.search(r"launch\((?:true|overlap),\s*" + k, SRC), k
    for k, b in BODY.items():
        if "release_next()" in b and k not in full_order:
            assert 0 <= b.find("after_previous()") < b.index("release_next()"), k


def test_the_raster_behind_clipping_acquires_what_clipping_published():
    clip, raster = BODY["clip_kernel"], BODY["raster_kernel"]
    assert clip.index("after_previous()") < clip.index("publish(&cnt->set_up)") < clip.index("release_next()")
    assert re.search(r"if \(threadIdx\.x == 0\) \{\s*if \(blockIdx\.x == 0\) publish\(&cnt->set_up\);\s*release_next\(\);\s*\}", clip)
    at = raster.index("if (!published(&P.cnt->set_up)) after_previous();")
    assert at < raster.index("__syncthreads()") < raster.index("c->n_tasks")
    assert "st.release.gpu" in SRC and "ld.acquire.gpu" in SRC


def test_every_launch_is_checked():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
            for m in re.finditer(r"<<<", src):
                after = src[m.end():m.end() + 500].split("return ", 1)[1]
                assert after.startswith("check(cudaGetLastError())"), (name, src[m.start() - 60:m.end()])


def test_the_wait_for_submitted_outputs_ends():
    """A context that has submitted a frame waits for its outputs' copies until the host has waited itself."""
    api = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "pr_api.cpp")).read())
    frame = api[api.index("int render_impl("):]
    assert frame.index("cudaStreamWaitEvent(st, c->ev_d2h, 0)") < frame.index("cudaStreamSynchronize(st)") < frame.index("c->submitted = false;")
    upload = api[api.index("int pr_scene_upload("):]
    assert upload.index("cudaStreamSynchronize(c->stream_d)") < upload.index("c->submitted = false;") < upload.index("scene_fill(")


def test_device_functions_hide_none_of_the_header():
    """A function of pr_kernels.cu with the name of one of pr_devmath.cuh would take its calls from that line on."""
    def names(src):
        return set(re.findall(r"PR_DEV [\w:<>*& ]+?(\w+)\(", src))
    header = names(re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "pr_devmath.cuh")).read()))
    own = names(SRC)
    assert len(header) > 20 and len(own) > 60
    assert not header & own, header & own
