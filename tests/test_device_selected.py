"""Every entry point that allocates, copies, waits or launches for a context selects the
context's device first: buffers are kept between calls and cudaDeviceSynchronize only waits for
the current device, so with another one current a copy could overwrite arrays that kernels
of this context still read."""
import re

from conftest import ROOT

TEXT = (ROOT / "finiteelementcontainers.jl_gb300" / "csrc" / "fec_abi.cu").read_text()
WORK = re.compile(r"\b(upload|ensure|invalidate_pattern|release_pattern|build_affine|"
                  r"cuda(?:Malloc\w*|Free\w*|Memcpy\w*|Memset\w*|DeviceSynchronize|StreamSynchronize))\(|<<<|fec::(?:launch|pattern|pcg)\w*\(")


def entry_points():
    for m in re.finditer(r"^int (fec_\w+)\(([^;{]*?)\) \{\n(.*?)^\}", TEXT, re.M | re.S):
        if "fec_ctx* c" in m[2]:
            yield m[1], m[3]


def test_device_is_selected_before_any_work():
    seen, late = 0, []
    for name, body in entry_points():
        work = WORK.search(body)
        if not work or name == "fec_ctx_create":
            continue
        seen += 1
        selected = re.search(r"cudaSetDevice\(c->device\)", body)
        if not selected or selected.start() > work.start():
            late.append(name)
    assert seen >= 12 and late == []
