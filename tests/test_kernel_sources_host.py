"""Orders that the CUDA sources have to keep and that no run can be relied on to show."""
import glob
import os

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nano-vllm-ascend_b200", "csrc")


def test_tensor_memory_is_allocated_after_the_kernel_before_has_finished():
    """Kernels are launched as programmatic dependents and let their own dependents in at their start: one that took tensor
    memory before its wait could hold the columns that a CTA of the kernel before is still to allocate."""
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            text = f.read()
        at = text.find("umma::tmem_alloc(")
        while at >= 0:
            body = text[text.rfind("__global__", 0, at):at]
            assert "pdl_wait();" in body, (os.path.basename(path), text.count("\n", 0, at) + 1)
            seen += 1
            at = text.find("umma::tmem_alloc(", at + 1)
    assert seen >= 3


def test_shared_memory_is_asked_for_on_every_device():
    """A kernel's attributes hold for one device: a launcher that remembers per process that it has asked refuses every call on
    the second device. The launchers of these files serve calls that needed no such memory before, or asked each time."""
    for name in ("attn_tiled.cu", "moe_umma.cu", "seq_mixers.cu"):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        assert "static const cudaError_t" not in text, name
        assert text.count("allow_smem(") >= 1, name
