"""The bench's count of what the MLP kernels issue to the tensor cores, from the shapes of their MMAs in the folded form:
128 samples a tile, forward M = 128, K = 8 a step; adjoint M = 128, K = 16 a step."""

from test_bench_accounting import _bench


def test_issued_flops_per_sample():
    b = _bench()
    tile = 128
    forward = sum(2 * 128 * n * 8 for _ in range(5) for n in (128, 64))  # 5 K steps, hi and lo operand
    g = 3 * 8 * 2 * 128 * 64 * 16  # three parts, 8 steps over the tile's samples
    dx = 3 * 4 * 2 * 128 * 112 * 16  # three parts, 4 steps over the hidden units
    assert b.MLP_ISSUED["vx_appearance_mlp_forward_masked"] == (forward // tile, "tf32") == (15360, "tf32")
    assert b.MLP_ISSUED["vx_appearance_mlp_backward_masked"] == ((g + dx) // tile, "bf16") == (92160, "bf16")


def test_tensor_rate_is_the_issued_one():
    b = _bench()
    name = "vx_appearance_mlp_backward_masked"
    r = b.mlp_tensor({name: 0.135}, 1 << 20)[name]
    assert abs(r["issued_tflops"] - 92160 * (1 << 20) / 0.135e-3 / 1e12) < 1e-6
    assert abs(r["frac"] - r["issued_tflops"] / r["peak_tflops"]) < 1e-12
    assert r["fp32_equiv_tflops"] < r["issued_tflops"] / 7
