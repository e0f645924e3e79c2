"""The tensor-core expectation's CTAs per SM: never more than tensor memory holds
(512 columns), whatever part of its static shared memory a shape lays out, and
no fewer than that where shared memory allows."""

from pylcm_b200.codegen import RegimeKernels

PER_SM, RESERVED = 233472, 1024  # bytes of an SM; reserved per CTA


def _static(K: int, J: int) -> int:
    """Weights, row scales, sums and node bits where they fit, barrier and two
    words, as lcm_tc_expect lays them out."""
    sums = K * (8 * J + 12) + 256 <= 49152
    bits = K > 8 and K * (8 * J + 20) + 256 <= 49152
    return K * J * 8 + K * 4 + 8 * ((K if sums else 0) + (K + 1 if bits else 0) + 1) + 8


def test_no_more_ctas_than_tensor_memory_holds():
    for K in range(1, RegimeKernels.TC_MAX_K + 1):
        for J in range(1, RegimeKernels.TC_MAX_J + 1):
            static = _static(K, J)
            if static > 49152:
                continue
            sh = RegimeKernels.tc_shape(K, J)
            plain = 2 * 128 * sh["JP"] * 4 + 2 * sh["NP"] * sh["JP"] * 4 + 128
            assert sh["ncol"] >= sh["NP"] and sh["smem"] >= plain
            assert PER_SM // (sh["smem"] + static + RESERVED) <= 512 // sh["ncol"], (K, J)
            units = lambda b: (b + static + 127) // 128 * 128 + RESERVED  # noqa: E731
            assert PER_SM // units(sh["smem"]) >= min(512 // sh["ncol"], PER_SM // units(plain)), (K, J)
