"""The row kernels of prompt slices at the ends of the sizes that go by them, against the forms of few rows, to the bit."""
import pytest
import torch

import test_gpu_aux_rows as aux

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(297, 1152), (511, 2048), (593, 2048), (297, 4096)])
def test_residual_finish(M, N):
    aux.test_finish_of_a_slice_equals_the_general_form(M, N, True, True, True)
