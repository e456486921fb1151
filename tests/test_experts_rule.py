"""Which steps' experts are multiplied with the tokens that chose them: those where it was measured to be the faster form."""

import pytest


# (width, experts, chosen, features, shared features, tokens), us grouped / over all tokens
@pytest.mark.parametrize("sizes,grouped,dense", [
    ((2048, 32, 4, 256, 2048, 3577), 226, 329), ((2048, 32, 1, 256, 2048, 3577), 172, 325), ((1024, 64, 8, 256, 1024, 1431), 133, 160),
    ((1024, 256, 8, 128, 1024, 1789), 161, 316), ((4096, 8, 2, 2048, 4096, 895), 269, 336), ((512, 64, 16, 512, 512, 1431), 154, 208),
    ((2048, 256, 16, 128, 128, 895), 224, 283), ((2048, 32, 4, 256, 2048, 895), 116, 104), ((2048, 32, 8, 256, 2048, 1431), 165, 151),
    ((2048, 64, 16, 128, 512, 3577), 377, 300), ((2048, 64, 16, 128, 512, 1431), 203, 138), ((2048, 256, 16, 128, 128, 224), 176, 133),
    ((1024, 32, 8, 128, 1024, 3970), 224, 141), ((4096, 8, 2, 1024, 512, 551), 127, 110), ((3072, 32, 4, 512, 2048, 350), 149, 125)])
def test_the_faster_form(sizes, grouped, dense):
    from kv_cache_optimization_for_llm_b200 import ops
    H, E, top, F, S, T = sizes
    assert ops.experts_grouped_faster(T, H, E, F, S, top) == (grouped < dense)


@pytest.mark.parametrize("most", [100, 900, 1430, 4096])
@pytest.mark.parametrize("sizes", [(2048, 32, 4, 256, 2048), (2048, 64, 16, 128, 512), (1024, 8, 2, 768, 2048), (2048, 8, 2, 512, 128), (4096, 8, 1, 256, 1024),
                                   (2048, 256, 16, 128, 128), (512, 128, 3, 512, 4096), (3072, 16, 4, 256, 512)])
def test_room_is_declared_where_some_step_is_grouped(sizes, most):
    from kv_cache_optimization_for_llm_b200 import ops
    H, E, top, F, S = sizes
    grouped = any(ops.experts_grouped_faster(t, H, E, F, S, top) for t in range(1, most + 1))
    assert (ops.experts_grouped_widths(H, E, F, S, top, most) > 0) == grouped
