"""Under an SM budget the expert layer runs in the kernels that keep to it."""


def test_two_launch_expert_layer_is_not_taken_under_an_sm_budget():
    import dsv3_b200
    from dsv3_b200 import _lib
    pay = _lib.lib.dsv3_few_experts_pay
    try:
        dsv3_b200.set_num_sms(64)
        assert pay(1, 8, 32, 256, 7168, 2048, 256) == 0
    finally:
        dsv3_b200.set_num_sms(0)
    assert pay(1, 8, 32, 256, 7168, 2048, 256) == 1
