// Prints what csu_b200/csrc/cuda/launch_rules.h chooses: model fp32 cells multiprocessors -> wide tune_class early grad_small, per line of stdin.
#include <cstdio>

#include "../../csu_b200/csrc/cuda/launch_rules.h"

int main()
{
    int model, fp32, cells, sms;
    while (scanf("%d %d %d %d", &model, &fp32, &cells, &sms) == 4)
        printf("%d %d %d %d\n", (int)csu::sweep_wide(model, fp32 != 0, cells, sms),
               csu::tune_class(model, fp32 != 0, cells, sms), (int)csu::sweep_early(model, fp32 != 0, cells, sms),
               (int)csu::grad_small(model, (cells + 31) / 32, sms));
    return 0;
}
