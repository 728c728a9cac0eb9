// Prints what csu_b200/csrc/cuda/launch_rules.h chooses: model fp32 cells multiprocessors -> wide tune_class early, per line of stdin.
#include <cstdio>

#include "../../csu_b200/csrc/cuda/launch_rules.h"

int main()
{
    int model, fp32, cells, sms;
    while (scanf("%d %d %d %d", &model, &fp32, &cells, &sms) == 4)
        printf("%d %d %d\n", (int)csu::sweep_wide(model, fp32 != 0, cells, sms),
               csu::tune_class(model, fp32 != 0, cells, sms), (int)csu::sweep_early(model, fp32 != 0, cells, sms));
    return 0;
}
