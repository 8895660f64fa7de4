// The mixed variant's clamped plasticity update (precompute<float, double>: the first-order
// correction of the FP32 SVD) against the FP64 one on the same FP32 inputs. Per family of
// singular values, the largest difference of Fe, Re (absolute), Jp and Je (relative) in
// units of 2^-24. Prints "name value" pairs.
//   wide    0.8 .. 1.2            band    0.97 .. 1.03 (mixed sides of the limits)
//   equal   0.97 +- 1e-6          lower, upper: within 3e-7 of a limit, all three
//   near    within 1e-4 of the lower limit    pair: two equal to 1e-7, one apart
//   far     exp(+-1.2): beyond the range the correction is used for, too
#include "mpm_math.cuh"
#include <cmath>
#include <cstdio>
#include <random>

using namespace mpm;

static void rotation(std::mt19937_64& g,double* R)
{
    std::normal_distribution<double> n(0.,1.);
    double q[4],s=0;
    for(double& x:q){x=n(g);s+=x*x;}
    for(double& x:q) x/=std::sqrt(s);
    for(int c=0;c<3;++c){                       // columns q e_c q*
        const double e[3]={c==0?1.:0.,c==1?1.:0.,c==2?1.:0.};
        const double t[3]={2*(q[2]*e[2]-q[3]*e[1]),2*(q[3]*e[0]-q[1]*e[2]),2*(q[1]*e[1]-q[2]*e[0])};
        R[c]=e[0]+q[0]*t[0]+q[2]*t[2]-q[3]*t[1];
        R[3+c]=e[1]+q[0]*t[1]+q[3]*t[0]-q[1]*t[2];
        R[6+c]=e[2]+q[0]*t[2]+q[1]*t[1]-q[2]*t[0];}
}

int main()
{
    const float cy=0.975f,sy=1.0075f;
    const char* names[]={"wide","band","equal","lower","upper","near","pair","far"};
    for(int mode=0;mode<8;++mode){
        std::mt19937_64 g(11+mode);
        std::uniform_real_distribution<double> u(-1.,1.);
        double worst=0;
        for(int it=0;it<20000;++it){
            double A[9],B[9],s[3],F[9];
            rotation(g,A);rotation(g,B);
            for(double& x:s){
                const double r=u(g);
                x=mode==0?1+.2*r:mode==1?1+.03*r:mode==2?.97+1e-6*r:mode==3?cy+3e-7*r:mode==4?sy+3e-7*r:mode==5?cy+1e-4*r:
                  mode==6?1+.05*r:std::exp(1.2*r);}
            if(mode==6) s[1]=s[0]+1e-7*u(g);
            for(int i=0;i<3;++i) for(int j=0;j<3;++j) F[3*i+j]=A[3*i]*s[0]*B[3*j]+A[3*i+1]*s[1]*B[3*j+1]+A[3*i+2]*s[2]*B[3*j+2];
            float Fm[9],Rm[9],lam,mu,Je,Jp=1.f+.1f*(float)u(g);
            double Fx[9],Rx[9],lx,mx,Jx,Jq=Jp;
            for(int k=0;k<9;++k){Fm[k]=(float)F[k];Fx[k]=Fm[k];}
            precompute<float,double>(Fm,Jp,1e4f,2e4f,1,10.f,cy,sy,10.f,Rm,lam,mu,Je);
            precompute<double,double>(Fx,Jq,1e4,2e4,1,10.,(double)cy,(double)sy,10.,Rx,lx,mx,Jx);
            bool clamped=false;               // the others keep Fe and take the polar refinement
            for(int k=0;k<9;++k) clamped|=Fm[k]!=(float)F[k];
            if(!clamped) continue;
            double d=std::fmax(std::fabs(Jp-Jq)/std::fabs(Jq),std::fabs(Je-Jx)/std::fabs(Jx));
            for(int k=0;k<9;++k) d=std::fmax(d,std::fmax(std::fabs(Fm[k]-Fx[k]),std::fabs(Rm[k]-Rx[k])));
            worst=std::fmax(worst,d*std::ldexp(1.,24));}
        std::printf("%s %.4f ",names[mode],worst);}
    // the rotation near a rotation (polar_near, FP32 storage in both variants): Re and Je
    for(int mode=0;mode<3;++mode){
        std::mt19937_64 g(31+mode);
        std::uniform_real_distribution<double> u(-1.,1.);
        const double strain=mode==0?1e-7:mode==1?1e-3:0.007;     // the last reaches the series' limit
        double worst=0;
        for(int it=0;it<20000;++it){
            double A[9],B[9],s[3],F[9];
            rotation(g,A);rotation(g,B);
            for(double& x:s) x=1+strain*u(g);
            for(int i=0;i<3;++i) for(int j=0;j<3;++j) F[3*i+j]=A[3*i]*s[0]*B[3*j]+A[3*i+1]*s[1]*B[3*j+1]+A[3*i+2]*s[2]*B[3*j+2];
            float Ff[9],R[9];double Fx[9],Rx[9],lx,mx,Jx,Jq=1.;
            for(int k=0;k<9;++k){Ff[k]=(float)F[k];Fx[k]=Ff[k];}
            if(!polar_near(Ff,POLAR_SERIES_MAX*POLAR_SERIES_MAX,R)) continue;
            precompute<double,double>(Fx,Jq,1e4,2e4,0,10.,(double)cy,(double)sy,10.,Rx,lx,mx,Jx);
            for(int k=0;k<9;++k) worst=std::fmax(worst,std::fabs(R[k]-Rx[k])*std::ldexp(1.,24));}
        std::printf("%s %.4f ",mode==0?"rigid":mode==1?"light":"limit",worst);}
    std::printf("\n");
    return 0;
}
